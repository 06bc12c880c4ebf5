"""The prefill's wait for other blocks' items (csrc/kda_prefill_sp.cu, count_wait), compiled for the host against a clock and a count of the test's own:
while the count rises, the block's progress counter, which renews the limit of the block's other waits, moves with it; a count that stands
still ends the wait at the limit.  No GPU."""
import os
import re
import shutil
import subprocess

import pytest

SOURCE = os.path.join(os.path.dirname(__file__), "..", "glm53f-afd_b200", "csrc", "kda_prefill_sp.cu")

HARNESS = r"""
#include <cstdint>
#include <cstdio>
#include <cstdlib>
struct WaitCtx { volatile uint32_t* progress; volatile uint32_t* abort; int* status; uint64_t limit_ns; };
static uint64_t now_ns = 0, step_ns, quiet_ns = 0, longest_ns = 0;
static unsigned stop_at;
static uint32_t progress = 0, last_progress = 0, raised = 0;
static int status_word = 0;
static uint64_t global_timer_ns() { return now_ns; }
static void atomicAdd(uint32_t* p, uint32_t x) { *p += x; }
static void atomicCAS(int* p, int want, int x) { if (*p == want) *p = x; }
static unsigned load(const unsigned*) {  // the count rises by one every step_ns, up to stop_at
    const uint64_t n = now_ns / step_ns;
    return n < stop_at ? (unsigned)n : stop_at;
}
static void __nanosleep(unsigned) {  // a tenth of a second passes
    now_ns += 100000000ull;
    quiet_ns = progress == last_progress ? quiet_ns + 100000000ull : 0;
    last_progress = progress;
    if (quiet_ns > longest_ns) longest_ns = quiet_ns;
}
COUNT_WAIT
int main(int, char** argv) {
    step_ns = strtoull(argv[1], nullptr, 10);
    stop_at = (unsigned)atoi(argv[2]);
    unsigned at = 0;
    const bool there = count_wait(&at, (unsigned)atoi(argv[3]), WaitCtx{&progress, &raised, &status_word, 2000000000ull}, 120);
    printf("%d %d %llu %llu\n", (int)there, status_word, (unsigned long long)longest_ns, (unsigned long long)now_ns);
}
"""


@pytest.fixture(scope="module")
def harness(tmp_path_factory):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("no g++")
    with open(SOURCE) as f:
        body = re.search(r"__device__ __forceinline__ (bool count_wait\(.*?\n\})\n", f.read(), re.S).group(1)
    body, loads = re.subn(r'asm volatile\("ld\.acquire\.gpu\.global\.u32[^;]*;"[^;]*;', "v = load(at);", body)
    assert loads == 1
    where = tmp_path_factory.mktemp("count_wait")
    (where / "x.cpp").write_text(HARNESS.replace("COUNT_WAIT", "static " + body))
    subprocess.check_call([gxx, "-std=c++17", "-O1", "-o", str(where / "x"), str(where / "x.cpp")])
    return lambda *a: [int(x) for x in subprocess.check_output([str(where / "x"), *map(str, a)]).split()]


def test_a_rising_count_renews_the_block_s_limit(harness):
    there, status, longest, now = harness(1_500_000_000, 20, 8)  # eight items, one every 1.5 s, with a limit of 2 s
    assert there and status == 0 and now >= 8 * 1_500_000_000
    assert longest < 2_000_000_000


def test_a_count_that_stands_still_ends_the_wait(harness):
    there, status, _, now = harness(1_500_000_000, 3, 8)
    assert not there and status == 120
    assert now <= 3 * 1_500_000_000 + 2_500_000_000
