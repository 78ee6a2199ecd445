"""The sets of words that measurements of ranges share, compiled against stand-ins for the CUDA calls: no GPU."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#include <atomic>
#include <set>
#include <thread>
#include <vector>

enum cudaError_t { cudaSuccess = 0, failed = 1 };
static int memset_fails, sync_fails, words_missing;
static uint64_t words[64];
static unsigned char *ws;
static size_t cap;
cudaError_t cudaGetDevice(int *d) { *d = 0; return cudaSuccess; }
cudaError_t cudaMemset(void *p, int v, size_t n) { if (memset_fails) return failed; memset(p, v, n); return cudaSuccess; }
cudaError_t cudaDeviceSynchronize() { return sync_fails ? failed : cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
namespace zkds {
int sm_count() { return 148; }
void *workspace_fresh(size_t bytes, int, size_t *fresh)
{
    *fresh = 0;
    if (!ws) { ws = (unsigned char *)malloc(bytes); memset(ws, 0x5A, bytes); cap = *fresh = bytes; }
    return cap >= bytes ? ws : nullptr;
}
bool range_words(uint64_t **, uint64_t **);
}
#include "range_answer.h"
bool zkds::range_words(uint64_t **host, uint64_t **dev) { *host = *dev = words; return !words_missing; }

#define CHECK(x) do { if (!(x)) { printf("line %d: %s\n", __LINE__, #x); return 1; } } while (0)

int main()
{
    using zkds::RangeAnswer;
    // new words that could not be cleared are cleared by the first call that can, whichever step failed
    for (int *what : {&words_missing, &memset_fails, &sync_fails}) {
        free(ws); ws = nullptr;
        *what = 1;
        { RangeAnswer a; CHECK(!a.claim()); }
        *what = 0;
        if (ws) memset(ws, 0x5A, cap);
        RangeAnswer a;
        CHECK(a.claim() && *a.arrived == 0);
    }
    // words that were cleared once keep what the kernels leave in them, and a new arena is cleared again
    { RangeAnswer a; CHECK(a.claim()); a.partial[0] = 7; }
    { RangeAnswer a; CHECK(a.claim() && a.partial[0] == 7); }
    free(ws); ws = nullptr;
    { RangeAnswer a; CHECK(a.claim() && a.partial[0] == 0 && *a.arrived == 0); }
    // ten callers at once: eight get sets of their own, two are sent away and get one later
    std::atomic<int> here{0}, given{0}, clashes{0};
    std::atomic<unsigned> taken{0};
    std::atomic<unsigned long long> tickets{0};
    std::vector<std::thread> threads;
    for (int t = 0; t < 10; ++t)
        threads.emplace_back([&] {
            RangeAnswer a;
            const bool got = a.claim();
            if (got) {
                ++given;
                const unsigned bit = 1u << ((a.host - words) / 4);
                if (taken.fetch_or(bit) & bit) ++clashes;
                if (tickets.fetch_or(1ull << a.ticket) >> a.ticket & 1) ++clashes;
            }
            ++here;
            while (here < 10) std::this_thread::yield();
        });
    for (auto &t : threads) t.join();
    CHECK(given == 8 && clashes == 0 && taken == 255);
    RangeAnswer late;
    CHECK(late.claim());
    return 0;
}
"""


def test_sets_of_words(tmp_path):
    """cleared before their first use also when a first attempt to clear them failed; one owner at a time; refused when all are taken"""
    src = tmp_path / "sets.cpp"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-pthread", "-include", "stdint.h", "-include", "stddef.h", "-I",
                    os.path.join(ROOT, "zk-deepseek_b200", "csrc"), str(src), "-o", str(tmp_path / "sets")], check=True)
    r = subprocess.run([str(tmp_path / "sets")], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout
