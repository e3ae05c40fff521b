"""Page-locked blocks that a context keeps for results (no GPU: allocations counted by stand-ins)."""
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parents[1]

SOURCE = r"""
#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <memory>
#include <mutex>
#include <vector>
enum cudaError_t { cudaSuccess, cudaErrorMemoryAllocation };
constexpr unsigned cudaHostAllocPortable = 1;
static size_t made = 0, live = 0;
static bool full = false;
static cudaError_t cudaHostAlloc(void **p, size_t, unsigned) {
    if (full) return cudaErrorMemoryAllocation;
    *p = malloc(1);
    ++made, ++live;
    return cudaSuccess;
}
static cudaError_t cudaFreeHost(void *p) { free(p); --live; return cudaSuccess; }
static cudaError_t cudaGetLastError() { return cudaSuccess; }
#include "rt_hostpool.inc"
#define WANT(c) do { if (!(c)) { printf("line %d: %s\n", __LINE__, #c); return 1; } } while (0)
int main() {
    const size_t MB = 1 << 20;
    auto pool = std::make_shared<HostPool>();
    void *big;
    { auto a = pool->take(400 * MB); big = a->p; WANT(a->pinned && a->bytes >= 400 * MB); }
    WANT(made == 1 && live == 1);
    auto small = pool->take(MB);  // lives on
    WANT(small->pinned && small->bytes < 3 * MB && made == 2);
    { auto a = pool->take(380 * MB); WANT(a->p == big && made == 2); }
    { auto a = pool->take(MB); auto c = pool->take(100 * 1024); WANT(a->p != small->p && !c->pinned && made == 3); }
    { auto a = pool->take(MB); WANT(made == 3); }
    // kept blocks of up to 128 MB serve any smaller request
    { auto a = pool->take(100 * MB); WANT(made == 4); }
    { auto a = pool->take(3 * MB), c = pool->take(40 * MB); WANT(made <= 5 && a->p != c->p); }
    // kept: at most four, of 512 MB together
    for (size_t mb : {8, 32, 128, 500, 2}) pool->take(mb * MB);
    WANT(live <= 5);
    { auto a = pool->take(500 * MB), c = pool->take(450 * MB); WANT(a->p != c->p); }
    { auto a = pool->take(600 * MB); WANT(!a->pinned); }
    {   // page-locked memory stops at 2 GB, whatever is held
        std::vector<std::shared_ptr<HostBlock>> held;
        size_t pinned = 0;
        for (int k = 0; k < 40; ++k) {
            held.push_back(pool->take(100 * MB));
            pinned += held.back()->pinned ? held.back()->bytes : 0;
        }
        WANT(pinned > 1900 * MB && pinned <= 2048 * MB && !held.back()->pinned);
    }
    { auto a = pool->take(100 * MB); WANT(a->pinned); }
    full = true;
    { auto a = pool->take(300 * MB); WANT(!a->pinned); }
    pool.reset();
    WANT(live == 1);
    small.reset();
    WANT(live == 0);
    return 0;
}
"""


def test_blocks_are_kept_by_size_and_given_back(tmp_path):
    src = tmp_path / "pool.cpp"
    src.write_text(SOURCE)
    exe = tmp_path / "pool"
    subprocess.check_call(["g++", "-std=c++17", "-Wall", "-I", str(ROOT / "cupami_b200" / "csrc"), str(src), "-o",
                           str(exe), "-pthread"])
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert out.returncode == 0, out.stdout + out.stderr
