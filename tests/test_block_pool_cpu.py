"""The block pool of the cache objects against a counting stand-in for the CUDA allocator (no GPU)."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")

PROGRAM = r"""
#include "tqb_block_pool.h"
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>

static std::map<char*, size_t> g_live;
static size_t g_bytes = 0, g_limit = ~(size_t)0, g_calls = 0;
static char* g_next = (char*)0x100000000;
extern "C" cudaError_t cudaMalloc(void** p, size_t n) {
    ++g_calls;
    if (g_bytes + n > g_limit) return cudaErrorMemoryAllocation;
    *p = g_next;
    g_next += (n + 4095) / 4096 * 4096;
    g_live[(char*)*p] = n;
    g_bytes += n;
    return cudaSuccess;
}
extern "C" cudaError_t cudaFree(void* p) {
    auto it = g_live.find((char*)p);
    if (it == g_live.end()) { std::puts("cudaFree of what is not allocated"); std::exit(1); }
    g_bytes -= it->second;
    g_live.erase(it);
    return cudaSuccess;
}
extern "C" cudaError_t cudaGetLastError() { return cudaSuccess; }

using namespace tqb;
typedef BlockPool::Block Block;
#define CHECK(c) do { if (!(c)) { std::printf("line %d: %s\n", __LINE__, #c); std::exit(1); } } while (0)
[[maybe_unused]] static const size_t MB = 1 << 20;
[[maybe_unused]] static Block take(BlockPool& p, size_t n, int alike = 1, bool use_idle = true) {
    Block b;
    CHECK(p.take(n, alike, use_idle, &b) == cudaSuccess);
    auto it = g_live.upper_bound((char*)b.p);
    CHECK(it != g_live.begin());
    --it;
    CHECK((char*)b.p + n <= it->first + it->second);      // inside an allocation
    return b;
}
"""

RETIRE = """
int main() {
    BlockPool p;
    Block a = take(p, 3 * MB, 4);
    p.retire(a);                                          // outgrown: queued work may still read it
    Block b[4];
    for (auto& x : b) { x = take(p, 3 * MB); CHECK(x.p != a.p); }
    p.settle();                                           // the device has been waited for
    CHECK(take(p, 3 * MB).p == a.p);
    p.release();
    CHECK(g_bytes == 0);
}
"""

BOUND = """
int main() {
    BlockPool p;
    const size_t keep = BlockPool::kKeepBytes;
    // 28 layers of 40 MB, 1,120 MB: what the pool holds after a reset is the bound's worth of blocks, and the next request
    // allocates the rest only
    std::vector<Block> b(28);
    for (int request = 0; request < 5; ++request) {
        const size_t before = g_calls;
        for (auto& x : b) x = take(p, 40 * MB);
        CHECK(g_calls - before == (request == 0 ? 28u : 28u - keep / (40 * MB)));
        CHECK(g_bytes == 28 * 40 * MB);
        for (auto& x : b) p.put(x);
        p.settle();
        CHECK(g_bytes <= keep && g_bytes > keep - 40 * MB);
    }
    // idle blocks beside a live one come on top of the bound and go with it
    Block one = take(p, 16 * MB, 4);
    for (auto& x : b) x = take(p, 40 * MB);
    for (auto& x : b) p.put(x);
    CHECK(g_bytes <= keep + 4 * 16 * MB);
    p.put(one);
    CHECK(g_bytes <= keep);
    // an allocation that fails gives back everything unused first
    g_limit = keep + 8 * MB;
    take(p, keep);
    CHECK(g_bytes == keep);
    p.release();
    CHECK(g_bytes == 0);
}
"""

RECORDS = """
int main() {
    BlockPool p;
    std::vector<Block> b(28);
    for (int request = 0; request < 200; ++request) {     // above the bound: slabs come and go with every request
        for (auto& x : b) x = take(p, (30 + request % 7) * MB, request % 3 + 1);
        for (auto& x : b) { if (request % 2) p.retire(x); else p.put(x); }
        p.settle();
        CHECK(p.slabs() == g_live.size());
        CHECK(p.slabs() <= 28);
    }
    p.release();
    CHECK(g_bytes == 0 && p.slabs() == 0);
}
"""

AHEAD = """
struct Layer { int64_t cap; };
int main() {
    std::vector<Layer> l(80, Layer{0});
    CHECK(blocks_ahead(l, 0, 100) == 80);                 // a new cache's first prompt
    l[0].cap = 228;
    CHECK(blocks_ahead(l, 0, 100) == 79);                 // the second layer's: the first one has its rows
    CHECK(blocks_ahead(l, l[0].cap, 300) == 2);           // a layer used alone
    for (int i = 0; i < 28; ++i) l[i].cap = 228;
    CHECK(blocks_ahead(l, l[0].cap, 300) == 28 + 28);
    for (auto& x : l) x.cap = 228;
    l[0].cap = 428;
    CHECK(blocks_ahead(l, l[1].cap, 300) == 79);
    std::vector<Layer> one(1, Layer{0});
    CHECK(blocks_ahead(one, 0, 1) == 1);
    one[0].cap = 129;
    CHECK(blocks_ahead(one, 129, 200) == 1);
}
"""


def run(tmp_path, main):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None or not os.path.exists(os.path.join(CUDA, "include", "cuda_runtime_api.h")):
        pytest.skip("needs a C++ compiler and the CUDA headers")
    src, exe = tmp_path / "pool.cpp", tmp_path / "pool"
    src.write_text(PROGRAM + main)
    r = subprocess.run([cxx, "-std=c++17", "-Wall", "-Werror", "-I", os.path.join(ROOT, "turboquant_b200", "csrc"), "-isystem",
                        os.path.join(CUDA, "include"), str(src), "-o", str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout


def test_a_retired_block_waits_for_the_device(tmp_path):
    run(tmp_path, RETIRE)


def test_what_the_pool_holds_is_bounded_and_kept_up_to_the_bound(tmp_path):
    run(tmp_path, BOUND)


def test_many_resets_above_the_bound_leave_no_records(tmp_path):
    run(tmp_path, RECORDS)


def test_memory_for_layers_that_are_never_used_is_bounded(tmp_path):
    run(tmp_path, AHEAD)
