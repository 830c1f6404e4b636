"""The caching allocator on the CPU, over stand-ins of the driver's calls: memory that runs out while a capture is open must not give back
blocks that the kernels captured so far address."""
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parent.parent

PROGRAM = r"""
#include "ctx.h"
#include <cstdlib>
#include <set>
static size_t room = 64u << 20;
static std::map<void*, size_t> live;
static size_t used() { size_t s = 0; for (auto& kv : live) s += kv.second; return s; }
extern "C" cudaError_t cudaMalloc(void** p, size_t n) {
    if (used() + n > room) return cudaErrorMemoryAllocation;
    *p = std::malloc(16); live[*p] = n; return cudaSuccess;
}
extern "C" cudaError_t cudaFree(void* p) { live.erase(p); std::free(p); return cudaSuccess; }
extern "C" cudaError_t cudaGetLastError() { return cudaSuccess; }
extern "C" cudaError_t cudaMemset(void*, int, size_t) { return cudaSuccess; }
extern "C" cudaError_t cudaMemcpy(void*, const void*, size_t, cudaMemcpyKind) { return cudaSuccess; }
#define CHECK(x) do { if (!(x)) { std::printf("line %d: %s\n", __LINE__, #x); return 1; } } while (0)
int main() {
    DeviceCachingAllocator a(0);
    void *idle, *p, *q, *r;
    CHECK(a.allocate(16u << 20, &idle) == cudaSuccess && a.free(idle));       // cached, addressed by nobody
    a.begin_log();
    CHECK(a.allocate(24u << 20, &p) == cudaSuccess && a.free(p));            // a temporary of the forward that is being captured
    CHECK(a.allocate(32u << 20, &q) == cudaSuccess);                         // fits once the idle block is given back
    CHECK(live.count(p) == 1 && live.count(idle) == 0);                       // ... and only that one
    CHECK(a.allocate(32u << 20, &r) == cudaErrorMemoryAllocation);           // the temporary may not make room
    CHECK(live.count(p) == 1);
    a.free(q);
    std::vector<void*> kept = a.take_logged();
    CHECK(kept.size() == 2);
    uint64_t in_use = 0, cached = 0;
    a.stats(nullptr, nullptr, &in_use, &cached);
    CHECK(in_use == (56u << 20) && cached == 0);
    a.give_back(kept);
    a.release_cached();
    CHECK(live.empty());
    return 0;
}
"""


def test_memory_that_runs_out_during_a_capture(tmp_path):
    src, exe = tmp_path / "alloc.cpp", tmp_path / "alloc"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O0", "-I", str(ROOT / "tensor_b200" / "csrc"), "-I", "/usr/local/cuda/include", str(src), "-o", str(exe)], check=True)
    done = subprocess.run([str(exe)], capture_output=True, text=True)
    assert done.returncode == 0, done.stdout
