"""Which host buffers are copied through the pinned ring, on the CPU over stand-ins of the driver's calls: pageable memory only, and only
while the ring's own memory can be had; everything else goes to the driver as the caller gave it."""
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parent.parent

PROGRAM = r"""
#include "ctx.h"
#include <cstdlib>
static cudaMemoryType kind = cudaMemoryTypeUnregistered;
static bool pinned_left = false, known = true;
static int errors_cleared = 0;
extern "C" cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void*) { a->type = kind; return known ? cudaSuccess : cudaErrorInvalidValue; }
extern "C" cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { *e = (cudaEvent_t)1; return cudaSuccess; }
extern "C" cudaError_t cudaMallocHost(void** p, size_t n) { if (!pinned_left) return cudaErrorMemoryAllocation; *p = std::malloc(n); return cudaSuccess; }
extern "C" cudaError_t cudaGetLastError() { ++errors_cleared; return cudaSuccess; }
#define CHECK(x) do { if (!(x)) { std::printf("line %d: %s\n", __LINE__, #x); return 1; } } while (0)
int main() {
    HostStaging ring;
    int host;
    CHECK(!ring.takes(&host) && errors_cleared == 1);  // no pinned memory: the driver's own path, and no error left behind
    pinned_left = true;
    for (cudaMemoryType k : {cudaMemoryTypeHost, cudaMemoryTypeDevice, cudaMemoryTypeManaged}) {
        kind = k;
        CHECK(!ring.takes(&host) && ring.mem == nullptr);
    }
    kind = cudaMemoryTypeUnregistered;
    known = false;
    CHECK(!ring.takes(&host));
    known = true;
    CHECK(ring.takes(&host) && ring.mem != nullptr);
    return 0;
}
"""


def test_what_goes_through_the_ring(tmp_path):
    src, exe = tmp_path / "staging.cpp", tmp_path / "staging"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O0", "-I", str(ROOT / "tensor_b200" / "csrc"), "-I", "/usr/local/cuda/include", str(src), "-o", str(exe)], check=True)
    done = subprocess.run([str(exe)], capture_output=True, text=True)
    assert done.returncode == 0, done.stdout
