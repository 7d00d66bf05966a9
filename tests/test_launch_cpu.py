"""The host side of a launch, on the CPU: `csrc/pdl.cuh` over a CUDA runtime whose calls are answered by the test program."""

import os
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]

PROGRAM = r"""
#include <cuda_runtime.h>
#include <stdio.h>
#include <string.h>
#include <thread>
#include <vector>

// what nvcc's headers add to the C calls
template <class T> cudaError_t cudaFuncGetAttributes(cudaFuncAttributes* a, T* f) { return cudaFuncGetAttributes(a, (const void*)f); }
template <class T> cudaError_t cudaFuncSetAttribute(T* f, cudaFuncAttribute a, int v) { return cudaFuncSetAttribute((const void*)f, a, v); }
template <class T> cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int* n, T* f, int threads, size_t smem) {
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(n, (const void*)f, threads, smem);
}
#include "pdl.cuh"

constexpr int kStatic = 512, kBlocks = 8;
thread_local size_t dynamic_bytes;
extern "C" {
cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
cudaError_t cudaFuncGetAttributes(cudaFuncAttributes* a, const void*) { memset(a, 0, sizeof *a); a->sharedSizeBytes = kStatic; return cudaSuccess; }
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int* n, const void*, int, size_t) { *n = kBlocks; return cudaSuccess; }
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void*, void**) {
    dynamic_bytes = c->dynamicSmemBytes;
    return c->gridDim.x && c->gridDim.y && c->gridDim.z ? cudaSuccess : cudaErrorInvalidConfiguration;
}
}
namespace kge { bool dependent_launch_enabled() { return false; } }
void kernel(int) {}

static bool spread(unsigned blocks) {
    if (kge::launch_spread<kernel>(dim3(blocks), dim3(256), nullptr, 1) != cudaSuccess) return false;
    const size_t sm = 228 * 1024, each = dynamic_bytes + kStatic + 1024, share = (blocks + 147) / 148;
    if (share >= (size_t)kBlocks) return dynamic_bytes == 0;
    // an SM's share of the blocks fits, one more does not (where a block can be given that much: 227 KB)
    return share * each <= sm && ((share + 1) * each > sm || dynamic_bytes + kStatic >= 227 * 1024 - 128);
}

static bool not_spread() { return kge::launch_spread_if<kernel>(false, dim3(160), dim3(256), nullptr, 1) == cudaSuccess && dynamic_bytes == 0; }

int main(int argc, char** argv) {
    if (argc > 1 && !strcmp(argv[1], "beside")) return not_spread() ? 0 : 1;
    if (argc > 1) return kge::launch_spread<kernel>(dim3(0), dim3(256), nullptr, 1) == cudaErrorInvalidConfiguration ? 0 : 1;
    std::vector<std::thread> threads;
    bool ok[4] = {};
    for (int t = 0; t < 4; ++t)
        threads.emplace_back([t, &ok] {
            bool all = true;
            for (unsigned blocks = 1 + (unsigned)t; blocks < 1500; blocks += 4) all = spread(blocks) && all;
            ok[t] = all;
        });
    for (std::thread& t : threads) t.join();
    return ok[0] && ok[1] && ok[2] && ok[3] ? 0 : 1;
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    folder = tmp_path_factory.mktemp("launch")
    cuda = next((p for p in (os.environ.get("CUDA_HOME"), "/usr/local/cuda") if p and Path(p, "include/cuda_runtime.h").exists()), None)
    if cuda is None:
        pytest.skip("no CUDA headers")
    source, sanitized = folder / "launch.cpp", ["g++", "-std=c++17", "-g", "-O1", "-fsanitize=thread"]
    source.write_text("int main() { return 0; }")
    if subprocess.run([*sanitized, source, "-o", folder / "empty"], capture_output=True).returncode or subprocess.run([folder / "empty"], capture_output=True).returncode:
        pytest.skip("no thread sanitizer")
    source.write_text(PROGRAM)
    subprocess.run([*sanitized, f"-I{cuda}/include", f"-I{ROOT / 'distributed-kge-poplar_b200' / 'csrc'}", source, "-o", folder / "launch", "-lpthread"], check=True)
    return folder / "launch"


def test_spread_launches_on_several_threads(program):
    """Engines on several threads make their first launches of a kernel at the same time: no data race, and every SM gets room for
    its share of the blocks and no more."""
    run = subprocess.run([program], capture_output=True, text=True)
    assert run.returncode == 0, run.stderr[-3000:]


def test_a_launch_beside_others_leaves_them_room(program):
    """Where shards run side by side, no block takes an SM's shared memory for itself."""
    run = subprocess.run([program, "beside"], capture_output=True, text=True)
    assert run.returncode == 0, run


def test_a_launch_of_no_blocks_is_an_error_status(program):
    run = subprocess.run([program, "empty"], capture_output=True, text=True)
    assert run.returncode == 0, run
