"""A restart cycle's graph whose capture fails: the error comes back as a status, and the
next graph on the same stream is built and runs."""
import os
import subprocess

import pytest

from conftest import ROOT
from cugmres_b200 import build

pytestmark = pytest.mark.gpu

PROGRAM = r"""
#include <cstdio>
#include "cg_internal.h"

__global__ void k_count(int *n) { atomicAdd(n, 1); }
__global__ void k_test(int *n, cudaGraphConditionalHandle h) { cudaGraphSetConditional(h, *n < 12 ? 1u : 0u); }
static int *count;

namespace cg {  // the loop ends once the body's kernels have counted to twelve
int add_loop_test(const KrylovPtrs &, cudaGraphConditionalHandle h, cudaGraph_t in, cudaGraphNode_t after,
                  cudaGraphNode_t *node) {
    void *args[] = {&count, &h};
    cudaKernelNodeParams p = {};
    p.func = (void *)k_test;
    p.gridDim = dim3(1);
    p.blockDim = dim3(1);
    p.kernelParams = args;
    return (int)cudaGraphAddKernelNode(node, in, &after, 1, &p);
}
}  // namespace cg

int main() {
    cudaStream_t s;
    cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking);
    cudaMalloc(&count, sizeof(int));
    cudaMemset(count, 0, sizeof(int));
    cudaDeviceSynchronize();
    auto launch = [](cudaStream_t q, size_t smem) -> int {
        k_count<<<1, 1, smem, q>>>(count);
        return cudaGetLastError() == cudaSuccess ? 0 : 2;
    };
    auto good = [&](cudaStream_t q) -> int { return launch(q, 0) + launch(q, 0); };
    // more shared memory than a launch may have without opting in: refused by the runtime
    auto refused = [&](cudaStream_t q) -> int {
        const int e = launch(q, 0);
        return e ? e : launch(q, 100 * 1024);
    };
    auto stops = [&](cudaStream_t q) -> int { return launch(q, 0) ? 2 : 9; };
    cg::KrylovPtrs kp{};
    cudaGraphExec_t x = nullptr;
    printf("%d", cg::cycle_graph(kp, s, refused, good, &x));
    printf(" %d", cg::cycle_graph(kp, s, good, refused, &x));
    printf(" %d", cg::cycle_graph(kp, s, stops, good, &x));
    printf(" %d", x == nullptr);
    printf(" %d", cg::cycle_graph(kp, s, good, good, &x));
    int n = -1;
    printf(" %d", (int)cudaGraphLaunch(x, s));
    cudaStreamSynchronize(s);
    cudaMemcpy(&n, count, sizeof(int), cudaMemcpyDeviceToHost);
    cudaGraphExecDestroy(x);
    printf(" %d %d\n", n, (int)cudaGetLastError());
}
"""


def test_failed_captures_return_their_status(cuda_device, tmp_path):
    src, exe = tmp_path / "capture.cu", tmp_path / "capture"
    src.write_text(PROGRAM)
    subprocess.run([build.nvcc(), "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "--extended-lambda", "-I",
                    os.path.join(ROOT, "cugmres_b200", "csrc"), str(src), "-o", str(exe)], check=True, timeout=300)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stderr
    # two refused launches, an error of the callback's own, then a loop of six bodies and a tail
    assert r.stdout.split() == ["2", "2", "9", "1", "0", "0", "14", "0"]
