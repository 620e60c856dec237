"""The bounded mbarrier waits of csrc/tma.cuh run out after a second of the GPU's clock, whatever a try_wait or a nanosleep takes, and
roles that wait beside them leave with them.  A kernel of one block waits for barriers that nobody completes."""
import ctypes
import os
import subprocess

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SOURCE = r"""
#include "tma.cuh"
using namespace mt;
static __device__ __forceinline__ unsigned long long clock_ns() { unsigned long long t; asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t)); return t; }
// warp w waits in its own way; out[3 w] = what the wait said, [3 w + 1] = how long it took, [3 w + 2] = the abort flag afterwards
__global__ void waits(long long* out) {
    __shared__ __align__(8) uint64_t bars[4];
    __shared__ int abort_flag;
    if (threadIdx.x == 0) {
        abort_flag = 0;
        for (int i = 0; i < 4; ++i) mbar_init(smem_u32(bars + i), 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    const int w = threadIdx.x >> 5;
    if ((threadIdx.x & 31) == 0) {
        const unsigned long long t0 = clock_ns();
        bool said;
        if (w == 0) said = mbar_wait(smem_u32(bars), 0, &abort_flag);
        else if (w == 1) said = mbar_wait_sleep<40>(smem_u32(bars + 1), 0, &abort_flag);
        else if (w == 2) said = mbar_wait_sleep<500>(smem_u32(bars + 2), 0, &abort_flag);
        else { mbar_arrive(smem_u32(bars + 3)); said = mbar_wait(smem_u32(bars + 3), 0, &abort_flag); }     // complete: at once
        out[3 * w] = said; out[3 * w + 1] = (long long)(clock_ns() - t0); out[3 * w + 2] = *(volatile int*)&abort_flag;
    }
}
extern "C" int run(long long* host) {
    long long* dev = nullptr;
    if (cudaMalloc(&dev, 12 * sizeof(long long)) != cudaSuccess) return 1;
    waits<<<1, 128>>>(dev);
    const int rc = cudaDeviceSynchronize() != cudaSuccess || cudaMemcpy(host, dev, 12 * sizeof(long long), cudaMemcpyDeviceToHost) != cudaSuccess;
    cudaFree(dev);
    return rc;
}
"""


def test_waits_run_out_after_a_second(lib_built, tmp_path):
    import torch
    nvcc = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "bin", "nvcc")
    (tmp_path / "waits.cu").write_text(SOURCE)
    so = tmp_path / "libwaits.so"
    r = subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-shared", "-Xcompiler", "-fPIC",
                        "-I" + os.path.join(ROOT, "minit_b200", "csrc"), str(tmp_path / "waits.cu"), "-o", str(so)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
    torch.zeros(1, device="cuda:0")
    out = (ctypes.c_longlong * 12)()
    assert ctypes.CDLL(str(so)).run(out) == 0
    said, took, flag = out[0::3], out[1::3], out[2::3]
    assert list(said) == [0, 0, 0, 1] and list(flag)[:3] == [1, 1, 1]
    assert all(0.9e9 <= t <= 1.3e9 for t in took[:3]), list(took)
    assert took[3] < 1e6
