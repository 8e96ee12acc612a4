"""GPU: the activation quantizer's wait for its row, made to run out: a barrier whose copy is never issued, a short limit.  Every
thread of the CTA has to come back from the wait and meet the barrier behind it, and the error word has to say what happened."""
import ctypes
import os
import subprocess

import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "ruquant_b200", "csrc")
PROGRAM = r"""
#include "rq_common.cuh"
#include "rq_act_dev.cuh"
__global__ void probe(int32_t * status, int32_t * seen, long long cycles, int arrive) {
    __shared__ uint64_t bar;
    __shared__ int n;
    const uint32_t b = (uint32_t) __cvta_generic_to_shared(&bar);
    if (threadIdx.x == 0) {
        n = 0;
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" :: "r"(b) : "memory");
    }
    __syncthreads();
    if (threadIdx.x == 0 && arrive) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" :: "r"(b) : "memory");
    rq_act_dev::await_row(b, status, cycles);
    atomicAdd(&n, 1);
    __syncthreads();
    seen[threadIdx.x] = n;
}
extern "C" __attribute__((visibility("default"))) int run_probe(int32_t * status, int32_t * seen, int threads, long long cycles, int arrive) {
    probe<<<1, threads>>>(status, seen, cycles, arrive);
    return (int) cudaDeviceSynchronize();
}
"""


@pytest.mark.parametrize("threads", [128, 1024])
def test_a_wait_that_runs_out_is_reported_and_keeps_the_threads_together(tmp_path, threads):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from ruquant_b200 import build
    (tmp_path / "probe.cu").write_text(PROGRAM)
    so = str(tmp_path / "probe.so")
    subprocess.check_call([os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")] + build.NVCC_FLAGS + ["-shared", "-I", CSRC, str(tmp_path / "probe.cu"), "-o", so])
    run = ctypes.CDLL(so).run_probe
    run.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_int, ctypes.c_longlong, ctypes.c_int]
    for arrive, word in ((1, 0), (0, 1)):
        status = torch.zeros(64, dtype=torch.int32, device="cuda")
        seen = torch.zeros(threads, dtype=torch.int32, device="cuda")
        torch.cuda.synchronize()
        assert run(status.data_ptr(), seen.data_ptr(), threads, 2000000, arrive) == 0      # (about a millisecond)
        assert int(status[0]) == word
        assert (seen == threads).all()
