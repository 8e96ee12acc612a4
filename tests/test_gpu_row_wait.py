"""GPU: the wait for a row, made to run out: a barrier whose copy is never issued, a short limit.  Every thread of the CTA has to
come back from it and meet the barrier behind it; with an error word, the word has to say what happened, without one the row
has to be there all the same."""
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
    rq_act_dev::await_row(b, nullptr, nullptr, 0, threadIdx.x, blockDim.x, status, cycles);
    atomicAdd(&n, 1);
    __syncthreads();
    seen[threadIdx.x] = n;
}
// the wait that copies the row itself: a barrier whose copy is never issued, or the whole load
__global__ void surely(const float * src, float * out, int len, long long cycles, int issue) {
    extern __shared__ __align__(16) float buf[];
    __shared__ uint64_t bar;
    const uint32_t b = (uint32_t) __cvta_generic_to_shared(&bar);
    for (int i = threadIdx.x; i < len; i += blockDim.x) buf[i] = -1.0f;
    if (threadIdx.x == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" :: "r"(b) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    if (issue) rq_act_dev::bulk_load_row(buf, src, len, &bar, threadIdx.x, blockDim.x, nullptr);
    else rq_act_dev::await_row(b, buf, src, len, threadIdx.x, blockDim.x, nullptr, cycles);
    for (int i = threadIdx.x; i < len; i += blockDim.x) out[i] = buf[len - 1 - i];
}
extern "C" __attribute__((visibility("default"))) int run_surely(const float * src, float * out, int len, int threads, long long cycles, int issue) {
    surely<<<1, threads, len * sizeof(float)>>>(src, out, len, cycles, issue);
    return (int) cudaDeviceSynchronize();
}
extern "C" __attribute__((visibility("default"))) int run_probe(int32_t * status, int32_t * seen, int threads, long long cycles, int arrive) {
    probe<<<1, threads>>>(status, seen, cycles, arrive);
    return (int) cudaDeviceSynchronize();
}
"""


@pytest.fixture(scope="module")
def probe(tmp_path_factory):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from ruquant_b200 import build
    d = tmp_path_factory.mktemp("wait")
    (d / "probe.cu").write_text(PROGRAM)
    subprocess.check_call([os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")] + build.NVCC_FLAGS + ["-shared", "-I", CSRC, str(d / "probe.cu"), "-o", str(d / "probe.so")])
    return ctypes.CDLL(str(d / "probe.so"))


@pytest.mark.parametrize("threads", [128, 1024])
def test_a_wait_that_runs_out_is_reported_and_keeps_the_threads_together(probe, threads):
    run = probe.run_probe
    run.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_int, ctypes.c_longlong, ctypes.c_int]
    for arrive, word in ((1, 0), (0, 1)):
        status = torch.zeros(64, dtype=torch.int32, device="cuda")
        seen = torch.zeros(threads, dtype=torch.int32, device="cuda")
        torch.cuda.synchronize()
        assert run(status.data_ptr(), seen.data_ptr(), threads, 2000000, arrive) == 0      # (about a millisecond)
        assert int(status[0]) == word
        assert (seen == threads).all()


@pytest.mark.parametrize("issue", [0, 1])
@pytest.mark.parametrize("threads,length", [(128, 256), (128, 5120), (1024, 768), (256, 11264)])
def test_a_row_without_an_error_word_always_arrives(probe, threads, length, issue):
    """the wait runs out (no copy is issued): the threads copy the row themselves; and the load as the kernels call it"""
    run = probe.run_surely
    run.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_int, ctypes.c_int, ctypes.c_longlong, ctypes.c_int]
    src = torch.randn(length, device="cuda")
    out = torch.zeros(length, device="cuda")
    torch.cuda.synchronize()
    assert run(src.data_ptr(), out.data_ptr(), length, threads, 2000000, issue) == 0
    assert (out == src.flip(0)).all()
