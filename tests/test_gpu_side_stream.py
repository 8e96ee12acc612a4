"""GPU: calls on a side stream without a workspace.  The scratch of such a call must not be handed to the current stream while
the side stream still has the call ahead of it, and the results are those of a call on the current stream."""
import pytest

from tests import inputs
from tests.test_gpu_parity import dev

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

BUSY = 40_000_000        # cycles the side stream is kept busy with: 20 ms


@pytest.fixture(scope="module")
def rq():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import ruquant_b200
    ruquant_b200.lib()
    return ruquant_b200


def spy(monkeypatch, rq, name, index, seen):
    real = getattr(rq.lib(), name)

    def call(*a):
        seen.append(a[index])
        return real(*a)

    monkeypatch.setattr(rq.lib(), name, call)


def taken_by_current_stream(ptr, nbytes):
    """whether an allocation of the same size on the current stream gets the memory at ptr"""
    held = [torch.empty(nbytes, dtype=torch.uint8, device="cuda") for _ in range(4)]
    return any(h.data_ptr() <= ptr < h.data_ptr() + nbytes for h in held)


@pytest.mark.parametrize("M", [1, 40, 200])
def test_mul_mat(rq, port, monkeypatch, M):
    K, N = 5120, 512
    wb = port.quantize_weights(inputs.normal_weights(N, K, 9300), 45)
    w = rq.Weight(dev(wb).view(-1), 45, K, N=N)
    x = dev(inputs.outlier_activations(M, K, 9301))
    want = rq.mul_mat(w, x)
    seen, side = [], torch.cuda.Stream()
    spy(monkeypatch, rq, "rq_w4a4_mul_mat", 10, seen)
    torch.cuda.synchronize()
    with torch.cuda.stream(side):
        torch.cuda._sleep(BUSY)
    got = rq.mul_mat(w, x, stream=side)
    assert not side.query()
    assert not taken_by_current_stream(seen[0], rq.workspace_bytes(K, M))
    side.synchronize()
    assert (got.view(torch.int32) == want.view(torch.int32)).all()


@pytest.mark.parametrize("type_", [44, 45])
def test_quantize_weights(rq, monkeypatch, type_):
    K, N = 5120, 96
    w = dev(inputs.normal_weights(N, K, 9302))
    want = rq.quantize_weights(w, type_)
    seen, side = [], torch.cuda.Stream()
    spy(monkeypatch, rq, "rq_w4a4_quantize_weights", 8, seen)
    torch.cuda.synchronize()
    with torch.cuda.stream(side):
        torch.cuda._sleep(BUSY)
    got = rq.quantize_weights(w, type_, stream=side)
    assert not side.query()
    assert not taken_by_current_stream(seen[0], rq.lib().rq_w4a4_quantize_weights_scratch_bytes(type_, K, N, 0))
    side.synchronize()
    assert (got == want).all()
