"""GPU: the prefill GEMM's tile widths (256, 192, 160 and 128 weight rows, chosen by how the units fill the chip) and its
launches of several weights, bit for bit against the oracle on sampled tokens: ragged rows and tokens, both operand formats,
activation groups that are whole slices, totals large enough to leave the fold's window, strided and unaligned outputs."""
import numpy as np
import pytest

from tests import inputs
from tests.test_gpu_parity import assert_bits, dev, gpu_mul_mat

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.fixture(scope="module")
def rq():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import ruquant_b200
    ruquant_b200.lib()
    return ruquant_b200


# rows and tokens with which the rule takes tiles of 128, 160, 192 and 256 rows on 148 SMs
WIDTHS = {128: (2117, 300), 160: (5107, 500), 192: (6113, 512), 256: (9001, 500)}


def blocks(port, K, N, wgroup, distinct=160):
    """N rows out of `distinct` adversarial ones: the oracle multiplies those, the rest follows"""
    w = inputs.reference_test_weights(distinct, K)
    return w, np.resize(port.quantize_weights(w, 44, wgroup=wgroup), (N, K // 256 * 144))


def check(port, wb, K, x, got, group, what, distinct=160):
    pick = np.unique(np.concatenate([[0, 127, 128, x.shape[0] - 1], np.arange(5, x.shape[0], 61)]))
    want = port.mul_mat(wb[:distinct], 44, K, x[pick], group=group)
    assert_bits(got[pick], want[:, np.arange(got.shape[1]) % distinct], what)


@pytest.mark.parametrize("wgroup,group", [(0, 64), (64, 64), (0, 128), (256, 256)])
@pytest.mark.parametrize("rows", sorted(WIDTHS))
def test_tile_widths(rq, port, rows, wgroup, group):
    N, M = WIDTHS[rows]
    for K in (256, 1792):          # K / 64 = 28 groups of 64; 14 of 128 and 7 of 256 are not multiples of four
        w, wb = blocks(port, K, N, wgroup)
        x = inputs.reference_test_activations(M, K, w, True, 31)
        check(port, wb, K, x, gpu_mul_mat(rq, wb, 44, K, x, group=group), group, "tile %d K=%d" % (rows, K))


@pytest.mark.parametrize("rows", sorted(WIDTHS))
def test_totals_beyond_the_window(rq, port, rows):
    """flat rows and tokens that carry the same signs: totals of 2^27, digits move into the carry words"""
    N, M = WIDTHS[rows]
    K = 17408
    w, wb = blocks(port, K, N, 0)
    x = inputs.reference_test_activations(M, K, w, True, 37)
    check(port, wb, K, x, gpu_mul_mat(rq, wb, 44, K, x), 64, "tile %d" % rows)


@pytest.mark.parametrize("wgroup", [0, 64])
def test_weights_of_one_launch(rq, port, wgroup):
    """three ragged weights in one launch; outputs inside wider buffers, one 4 bytes off a 16-byte boundary; what lies beyond
    a weight's rows and tokens stays as it was"""
    K, M, rows = 1024, 270, (1000, 130, 257)
    wbs = [blocks(port, K, N, wgroup) for N in rows]
    x = inputs.reference_test_activations(M, K, wbs[0][0], True, 41)
    ws = [rq.Weight(dev(wb).view(-1), 44, K, N=N) for (_, wb), N in zip(wbs, rows)]
    bufs = [torch.full((M + 1, N + 9), -7.0, device="cuda") for N in rows]
    outs = [b[:M, o:o + N] for b, N, o in zip(bufs, rows, (0, 1, 4))]
    work = rq.new_workspace(K, M)
    rq.mul_mat(ws, dev(x), out=outs, workspace=work, act_group=64)
    torch.cuda.synchronize()
    rq.device_status(work, K, M)
    for (_, wb), b, y, N in zip(wbs, bufs, outs, rows):
        check(port, wb, K, x, y.cpu().numpy(), 64, "N=%d" % N)
        assert int((b == -7.0).sum()) >= b.numel() - M * N
        assert (b[M] == -7.0).all()
