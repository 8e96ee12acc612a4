"""GPU: the batch-width contraction (9 to 64 tokens straight from the int4 stream) at the edges of its tiles, bit for bit
against the oracle: token counts around the multiples of 16, row counts around the 128-row tile and its 16-row parts, inputs
from one slice of 256 to the longest row, every activation group and multiplier mode, one and several weights, K split over
a cluster and not."""
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


def case(port, type_, N, M, K, wgroup, seed):
    w = inputs.reference_test_weights(N, K)
    return port.quantize_weights(w, type_, wgroup=wgroup), inputs.reference_test_activations(M, K, w, type_ == 44, seed)


@pytest.mark.parametrize("M", [9, 15, 16, 17, 32, 33, 47, 48, 49, 63, 64])
@pytest.mark.parametrize("N,K", [(1, 256), (16, 512), (113, 2048), (129, 5120), (272, 768)])
def test_edges_of_the_tiles(rq, port, M, N, K):
    wb, x = case(port, 44, N, M, K, 0, M)
    assert_bits(gpu_mul_mat(rq, wb, 44, K, x, path=1), port.mul_mat(wb, 44, K, x), "N=%d M=%d K=%d" % (N, M, K))


@pytest.mark.parametrize("M", [9, 32, 50])
@pytest.mark.parametrize("group,wgroup", [(64, 0), (128, 0), (256, 0), (64, 64), (64, 256), (128, 256), (256, 256)])
def test_groups_and_multipliers(rq, port, M, group, wgroup):
    wb, x = case(port, 45, 144, M, 3072, wgroup, 7)
    want = port.mul_mat(wb, 45, 3072, x, group=group)
    assert_bits(gpu_mul_mat(rq, wb, 45, 3072, x, group=group, path=1), want, "M=%d group=%d wgroup=%d" % (M, group, wgroup))


@pytest.mark.parametrize("K", [17408, 32768])
def test_longest_rows(rq, port, K):
    wb, x = case(port, 44, 130, 33, K, 0, 5)
    assert_bits(gpu_mul_mat(rq, wb, 44, K, x, path=1), port.mul_mat(wb, 44, K, x), "K=%d" % K)


def test_more_row_tiles_than_sms(rq, port):
    """one CTA walks several tiles: ring slots, phases and accumulators carry over (tiled weight rows: a property check)"""
    K, N, M = 1024, 20000, 40
    wb, x = case(port, 45, 160, M, K, 0, 11)
    got = gpu_mul_mat(rq, np.tile(wb, (N // 160, 1)), 45, K, x)
    assert_bits(got[:, :160], port.mul_mat(wb, 45, K, x), "first rows")
    assert (inputs.bits(got).reshape(M, N // 160, 160) == inputs.bits(got)[:, None, :160]).all()


def test_three_weights_and_token_passes(rq, port):
    """a shared activation with three ragged weights in one launch; 70 tokens on the forced path: a pass of 64 and one of 6"""
    K, rows = 1024, (200, 16, 129)
    for M, path in [(24, 0), (70, 1)]:
        wbs = [case(port, 45, N, M, K, 0, 3)[0] for N in rows]
        x = inputs.outlier_activations(M, K, 21)
        ws = [rq.Weight(dev(wb).view(-1), 45, K, N=N) for wb, N in zip(wbs, rows)]
        work = rq.new_workspace(K, M)
        ys = rq.mul_mat(ws, dev(x), path=path, workspace=work)
        torch.cuda.synchronize()
        rq.device_status(work, K, M)
        for wb, y, N in zip(wbs, ys, rows):
            assert_bits(y.cpu().numpy(), port.mul_mat(wb, 45, K, x), "M=%d N=%d" % (M, N))


GROUPS = [(64, 0), (128, 0), (256, 0), (64, 64), (64, 256), (128, 256), (256, 256)]
DISTINCT = 160


def tiled_weight(rq, port, type_, N, M, K, wgroup, seed):
    """N rows out of DISTINCT that repeat: the oracle multiplies those, the copies have to agree with them"""
    wb, x = case(port, type_, DISTINCT, M, K, wgroup, seed)
    blocks = dev(wb).repeat((N + DISTINCT - 1) // DISTINCT, 1)[:N].contiguous()
    return rq.Weight(blocks.view(-1), type_, K, N=N, layouts=rq.PREPACK_DECODE), wb, x


def check_tiled(port, wb, type_, K, x, y, group, what):
    assert_bits(y[:, :DISTINCT].cpu().numpy(), port.mul_mat(wb, type_, K, x, group=group), what)
    whole = y.shape[1] // DISTINCT * DISTINCT
    bits = y.contiguous().view(torch.int32)
    assert (bits[:, :whole].view(y.shape[0], -1, DISTINCT) == bits[:, None, :DISTINCT]).all(), what
    assert (bits[:, whole:] == bits[:, :y.shape[1] - whole]).all(), what


@pytest.mark.parametrize("M", [16, 30, 47, 64])
@pytest.mark.parametrize("group,wgroup", GROUPS)
def test_many_tiles_a_cta_in_every_mode(rq, port, M, group, wgroup):
    """more row tiles than CTAs (K not split) and 16 slices of K a tile: every ring, the accumulator sets and the multiplier slots
    wrap several times, for each tile width, activation group and multiplier mode"""
    K, N = 4096, 40000
    w, wb, x = tiled_weight(rq, port, 44, N, M, K, wgroup, 13)
    work = rq.new_workspace(K, M)
    y = rq.mul_mat(w, dev(x), act_group=group, workspace=work)
    torch.cuda.synchronize()
    rq.device_status(work, K, M)
    check_tiled(port, wb, 44, K, x, y, group, "M=%d group=%d wgroup=%d" % (M, group, wgroup))


@pytest.mark.parametrize("M", [2, 8, 9, 16])
@pytest.mark.parametrize("group,wgroup", GROUPS)
@pytest.mark.parametrize("N", [1000, 8200])
def test_gemv_tiles(rq, port, M, group, wgroup, N):
    """the GEMV with one and two tiles of 8 tokens: one and several rounds of row tiles a CTA, a ragged last tile"""
    K = 1024
    w, wb, x = tiled_weight(rq, port, 44, N, M, K, wgroup, 17)
    work = rq.new_workspace(K, M)
    y = rq.mul_mat(w, dev(x), act_group=group, workspace=work)
    torch.cuda.synchronize()
    rq.device_status(work, K, M)
    check_tiled(port, wb, 44, K, x, y, group, "M=%d N=%d group=%d wgroup=%d" % (M, N, group, wgroup))


@pytest.mark.parametrize("wgroup", [0, 64])
@pytest.mark.parametrize("M,N,K", [(12, 328, 1024), (16, 328, 5120), (47, 328, 5120), (64, 328, 5120), (16, 20008, 1024), (47, 20008, 1024), (64, 20008, 1024)])
def test_push(rq, port, M, N, K, wgroup):
    """outputs into two destinations, the second 4 bytes off a 16-byte boundary and both wider than the weight: from the GEMV's
    two tiles (12 tokens), from clusters that split K (328 rows) and from CTAs that walk whole tiles (20008 rows)"""
    w, wb, x = tiled_weight(rq, port, 44, N, M, K, wgroup, 19)
    ld = N + 8
    a = torch.full((M, ld), -1.0, device="cuda")
    b = torch.full((M * ld + 1,), -1.0, device="cuda")
    work = rq.new_workspace(K, M)
    rq.mul_mat_push([w], dev(x), [[a.data_ptr()], [b.data_ptr() + 4]], [ld], workspace=work)
    torch.cuda.synchronize()
    rq.device_status(work, K, M)
    for got in (a, b[1:].view(M, ld)):
        check_tiled(port, wb, 44, K, x, got[:, :N], 64, "push M=%d N=%d wgroup=%d" % (M, N, wgroup))
        assert (got[:, N:] == -1.0).all()
    assert float(b[0]) == -1.0
