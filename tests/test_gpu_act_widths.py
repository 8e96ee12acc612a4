"""GPU: the activation quantizer over its launch shapes -- cluster widths by the number of tokens, one CTA per token with 128,
256 or 1024 threads, every Paley order's prefill kernel -- against the oracle, bit for bit: codes through both formats, group
multipliers and units; values on the rounding boundary of the codes, infinities of range (all-zero rows), odd token counts."""
import numpy as np
import pytest

import oracle
from tests import inputs
from tests.test_gpu_parity import dev

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.fixture(scope="module")
def rq():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import ruquant_b200
    ruquant_b200.lib()
    return ruquant_b200


def fields(rq, x, n_rot, clip, group, fmt):
    ws, a8, msh, u = rq.quantize(dev(x), n_rot, clip, group, fmt=fmt)
    torch.cuda.synchronize()
    rq.device_status(ws, x.shape[1], x.shape[0])
    return a8.cpu().numpy().view(np.uint8), msh.cpu().numpy(), u.cpu().numpy()


def check(rq, port, x, n_rot, clip, group, pick):
    """the int8 format against the oracle's fields for the picked tokens, the fp8 format against the int8 one for all"""
    M, K = x.shape
    a8, msh, u = fields(rq, x, n_rot, clip, group, rq.FMT_I8)
    f8, msf, uf = fields(rq, x, n_rot, clip, group, rq.FMT_E4M3)
    assert (u.view(np.uint32) == uf.view(np.uint32)).all() and (msf.view(np.float32) * 16 == msh).all()
    table = torch.arange(256, dtype=torch.uint8).view(torch.float8_e4m3fn).float().numpy()
    assert (table[f8] * 8 == a8.view(np.int8)).all()
    pos = np.array([16 * ((p % 16) // 4) + 4 * (p // 16) + p % 4 for p in range(64)])        # input at byte p of a run of 64
    got = np.empty_like(a8)
    for r in range(K // 64):
        got[:, 64 * r + pos] = a8[:, 64 * r:64 * r + 64]
    pick = np.array(pick)
    uo, mo, zo, qo = oracle.act_fields(port.quantize_act(x[pick], clip, group, n_rot), group)
    assert (got[pick].view(np.int8).astype(np.int32) == 8 * (qo - np.repeat(zo, group, axis=1))).all()
    assert (msh[pick] == mo).all() and (u[pick].view(np.uint32) == uo.view(np.uint32)).all()


@pytest.mark.parametrize("M", [2, 13, 17, 33, 41, 75])
@pytest.mark.parametrize("K", [768, 5120, 17408])
def test_cluster_widths(rq, port, K, M):
    x = inputs.outlier_activations(M, K, 50 + M)
    x[M - 1] = 0.0
    check(rq, port, x, K, 0.9, 64, sorted({0, M // 2, M - 1}))


# one rotation per Paley order, the power-of-two ones of one and several register runs, block-diagonal and narrow ones
ROTATIONS = [(256, 256), (4096, 4096), (8192, 8192), (3072, 3072), (5120, 2560), (11264, 11264), (15360, 15360), (17408, 17408),
             (18432, 18432), (21504, 21504), (26624, 26624), (27648, 27648), (768, 12), (4096, 0), (1536, 24), (32768, 32768)]


@pytest.mark.parametrize("K,n_rot", ROTATIONS)
@pytest.mark.parametrize("M", [130, 600])
def test_one_cta_per_token(rq, port, K, n_rot, M):
    x = inputs.student_t_activations(M, K, 60)
    x[5] = 0.0
    x[6] = np.round(x[6] * 2) / 2         # many values halfway between codes
    check(rq, port, x, n_rot, 0.95, 64, [0, 5, 6, M - 1])


@pytest.mark.parametrize("group", [128, 256])
def test_wider_groups(rq, port, group):
    x = inputs.spiky_activations(90, 5120, 70)
    check(rq, port, x, 5120, 1.0, group, [0, 44, 89])
