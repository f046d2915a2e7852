"""Single-kernel backward (csrc/bwd_fused.cuh, bwd_fused64.cuh): the query steps of a key tile start at the 32-row group of the
first query that sees it, earlier where the last step would otherwise reach beyond the dQ accumulator."""
import pytest
import torch

from helpers import bwd_kernels, check_grads, ensure_built, make_inputs, oracle_all

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built():
    ensure_built()


@pytest.mark.parametrize("D,B,H,Hkv", [(64, 50, 3, 3), (64, 2, 4, 2), (32, 40, 4, 4), (128, 2, 4, 2)])
@pytest.mark.parametrize("L", [129, 160, 255, 256, 289, 384])
@pytest.mark.parametrize("left,right", [(16, 16), (0, 40), (33, 5), (70, 70)])
def test_windows(left, right, L, D, B, H, Hkv):
    import chill_attention as ca
    from chill_attention import _cabi

    mask, dtype = ca.SlidingWindowChillMask(left, right), torch.float16
    q, k, v, do = make_inputs(B, H, Hkv, L, D, dtype, seed=L + left)
    lens = torch.tensor(([L, L - 40, 32, 1] * B)[:B], dtype=torch.int32)
    o_ref, lse_ref, *g_ref = oracle_all(mask, q, k, v, do, lens)
    qd, kd, vd = (t.cuda().requires_grad_(True) for t in (q, k, v))
    o = ca.chill_attention(qd, kd, vd, mask=mask, lens=lens.cuda())
    grads = torch.autograd.grad(o, (qd, kd, vd), do.cuda())
    lib = _cabi.load_library()
    assert lib.chill_read_device_status() == 0
    pair = bwd_kernels(lib, mask, B, H, Hkv, L, D, dtype, flags=_cabi.FLAG_NARROW_HEAD) == _cabi.BWD_SINGLE_PAIR
    assert pair == (B >= 40 and B * Hkv * -(-L // 128) >= 296)
    check_grads(grads, g_ref, dtype, lens)
