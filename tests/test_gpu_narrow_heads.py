"""16-bit head dims 16 and 32 on the 64-channel tensor-core tiles: TMA supplies the missing channels as zeros and drops them
on store, the threads' own stores (padded rows, dQ conversion) stop at the true width."""
import pytest
import torch

from helpers import big_masks, bwd_kernels, check_forward, check_grads, ensure_built, make_inputs, oracle_all

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _lib():
    ensure_built()
    from chill_attention import _cabi

    lib = _cabi.load_library()
    yield lib
    assert lib.chill_read_device_status() == 0


def blhd(t):  # [B, L, H, D] in memory, every row between two rows of NaN guards
    B, H, n, d = t.shape
    buf = torch.full((B, n, H + 2, d), float("nan"), dtype=t.dtype, device="cuda")
    buf[:, :, 1:-1] = t.transpose(1, 2).cuda()
    return buf[:, :, 1:-1].transpose(1, 2)


@pytest.mark.parametrize("deterministic", [False, True], ids=["one_kernel", "two_kernels"])
@pytest.mark.parametrize("D", [16, 32])
@pytest.mark.parametrize("L", [1, 127, 128, 129, 400])
def test_width_edges(D, L, deterministic):
    import chill_attention as ca

    mask = big_masks()[(L + D) % 7]
    dtype = torch.float16 if D == 16 else torch.bfloat16
    q, k, v, do = make_inputs(3, 4, 2, L, D, dtype, seed=L + D)
    lens = torch.tensor([L, max(1, L // 3), 0], dtype=torch.int32)
    o_ref, lse_ref, *g_ref = oracle_all(mask, q, k, v, do, lens)

    qd, kd, vd = (blhd(t).requires_grad_(True) for t in (q, k, v))
    before = ca.is_deterministic()
    ca.set_deterministic(deterministic)
    try:
        o, lse = ca.chill_attention(qd, kd, vd, mask=mask, lens=lens.cuda(), return_lse=True)
        grads = torch.autograd.grad(o, (qd, kd, vd), blhd(do))
    finally:
        ca.set_deterministic(before)
    assert o.shape == q.shape and o.is_contiguous()
    check_forward(o, lse, o_ref, lse_ref, lens, dtype)
    if L > 1:
        check_grads(grads, g_ref, dtype, lens)
    else:  # one key: dQ = dK = 0 up to the rounding of P and dP - delta, only dV carries a value
        check_grads((grads[2],), (g_ref[2],), dtype)


@pytest.mark.parametrize("D", [16, 32])
def test_two_ctas_per_sm(D, _lib):
    """Large enough grids and few enough query tiles for the form of the backward that shares an SM between two CTAs."""
    import chill_attention as ca
    from chill_attention import _cabi

    mask, dtype, L = ca.SlidingWindowChillMask(40, 5), torch.bfloat16 if D == 16 else torch.float16, 330
    assert bwd_kernels(_lib, mask, 5, 30, 30, L, D, dtype, flags=_cabi.FLAG_NARROW_HEAD) == _cabi.BWD_SINGLE_PAIR
    q, k, v, do = make_inputs(5, 30, 30, L, D, dtype, seed=D)
    lens = torch.tensor([L, 0, 129, 64, 2], dtype=torch.int32)
    o_ref, lse_ref, *g_ref = oracle_all(mask, q, k, v, do, lens)
    qd, kd, vd = (blhd(t).requires_grad_(True) for t in (q, k, v))
    o, lse = ca.chill_attention(qd, kd, vd, mask=mask, lens=lens.cuda(), return_lse=True)
    check_forward(o, lse, o_ref, lse_ref, lens, dtype)
    check_grads(torch.autograd.grad(o, (qd, kd, vd), blhd(do)), g_ref, dtype, lens)
