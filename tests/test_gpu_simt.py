"""CUDA-core kernels (csrc/simt.cuh) at the edges of their tiles: fp32 in IEEE arithmetic against the fp64 oracle.

A CTA owns 16 rows when few CTAs would be in flight and 64 (32 for head dims 128 / 256) otherwise; the streamed axis comes
in tiles of 64 positions; head dims are padded to 32, 64, 128 or 256 channels in shared memory."""
import pytest
import torch

from helpers import all_masks, check_forward, check_grads, ensure_built, make_inputs, oracle_all

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built():
    ensure_built()


def run(q, k, v, do, mask, lens):
    from chill_attention import chill_attention

    qd, kd, vd = (t.cuda().requires_grad_(True) for t in (q, k, v))
    o, lse = chill_attention(qd, kd, vd, mask=mask, lens=None if lens is None else lens.cuda(), return_lse=True)
    return o, lse, torch.autograd.grad(o, (qd, kd, vd), do.cuda())


@pytest.mark.parametrize("D", [16, 32, 64, 128, 256])
@pytest.mark.parametrize("L", [1, 15, 16, 17, 63, 64, 65, 130])
@pytest.mark.parametrize("heads", [(2, 1), (24, 12)], ids=["small_tiles", "large_tiles"])
def test_tile_edges(D, L, heads):
    H, Hkv = heads
    mask = all_masks()[(L + D // 16 + H) % 5]
    q, k, v, do = make_inputs(3, H, Hkv, L, D, torch.float32, seed=L + D)
    lens = torch.tensor([L, max(1, L // 2), L + 1], dtype=torch.int32) if L % 2 else None
    o_ref, lse_ref, *g_ref = oracle_all(mask, q, k, v, do, lens)
    o, lse, grads = run(q, k, v, do, mask, lens)
    check_forward(o, lse, o_ref, lse_ref, lens, torch.float32)
    if L > 1:
        check_grads(grads, g_ref, torch.float32, lens)
    else:
        # One key: P = 1 and dQ = dK = 0 because dP and delta are the same sum of D products.  Each of the two fp32 sums
        # is off by at most D * 2^-24 times the sum of the products' magnitudes.
        check_grads(grads[2:], g_ref[2:], torch.float32, lens)
        kv = lambda t: t.double().abs().repeat_interleave(H // Hkv, dim=1)  # noqa: E731
        ds = 2 * D * 2.0 ** -24 * D ** -0.5 * (do.double().abs() * kv(v)).sum(-1, keepdim=True)
        assert (grads[0].cpu().abs() <= ds * kv(k)).all()
        assert (grads[1].cpu().abs() <= (ds * q.double().abs()).unflatten(1, (Hkv, H // Hkv)).sum(2)).all()


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16], ids=str)
def test_element_types_and_strides_through_the_c_abi(dtype):
    """The same kernels for every element type (loads and stores convert), with a channel stride of 2."""
    from chill_attention import CausalChillMask, _cabi

    B, H, L, D = 2, 3, 70, 24
    mask, lib = CausalChillMask(), _cabi.load_library()
    q, k, v, do = make_inputs(B, H, H, L, D, dtype, seed=7)
    o_ref, lse_ref, *g_ref = oracle_all(mask, q, k, v, do)
    wide = [torch.zeros(B, H, L, 2 * D, dtype=dtype, device="cuda")[..., ::2] for _ in range(8)]
    for t, x in zip(wide, (q, k, v, do)):
        t.copy_(x)
    qd, kd, vd, dod, o, dq, dk, dv = wide
    lse, delta = (torch.empty(B, H, L, device="cuda") for _ in range(2))
    shape = _cabi.make_shape(qd, kd, _cabi.MASK_CAUSAL, (), None, D ** -0.5)
    _cabi.forward(lib, qd, kd, vd, o, lse, shape)
    _cabi.backward(lib, qd, kd, vd, o, dod, lse, delta, dq, dk, dv, shape)
    check_forward(o, lse, o_ref, lse_ref, None, dtype)
    check_grads((dq, dk, dv), g_ref, dtype)
