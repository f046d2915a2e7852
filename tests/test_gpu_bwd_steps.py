"""Single-kernel backward (csrc/bwd_fused.cuh, bwd_fused64.cuh): the query steps of a key tile start at the 32-row group of the
first query that sees it, earlier where the last step would otherwise reach beyond the dQ accumulator."""
import pytest
import torch

from helpers import bwd_kernels, check_forward, check_grads, ensure_built, make_inputs, oracle_all
from oracle import attention_oracle as orc

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


def test_rows_whose_offset_needs_64_bits():
    """More than 2^24 query rows of 128 channels: the fp32 sums of the last rows lie beyond element 2^31 of their head.  The keys are
    the last 256 positions of the sequence; all queries but the last 512 are zero and see none of them (26 GB on the device)."""
    import chill_attention as ca
    from chill_attention import _cabi

    if torch.cuda.mem_get_info()[0] < 40e9:
        pytest.skip("needs 40 GB")
    mask, L, Lk, live, D, dtype = ca.SlidingWindowChillMask(100, 30), 2**24 + 256, 256, 512, 128, torch.bfloat16
    q_l, k, v, do_l = make_inputs(1, 1, 1, live, D, dtype, seed=24)
    k, v = k[:, :, :Lk].cuda(), v[:, :, :Lk].cuda()
    q, o, do, dq = (torch.zeros(1, 1, L, D, dtype=dtype, device="cuda") for _ in range(4))
    q[:, :, -live:], do[:, :, -live:] = q_l.cuda(), do_l.cuda()
    dq.fill_(7.0)
    dk, dv = torch.empty_like(k), torch.empty_like(v)
    lse, delta = (torch.empty(1, 1, L, device="cuda") for _ in range(2))
    lib = _cabi.load_library()
    shape = _cabi.make_shape(q, k, _cabi.BUILTIN_FUNCTOR_IDS[mask.cuda_functor], mask.constargs, None, D ** -0.5, k_offset=L - Lk, seq_len=L)
    _cabi.forward(lib, q, k, v, o, lse, shape)
    before = lib.chill_launch_count()
    _cabi.backward(lib, q, k, v, o, do, lse, delta, dq, dk, dv, shape)
    assert lib.chill_launch_count() - before == 3 and lib.chill_read_device_status() == 0  # delta, single kernel, dQ conversion
    q_pos, k_pos = torch.arange(L - live, L), torch.arange(L - Lk, L)
    md = orc.builtin_mask_dense(mask.name, mask.constargs, q_pos, k_pos)
    where = dict(q_pos=q_pos, k_pos=k_pos, seq_len=L)
    kc, vc = k.cpu().double(), v.cpu().double()
    o_ref, lse_ref = orc.attention_forward(md, q_l.double(), kc, vc, **where)
    check_forward(o[:, :, -live:], None, o_ref, lse_ref, None, dtype)
    g_ref = orc.attention_backward(md, q_l.double(), kc, vc, do_l.double(), **where)
    check_grads((dq[:, :, -live:], dk, dv), g_ref, dtype)
    assert not dq[:, :, :-live].any()


@pytest.mark.parametrize("D,B", [(32, 40), (64, 2), (64, 40), (128, 2), (256, 2)])
@pytest.mark.parametrize("mask_no", range(4))
def test_padding_behind_the_last_tile_may_hold_anything(mask_no, D, B):
    """lens at multiples of 128, NaN in all padded rows: tiles and steps that start between such multiples do not reach beyond them."""
    import chill_attention as ca

    mask = (ca.SlidingWindowChillMask(16, 16), ca.SlidingWindowChillMask(100, 0), ca.SlidingWindowChillMask(0, 70), ca.ChunkwiseChillMask(96, 1))[mask_no]
    L, dtype = 512, torch.float16
    clean = make_inputs(B, 3, 3, L, D, dtype, seed=D)
    lens = torch.tensor(([384, 512, 128, 256] * B)[:B], dtype=torch.int32)
    o_ref, lse_ref, *g_ref = oracle_all(mask, *clean, lens)
    dirty = [t.masked_fill(torch.arange(L)[None, None, :, None] >= lens[:, None, None, None], float("nan")).cuda() for t in clean]
    q, k, v = (t.requires_grad_(True) for t in dirty[:3])
    o, lse = ca.chill_attention(q, k, v, mask=mask, lens=lens.cuda(), return_lse=True)
    grads = torch.autograd.grad(o, (q, k, v), dirty[3])
    check_forward(o, lse, o_ref, lse_ref, lens, dtype)
    check_grads(grads, g_ref, dtype, lens)
