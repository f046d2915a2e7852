"""Forward with two streams of key tiles per tile of queries (csrc/fwd_tc.cuh, chosen by fwd_two_streams: all CTAs resident at
once, loops of 7 64-key steps at head dim 64 and 16 at 128), merged at the end; and key tiles that start between multiples of 64."""
import pytest
import torch

from helpers import big_masks, check_forward, ensure_built, fwd_kernel, make_inputs, oracle_all

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built():
    ensure_built()


def most_steps(mask, L):
    """Steps of 64 keys of the longest tile of 128 queries."""
    lo, hi = (torch.as_tensor(x).expand(L) for x in type(mask).k_range_for_q(torch.arange(L), L, mask.constargs))
    return max(int(hi[t:t + 128].max().clamp(max=L - 1) - lo[t:t + 128].min().clamp(min=0)) // 64 + 1 for t in range(0, L, 128))


def check(mask, B, H, Hkv, L, D, dtype, lens=None, two=None):
    from chill_attention import _cabi, chill_attention

    route = fwd_kernel(_cabi.load_library(), mask, B, H, Hkv, L, D, dtype, flags=_cabi.FLAG_NARROW_HEAD)
    if two is None:  # tests of few tiles: the steps decide
        two = D < 256 and most_steps(mask, L) >= (16 if D == 128 else 7)
    assert route == (_cabi.FWD_TWO_STREAMS if two else _cabi.FWD_ONE_STREAM)
    q, k, v, do = make_inputs(B, H, Hkv, L, D, dtype, seed=L + D)
    o_ref, lse_ref, *_ = oracle_all(mask, q, k, v, do, lens)
    o, lse = chill_attention(q.cuda(), k.cuda(), v.cuda(), mask=mask, lens=None if lens is None else lens.cuda(), return_lse=True)
    assert _cabi.load_library().chill_read_device_status() == 0
    check_forward(o, lse, o_ref, lse_ref, lens, dtype)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16], ids=str)
@pytest.mark.parametrize("D,L", [(32, 385), (64, 321), (64, 384), (64, 385), (64, 448), (64, 449), (64, 640), (128, 961), (128, 1024), (128, 1090)])
@pytest.mark.parametrize("mask_no", range(7))
def test_two_streams(mask_no, D, L, dtype):
    """Even and odd numbers of steps; lens that leaves a tile of queries one step, or none, or a last step of one key."""
    lens = torch.tensor([L, L // 3, 130, 65, 0], dtype=torch.int32)
    check(big_masks()[mask_no], 5, 2, 1, L, D, dtype, lens)


@pytest.mark.parametrize("D,L", [(64, 4200), (128, 2100)])
def test_long_loops(D, L):
    """Running maxima that rise and fall between the streams: one stream's part of the row dominates by far."""
    import chill_attention as ca

    check(ca.CausalChillMask(), 1, 2, 2, L, D, torch.bfloat16)
    q, k, v, do = make_inputs(1, 1, 1, 1100, D, torch.float16, seed=9)
    k[:, :, 64:128] *= 8  # tile 1: scores of +-30 and more
    q *= 4
    o_ref, lse_ref, *_ = oracle_all(ca.FullChillMask(), q, k, v, do)
    o, lse = ca.chill_attention(q.cuda(), k.cuda(), v.cuda(), mask=ca.FullChillMask(), return_lse=True)
    check_forward(o, lse, o_ref, lse_ref, None, torch.float16)


@pytest.mark.parametrize("D", [64, 128, 256])
@pytest.mark.parametrize("left,right", [(16, 16), (1, 0), (0, 0), (63, 65), (100, 3)])
def test_key_tiles_start_anywhere(left, right, D):
    import chill_attention as ca

    check(ca.SlidingWindowChillMask(left, right), 2, 4, 2, 333, D, torch.float16, torch.tensor([333, 200], dtype=torch.int32))
    check(ca.ChunkwiseChillMask(left + 7, 1), 1, 2, 2, 301, D, torch.bfloat16)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16], ids=str)
def test_more_tiles_than_fit_at_once(dtype):
    """Causal, head dim 64, 320 tiles of queries: a few long loops outlast the rest; the full mask takes one stream there."""
    import chill_attention as ca

    check(ca.CausalChillMask(), 2, 10, 5, 2048, 64, dtype, two=True)
    check(ca.FullChillMask(), 2, 10, 5, 2048, 64, dtype, torch.tensor([2048, 700], dtype=torch.int32), two=False)
