"""Forward with two streams of key tiles per tile of queries (csrc/fwd_tc.cuh, chosen by fwd_two_streams: all CTAs resident at
once, loops of 6 64-key steps at head dim 64 and 16 at 128), merged at the end; and key tiles that start between multiples of 64."""
import pytest
import torch

from helpers import big_masks, check_forward, ensure_built, make_inputs, oracle_all

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built():
    ensure_built()


def check(mask, B, H, Hkv, L, D, dtype, lens=None):
    from chill_attention import _cabi, chill_attention

    q, k, v, do = make_inputs(B, H, Hkv, L, D, dtype, seed=L + D)
    o_ref, lse_ref, *_ = oracle_all(mask, q, k, v, do, lens)
    o, lse = chill_attention(q.cuda(), k.cuda(), v.cuda(), mask=mask, lens=None if lens is None else lens.cuda(), return_lse=True)
    assert _cabi.load_library().chill_read_device_status() == 0
    check_forward(o, lse, o_ref, lse_ref, lens, dtype)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16], ids=str)
@pytest.mark.parametrize("D,L", [(32, 385), (64, 321), (64, 384), (64, 449), (64, 640), (128, 961), (128, 1024), (128, 1090)])
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
