"""Backward of 16-bit head dim 256 (csrc/bwd_wide.cuh) at the edges of its pipeline: streamed tiles of 64 positions in two
stages (the tile that only a score GEMM reads in one, for dV in two), row tiles of 128, several heads of a group in one walk."""
import pytest
import torch

from helpers import all_masks, check_forward, check_grads, ensure_built, make_inputs, oracle_all

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built():
    ensure_built()


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16], ids=str)
@pytest.mark.parametrize("heads", [(2, 2), (3, 1)], ids=str)
@pytest.mark.parametrize("L", [33, 64, 65, 128, 129, 192, 193, 257, 385])
def test_tile_edges(L, heads, dtype):
    from chill_attention import _cabi, chill_attention

    H, Hkv = heads
    mask = all_masks()[(L + H) % 5]
    q, k, v, do = make_inputs(2, H, Hkv, L, 256, dtype, seed=L)
    lens = torch.tensor([L, L // 2], dtype=torch.int32) if L % 2 else None
    o_ref, lse_ref, *g_ref = oracle_all(mask, q, k, v, do, lens)
    qd, kd, vd = (t.cuda().requires_grad_(True) for t in (q, k, v))
    o, lse = chill_attention(qd, kd, vd, mask=mask, lens=None if lens is None else lens.cuda(), return_lse=True)
    grads = torch.autograd.grad(o, (qd, kd, vd), do.cuda())
    assert _cabi.load_library().chill_read_device_status() == 0
    check_forward(o, lse, o_ref, lse_ref, lens, dtype)
    check_grads(grads, g_ref, dtype, lens)
