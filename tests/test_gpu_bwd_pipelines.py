"""Pipelined backward kernels at the sizes where a ring, a step or a half tile can go wrong: one to a few steps (so that the
first round of every ring, the wrap-around and the last step are each reached), ragged ends, several heads per key tile."""
import pytest
import torch

from helpers import G_RTOL, big_masks, ensure_built, make_inputs, oracle_all

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _lib():
    ensure_built()
    from chill_attention import _cabi

    lib = _cabi.load_library()
    yield lib
    assert lib.chill_read_device_status() == 0


def _gradients(mask, lens, q, k, v, do, precision):
    import chill_attention as ca

    qd, kd, vd = (t.cuda().requires_grad_(True) for t in (q, k, v))
    o = ca.chill_attention(qd, kd, vd, mask=mask, lens=lens.cuda(), precision=precision)
    return torch.autograd.grad(o, (qd, kd, vd), do.cuda())


def _check(grads, refs, lens, rtol):
    for name, g, r in zip(("dq", "dk", "dv"), grads, refs):
        g = g.cpu().double()
        assert torch.isfinite(g).all(), name
        rel = ((g - r).norm() / r.norm()).item()
        assert rel <= rtol, f"{name} relative error {rel}"
        for b, n in enumerate(lens.tolist()):
            assert (g[b, :, n:] == 0).all(), f"{name}: padded rows must be exactly zero"


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("L", [32, 33, 64, 65, 96, 97, 129, 191, 260])
def test_tf32_steps(D, L):
    """Steps of 64 (head dim 64) or 32 positions, two stages; tolerance as stated for TF32 (operands lose all but 10 mantissa
    bits, i.e. 2^-10 relative each, through two GEMMs in a row)."""
    for mask in (big_masks()[L % 7], big_masks()[(L + 3) % 7]):
        q, k, v, do = make_inputs(2, 4, 2, L, D, torch.float32, seed=L + D)
        lens = torch.tensor([L, max(20, L // 3)], dtype=torch.int32)
        _, _, *refs = oracle_all(mask, q, k, v, do, lens)
        _check(_gradients(mask, lens, q, k, v, do, "tf32"), refs, lens, 5e-3)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16], ids=str)
@pytest.mark.parametrize("L", [2, 127, 128, 129, 257, 385, 513])
def test_head_dim_64_tiles(L, dtype):
    """1 to 10 query tiles per key tile (a ring of three stages, two dS tiles, dQ columns of their own), ragged ends."""
    for mask in (big_masks()[L % 7], big_masks()[(L + 2) % 7]):
        q, k, v, do = make_inputs(2, 4, 2, L, 64, dtype, seed=L)
        lens = torch.tensor([L, max(2, L // 3)], dtype=torch.int32)
        _, _, *refs = oracle_all(mask, q, k, v, do, lens)
        _check(_gradients(mask, lens, q, k, v, do, "ieee"), refs, lens, G_RTOL[dtype])


@pytest.mark.parametrize("kind", ["window", "one_sided", "chunkwise", "off_grid_chunks", "full", "causal"])
def test_head_dim_64_short_loops(kind):
    """Enough key tiles and few enough query tiles for the form with two CTAs per SM (steps of 64 queries, two to a dQ tile):
    first or last half of a query tile missing, ragged last step, rows of padding only, one or two heads per key head."""
    import chill_attention as ca

    mask = {"window": ca.SlidingWindowChillMask(40, 5), "one_sided": ca.SlidingWindowChillMask(0, 70), "chunkwise": ca.ChunkwiseChillMask(64, 1),
            "off_grid_chunks": ca.ChunkwiseChillMask(48, 0), "full": ca.FullChillMask(), "causal": ca.CausalChillMask()}[kind]
    L, dtype = (200, torch.bfloat16) if kind in ("full", "causal") else (330, torch.float16)
    heads = 30 if kind in ("window", "off_grid_chunks") else 60  # these see three query tiles per key tile, the others two
    q, k, v, do = make_inputs(5, heads, 30, L, 64, dtype, seed=7)
    lens = torch.tensor([L, L - 1, 129, 64, 2], dtype=torch.int32)
    _, _, *refs = oracle_all(mask, q, k, v, do, lens)
    _check(_gradients(mask, lens, q, k, v, do, "ieee"), refs, lens, G_RTOL[dtype])
