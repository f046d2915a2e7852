"""Pipelined backward kernels at the sizes where a ring, a step or a half tile can go wrong: one to a few steps (so that the
first round of every ring, the wrap-around and the last step are each reached), ragged ends, several heads per key tile."""
import pytest
import torch

from helpers import G_RTOL, big_masks, bwd_kernels, ensure_built, make_inputs, oracle_all

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
def test_head_dim_64_short_loops(kind, _lib):
    """Enough key tiles and few enough query tiles for the form with two CTAs per SM (steps of 64 queries, two to a dQ tile):
    first or last half of a query tile missing, ragged last step, rows of padding only, one or two heads per key head."""
    import chill_attention as ca
    from chill_attention import _cabi

    mask = {"window": ca.SlidingWindowChillMask(40, 5), "one_sided": ca.SlidingWindowChillMask(0, 70), "chunkwise": ca.ChunkwiseChillMask(64, 1),
            "off_grid_chunks": ca.ChunkwiseChillMask(48, 0), "full": ca.FullChillMask(), "causal": ca.CausalChillMask()}[kind]
    L, dtype = (200, torch.bfloat16) if kind in ("full", "causal") else (330, torch.float16)
    heads = 30 if kind in ("window", "off_grid_chunks") else 60  # these see three query tiles per key tile, the others two
    assert bwd_kernels(_lib, mask, 5, heads, 30, L, 64, dtype) == _cabi.BWD_SINGLE_PAIR
    q, k, v, do = make_inputs(5, heads, 30, L, 64, dtype, seed=7)
    lens = torch.tensor([L, L - 1, 129, 64, 2], dtype=torch.int32)
    _, _, *refs = oracle_all(mask, q, k, v, do, lens)
    _check(_gradients(mask, lens, q, k, v, do, "ieee"), refs, lens, G_RTOL[dtype])


def test_head_dim_64_short_loops_of_a_shard(_lib):
    """The same form for a shard: queries [q0, L) against keys [k0, L) (neither on a tile boundary), with the un-rounded fp32
    copies of the first and last dK / dV rows, which must round to the 16-bit outputs."""
    import ctypes as C

    import chill_attention as ca
    from chill_attention import _cabi

    L, q0, k0, H, D, dtype, head, tail = 330, 100, 20, 100, 64, torch.float16, 40, 30
    mask = ca.SlidingWindowChillMask(40, 5)
    q, k, v, do = make_inputs(1, H, H, L, D, dtype, seed=9)
    _, _, dq_ref, dk_ref, dv_ref = oracle_all(mask, q, k, v, do)
    qs, dos = (t[:, :, q0:].contiguous().cuda() for t in (q, do))
    ks, vs = (t[:, :, k0:].contiguous().cuda() for t in (k, v))
    shape = _cabi.make_shape(qs, ks, _cabi.BUILTIN_FUNCTOR_IDS[mask.cuda_functor], mask.constargs, None, D ** -0.5,
                             q_offset=q0, k_offset=k0, seq_len=L)
    o, lse = torch.empty_like(qs), torch.empty(1, H, L - q0, dtype=torch.float32, device="cuda")
    _cabi.forward(_lib, qs, ks, vs, o, lse, shape)
    delta = torch.empty_like(lse)
    accum = torch.empty(_lib.chill_bwd_dq_accum_bytes(C.byref(shape)) // 4, dtype=torch.float32, device="cuda")
    part = [torch.full((1, H, head + tail, D), float("nan"), dtype=torch.float32, device="cuda") for _ in range(2)]
    g = [torch.full_like(t, float("nan")) for t in (qs, ks, vs)]
    a = _cabi.backward_args(qs, ks, vs, o, dos, lse, delta, *g, shape, accum, part=(part[0], part[1], head, tail))
    assert _lib.chill_bwd_kernels(C.byref(a)) == _cabi.BWD_SINGLE_PAIR
    _cabi.check(_lib, _lib.chill_bwd_delta(C.byref(a), _cabi._stream()), "chill_bwd_delta")
    _cabi.check(_lib, _lib.chill_bwd(C.byref(a), _cabi._stream()), "chill_bwd")
    torch.cuda.synchronize()
    own = q0 + 5 - k0  # keys from here on are seen by queries of this shard only
    for name, got, ref in (("dq", g[0], dq_ref[:, :, q0:]), ("dk", g[1][:, :, own:], dk_ref[:, :, own + k0:]),
                           ("dv", g[2][:, :, own:], dv_ref[:, :, own + k0:])):
        got = got.cpu().double()
        assert torch.isfinite(got).all(), name
        assert ((got - ref).norm() / ref.norm()).item() <= G_RTOL[dtype], name
    for p, out in zip(part, g[1:]):
        assert torch.equal(p.to(dtype), torch.cat([out[:, :, :head], out[:, :, out.shape[2] - tail:]], dim=2))
