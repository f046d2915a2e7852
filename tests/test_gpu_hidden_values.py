"""fp32 attention on the CUDA cores (csrc/simt.cuh): what a row may not see does not reach it, whatever the value.

Padding comes from torch.empty or an unfilled cache as a rule, so rows at or beyond lens[b] may hold NaN and Inf; a value hidden
by the mask may be non-finite too.  A weight of zero times such a value is NaN, so the kernels must not form that product."""
import pytest
import torch

from helpers import all_masks, check_forward, check_grads, ensure_built, make_inputs, oracle_all

pytestmark = pytest.mark.gpu

BAD = (float("nan"), float("inf"), -float("inf"))


@pytest.fixture(scope="module", autouse=True)
def _built():
    ensure_built()


def run(tensors, mask, lens, strided=False):
    from chill_attention import chill_attention

    def place(t):
        if not strided:
            return t.cuda()
        wide = torch.full((*t.shape[:3], 2 * t.shape[3]), float("nan"), device="cuda")[..., ::2]
        return wide.copy_(t)

    q, k, v, do = (place(t) for t in tensors)
    qd, kd, vd = (t.detach().requires_grad_(True) for t in (q, k, v))
    o, lse = chill_attention(qd, kd, vd, mask=mask, lens=None if lens is None else lens.cuda(), return_lse=True)
    return o.detach(), lse.detach(), torch.autograd.grad(o, (qd, kd, vd), do)


@pytest.mark.parametrize("strided", [False, True], ids=["packed", "strided"])
@pytest.mark.parametrize("D", [16, 64, 128, 256])
@pytest.mark.parametrize("heads", [(2, 1), (24, 12)], ids=["small_tiles", "large_tiles"])
@pytest.mark.parametrize("mask_no", range(5))
def test_non_finite_padding(mask_no, heads, D, strided):
    """NaN, +Inf and -Inf in every padded row of q, k, v and dO; sequence lengths inside, at the end of and beyond a tile."""
    mask, (H, Hkv), L = all_masks()[mask_no], heads, 130
    clean = make_inputs(4, H, Hkv, L, D, torch.float32, seed=3 + D)
    lens = torch.tensor([L, 97, 64, 0], dtype=torch.int32)
    o_ref, lse_ref, *g_ref = oracle_all(mask, *clean, lens)
    dirty = [t.clone() for t in clean]
    for t in dirty:
        for b, n in enumerate(lens.tolist()):
            t[b, :, n:] = torch.tensor(BAD).repeat(D)[:D]
    o, lse, grads = run(dirty, mask, lens, strided)
    check_forward(o, lse, o_ref, lse_ref, lens, torch.float32)
    check_grads(grads, g_ref, torch.float32, lens)


@pytest.mark.parametrize("value", BAD, ids=str)
@pytest.mark.parametrize("where", ["q", "k", "v", "do"])
@pytest.mark.parametrize("D,heads", [(32, 2), (64, 24), (128, 24), (256, 2)], ids=str)
def test_non_finite_value_behind_the_mask(D, heads, where, value):
    """One non-finite element at a position that most rows of its tile cannot see: every result outside its reach is bitwise
    what it is without that element, and the rows that do see a non-finite V carry it."""
    import chill_attention as ca

    L, pos, ch = 150, 70, 5
    mask = ca.SlidingWindowChillMask(10, 4)
    clean = make_inputs(3, heads, heads, L, D, torch.float32, seed=D)
    dirty = [t.clone() for t in clean]
    dirty["q k v do".split().index(where)][:, :, pos, ch] = value
    o0, lse0, g0 = run(clean, mask, None)
    o1, lse1, g1 = run(dirty, mask, None)
    see = mask.make_mask(L, device="cpu")  # [query, key]
    rows = see[:, pos] if where in "kv" else torch.arange(L) == pos  # queries whose row of results the element can reach
    keys = see[rows].any(0)
    out = torch.zeros(L, dtype=torch.bool) if where == "do" else rows
    same = lambda a, b, hit: torch.equal(a[:, :, ~hit.to(a.device)], b[:, :, ~hit.to(a.device)])  # noqa: E731
    assert same(o0, o1, out) and same(lse0, lse1, out if where in "qk" else torch.zeros_like(out))
    assert same(g0[0], g1[0], rows) and same(g0[1], g1[1], keys) and same(g0[2], g1[2], keys)
    if where == "v":
        assert not torch.isfinite(o1[:, :, rows][..., ch]).any()
        rest = torch.arange(D) != ch
        assert torch.equal(o1[..., rest], o0[..., rest])
