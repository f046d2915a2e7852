"""fp32 attention of IEEE accuracy on the tensor cores (csrc/split.cuh: every operand as three bf16 parts, head dim <= 64).

A CTA owns 128 rows and takes the other axis in steps of 64 positions (the forward in two streams of alternate steps); the
CUDA-core kernels (FLAG_FORCE_GENERIC) serve as the reference for accuracy and for non-finite values."""
import pytest
import torch

from helpers import all_masks, big_masks, check_forward, check_grads, ensure_built, make_inputs, oracle_all

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built():
    ensure_built()


def run(q, k, v, do, mask, lens=None, split=True, blhd=False, **where):
    """O, LSE, dQ, dK, dV through the C ABI, and which route was taken (the split kernels launch the CUDA-core ones behind them)."""
    from chill_attention import _cabi

    def place(t):
        return t.transpose(1, 2).contiguous().cuda().transpose(1, 2) if blhd else t.cuda()

    lib = _cabi.load_library()
    q, k, v, do = (place(t) for t in (q, k, v, do))
    lens = None if lens is None else lens.cuda()
    o, dq, dk, dv = (torch.full_like(t, float("nan")) for t in (q, q, k, v))
    lse, delta = (torch.empty(q.shape[:3], device="cuda") for _ in range(2))
    shape = _cabi.make_shape(q, k, _cabi.BUILTIN_FUNCTOR_IDS[mask.cuda_functor], mask.constargs, lens, q.shape[-1] ** -0.5,
                             flags=0 if split else _cabi.FLAG_FORCE_GENERIC, **where)
    before = lib.chill_launch_count()
    _cabi.forward(lib, q, k, v, o, lse, shape)
    middle = lib.chill_launch_count()
    _cabi.backward(lib, q, k, v, o, do, lse, delta, dq, dk, dv, shape)
    routes = middle - before == 2, lib.chill_launch_count() - middle == 3
    torch.cuda.synchronize()
    assert lib.chill_read_device_status() == 0
    return (o, lse, dq, dk, dv), routes


@pytest.mark.parametrize("D", [16, 32, 64])
@pytest.mark.parametrize("L", [65, 127, 128, 129, 192, 193, 320, 511])
@pytest.mark.parametrize("mask_no", range(5))
def test_tile_edges(mask_no, L, D):
    mask = all_masks()[mask_no]
    q, k, v, do = make_inputs(6, 24, 12, L, D, torch.float32, seed=L + D)
    lens = torch.tensor([L, L // 2, 1, 0, L + 1, 64], dtype=torch.int32) if L % 2 else None
    o_ref, lse_ref, *g_ref = oracle_all(mask, q, k, v, do, lens)
    (o, lse, *grads), routes = run(q, k, v, do, mask, lens, blhd=L % 3 == 0)
    assert routes == (True, True)
    check_forward(o, lse, o_ref, lse_ref, lens, torch.float32)
    check_grads(grads, g_ref, torch.float32, lens)


@pytest.mark.parametrize("mask_no", range(7))
def test_no_further_from_the_exact_result_than_rounded_fma_chains(mask_no):
    """N(0, 1) inputs: each result at most as far from the 64-bit one as the CUDA-core kernels' (measured 0.3 to 0.95 of it)."""
    mask = big_masks()[mask_no]
    for L, D in ((700, 64), (500, 32)):
        inputs = make_inputs(2, 16, 8, L, D, torch.float32, seed=L)
        exact = oracle_all(mask, *inputs)
        mine, routes = run(*inputs, mask)
        fma, _ = run(*inputs, mask, split=False)
        assert routes == (True, True)
        for name, a, b, r in zip(("o", "lse", "dq", "dk", "dv"), mine, fma, exact):
            if name != "lse":
                assert (a.cpu().double() - r).norm() <= (b.cpu().double() - r).norm(), name


def test_sequence_shard():
    """Global offsets: queries 100.. of the sequence against keys 150.., rows of the shard that see none of its keys."""
    import chill_attention as ca

    mask, L = ca.SlidingWindowChillMask(90, 20), 400
    q, k, v, do = make_inputs(4, 16, 8, L, 64, torch.float32, seed=5)
    where = dict(q_offset=100, k_offset=150, seq_len=900)
    a, routes = run(q, k, v, do, mask, **where)
    b, _ = run(q, k, v, do, mask, split=False, **where)
    assert routes == (True, True)
    assert torch.equal(torch.isfinite(a[1]), torch.isfinite(b[1])) and not torch.isfinite(a[1]).all()
    for x, y in zip((a[0], *a[2:]), (b[0], *b[2:])):
        assert (x - y).norm() <= 2e-6 * y.norm()  # each within 1e-6 of the exact result


@pytest.mark.parametrize("value", [float("nan"), float("inf"), -float("inf"), 3.4e38], ids=str)
@pytest.mark.parametrize("where", ["q", "k", "v", "do"])
@pytest.mark.parametrize("D", [32, 64])
def test_values_bf16_cannot_hold(D, where, value):
    """The same results, non-finite ones included, as the CUDA-core kernels; bitwise those without the value out of its reach."""
    import chill_attention as ca

    mask, L, pos, ch = ca.SlidingWindowChillMask(40, 30), 330, 200, 3
    clean = make_inputs(4, 16, 16, L, D, torch.float32, seed=D)
    dirty = [t.clone() for t in clean]
    dirty["q k v do".split().index(where)][:, 3:, pos, ch] = value
    base, routes = run(*clean, mask)
    a, _ = run(*dirty, mask)
    b, _ = run(*dirty, mask, split=False)
    assert routes == (True, True)
    for name, x, y in zip(("o", "lse", "dq", "dk", "dv"), a, b):
        assert torch.equal(torch.isnan(x), torch.isnan(y)), name
        fin = torch.isfinite(y)
        assert torch.equal(x[~fin].nan_to_num(7.0), y[~fin].nan_to_num(7.0)), name
        assert ((x[fin].double() - y[fin].double()).abs() <= 1e-5 * y[fin].double().abs().max()).all(), name
    see = mask.make_mask(L, device="cpu")
    rows = see[:, pos] if where in "kv" else torch.arange(L) == pos
    keys = see[rows].any(0)
    for x, y, hit in zip(a, base, (rows, rows, rows, keys, keys)):
        assert torch.equal(x[:, :, ~hit.to(x.device)], y[:, :, ~hit.to(x.device)])


@pytest.mark.parametrize("mask_no", [0, 2])
@pytest.mark.parametrize("layout", ["bhld", "blhd", "wide_rows"])
@pytest.mark.parametrize("D", [16, 32, 48, 64])
def test_nothing_but_the_rows_is_written(D, layout, mask_no):
    """Every head dim the kernels take, 48 among them: results inside buffers whose other elements (before, between and behind the
    rows) keep their value.  Rows 4 channels apart, heads in between ([batch, position, head, channel]), packed."""
    from chill_attention import _cabi

    mask, B, H, L, guard, fill = all_masks()[mask_no], 6, 24, 193, 256, 7.0
    row = D + 4 if layout == "wide_rows" else D

    def buffer(heads):
        return torch.full((B * heads * L * row + 2 * guard,), fill, device="cuda"), heads

    def view(buf, heads):
        strides = (L * heads * row, row, heads * row, 1) if layout == "blhd" else (heads * L * row, L * row, row, 1)
        return buf.as_strided((B, heads, L, D), strides, guard)

    q, k, v, do = make_inputs(B, H, H // 2, L, D, torch.float32, seed=D)
    o_ref, lse_ref, *g_ref = oracle_all(mask, q, k, v, do)
    q, k, v, do = (t.cuda() for t in (q, k, v, do))
    buffers = [buffer(heads) for heads in (H, H, H // 2, H // 2)]
    o, dq, dk, dv = (view(*b) for b in buffers)
    lse, delta = (torch.empty(B, H, L, device="cuda") for _ in range(2))
    lib = _cabi.load_library()
    shape = _cabi.make_shape(q, k, _cabi.BUILTIN_FUNCTOR_IDS[mask.cuda_functor], mask.constargs, None, D ** -0.5)
    before = lib.chill_launch_count()
    _cabi.forward(lib, q, k, v, o, lse, shape)
    _cabi.backward(lib, q, k, v, o, do, lse, delta, dq, dk, dv, shape)
    assert lib.chill_launch_count() - before == 5  # the split kernels ran, forward and backward
    check_forward(o, lse, o_ref, lse_ref, None, torch.float32)
    check_grads((dq, dk, dv), g_ref, torch.float32)
    for buf, heads in buffers:
        view(buf, heads).fill_(fill)
        assert (buf == fill).all()


def test_head_dim_48_from_host_memory():
    """attention_fwd_bwd_host takes any head dim: packed heads, so that a row's neighbour is the next one."""
    from chill_attention.host import attention_fwd_bwd_host

    mask = all_masks()[1]
    inputs = make_inputs(2, 16, 8, 257, 48, torch.float32, seed=48)
    o_ref, _, *g_ref = oracle_all(mask, *inputs)
    o, *grads = attention_fwd_bwd_host(*(t.pin_memory() for t in inputs), mask)
    check_forward(o, None, o_ref, None, None, torch.float32)
    check_grads(grads, g_ref, torch.float32)


@pytest.mark.parametrize("kind", ["all", "one_channel", "one_position"])
@pytest.mark.parametrize("where", ["v", "k", "q", "do"])
def test_non_finite_inputs_cost_no_more_than_on_the_cuda_cores(where, kind):
    """NaN everywhere, in one channel of every position, in one position that all queries see.  Measured, split / CUDA cores: forward
    0.2 to 0.9, backward 0.9; a walk of every row over all its keys took 9 to 25 times as long.  Bound: twice."""
    import chill_attention as ca

    mask = ca.FullChillMask()
    inputs = [t.cuda() for t in make_inputs(2, 8, 8, 1000, 64, torch.float32, seed=1)]
    bad = inputs["q k v do".split().index(where)]
    bad[{"all": (...,), "one_channel": (..., 7), "one_position": (slice(None), slice(None), 5)}[kind]] = float("nan")

    def fastest(split):
        times = []
        for _ in range(4):
            start, end = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            start.record()
            run(*inputs, mask, split=split)
            end.record()
            torch.cuda.synchronize()
            times.append(start.elapsed_time(end))
        return min(times[1:])

    assert fastest(True) <= 2 * fastest(False)


@pytest.mark.parametrize("positions", [1, 4, 5, 9])
@pytest.mark.parametrize("value", [float("nan"), float("inf"), -float("inf")], ids=str)
def test_some_non_finite_positions_of_v(value, positions):
    """Up to four per row and stream are looked up by the row itself, rows with more are left to the CUDA cores: the same results."""
    import chill_attention as ca

    clean = make_inputs(2, 8, 4, 700, 64, torch.float32, seed=2)
    for at in (torch.arange(positions) * 3 + 65, torch.arange(positions) * 128 % 700):  # in one tile; all over the keys
        q, k, v, do = (t.clone() for t in clean)
        v[:, :, at, 11] = value
        mine, routes = run(q, k, v, do, ca.FullChillMask())
        ref, _ = run(q, k, v, do, ca.FullChillMask(), split=False)
        assert routes == (True, True)
        for a, b in zip(mine, ref):
            assert torch.equal(torch.isfinite(a), torch.isfinite(b)) and torch.equal(torch.isnan(a), torch.isnan(b))
            fin = torch.isfinite(b)
            assert (a[fin] - b[fin]).norm() <= 2e-6 * b[fin].norm()
        assert not torch.isfinite(mine[0][..., 11]).any() and torch.isfinite(mine[0][..., :11]).all()


#: factors of q, k, v, dO
SCALES = {"v tiny": (1, 1, 1e-36, 1), "dO tiny": (1, 1, 1, 1e-36), "dO tiny, v large": (1, 1, 1e30, 1e-37), "q tiny": (1e-36, 1, 1, 1),
          "k tiny": (1, 1e-36, 1, 1), "dO subnormal": (1, 1, 1, 1e-40), "v and dO small": (1, 1, 1e-30, 1e-5),
          "q and k beyond the scores' limit": (1e-15, 1e15, 1, 1), "v and dO large": (1, 1, 1e15, 1e15), "v beyond the limit": (1, 1, 1e35, 1)}


@pytest.mark.parametrize("scales", SCALES)
@pytest.mark.parametrize("mask_no,L,D", [(0, 700, 64), (3, 500, 32)])
def test_as_exact_at_any_scale(mask_no, L, D, scales):
    """Each result at most as far from the 64-bit one as the CUDA-core kernels' (measured 0.1 to 0.9 of it; rows that they compute: the
    same up to what they take from the forward, 1.1)."""
    mask = big_masks()[mask_no]
    inputs = [(t.double() * f).float() for t, f in zip(make_inputs(2, 16, 8, L, D, torch.float32, seed=L), SCALES[scales])]
    exact = oracle_all(mask, *inputs)
    mine, routes = run(*inputs, mask)
    fma, _ = run(*inputs, mask, split=False)
    assert routes == (True, True)
    for name, a, b, r in zip(("o", "lse", "dq", "dk", "dv"), mine, fma, exact):
        if name != "lse" and torch.isfinite(b).all():
            assert (a.cpu().double() - r).norm() <= 1.1 * (b.cpu().double() - r).norm(), name
        else:
            assert torch.equal(torch.isfinite(a), torch.isfinite(b)), name


def test_mixed_scales_within_a_row():
    """Some positions have eight tiny channels beside ordinary ones: every channel of every row as exact as on the CUDA cores."""
    import chill_attention as ca

    mask = ca.SlidingWindowChillMask(90, 40)
    q, k, v, do = make_inputs(2, 16, 16, 600, 64, torch.float32, seed=4)
    for t in (v, do):
        t[..., 8:16] *= 1e-36
        t[:, :, ::7, 40:48] *= 1e-35
    inputs = (q, k, v, do)
    exact = oracle_all(mask, *inputs)
    mine, _ = run(*inputs, mask)
    fma, _ = run(*inputs, mask, split=False)
    for i in (0, 4):  # O, dV: channel by channel
        err = lambda x: (x.cpu().double() - exact[i]).norm(dim=2) / exact[i].norm(dim=2)  # noqa: E731, B023
        assert (err(mine[i]) <= 1.2 * err(fma[i]).clamp(min=2e-7)).all()



@pytest.mark.parametrize("D,B,H,Hkv,L,window,split", [
    (64, 1, 16, 2, 256, 32, (False, False)),   # 4 key tiles of 24 steps each; the CUDA cores' 16-row tiles have 16
    (64, 1, 8, 1, 512, None, (True, True)),    # few tiles, but as many steps for 16 rows as for 128
    (32, 1, 8, 1, 512, None, (False, False)),
    (32, 1, 2, 1, 2048, None, (True, True)),   # forward: 256 tiles of 16 rows, 32 steps; backward: 96 tiles of 64 rows
    (32, 1, 1, 1, 2048, None, (False, False)),
    (64, 1, 8, 8, 1024, 32, (False, True)),    # narrow: 184 steps, 256 needed
    (64, 1, 8, 8, 2048, 32, (True, True)),
    (32, 2, 8, 8, 2048, 32, (True, False)),
    (32, 1, 8, 1, 4096, 32, (True, True)),
    (16, 2, 8, 8, 2048, 32, (True, True)),
    (64, 1, 8, 8, 256, None, (False, False)),  # 64 steps
])
def test_route(D, B, H, Hkv, L, window, split):
    """Both sides of each line of the dispatch rule, with results within each other's error."""
    import chill_attention as ca

    mask = ca.FullChillMask() if window is None else ca.SlidingWindowChillMask(window, 0)
    inputs = make_inputs(B, H, Hkv, L, D, torch.float32, seed=L)
    mine, routes = run(*inputs, mask)
    ref, _ = run(*inputs, mask, split=False)
    assert routes == split
    for a, b in zip(mine, ref):
        assert (a - b).norm() <= 3e-6 * b.norm()


@pytest.mark.parametrize("mask_no", [0, 1, 4])
@pytest.mark.parametrize("L", [129, 1000])
def test_inputs_of_one_sign(L, mask_no):
    """What the tensor core's truncation takes is one-sided, so it does not average out here.  Measured, distance from the 64-bit result
    over the CUDA cores': O 0.65, dQ 1.0, dK 1.3 (2.8e-7 and 2.2e-7), dV 0.6; bound: 1.5."""
    mask = big_masks()[mask_no]
    inputs = [t.abs() for t in make_inputs(4, 16, 16, L, 64, torch.float32, seed=L)]
    exact = oracle_all(mask, *inputs)
    mine, routes = run(*inputs, mask)
    fma, _ = run(*inputs, mask, split=False)
    assert routes == (True, True)
    for i in (0, 2, 3, 4):
        assert (mine[i].cpu().double() - exact[i]).norm() <= 1.5 * (fma[i].cpu().double() - exact[i]).norm(), "o lse dq dk dv".split()[i]
