"""Which kernels serve a backward call (chill_bwd_kernels; a host-side decision, asked without a GPU)."""
import pytest
import torch

from helpers import bwd_kernels, ensure_built


@pytest.fixture(scope="module")
def lib():
    ensure_built()
    from chill_attention import _cabi

    return _cabi.load_library()


def test_families(lib):
    import chill_attention as ca
    from chill_attention import _cabi

    full, h, b, f = ca.FullChillMask(), torch.float16, torch.bfloat16, torch.float32
    shape = (2, 4, 2, 300)
    ask = lambda D, dtype, **kw: bwd_kernels(lib, full, *shape, D, dtype, **kw)  # noqa: E731
    for D in (64, 128):
        assert ask(D, b) == _cabi.BWD_SINGLE
        assert ask(D, h, accum=False) == ask(D, h, flags=_cabi.FLAG_BWD_ONLY_DQ) == _cabi.BWD_TWO_KERNELS
        assert ask(D, f, flags=_cabi.FLAG_ALLOW_TF32) == _cabi.BWD_TF32
        assert ask(D, f) == ask(D, h, pointer=4098) == ask(D, h, flags=_cabi.FLAG_FORCE_GENERIC) == _cabi.BWD_CUDA_CORES
    for D in (16, 32):
        assert ask(D, h, flags=_cabi.FLAG_NARROW_HEAD) == _cabi.BWD_SINGLE
        assert ask(D, h) == ask(D, f) == _cabi.BWD_CUDA_CORES
    assert ask(256, b) == ask(256, b, accum=False) == _cabi.BWD_WIDE
    assert ask(256, b, flags=_cabi.FLAG_BWD_ONLY_DKDV) == ask(96, h) == _cabi.BWD_CUDA_CORES
    assert bwd_kernels(lib, full, 2, 3, 2, 300, 64, h) < 0  # H % H_kv != 0


def test_rule_of_the_form_with_two_ctas_per_sm(lib):
    """148 SMs (also what the library assumes without a GPU): 296 key tiles at least, four query tiles at most for a key tile in
    the middle, counted over the heads of its group; head dims up to 64."""
    import chill_attention as ca
    from chill_attention import _cabi

    def pair(mask, B, H, Hkv, L, D, flags=0):
        got = bwd_kernels(lib, mask, B, H, Hkv, L, D, torch.float16, flags)
        assert got in (_cabi.BWD_SINGLE, _cabi.BWD_SINGLE_PAIR)
        return got == _cabi.BWD_SINGLE_PAIR

    full, causal = ca.FullChillMask(), ca.CausalChillMask()
    assert pair(full, 37, 2, 2, 512, 64) and not pair(full, 1, 73, 73, 512, 64)          # 296 and 292 key tiles of four query tiles
    assert not pair(full, 37, 2, 2, 513, 64) and not pair(full, 37, 2, 2, 512, 128)      # five query tiles; head dim 128
    assert pair(full, 74, 4, 2, 256, 64) and not pair(full, 74, 6, 2, 256, 64)           # two tiles of two heads, of three heads
    assert pair(causal, 64, 1, 1, 896, 64) and not pair(causal, 64, 1, 1, 1024, 64)      # middle tile 3 of 7 sees four, 3 of 8 five
    assert pair(ca.ChunkwiseChillMask(128, 2), 1, 8, 8, 8192, 64) and pair(ca.SlidingWindowChillMask(16, 16), 8, 12, 12, 2085, 64)
    assert pair(ca.SlidingWindowChillMask(16, 16), 8, 12, 12, 2085, 32, _cabi.FLAG_NARROW_HEAD)
    assert not pair(ca.SlidingWindowChillMask(1024, 0), 1, 32, 32, 8192, 64)
