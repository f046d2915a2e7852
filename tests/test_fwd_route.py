"""Which kernel serves a forward call (chill_fwd_kernel; a host-side decision, asked without a GPU)."""
import pytest
import torch

from helpers import ensure_built, fwd_kernel


@pytest.fixture(scope="module")
def lib():
    ensure_built()
    from chill_attention import _cabi

    return _cabi.load_library()


def test_families(lib):
    import chill_attention as ca
    from chill_attention import _cabi

    ask = lambda D, dtype, **kw: fwd_kernel(lib, ca.FullChillMask(), 2, 4, 2, 300, D, dtype, **kw)  # noqa: E731
    h, f = torch.float16, torch.float32
    for D in (64, 128, 256):
        assert ask(D, h) == ask(D, torch.bfloat16) == _cabi.FWD_ONE_STREAM
        assert ask(D, f) == ask(D, h, pointer=4098) == ask(D, h, flags=_cabi.FLAG_FORCE_GENERIC) == _cabi.FWD_CUDA_CORES
    assert ask(32, h, flags=_cabi.FLAG_NARROW_HEAD) == _cabi.FWD_ONE_STREAM and ask(32, h) == _cabi.FWD_CUDA_CORES
    assert ask(128, f, flags=_cabi.FLAG_ALLOW_TF32) == _cabi.FWD_TF32 and ask(32, f, flags=_cabi.FLAG_ALLOW_TF32) == _cabi.FWD_CUDA_CORES
    assert fwd_kernel(lib, ca.FullChillMask(), 2, 3, 2, 300, 64, h) < 0  # H % H_kv != 0


def test_rule_of_the_form_with_two_streams(lib):
    """148 SMs (also what the library assumes without a GPU).  Head dim 128: one wave of 148 tiles of 128 queries, 16 steps of 64
    keys.  Head dim 64: 296 tiles and 7 steps, or 592 tiles and 32 steps if the average is two thirds of the longest at most."""
    import chill_attention as ca
    from chill_attention import _cabi

    def two(mask, B, H, L, D, flags=0):
        got = fwd_kernel(lib, mask, B, H, H, L, D, torch.bfloat16, flags=flags)
        assert got in (_cabi.FWD_ONE_STREAM, _cabi.FWD_TWO_STREAMS)
        return got == _cabi.FWD_TWO_STREAMS

    full, causal, window = ca.FullChillMask(), ca.CausalChillMask(), ca.SlidingWindowChillMask
    assert two(full, 1, 16, 961, 128) and not two(full, 1, 16, 960, 128)                       # 16 and 15 steps
    assert two(full, 1, 18, 1024, 128) and not two(full, 1, 19, 1024, 128)                     # 144 and 152 tiles
    assert two(full, 1, 16, 385, 64) and not two(full, 1, 16, 384, 64)                         # 7 and 6 steps
    assert two(full, 1, 37, 1024, 64) and not two(full, 1, 38, 1024, 64)                       # 296 and 304 tiles
    assert two(full, 1, 37, 1024, 32, _cabi.FLAG_NARROW_HEAD) and not two(full, 1, 37, 1024, 256)
    assert two(causal, 1, 37, 2048, 64) and not two(causal, 1, 38, 2048, 64)                   # 592 and 608 tiles, 32 steps
    assert not two(causal, 1, 37, 1920, 64) and not two(full, 1, 30, 2048, 64)                 # 30 steps; all tiles alike
    assert two(window(256, 0), 2, 8, 1000, 64) is False and two(window(300, 0), 2, 8, 1000, 64)  # 6 and 7 steps
    assert not two(ca.ChunkwiseChillMask(128, 2), 1, 8, 4096, 64)
