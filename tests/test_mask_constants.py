"""Mask constants on their way to the kernels: the eager call path (csrc/torch_ext.cpp) and the dispatcher ops (_cabi.mask_desc)
must read them alike, whatever number a user passes for "unbounded"."""
import pytest
import torch

from helpers import ensure_built, make_inputs


@pytest.fixture(scope="module", autouse=True)
def _built():
    ensure_built()


def both(constants):
    from chill_attention import _cabi, _eager

    d = _cabi.mask_desc(0, constants)
    return _eager.extension().mask_constants(constants), list(zip(d.i, d.f))[:d.n_args]


def test_whole_numbers_truncate_and_saturate():
    top, bottom = 2**63 - 1, -2**63
    given = {0: 0, -3: -3, True: 1, 2.7: 2, -2.7: -2, 2**31 - 1: 2**31 - 1, 2**40: 2**40, top: top, bottom: bottom, 2**63: top,
             2**70: top, -2**70: bottom, 1e20: top, -1e20: bottom, 1e300: top, -1e300: bottom}
    for value, whole in given.items():
        native, ops = both((value, 5))
        assert native == ops == [(whole, float(value)), (5, 5.0)], value


@pytest.mark.parametrize("value,error", [(float("inf"), OverflowError), (-float("inf"), OverflowError), (float("nan"), ValueError)], ids=str)
def test_non_finite_constants_are_refused(value, error):
    from chill_attention import _cabi, _eager

    with pytest.raises(error):
        _cabi.mask_desc(0, (4, value))
    with pytest.raises(error):
        _eager.extension().mask_constants((4, value))


def test_at_most_eight():
    from chill_attention import _cabi, _eager

    for read in (lambda c: _cabi.mask_desc(0, c), _eager.extension().mask_constants):
        read(tuple(range(8)))
        with pytest.raises(ValueError):
            read(tuple(range(9)))


@pytest.mark.gpu
@pytest.mark.parametrize("eager", [True, False], ids=["eager", "ops"])
def test_unbounded_window_written_as_a_float(eager, monkeypatch):
    import chill_attention as ca
    from chill_attention import _eager

    monkeypatch.setattr(_eager, "ENABLED", eager)
    q, k, v, _ = (t.cuda() for t in make_inputs(2, 3, 3, 150, 32, torch.float32))
    window = lambda left: ca.chill_attention(q, k, v, mask=ca.SlidingWindowChillMask(left, 0))  # noqa: E731
    for left in (1e20, 1e300, 2**40):
        assert torch.equal(window(left), window(150)), left
    for left, error in ((float("inf"), OverflowError), (float("nan"), ValueError)):
        with pytest.raises(error):
            window(left)
