"""The native eager call path (chill_attention/_eager.py, csrc/torch_ext.cpp): what happens when it cannot serve a call."""
import warnings

import pytest
import torch

from helpers import check_forward, check_grads, ensure_built, make_inputs, oracle_all


@pytest.fixture(scope="module", autouse=True)
def _built():
    ensure_built()


@pytest.fixture(params=["missing", "not_a_library"])
def no_module(request, monkeypatch, tmp_path):
    """A tree in which only the kernel library was built, or whose native module was built for another torch."""
    from chill_attention import _eager, chill

    path = tmp_path / "_chill_torch.so"
    if request.param == "not_a_library":
        path.write_bytes(b"nothing the loader takes")
    monkeypatch.setattr(_eager, "EXTENSION", str(path))
    monkeypatch.setattr(_eager, "_extension", None)
    monkeypatch.setattr(_eager, "ENABLED", True)
    monkeypatch.setattr(chill, "_NATIVE", {})


def test_no_native_module_switches_the_path_off(no_module):
    from chill_attention import _cabi, _eager

    with pytest.raises((ImportError, _cabi.ChillLibraryError)):
        _eager.extension()
    with pytest.warns(UserWarning, match="dispatcher ops"):
        assert _eager.native_library(_cabi.load_library(), 0) is None
    assert _eager.ENABLED is False


@pytest.mark.gpu
def test_calls_without_a_native_module(no_module):
    import chill_attention as ca

    mask, dtype = ca.CausalChillMask(), torch.float16
    q, k, v, do = make_inputs(2, 4, 2, 150, 64, dtype)
    o_ref, lse_ref, *g_ref = oracle_all(mask, q, k, v, do)
    qd, kd, vd = (t.cuda().requires_grad_(True) for t in (q, k, v))
    with pytest.warns(UserWarning, match="dispatcher ops"):
        ca.chill_attention(qd, kd, vd, mask=mask)
    with warnings.catch_warnings():
        warnings.simplefilter("error")  # said once
        o, lse = ca.chill_attention(qd, kd, vd, mask=mask, return_lse=True)
    check_forward(o, lse, o_ref, lse_ref, None, dtype)
    check_grads(torch.autograd.grad(o, (qd, kd, vd), do.cuda()), g_ref, dtype)


def test_set_deterministic_while_the_module_loads(monkeypatch):
    """The flag is set by one thread between the moment another one hands it to the module and the moment the module is
    published; the module must end up with the new value."""
    import importlib.util
    import threading
    from types import SimpleNamespace

    from chill_attention import _cabi, _eager

    class Module:
        abi_version, flag, setter = _cabi.ABI_VERSION, None, None

        def set_deterministic(self, flag):
            self.flag = flag
            if self.setter is None:
                self.setter = threading.Thread(target=_cabi.set_deterministic, args=(True,))
                self.setter.start()
                self.setter.join(0.3)  # without a lock it is through by then

    module, spec = Module(), SimpleNamespace(loader=SimpleNamespace(exec_module=lambda m: None))
    monkeypatch.setattr(importlib.util, "spec_from_file_location", lambda *a: spec)
    monkeypatch.setattr(importlib.util, "module_from_spec", lambda s: module)
    monkeypatch.setattr(_eager, "EXTENSION", __file__)
    monkeypatch.setattr(_eager, "_extension", None)
    monkeypatch.setattr(_cabi, "_deterministic", False)
    assert _eager.extension() is module
    module.setter.join()
    assert _cabi.is_deterministic() and module.flag is True


@pytest.mark.gpu
def test_an_error_of_the_library_has_its_own_type_in_both_directions(monkeypatch):
    """chill_fwd or chill_bwd replaced by a host function that only returns a status."""
    import ctypes as C

    import chill_attention as ca
    from chill_attention import _cabi, _eager, chill

    refuse = C.CFUNCTYPE(C.c_int, C.c_void_p, C.c_void_p)(lambda args, stream: -4)
    mask, lib = ca.CausalChillMask(), _cabi.load_library()
    q = make_inputs(1, 2, 2, 64, 64, torch.float16)[0].cuda().requires_grad_(True)
    o = ca.chill_attention(q, q, q, mask=mask)  # registers the mask
    for name in ("chill_fwd", "chill_bwd"):
        addresses = [C.cast(refuse if n == name else getattr(lib, n), C.c_void_p).value for n in _eager._ENTRY_POINTS]
        monkeypatch.setitem(chill._NATIVE, mask.name, _eager.extension().Library(addresses, _cabi.MASK_CAUSAL))
        with pytest.raises(_cabi.ChillLibraryError, match=f"{name} failed: size exceeds"):
            o = ca.chill_attention(q, q, q, mask=mask)
            o.sum().backward()
    assert q.grad is None
