"""CPU checks of the module-level part of the Python surface: the constants
and free functions that the reference's Python module exposes from shtns.h
(shtns_numpy.i:115-135), with the reference's names."""
import types

import pytest

import shtns_b200


def test_module_exposes_reference_names():
    for name in ("sht", "rotation", "nlm_calc", "nlm_cplx_calc", "set_verbosity", "print_version", "build_info",
                 "shtns_use_threads", "shtns_use_gpu",
                 "sht_orthonormal", "sht_fourpi", "sht_schmidt", "SHT_NO_CS_PHASE", "SHT_REAL_NORM",
                 "sht_gauss", "sht_auto", "sht_reg_fast", "sht_reg_dct", "sht_quick_init", "sht_reg_poles",
                 "sht_gauss_fly", "SHT_NATIVE_LAYOUT", "SHT_THETA_CONTIGUOUS", "SHT_PHI_CONTIGUOUS",
                 "SHT_SOUTH_POLE_FIRST", "SHT_SCALAR_ONLY", "SHT_LOAD_SAVE_CFG", "SHT_ALLOW_GPU", "SHT_ALLOW_PADDING"):
        assert hasattr(shtns_b200, name), name
    # enum values as in shtns.h:48-75
    assert (shtns_b200.sht_gauss, shtns_b200.sht_reg_fast, shtns_b200.sht_gauss_fly) == (0, 2, 6)
    assert shtns_b200.SHT_PHI_CONTIGUOUS == 512 and shtns_b200.SHT_ALLOW_PADDING == 65536


def test_module_functions():
    for lmax, mmax, mres in [(127, 127, 1), (40, 16, 2), (31, 10, 3)]:
        assert shtns_b200.nlm_calc(lmax, mmax, mres) == (mmax + 1) * (lmax + 1) - mres * mmax * (mmax + 1) // 2
    # complex fields: orders -mmax..mmax, (lmax+1)^2 for a full triangle
    assert shtns_b200.nlm_cplx_calc(10, 10, 1) == 121
    assert "SHTns" in shtns_b200.build_info()
    shtns_b200.set_verbosity(0)
    shtns_b200.print_version()


class _FakeTensor:
    def __init__(self, ptr, n):
        self.ptr, self.n = ptr, n

    def data_ptr(self):
        return self.ptr

    def numel(self):
        return self.n


def test_into_forms_take_as_many_outputs_as_components(monkeypatch):
    """synth_into / analys_into on a library that records its calls: a missing
    output tensor is an IndexError (a null grid would be written), tensors
    beyond the components or beyond three of them are left out."""
    torch = pytest.importorskip("torch")
    sh = shtns_b200.sht(7)
    calls = []
    monkeypatch.setattr(sh, "_lib", types.SimpleNamespace(shtns_b200_transform=lambda cfg, st, nf, kind, *a: calls.append((nf, kind) + a) or 0))
    monkeypatch.setattr(sh, "nspat", 5, raising=False)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda: types.SimpleNamespace(cuda_stream=0))
    q = [_FakeTensor(10 + i, 2 * sh.nlm) for i in range(4)]
    v = [_FakeTensor(20 + i, 10) for i in range(4)]
    for n in (1, 2, 3):
        for call in (sh.synth_into, sh.analys_into):
            src, dst = (q, v) if call == sh.synth_into else (v, q)
            with pytest.raises(IndexError):
                call(src[:n], dst[:n - 1])
            assert not calls
            call(src[:n], dst)
            ptrs = tuple(x.ptr for x in src[:n] + dst[:n])
            assert calls.pop() == (2, n - 1 if src is q else n + 2) + ptrs + (None,) * (6 - 2 * n) + (7,)
    sh.synth_into(q, v)
    assert calls.pop()[:8] == (2, 2, 10, 11, 12, 20, 21, 22)
