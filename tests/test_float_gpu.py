"""Single-precision arrays: the kernels read and write them themselves and
compute in FP64, so a result is the FP64 result of the same (widened) input
rounded once, bit for bit.  Layouts, FFT families (prefetched, direct,
generic, four-step), latitude counts that tensor copies of floats cannot
address (not a multiple of 4), unaligned arrays, both adjoints."""
import ctypes as C

import pytest
import torch

from tests.common import rand_spec

pytestmark = pytest.mark.gpu

GRIDS = [(127, 192, 384, "theta"), (127, 190, 384, "theta"), (127, 192, 384, "phi"), (63, 66, 128, "theta"), (63, 66, 128, "phi"), (40, 42, 125, "theta"),
         (255, 384, 768, "theta"), (511, 514, 1536, "theta"), (63, 64, 6144, "theta"), (63, 64, 6144, "phi"), (31, 34, 12288, "phi"), (31, 34, 3072, "theta"), (31, 36, 3072, "phi"),
         (31, 1536, 3072, "theta"), (40, 128, 360, "theta"), (40, 130, 360, "theta"), (40, 128, 360, "phi"), (40, 128, 4096, "theta"),
         (40, 128, 4096, "phi"), (63, 66, 192, "phi"), (63, 66, 768, "phi"), (63, 66, 1536, "theta"), (63, 64, 1536, "phi")]


@pytest.mark.parametrize("lmax,nlat,nphi,layout", GRIDS)
@pytest.mark.parametrize("nf", [1, 3, 20])
def test_float_arrays_are_rounded_fp64_results(lmax, nlat, nphi, layout, nf):
    import shtns_b200
    from shtns_b200 import autograd
    dev = torch.device("cuda:0")
    sh = shtns_b200.sht(lmax)
    sh.set_grid(nlat, nphi, flags=shtns_b200.sht_quick_init | (shtns_b200.SHT_THETA_CONTIGUOUS if layout == "theta" else shtns_b200.SHT_PHI_CONTIGUOUS),
                polar_opt=1e-10)
    q = torch.from_numpy(rand_spec(lmax, lmax, 1, 5, nfields=nf)).to(dev).to(torch.complex64).requires_grad_(True)
    v = autograd.synth(sh, q)
    d = q.detach().to(torch.complex128).requires_grad_(True)
    w = autograd.synth(sh, d)
    # the grid through the four-step kernels and through the direct float kernels differs by rounding before the last rounding
    same = (lambda a, b: float((a.double() - b).abs().max()) <= 2.0 ** -22 * float(b.abs().max())) if nphi == 6144 else \
        (lambda a, b: torch.equal(a, b.to(a.dtype)))
    cplx = lambda x: torch.view_as_real(x) if x.is_complex() else x  # noqa: E731
    assert v.dtype == torch.float32 and same(v.detach(), w.detach())
    g = torch.randn(v.shape, dtype=torch.float32, device=dev, generator=torch.Generator(device=dev).manual_seed(1))
    a, = torch.autograd.grad(v, q, g)
    b, = torch.autograd.grad(w, d, g.double())
    assert a.dtype == torch.complex64 and same(cplx(a), cplx(b))
    x = g.clone().requires_grad_(True)
    y = g.double().requires_grad_(True)
    r, s = autograd.analys(sh, x), autograd.analys(sh, y)
    assert same(cplx(r.detach()), cplx(s.detach()))
    h = q.detach().conj()                                     # a lazy conjugate: its values count, not its storage
    a, = torch.autograd.grad(r, x, h)
    b, = torch.autograd.grad(s, y, h.resolve_conj().to(torch.complex128))
    assert same(a, b)


def test_float_arrays_at_odd_addresses():
    """Grids that start at an odd float and coefficients aligned to 4 bytes only."""
    import shtns_b200
    from shtns_b200 import capi
    lib = capi.load()
    dev = torch.device("cuda:0")
    sh = shtns_b200.sht(63)
    for nphi in (192, 200):
        sh.set_grid(96, nphi, flags=shtns_b200.sht_quick_init | shtns_b200.SHT_THETA_CONTIGUOUS, polar_opt=0.0)
        sh._batch(1)
        sh._stream()
        q = torch.from_numpy(rand_spec(63, 63, 1, 8)).to(dev).to(torch.complex64)
        raw = torch.zeros(2 * sh.nlm + 1, dtype=torch.float32, device=dev)
        raw[1:] = torch.view_as_real(q).flatten()
        grid = torch.zeros(sh.nspat + 1, dtype=torch.float32, device=dev)
        lib.cu_SH_to_spat_float(sh._cfg, C.c_void_p(raw.data_ptr() + 4), C.c_void_p(grid.data_ptr() + 4), 63)
        want = torch.empty(sh.spat_shape, dtype=torch.float32, device=dev)
        lib.cu_SH_to_spat_float(sh._cfg, C.c_void_p(q.data_ptr()), C.c_void_p(want.data_ptr()), 63)
        assert torch.equal(grid[1:], want.flatten()) and float(grid[0]) == 0.0
        back = torch.zeros(2 * sh.nlm + 1, dtype=torch.float32, device=dev)
        lib.cu_spat_to_SH_float(sh._cfg, C.c_void_p(grid.data_ptr() + 4), C.c_void_p(back.data_ptr() + 4), 63)
        ref = torch.empty_like(q)
        lib.cu_spat_to_SH_float(sh._cfg, C.c_void_p(want.data_ptr()), C.c_void_p(ref.data_ptr()), 63)
        assert torch.equal(back[1:], torch.view_as_real(ref).flatten()) and float(back[0]) == 0.0
        assert lib.shtns_b200_status() == 0


@pytest.mark.parametrize("nphi,layout,fourstep", [(3072, "theta", False), (3072, "phi", False), (6144, "phi", False), (6144, "theta", True)])
def test_device_memory_of_four_step_lengths(nphi, layout, fourstep):
    """Only a call that takes the four-step kernels pays for them: the analysis
    with a scratch grid per field, the FP32 transforms with FP64 copies of their
    arrays.  Here: the theta-contiguous 6144 (3072 has a four-step synthesis only,
    for grids beyond 96 MB)."""
    import shtns_b200
    from shtns_b200 import autograd, capi
    lib = capi.load()
    dev = torch.device("cuda:0")
    sh = shtns_b200.sht(31)
    sh.set_grid(34, nphi, flags=shtns_b200.sht_quick_init | (shtns_b200.SHT_THETA_CONTIGUOUS if layout == "theta" else shtns_b200.SHT_PHI_CONTIGUOUS),
                polar_opt=1e-10)
    nf = 8
    grids = 8 * nf * sh.nspat
    q = torch.from_numpy(rand_spec(31, 31, 1, 5, nfields=nf)).to(dev)
    v = sh.synth(q)
    before = lib.shtns_b200_device_bytes(sh._cfg)
    sh.analys(v)
    after = lib.shtns_b200_device_bytes(sh._cfg)
    assert after - before == (grids if fourstep else 0)
    with torch.no_grad():
        autograd.analys(sh, autograd.synth(sh, q.to(torch.complex64)))
    staged = lib.shtns_b200_device_bytes(sh._cfg) - after
    assert staged >= grids if fourstep else staged == 0
