"""The generic phi-FFT kernels (sht_fft_gen.cu) against torch.fft, through the
FFT stage entry points, at sizes where their pass plans change: one radix, the
primes alone, two to seven passes, each register class, the largest sizes, and
row counts that end inside a tile.  Every size runs a call of few latitudes
(direct loads, short butterflies) and one of more than 1000 latitude pairs
(input staged by tensor copies), and the plan that ran is checked (option 11).
Bar: 1e-13 of the largest value (a pass of radix <= 16 adds a few 2^-53; at most
eight passes and their twiddle products)."""
import ctypes as C

import pytest
import torch

from tests.common import relerr

pytestmark = pytest.mark.gpu

# nphi: (values per thread, passes) of a large and of a small call
PLANS = {1: (82, 82), 2: (82, 82), 3: (82, 82), 5: (82, 82), 7: (82, 82), 9: (122, 82), 16: (82, 82), 18: (82, 82), 25: (82, 82), 49: (82, 82),
         64: (82, 82), 90: (122, 83), 125: (83, 83), 216: (83, 83), 243: (123, 85), 343: (83, 83), 360: (123, 84), 512: (83, 83), 720: (123, 84),
         1000: (123, 84), 1024: (84, 84), 1440: (123, 84), 1680: (84, 84), 2187: (124, 87), 2401: (84, 84), 3000: (124, 124), 3125: (125, 125),
         4050: (124, 124), 4096: (163, 163), 5040: (124, 124), 5832: (124, 124), 6250: (125, 125), 6300: (164, 164), 6400: (124, 124)}


@pytest.mark.parametrize("layout", ["theta", "phi"])
@pytest.mark.parametrize("nphi", PLANS)
def test_generic_fft_matches_torch(nphi, layout):
    import shtns_b200
    from shtns_b200 import capi
    lib = capi.load()
    dev = torch.device("cuda:0")
    phi = layout == "phi"
    mmax = (nphi - 1) // 2 if nphi % 2 else nphi // 3        # up to the last order below Nyquist, or a zero band
    if nphi > 1100 and nphi not in (2187, 5040):
        mmax = min(mmax, 150)                                # fewer orders: quicker plans
    nlat = 2 * ((mmax + 44) // 2)
    sh = shtns_b200.sht(max(mmax, 2), mmax)
    sh.set_grid(nlat, nphi, flags=shtns_b200.sht_quick_init | (shtns_b200.SHT_PHI_CONTIGUOUS if phi else shtns_b200.SHT_THETA_CONTIGUOUS),
                polar_opt=0.0)
    lib.shtns_b200_set_option(sh._cfg, 3, 1)
    lib.cushtns_set_streams(sh._cfg, C.c_void_p(torch.cuda.current_stream().cuda_stream), None)
    g = torch.Generator(device=dev).manual_seed(nphi)
    err = lambda a, b: float((a - b).abs().max() / a.abs().max())  # noqa: E731
    many = 2002 // nlat + 1                                  # fields of a call of more than 1000 pairs
    # (whole grids for several fields: fields of a block of rows lie nspat apart)
    for nrows, nf, pairs in ((nlat, 2, 0), (nlat, many, 0), (2, 1, 0), (10, 1, 0), (38, 1, 8), (38, 1, 1)):
        lib.shtns_b200_set_option(sh._cfg, 1, pairs)
        shape = (nf, nrows, nphi) if phi else (nf, nphi, nrows)
        lib.shtns_set_batch(sh._cfg, nf, sh.nlm, nrows * nphi)
        small = nf * nrows // 2 <= 1000
        plan = PLANS[nphi][small]
        F = torch.randn((nf, mmax + 1, nrows), dtype=torch.complex128, generator=g, device=dev)
        F[:, 0] = F[:, 0].real.to(torch.complex128)
        v = torch.full(shape, float("nan"), dtype=torch.float64, device=dev)
        lib.shtns_b200_status()
        lib.shtns_b200_fourier_synth(sh._cfg, 0, C.c_void_p(F.data_ptr()), C.c_void_p(v.data_ptr()), None, None, nrows, sh.lmax)
        torch.cuda.synchronize()
        assert lib.shtns_b200_status() == 0, lib.shtns_b200_last_error().decode()
        assert lib.shtns_b200_get_option(sh._cfg, 6) == 0
        # of the small calls the synthesis of long rows is staged, beyond 2^19 points and without a wide zero band
        long_rows = nphi > 1024 and nf * nrows // 2 * nphi > 2 ** 19 and 4 * (mmax + 1) >= nphi
        assert lib.shtns_b200_get_option(sh._cfg, 11) == 10 * plan + (not small or long_rows), (nrows, nf)
        z = torch.zeros((nf, nphi // 2 + 1, nrows), dtype=torch.complex128, device=dev)
        z[:, : mmax + 1] = F
        want = torch.fft.irfft(z, nphi, dim=1, norm="forward")
        want = want.transpose(1, 2) if phi else want
        assert err(want, v) < 1e-13, (nrows, nf, pairs)
        w = torch.randn(shape, dtype=torch.float64, generator=g, device=dev)
        G = torch.full((nf, mmax + 1, nrows), float("nan"), dtype=torch.complex128, device=dev)
        lib.shtns_b200_fourier_analys(sh._cfg, 0, C.c_void_p(w.data_ptr()), None, None, C.c_void_p(G.data_ptr()), nrows, sh.lmax)
        torch.cuda.synchronize()
        assert lib.shtns_b200_status() == 0, lib.shtns_b200_last_error().decode()
        assert lib.shtns_b200_get_option(sh._cfg, 11) == 10 * plan + (not small and not phi), (nrows, nf)
        R = torch.fft.rfft(w.transpose(1, 2) if phi else w, dim=1, norm="forward")[:, : mmax + 1]
        assert err(R, G) < 1e-13, (nrows, nf, pairs)
    assert lib.shtns_b200_kernel_errors(sh._cfg) == 0


def test_generic_fft_wait_limit_reports_and_recovers():
    """The staged kernels wait for their tensor copies with a time limit.
    Option 7 makes them expect 16 bytes more than arrive: the wait gives up
    after about a second, the flag is set, and the next call is right."""
    import shtns_b200
    from shtns_b200 import capi
    lib = capi.load()
    dev = torch.device("cuda:0")
    sh = shtns_b200.sht(40)
    sh.set_grid(64, 100, flags=shtns_b200.sht_quick_init | shtns_b200.SHT_THETA_CONTIGUOUS, polar_opt=0.0)
    q = torch.randn(300, sh.nlm, dtype=torch.complex128, device=dev)
    q.imag[:, :41] = 0
    v = sh.synth(q)
    assert lib.shtns_b200_kernel_errors(sh._cfg) == 0
    # a call of few latitudes reads directly: nothing to wait for
    assert lib.shtns_b200_set_option(sh._cfg, 7, 16) == 0
    few = sh.analys(v[:2])
    assert lib.shtns_b200_get_option(sh._cfg, 11) % 10 == 0
    assert lib.shtns_b200_kernel_errors(sh._cfg) == 0
    assert relerr(q[:2].cpu().numpy(), few.cpu().numpy()) < 1e-12
    assert lib.shtns_b200_set_option(sh._cfg, 7, 0) == 0
    sh2 = shtns_b200.sht(40)
    sh2.set_grid(64, 100, flags=shtns_b200.sht_quick_init | shtns_b200.SHT_THETA_CONTIGUOUS, polar_opt=0.0)
    lib.shtns_b200_set_option(sh2._cfg, 7, 16)
    sh2.analys(v)
    assert lib.shtns_b200_kernel_errors(sh2._cfg) == 1
    assert lib.shtns_b200_kernel_errors(sh2._cfg) == 0
    back = sh.analys(v)
    assert lib.shtns_b200_kernel_errors(sh._cfg) == 0
    assert relerr(q.cpu().numpy(), back.cpu().numpy()) < 1e-12
