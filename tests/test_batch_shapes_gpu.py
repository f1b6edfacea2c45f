"""The kernels that a call gets depend on its number of field-components
(prologue and epilogue tiles of 1 to 16, SIMT, 128 x 16, 128 x 32 and 64 x 64
Legendre tiles, the FP64 table): every field of a batch equals that field alone
to rounding, at field counts on both sides of each rule and at truncations that
end inside and on a tile."""
import numpy as np
import pytest
import torch

from tests.common import rand_spec, relerr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lmax,mres,nlat,nphi", [(2, 1, 4, 6), (62, 1, 64, 125), (127, 1, 192, 384), (128, 2, 130, 144), (255, 1, 384, 768),
                                                 (258, 3, 520, 200), (511, 1, 514, 1024)])
def test_batched_fields_equal_single_fields(lmax, mres, nlat, nphi):
    """Sums of up to lmax + 1 terms in two orders: they differ by at most about
    lmax 2^-53 of the largest value, with the random signs far less; bar 1e-13."""
    import shtns_b200
    dev = torch.device("cuda:0")
    sh = shtns_b200.sht(lmax, lmax // mres, mres)
    sh.set_grid(nlat, nphi, flags=shtns_b200.sht_quick_init | shtns_b200.SHT_THETA_CONTIGUOUS, polar_opt=1e-10)
    for comps, nfs in ((1, (2, 3, 4, 5, 8, 9, 13, 17, 33)), (2, (1, 2, 3, 5, 17)), (3, (1, 2, 5, 8, 12))):
        if lmax > 255:
            nfs = nfs[::2]
        q = [torch.from_numpy(rand_spec(lmax, lmax // mres, mres, 7 + c, nfields=max(nfs), zero_l0=(comps == 2 or c > 0), power=1.0)).to(dev)
             for c in range(comps)]
        tup = lambda x: list(x) if isinstance(x, tuple) else [x]  # noqa: E731
        one_v = [tup(sh.synth(*(a[i] for a in q))) for i in range(max(nfs))]
        one_q = [tup(sh.analys(*one_v[i])) for i in range(max(nfs))]
        for nf in nfs:
            v = tup(sh.synth(*(a[:nf] for a in q)))
            r = tup(sh.analys(*[torch.stack([one_v[i][c] for i in range(nf)]) for c in range(comps)]))
            for c in range(comps):
                a = torch.stack([one_v[i][c] for i in range(nf)]).cpu().numpy()
                assert relerr(a, v[c].cpu().numpy()) < 1e-13, (comps, nf, c)
                a = torch.stack([one_q[i][c] for i in range(nf)]).cpu().numpy()
                assert relerr(a, r[c].cpu().numpy()) < 1e-13, (comps, nf, c)


@pytest.mark.parametrize("comps,nf", [(1, 3), (3, 1), (1, 7), (3, 5)])
@pytest.mark.parametrize("ltr", [0, 1, 63, 64, 126, 127])
def test_truncations_equal_zeroed_coefficients(comps, nf, ltr):
    """A synthesis truncated at ltr equals the whole one of coefficients zeroed
    above ltr; an analysis truncated there equals the whole one up to ltr and
    is zero beyond (the same sums: bar 1e-13)."""
    import shtns_b200
    dev = torch.device("cuda:0")
    sh = shtns_b200.sht(127)
    sh.set_grid(192, 360, flags=shtns_b200.sht_quick_init | shtns_b200.SHT_PHI_CONTIGUOUS, polar_opt=1e-10)
    l = torch.from_numpy(sh.l.astype(np.int64)).to(dev)
    q = [torch.from_numpy(rand_spec(127, 127, 1, 3 + c, nfields=nf, zero_l0=c > 0)).to(dev) for c in range(comps)]
    tup = lambda x: list(x) if isinstance(x, tuple) else [x]  # noqa: E731
    cut = [torch.where(l <= ltr, a, torch.zeros_like(a)) for a in q]
    for a, b in zip(tup(sh.synth(*cut)), tup(sh.synth(*q, ltr=ltr))):
        assert float((a - b).abs().max()) <= 1e-13 * max(1e-300, float(a.abs().max()))
    v = tup(sh.synth(*q))
    for a, b in zip(tup(sh.analys(*v)), tup(sh.analys(*v, ltr=ltr))):
        assert float((a - b)[:, l <= ltr].abs().max()) <= 1e-13 * float(a.abs().max())
        assert not b[:, l > ltr].any()


@pytest.mark.parametrize("lmax,free_mb,table_mb,seg", [(1023, 5000, 403, 8), (2047, 3000, 1610, 32), (1023, 380, 403, 16)])
def test_plans_on_a_used_gpu(lmax, free_mb, table_mb, seg):
    """The checkpoint table (table_mb: at the spacing that an empty GPU would
    give) on a GPU with free_mb left: as dense as ever where it is small, coarser
    where it would take more than a quarter, and at the next spacing where the
    allocation fails.  The transforms are the same: bar as for any round trip."""
    import shtns_b200
    from shtns_b200 import capi
    lib = capi.load()
    dev = torch.device("cuda:0")
    sh = shtns_b200.sht(lmax)
    nlat = 3 * (lmax + 1) // 2
    lib.shtns_b200_status()
    torch.cuda.empty_cache()
    hold = torch.empty(torch.cuda.mem_get_info()[0] - (free_mb << 20), dtype=torch.uint8, device=dev)
    sh.set_grid(nlat, 2 * nlat, flags=shtns_b200.sht_quick_init | shtns_b200.SHT_THETA_CONTIGUOUS, polar_opt=1e-10)
    del hold
    torch.cuda.empty_cache()
    assert lib.shtns_b200_get_option(sh._cfg, 2) == seg
    assert lib.shtns_b200_status() == 0
    q = torch.from_numpy(rand_spec(lmax, lmax, 1, 3)).to(dev)
    assert relerr(q.cpu().numpy(), sh.analys(sh.synth(q)).cpu().numpy()) < 1e-11
