"""GPU tests of the Legendre kernels (scalar and spin-2) where their tiling can go wrong: block remainders in l,
order cut-offs, odd numbers of maps, ring-pair counts around the sets a warp holds, rings in no
particular order, pairs that are evanescent at every l; against the FP64 oracle.

Tolerances (as in test_gpu_sht.py): FP64 1e-10, FP32 1e-5 relative (L2)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def hb():
    import hellblast_b200
    return hellblast_b200


def rel2(a, b):
    return float(np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300))


def _alm(oracle, rng, nmaps, lmax, mmax):
    n = oracle.alm_size(lmax, mmax)
    a = rng.standard_normal((nmaps, n)) + 1j * rng.standard_normal((nmaps, n))
    a[:, : lmax + 1].imag = 0
    return a


def _pair(hb, oracle, geom, lmax, mmax, nmaps, to_map, to_alm, seed):
    rng = np.random.default_rng(seed)
    a = _alm(oracle, rng, nmaps, lmax, mmax)
    mp = rng.standard_normal((nmaps, geom["npix"]))
    ref_map = np.stack([oracle.alm2map(x, geom, lmax, mmax) for x in a])
    ref_alm = np.stack([oracle.map2alm(x, geom, lmax, mmax) for x in mp])
    for prec, tol in (("fp64", 1e-10), ("fp32", 1e-5)):
        got = to_map(torch.from_numpy(a).cuda(), prec).double().cpu().numpy()
        assert rel2(got, ref_map) < tol, prec
        got = to_alm(torch.from_numpy(mp).cuda(), prec).to(torch.complex128).cpu().numpy()
        assert rel2(got, ref_alm) < tol, prec


@pytest.mark.parametrize("nside,lmax,mmax,nmaps", [
    (1, 0, 0, 1), (2, 3, 1, 2), (16, 255, 2, 1), (16, 256, 3, 3), (16, 257, 257, 1), (32, 513, 130, 2),
    (64, 127, 127, 3), (128, 300, 299, 5), (512, 64, 64, 2), (1024, 40, 33, 3)])
def test_healpix_sizes(hb, oracle, nside, lmax, mmax, nmaps):
    g = oracle.ring_tables(nside)
    _pair(hb, oracle, g, lmax, mmax, nmaps,
          lambda a, p: hb.hp_compat.alm2map(a, nside, lmax=lmax, mmax=mmax, precision=p),
          lambda m, p: hb.hp_compat.map2alm(m, lmax=lmax, mmax=mmax, precision=p), nside + lmax)


@pytest.mark.parametrize("nrings,lmax", [(1, 5), (63, 40), (65, 300), (129, 70), (257, 120), (1025, 30)])
def test_unsorted_rings(hb, oracle, nrings, lmax):
    rng = np.random.default_rng(nrings)
    th = rng.permutation(np.linspace(0.004, 3.1, nrings)) if nrings > 1 else np.array([1.5707963267948966])
    nphi = (2 * rng.integers(2, 6, nrings)).astype(np.int32)
    w, phi0 = rng.uniform(0.01, 0.02, nrings), rng.uniform(0, 1, nrings)
    g = oracle.generic_geometry(th, nphi, phi0=phi0, weights=w)
    _pair(hb, oracle, g, lmax, lmax, 1,
          lambda a, p: hb.alm2map_gpu(a[0], th, nphi, lmax, phi0=phi0, flat=True, precision=p)[None],
          lambda m, p: hb.map2alm_gpu(m[0], th, nphi, w, lmax, phi0=phi0, precision=p)[None], nrings)


@pytest.mark.parametrize("nside,lmax,mmax,nmaps", [
    (2, 1, 1, 1), (2, 2, 0, 2), (8, 257, 4, 1), (16, 258, 258, 2), (64, 130, 127, 3), (128, 300, 3, 1), (512, 40, 40, 2)])
def test_spin_sizes(hb, oracle, nside, lmax, mmax, nmaps):
    g = oracle.ring_tables(nside)
    rng = np.random.default_rng(nside + lmax)
    a = [_alm(oracle, rng, nmaps, lmax, mmax) for _ in range(2)]
    q = [rng.standard_normal((nmaps, g["npix"])) for _ in range(2)]
    ref_map = [oracle.alm2map_spin2(e, b, g, lmax, mmax) for e, b in zip(*a)]
    ref_alm = [oracle.map2alm_spin2(x, y, g, lmax, mmax) for x, y in zip(*q)]
    for prec, tol in (("fp64", 1e-10), ("fp32", 1e-5)):
        got = hb.hp_compat.alm2map_spin(*(torch.from_numpy(x).cuda() for x in a), 2, nside=nside, lmax=lmax, mmax=mmax, precision=prec)
        back = hb.hp_compat.map2alm_spin(*(torch.from_numpy(x).cuda() for x in q), 2, lmax=lmax, mmax=mmax, precision=prec)
        for i in range(2):
            assert rel2(got[i].double().cpu().numpy(), np.stack([r[i] for r in ref_map])) < tol, (prec, "map")
            assert rel2(back[i].to(torch.complex128).cpu().numpy(), np.stack([r[i] for r in ref_alm])) < tol, (prec, "alm")
