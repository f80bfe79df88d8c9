"""GPU tests of the FP32 ring-FFT stage alone (hb_ring_analysis / hb_ring_synthesis through the
C ABI) against the oracle's numpy ring FFTs (sht_raw.py:38-43 and isht.py:16-24 of the
reference, with the phi0 phase and alias fold).

On HEALPix grids the equatorial belt and the polar rings from ring index 64 on run on the
pair-packed kernels (one complex FFT per ring pair; Bluestein for the polar rings, whose nphi = 4i
is not a power of two), the smaller polar rings on the general ring kernels.  The polar rings
with 2048 < nphi < 8192 (nside >= 513) run split in four quarter-length Bluestein transforms
(ring_quad_*_kernel); the nside 1024 and 2048 cases cover both of those classes.  The cases cover
both conventions of phi0 (HEALPix: s = 0 or 1 in phi0 = s pi / nphi; the reference's: s = 1 or
2), the unpaired equator ring, the flags, and the three alias regimes (mmax < nphi/2,
nphi/2 <= mmax < nphi, mmax >= nphi).  Tolerance: 1e-5 relative (L2), FP32.
"""
import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

TOL = 1e-5


@pytest.fixture(scope="module")
def hb():
    import hellblast_b200
    return hellblast_b200


def rel2(a, b):
    return float(np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300))


def _pairs(g):
    """ring index of the north / south ring of each pair of a HEALPix grid (south -1: unpaired)."""
    nr = g["nr"]
    npairs = (nr + 1) // 2
    north = np.arange(npairs)
    south = nr - 1 - north
    south[south == north] = -1
    return north, south


CASES = [(128, "healpix", 200, 0), (256, "healpix", 767, 0), (256, "reference", 767, 0), (256, "healpix", 1500, 0),
         (256, "healpix", 767, 1), (256, "reference", 300, 2), (256, "healpix", 1100, 3),
         (1024, "healpix", 2047, 0), (2048, "healpix", 4095, 0), (2048, "reference", 4095, 2)]


def _nmaps(nside):
    return 2 if nside <= 256 else 1


@pytest.mark.parametrize("nside,phi0,lmax,flags", CASES)
def test_ring_analysis_fp32_vs_oracle(hb, oracle, nside, phi0, lmax, flags):
    from hellblast_b200 import _lib as L
    from hellblast_b200 import geometry as G
    g = G.healpix(nside, phi0=phi0)
    p = G.plan(g, lmax, precision=64)
    go = oracle.ring_tables(nside, phi0=phi0)
    nmaps = _nmaps(nside)
    rng = np.random.default_rng(nside + lmax + flags)
    maps = rng.standard_normal((nmaps, g.npix)).astype(np.float32)
    F = torch.empty(nmaps, lmax + 1, g.npairs, 2, dtype=torch.complex64, device="cuda")
    L.call("hb_ring_analysis", p.handle, 32, nmaps, torch.from_numpy(maps).cuda().data_ptr(), None, F.data_ptr(), flags,
           torch.cuda.current_stream().cuda_stream)
    F = F.cpu().numpy()
    north, south = _pairs(go)
    for b in range(nmaps):
        ref = oracle.ring_analysis(maps[b].astype(np.float64), go, lmax, weights=go["weights_dz"],
                                   phase=not (flags & L.HB_F_NOPHASE), fold=not (flags & L.HB_F_NOFOLD))
        want = np.zeros((lmax + 1, g.npairs, 2), dtype=np.complex128)
        want[:, :, 0] = ref[:, north]
        has = south >= 0
        want[:, has, 1] = ref[:, south[has]]
        assert rel2(F[b], want) < TOL
        assert np.all(F[b][:, ~has, 1] == 0)


@pytest.mark.parametrize("nside,phi0,lmax,flags", [c for c in CASES if not (c[3] & 2)])
def test_ring_synthesis_fp32_vs_oracle(hb, oracle, nside, phi0, lmax, flags):
    from hellblast_b200 import _lib as L
    from hellblast_b200 import geometry as G
    g = G.healpix(nside, phi0=phi0)
    p = G.plan(g, lmax, precision=64)
    go = oracle.ring_tables(nside, phi0=phi0)
    nmaps = _nmaps(nside)
    rng = np.random.default_rng(3 * nside + lmax + flags)
    Gm = (rng.standard_normal((nmaps, lmax + 1, g.npairs, 2)) + 1j * rng.standard_normal((nmaps, lmax + 1, g.npairs, 2)))
    Gm = Gm.astype(np.complex64)
    north, south = _pairs(go)
    has = south >= 0
    Gm[:, :, ~has, 1] = 0  # the unpaired equator's south slot is not data
    out = torch.empty(nmaps, g.npix, dtype=torch.float32, device="cuda")
    L.call("hb_ring_synthesis", p.handle, 32, nmaps, torch.from_numpy(Gm).cuda().data_ptr(), out.data_ptr(), flags,
           torch.cuda.current_stream().cuda_stream)
    out = out.cpu().numpy()
    for b in range(nmaps):
        Go = np.zeros((lmax + 1, go["nr"]), dtype=np.complex128)
        Go[:, north] = Gm[b, :, :, 0]
        Go[:, south[has]] = Gm[b, :, has, 1].T
        ref = oracle.ring_synthesis(Go, go, phase=not (flags & L.HB_F_NOPHASE))
        assert rel2(out[b].astype(np.float64), ref) < TOL


def test_unpaired_south_slot_garbage_is_ignored(hb, oracle):
    """The south slot of the unpaired equator pair may hold anything (here NaN): the equator ring
    and every other ring come out finite and equal to the clean input's."""
    from hellblast_b200 import _lib as L
    from hellblast_b200 import geometry as G
    nside, lmax = 256, 600
    g = G.healpix(nside)
    p = G.plan(g, lmax, precision=64)
    rng = np.random.default_rng(11)
    Gm = (rng.standard_normal((1, lmax + 1, g.npairs, 2)) + 1j * rng.standard_normal((1, lmax + 1, g.npairs, 2)))
    Gm = Gm.astype(np.complex64)
    eq = g.npairs - 1
    clean = Gm.copy()
    clean[:, :, eq, 1] = 0
    dirty = Gm.copy()
    dirty[:, :, eq, 1] = np.nan
    outs = []
    for x in (clean, dirty):
        out = torch.empty(1, g.npix, dtype=torch.float32, device="cuda")
        L.call("hb_ring_synthesis", p.handle, 32, 1, torch.from_numpy(x).cuda().data_ptr(), out.data_ptr(), 0,
               torch.cuda.current_stream().cuda_stream)
        outs.append(out.cpu().numpy())
    assert np.all(np.isfinite(outs[1]))
    assert np.array_equal(outs[0], outs[1])


@pytest.mark.parametrize("nside,lmax,nmaps,phi0", [(128, 200, 176, "healpix"), (256, 37, 80, "reference"),
                                                  (1024, 300, 24, "healpix")])
def test_few_maps_match_large_batch(hb, nside, lmax, nmaps, phi0):
    """The short pair-packed classes of a call on few maps run in one launch, those of a large batch in
    one each (the line is at 32768 (pair, map) items): the same operations, so the same bits."""
    from hellblast_b200 import _lib as L
    from hellblast_b200 import geometry as G
    g = G.healpix(nside, phi0=phi0)
    p = G.plan(g, lmax, precision=64)
    gen = torch.Generator(device="cuda").manual_seed(nside)
    few = 3
    nphi = np.asarray(g.nphi)[:g.npairs]
    shared = int(np.sum((nphi > 256) & ((nphi <= 2048) | (nphi == 4096))))
    assert shared * few <= 4800 and shared * nmaps > 32768
    Gm = torch.view_as_complex(torch.randn(nmaps, lmax + 1, g.npairs, 2, 2, device="cuda", generator=gen))
    st = torch.cuda.current_stream().cuda_stream
    maps = {n: torch.full((n, g.npix), float("nan"), device="cuda") for n in (few, nmaps)}
    for n, out in maps.items():
        L.call("hb_ring_synthesis", p.handle, 32, n, Gm.data_ptr(), out.data_ptr(), 0, st)
    assert torch.equal(maps[few], maps[nmaps][:few])
    F = {n: torch.full((n, lmax + 1, g.npairs, 2), float("nan"), dtype=torch.complex64, device="cuda") for n in (few, nmaps)}
    for n, out in F.items():
        L.call("hb_ring_analysis", p.handle, 32, n, maps[nmaps].data_ptr(), None, out.data_ptr(), 0, st)
    assert torch.equal(torch.view_as_real(F[few]), torch.view_as_real(F[nmaps][:few]))


@pytest.mark.parametrize("nside,lmax", [(32, 100), (256, 300), (512, 40)])
def test_fp64_one_map_matches_many(hb, nside, lmax):
    """FP64 ring FFTs of small and of large calls are separate builds of the kernels, with more and with fewer
    registers per thread: the same formulas, so 1e-13 relative (L2) between them (FFT rounding is below 1e-14)."""
    from hellblast_b200 import _lib as L
    from hellblast_b200 import geometry as G
    g = G.healpix(nside)
    p = G.plan(g, lmax, precision=64)
    many = max(2, 80000 // (64 * g.npairs) + 1)
    gen = torch.Generator(device="cuda").manual_seed(nside)
    Gm = torch.view_as_complex(torch.randn(many, lmax + 1, g.npairs, 2, 2, device="cuda", generator=gen, dtype=torch.float64))
    st = torch.cuda.current_stream().cuda_stream
    maps, F = {}, {}
    for n in (1, many):
        maps[n] = torch.full((n, g.npix), float("nan"), device="cuda", dtype=torch.float64)
        L.call("hb_ring_synthesis", p.handle, 64, n, Gm.data_ptr(), maps[n].data_ptr(), 0, st)
    for n in (1, many):
        F[n] = torch.full((n, lmax + 1, g.npairs, 2), float("nan"), dtype=torch.complex128, device="cuda")
        L.call("hb_ring_analysis", p.handle, 64, n, maps[many].data_ptr(), None, F[n].data_ptr(), 0, st)
    assert rel2(maps[1][0].cpu().numpy(), maps[many][0].cpu().numpy()) < 1e-13
    assert rel2(F[1][0].cpu().numpy(), F[many][0].cpu().numpy()) < 1e-13


@pytest.mark.parametrize("nside,nmaps,prec", [(64, 1, 32), (256, 3, 32), (256, 300, 32), (128, 2, 64), (512, 40, 32)])
def test_fft_launches_counts_the_call(hb, nside, nmaps, prec):
    """Geometry.fft_launches is the number of ring kernels a call on that many maps makes."""
    from hellblast_b200 import _lib as L
    from hellblast_b200 import geometry as G
    g = G.healpix(nside)
    p = G.plan(g, 20, precision=64)
    Gm = torch.zeros(nmaps, 21, g.npairs, 2, dtype=torch.complex64 if prec == 32 else torch.complex128, device="cuda")
    out = torch.empty(nmaps, g.npix, dtype=torch.float32 if prec == 32 else torch.float64, device="cuda")
    st = torch.cuda.current_stream().cuda_stream
    L.call("hb_ring_synthesis", p.handle, prec, nmaps, Gm.data_ptr(), out.data_ptr(), 0, st)
    torch.cuda.synchronize()
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as prof:
        L.call("hb_ring_synthesis", p.handle, prec, nmaps, Gm.data_ptr(), out.data_ptr(), 0, st)
        torch.cuda.synchronize()
    seen = sum(e.count for e in prof.key_averages() if "synthesis" in e.key)
    assert seen == g.fft_launches(prec, nmaps)


@pytest.mark.parametrize("nside,lmax,nmaps", [(4, 9, 1), (64, 100, 2), (512, 300, 1), (1024, 100, 1)])
@pytest.mark.parametrize("prec", [32, 64])
def test_maps_at_any_element(hb, nside, lmax, nmaps, prec):
    """A map may be a view that starts at an odd element of a larger buffer, in either direction."""
    from hellblast_b200 import _lib as L
    from hellblast_b200 import geometry as G
    dt = torch.float32 if prec == 32 else torch.float64
    gen = torch.Generator(device="cuda").manual_seed(nside)
    npix = 12 * nside * nside
    buf = torch.randn(nmaps * npix + 1, dtype=dt, device="cuda", generator=gen)
    view = buf[1:].view(nmaps, npix)
    a = hb.hp_compat.map2alm(view, lmax=lmax)
    assert torch.equal(a, hb.hp_compat.map2alm(view.clone(), lmax=lmax))
    if nside <= 64:  # (above 512 ring pairs the FP64 spin-2 analysis adds its chunks by atomics, in no fixed order)
        q, w = (hb.hp_compat.map2alm_spin(x, x.flip(0), 2, lmax=lmax) for x in (view, view.clone()))
        assert torch.equal(q[0], w[0]) and torch.equal(q[1], w[1])
    p = G.plan(G.healpix(nside), lmax, precision=prec)
    st = torch.cuda.current_stream().cuda_stream
    Gm = torch.zeros(nmaps, lmax + 1, p.geom.npairs, 2, dtype=a.dtype, device="cuda")
    L.call("hb_legendre_synthesis", p.handle, prec, nmaps, a.data_ptr(), Gm.data_ptr(), st)
    out = torch.full_like(buf, float("nan"))
    L.call("hb_ring_synthesis", p.handle, prec, nmaps, Gm.data_ptr(), out[1:].data_ptr(), 0, st)
    assert torch.equal(out[1:].view(nmaps, npix), hb.hp_compat.alm2map(a, nside, lmax=lmax)) and torch.isnan(out[0])


def test_batched_maps_at_any_element(hb):
    nside, lmax, n = 64, 100, 3
    gen = torch.Generator(device="cuda").manual_seed(8)
    buf = torch.randn(n * 12 * nside * nside + 1, device="cuda", generator=gen)
    bp = hb.batched.plan(nside, lmax, n)
    a = bp.map2alm(buf[1:])
    assert torch.equal(a, bp.map2alm(buf[1:].clone()))
    out = torch.empty_like(buf)
    assert torch.equal(bp.alm2map(a, out=out[1:]), bp.alm2map(a))


def test_stage_buffers_at_8_bytes(hb):
    """F and G of the FP32 ring stages that start at an odd complex64: taken on grids of short rings, refused where the
    pair-packed kernels read 16-byte pairs."""
    from hellblast_b200 import _lib as L
    from hellblast_b200 import geometry as G
    st = torch.cuda.current_stream().cuda_stream
    gen = torch.Generator(device="cuda").manual_seed(9)
    lmax = 40
    for nside in (32, 256):
        p = G.plan(G.healpix(nside), lmax, precision=32)
        n = (lmax + 1) * p.geom.npairs * 2
        m = torch.randn(1, p.npix, device="cuda", generator=gen)
        F = torch.zeros(n + 1, dtype=torch.complex64, device="cuda")
        want = torch.zeros(n, dtype=torch.complex64, device="cuda")
        out, ref = torch.zeros_like(m), torch.zeros_like(m)
        L.call("hb_ring_analysis", p.handle, 32, 1, m.data_ptr(), None, want.data_ptr(), 0, st)
        L.call("hb_ring_synthesis", p.handle, 32, 1, want.data_ptr(), ref.data_ptr(), 0, st)
        if nside == 256:
            with pytest.raises(ValueError, match="16 bytes"):
                L.call("hb_ring_analysis", p.handle, 32, 1, m.data_ptr(), None, F[1:].data_ptr(), 0, st)
            with pytest.raises(ValueError, match="16 bytes"):
                L.call("hb_ring_synthesis", p.handle, 32, 1, F[1:].data_ptr(), out.data_ptr(), 0, st)
            continue
        L.call("hb_ring_analysis", p.handle, 32, 1, m.data_ptr(), None, F[1:].data_ptr(), 0, st)
        assert torch.equal(F[1:], want)
        L.call("hb_ring_synthesis", p.handle, 32, 1, F[1:].data_ptr(), out.data_ptr(), 0, st)
        assert torch.equal(out, ref)
