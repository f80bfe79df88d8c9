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


@pytest.mark.parametrize("nrings,lmax,nmaps", [(2047, 1023, 1), (2051, 1025, 3), (2048, 511, 2), (4097, 1100, 1)])
def test_orders_in_turn_match_a_list(hb, nrings, lmax, nmaps):
    """FP64 analysis on 1024 and more ring pairs: with many orders a CTA takes an order's chunks of pairs in
    turn (and maps in pairs), a list of orders has each order's pairs side by side.  The same products
    summed in another order, at most 2049 per value: 1e-12 relative (L2) is 2049 eps with room."""
    from hellblast_b200 import _lib as L
    from hellblast_b200 import geometry as G
    th = np.linspace(0.0007, np.pi / 2, (nrings + 1) // 2 + (nrings % 2 == 0))[:(nrings + 1) // 2]
    th = np.concatenate([th, np.pi - th[:nrings // 2][::-1]])
    g = G.generic(th, np.full(nrings, 4, dtype=np.int32), np.full(nrings, 2.0 / nrings))
    assert g.npairs == (nrings + 1) // 2 >= 1024
    p = G.plan(g, lmax, precision=64)
    gen = torch.Generator(device="cuda").manual_seed(nrings)
    F = torch.view_as_complex(torch.randn(nmaps, lmax + 1, g.npairs, 2, 2, device="cuda", generator=gen, dtype=torch.float64))
    nalm = L.lib().hb_alm_size(lmax, lmax)
    st = torch.cuda.current_stream().cuda_stream
    full = torch.full((nmaps, nalm), float("nan"), dtype=torch.complex128, device="cuda")
    L.call("hb_legendre_analysis", p.handle, 64, nmaps, F.data_ptr(), full.data_ptr(), st)
    orders = [0, 1, 2, lmax // 2, lmax - 1, lmax]
    lst = torch.tensor(orders, dtype=torch.int32, device="cuda")
    some = torch.zeros_like(full)
    L.call("hb_legendre_analysis_ms", p.handle, 64, nmaps, len(orders), lst.data_ptr(), F[:, orders].contiguous().data_ptr(),
           some.data_ptr(), st)
    assert torch.isfinite(torch.view_as_real(full)).all()
    for m in orders:
        i = m * (2 * lmax + 1 - m) // 2
        a, b = full[:, i + m:i + lmax + 1].cpu().numpy(), some[:, i + m:i + lmax + 1].cpu().numpy()
        assert rel2(a, b) < 1e-12, m


@pytest.mark.parametrize("lmax,mmax,nmaps", [(0, 0, 1), (31, 31, 2), (33, 39, 1), (64, 40, 3), (255, 255, 1), (256, 256, 1), (300, 5, 2),
                                             (517, 300, 1), (256, 256, 456)])
@pytest.mark.parametrize("cross", [False, True])
def test_alm2cl_sizes(hb, lmax, mmax, nmaps, cross):
    """alm2cl around the sizes where its CTAs change their number of warps, with order cut-offs; against NumPy in
    64 bits: at most 2 * 517 products per value, 1e-13 of the largest |a||b| / (2l+1)."""
    from hellblast_b200 import ops
    mmax = min(mmax, lmax)
    nalm = (mmax + 1) * (2 * lmax + 2 - mmax) // 2
    for dt in (torch.complex64, torch.complex128):
        gen = torch.Generator(device="cuda").manual_seed(lmax)
        a = torch.randn(nmaps, nalm, dtype=dt, device="cuda", generator=gen)
        b = torch.randn(nmaps, nalm, dtype=dt, device="cuda", generator=gen) if cross else None
        A = a.to(torch.complex128).cpu().numpy()
        B = A if b is None else b.to(torch.complex128).cpu().numpy()
        want, size = np.zeros((2, nmaps, lmax + 1))
        for m in range(mmax + 1):
            i = m * (2 * lmax + 1 - m) // 2
            p, q = A[:, i + m:i + lmax + 1], B[:, i + m:i + lmax + 1]
            want[:, m:] += (1 if m == 0 else 2) * (p * q.conj()).real
            size[:, m:] += 2 * np.abs(p) * np.abs(q)
        deg = 2 * np.arange(lmax + 1) + 1.0
        got = ops.alm2cl(a, b, lmax, mmax).cpu().numpy()
        assert np.all(np.abs(got - want / deg) <= 1e-13 * size / deg)


def _odd_grid(oracle, nrings, nphi):
    """Rings symmetric about the middle one, which lies at theta = pi/2 (cos = 6e-17, not zero)."""
    th = np.linspace(0.02, np.pi - 0.02, nrings)
    th[nrings // 2] = np.pi / 2
    n = np.full(nrings, nphi, dtype=np.int32)
    w = np.random.default_rng(nrings).uniform(0.5, 1.5, nrings) * 2.0 / nrings
    return th, n, w, oracle.generic_geometry(th, n, weights=w), slice((nrings // 2) * nphi, (nrings // 2 + 1) * nphi)


@pytest.mark.parametrize("nrings,lmax,mmax", [(129, 700, 700), (33, 600, 3), (2051, 520, 2)])
def test_equator_ring(hb, oracle, nrings, lmax, mmax):
    """On a ring at theta = pi/2 every second lambda_lm is near zero, also at the starts of the 256-l blocks: the
    ring by itself, in both directions (1e-5 relative (L2) in FP32, 1e-10 in FP64, as above)."""
    th, nphi, w, g, eq = _odd_grid(oracle, nrings, 16)
    rng = np.random.default_rng(lmax)
    a = _alm(oracle, rng, 1, lmax, mmax)[0]
    mp = np.zeros(g["npix"])
    mp[eq] = rng.standard_normal(16)
    ref_map, ref_alm = oracle.alm2map(a, g, lmax, mmax)[eq], oracle.map2alm(mp, g, lmax, mmax)
    G = hb.geometry.generic(th, nphi, w)
    for prec, tol in (("fp64", 1e-10), ("fp32", 1e-5)):
        got = hb.transforms.alm2map(torch.from_numpy(a).cuda(), G, lmax, mmax, precision=prec).double().cpu().numpy()[eq]
        assert rel2(got, ref_map) < tol, (prec, "map")
        got = hb.transforms.map2alm(torch.from_numpy(mp).cuda(), G, lmax, mmax, precision=prec).cpu().numpy()
        assert rel2(got, ref_alm) < tol, (prec, "alm")


@pytest.mark.parametrize("nrings,lmax,mmax", [(129, 700, 700), (33, 600, 3)])
def test_equator_ring_spin(hb, oracle, nrings, lmax, mmax):
    """The same for spin 2 (at m = 0 its functions have a definite parity, so one of two is near zero)."""
    th, nphi, w, g, eq = _odd_grid(oracle, nrings, 16)
    rng = np.random.default_rng(lmax)
    a = _alm(oracle, rng, 2, lmax, mmax)
    q = np.zeros((2, g["npix"]))
    q[:, eq] = rng.standard_normal((2, 16))
    ref_map = [x[eq] for x in oracle.alm2map_spin2(a[0], a[1], g, lmax, mmax)]
    ref_alm = oracle.map2alm_spin2(q[0], q[1], g, lmax, mmax)
    G = hb.geometry.generic(th, nphi, w)
    for prec, tol in (("fp64", 1e-10), ("fp32", 1e-5)):
        got = hb.transforms.alm2map_spin2(*(torch.from_numpy(x).cuda() for x in a), G, lmax, mmax, precision=prec)
        back = hb.transforms.map2alm_spin2(*(torch.from_numpy(x).cuda() for x in q), G, lmax, mmax, precision=prec)
        for i in range(2):
            assert rel2(got[i].double().cpu().numpy()[eq], ref_map[i]) < tol, (prec, "map")
            assert rel2(back[i].cpu().numpy(), ref_alm[i]) < tol, (prec, "alm")


def test_equator_ring_batched(hb, oracle):
    """The tensor-core path starts from the same checkpoints: the equator ring by itself (1e-5 relative (L2))."""
    lmax, mmax, n = 600, 600, 3
    th, nphi, w, g, eq = _odd_grid(oracle, 129, 16)
    rng = np.random.default_rng(n)
    a = _alm(oracle, rng, n, lmax, mmax)
    mp = np.zeros((n, g["npix"]), dtype=np.float32)
    mp[:, eq] = rng.standard_normal((n, 16))
    bp = hb.batched.BatchedPlan([(hb.geometry.generic(th, nphi, w), lmax, mmax, n)])
    got = bp.alm2map(torch.from_numpy(a).to("cuda", torch.complex64)).reshape(n, -1)[:, eq].double().cpu().numpy()
    assert rel2(got, np.stack([oracle.alm2map(x, g, lmax, mmax)[eq] for x in a])) < 1e-5
    got = bp.map2alm(torch.from_numpy(mp).cuda()).reshape(n, -1).to(torch.complex128).cpu().numpy()
    assert rel2(got, np.stack([oracle.map2alm(x, g, lmax, mmax) for x in mp.astype(np.float64)])) < 1e-5


def _orders(alm, lmax, mmax, m0):
    """The coefficients of the orders m0 .. mmax."""
    return alm[..., m0 * (2 * lmax + 1 - m0) // 2 + m0:]


@pytest.mark.parametrize("nside,lmax,nmaps,m0", [(64, 130, 1, 90), (128, 200, 2, 90), (512, 1100, 1, 90), (512, 600, 2, 90)])
@pytest.mark.parametrize("prec", ["fp64", "fp32"])
def test_nan_stays_where_the_ring_contributes(hb, nside, lmax, nmaps, m0, prec):
    """A NaN pixel on the ring next to the pole (theta < 0.013, l theta < 1.8): for m >= 90 the ring's lambda is
    below 2^-256 at every l, (l theta / 2)^m / m! < 2^-400, and a ring that counts as zero adds nothing, be its
    value finite or not."""
    gen = torch.Generator(device="cuda").manual_seed(nside)
    mp = torch.randn(nmaps, 12 * nside * nside, device="cuda", generator=gen, dtype=torch.float64)
    bad = mp.clone()
    mp[:, 1], bad[:, 1] = 0.0, float("nan")
    a, b = (hb.hp_compat.map2alm(x, lmax=lmax, precision=prec) for x in (mp, bad))
    assert torch.isnan(torch.view_as_real(b)).any()
    assert torch.equal(torch.view_as_real(_orders(a, lmax, lmax, m0)), torch.view_as_real(_orders(b, lmax, lmax, m0)))


@pytest.mark.parametrize("value", [float("nan"), float("inf")])
@pytest.mark.parametrize("nmaps", [1, 2])
def test_nan_reaches_the_orders_of_its_ring(hb, oracle, value, nmaps):
    """The same ring (theta = 0.0128) where it counts, in FP64: lambda is past 2^-256 at every l of m <= 30, at m = 45
    from some l on (2^-283 at l = 45, 2^-198 at l = 130)."""
    nside, lmax = 64, 130
    mp = torch.ones(nmaps, 12 * nside * nside, device="cuda", dtype=torch.float64)
    mp[-1, 1] = value
    a = hb.hp_compat.map2alm(mp, lmax=lmax)[-1].cpu().numpy()
    at = lambda l, m: a[oracle.alm_index(lmax, l, m)]
    assert not any(np.isfinite(at(l, m)) for m in (0, 1, 2, 30) for l in range(m, lmax + 1))
    assert np.isfinite(at(45, 45)) and not np.isfinite(at(lmax, 45))
    if nmaps > 1:
        assert torch.isfinite(torch.view_as_real(hb.hp_compat.map2alm(mp, lmax=lmax)[0])).all()


@pytest.mark.parametrize("nside,lmax", [(64, 130), (256, 300)])
@pytest.mark.parametrize("prec", ["fp64", "fp32"])
def test_nan_stays_where_the_ring_contributes_spin(hb, nside, lmax, prec):
    """The same for spin 2, whose functions are of order m - 2 in theta."""
    gen = torch.Generator(device="cuda").manual_seed(nside)
    q = torch.randn(2, 12 * nside * nside, device="cuda", generator=gen, dtype=torch.float64)
    bad = q.clone()
    q[:, 1], bad[:, 1] = 0.0, float("nan")
    a, b = (hb.hp_compat.map2alm_spin(x[0], x[1], 2, lmax=lmax, precision=prec) for x in (q, bad))
    for x, y in zip(a, b):
        assert torch.isnan(torch.view_as_real(y)).any()
        assert torch.equal(torch.view_as_real(_orders(x, lmax, lmax, 96)), torch.view_as_real(_orders(y, lmax, lmax, 96)))


@pytest.mark.parametrize("value", [float("nan"), float("inf")])
def test_nan_reaches_the_orders_of_its_ring_spin(hb, oracle, value):
    """Spin 2 counts from 2^-256 too, in FP64: P and M are of order m + 2 and m - 2 in theta."""
    nside, lmax = 64, 130
    q = torch.ones(2, 12 * nside * nside, device="cuda", dtype=torch.float64)
    q[0, 1] = value
    for a in hb.hp_compat.map2alm_spin(q[0], q[1], 2, lmax=lmax):
        a = a.cpu().numpy()
        at = lambda l, m: a[oracle.alm_index(lmax, l, m)]
        assert not any(np.isfinite(at(l, m)) for m in (0, 1, 2, 30) for l in range(max(m, 2), lmax + 1))
        assert np.isfinite(at(48, 48)) and not np.isfinite(at(lmax, 47))


@pytest.mark.parametrize("lmax,nmaps", [(22, 3), (23, 2), (24, 1), (39, 1), (40, 2), (100, 74), (100, 75), (256, 16), (256, 17), (256, 66),
                                        (511, 37), (511, 38), (512, 9), (1000, 19), (600, 216)])
def test_alm2cl_warps(hb, oracle, lmax, nmaps):
    """alm2cl where its CTAs change their number of warps with the number of CTAs; the first and the last spectrum
    (tolerance as in test_alm2cl_sizes: at most 2 * 1001 products per value)."""
    from hellblast_b200 import ops
    gen = torch.Generator(device="cuda").manual_seed(lmax)
    for dt in (torch.complex64, torch.complex128):
        a, b = (torch.randn(nmaps, oracle.alm_size(lmax), dtype=dt, device="cuda", generator=gen) for _ in range(2))
        for other in (None, b):
            got = ops.alm2cl(a, other, lmax, lmax)
            for i in (0, nmaps - 1):
                x, y = (t[i].to(torch.complex128).cpu().numpy() for t in (a, a if other is None else b))
                want = oracle.alm2cl(x, lmax, alm2=y)
                size = oracle.alm2cl(np.abs(x).astype(complex), lmax, alm2=np.abs(y).astype(complex))
                assert np.all(np.abs(got[i].cpu().numpy() - want) <= 1e-13 * size)


@pytest.mark.parametrize("npairs", [255, 256, 511, 513, 700, 1000, 1023, 1024, 1025, 2049])
def test_fp32_analysis_pair_counts(hb, npairs):
    """Numbers of ring pairs around those at which the FP32 analysis changes its chunks of pairs.  With one pair not zero
    no sum rounds, so alm has the bits that the pair gives in a grid of its own; and maps that share a recursion have the
    bits of single ones."""
    from hellblast_b200 import _lib as L
    from hellblast_b200 import geometry as G
    lmax, mmax, nrings = 300, 6, 2 * npairs - 1
    th = (np.arange(nrings) + 0.5) * np.pi / nrings
    st = torch.cuda.current_stream().cuda_stream
    gen = torch.Generator(device="cuda").manual_seed(npairs)
    nalm = L.lib().hb_alm_size(lmax, mmax)

    def analysis(theta, F):
        g = G.generic(theta, np.full(len(theta), 4, np.int32), np.ones(len(theta)))
        assert g.npairs == F.shape[2]
        alm = torch.full((F.shape[0], nalm), float("nan"), dtype=torch.complex64, device="cuda")
        L.call("hb_legendre_analysis", G.plan(g, lmax, mmax, precision=32).handle, 32, F.shape[0], F.data_ptr(), alm.data_ptr(), st)
        return torch.view_as_real(alm)

    full = torch.view_as_complex(torch.randn(3, mmax + 1, npairs, 2, 2, device="cuda", generator=gen))
    alone = analysis(th, full[:1].contiguous())
    assert torch.isfinite(alone).all()
    assert torch.equal(analysis(th, full)[0], alone[0]) and torch.equal(analysis(th, full[:2].contiguous())[0], alone[0])
    for p in {0, 63, 64, 127, 128, 255, 256, 511, 512, 1023, 1024, 2047, 2048, npairs - 2}:
        if p < npairs - 1:  # (the last pair is the equator, which has no south ring)
            F = torch.zeros_like(full[:1])
            F[:, :, p] = full[:1, :, p]
            assert torch.equal(analysis(th, F), analysis(th[[p, nrings - 1 - p]], full[:1, :, p:p + 1].contiguous())), p


@pytest.mark.parametrize("nside,lmax,nmaps", [(16, 40, 1), (64, 130, 2), (512, 300, 2), (1024, 270, 1)])
def test_stage_buffers_at_8_bytes(hb, nside, lmax, nmaps):
    """F and G of the FP32 Legendre stages are complex64 and may start at any multiple of 8 bytes."""
    from hellblast_b200 import _lib as L
    from hellblast_b200 import geometry as G
    g = G.healpix(nside)
    p = G.plan(g, lmax, precision=32)
    st = torch.cuda.current_stream().cuda_stream
    gen = torch.Generator(device="cuda").manual_seed(nside)
    n = nmaps * (lmax + 1) * g.npairs * 2
    F = torch.randn(n + 1, dtype=torch.complex64, device="cuda", generator=gen)
    nalm = L.lib().hb_alm_size(lmax, lmax)
    alm, out = [], []
    for f in (F[1:], F[1:].clone()):
        a = torch.empty(nmaps, nalm, dtype=torch.complex64, device="cuda")
        L.call("hb_legendre_analysis", p.handle, 32, nmaps, f.data_ptr(), a.data_ptr(), st)
        alm.append(a)
    assert torch.equal(alm[0], alm[1])
    for ofs in (1, 0):
        buf = torch.zeros(n + 1, dtype=torch.complex64, device="cuda")
        L.call("hb_legendre_synthesis", p.handle, 32, nmaps, alm[0].data_ptr(), buf[ofs:].data_ptr(), st)
        out.append(buf[ofs:ofs + n])
    assert torch.equal(out[0], out[1]) and out[0].abs().sum() > 0


@pytest.mark.parametrize("nphi,lmax", [([2], 3), ([2, 4, 2, 6, 2], 9), ([2, 2, 8, 2, 2, 2], 40)])
def test_rings_of_two_pixels(hb, oracle, nphi, lmax):
    """Two pixels are the smallest ring: its FFT has length one."""
    nphi = np.array(nphi, dtype=np.int32)
    th = np.linspace(0.3, 2.7, nphi.size)
    w, phi0 = np.linspace(0.2, 0.4, nphi.size), np.linspace(0, 1, nphi.size)
    g = oracle.generic_geometry(th, nphi, phi0=phi0, weights=w)
    _pair(hb, oracle, g, lmax, lmax, 2,
          lambda a, p: hb.transforms.alm2map(a, hb.geometry.generic(th, nphi, w, phi0), lmax, precision=p),
          lambda m, p: hb.transforms.map2alm(m, hb.geometry.generic(th, nphi, w, phi0), lmax, precision=p), lmax)
