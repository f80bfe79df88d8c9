"""The workloads this library's speed is judged by: what they are (`listed`, `draw`), what a program
has in hand before the call (`prepare`), one pass through the public entry points (`run`), the
bytes and flops the pass cannot do without (`work`) and its result in 64 bits from plain torch
(`exact`).

A case is {"kind", "nside", "lmax", "mmax", "nmaps", "dtype", "weights"} and, for the tensor-core
batches, "wide" and "bf16".  Kinds:

  synth       hp_compat.alm2map: maps simulated from alm
  anafast     hp_compat.anafast(alm=True): alm and power spectrum of maps
  roundtrip   alm2map, map2alm and alm2cl: the transform pair used for filtering and inpainting
  spin_synth  hp_compat.alm2map_spin: Q, U from E, B
  spin_anal   hp_compat.map2alm_spin: E, B from Q, U
  grad        gradient of a T, E, B power-spectrum loss with respect to T, Q, U maps
  batched     BatchedPlan alm2map then map2alm on the tensor cores
  smooth      smoothing.smooth_map with a Gaussian beam (float32 batches: the tensor-core path)
  rotate      rotate_alm_euler: alm moved to another coordinate frame
"""
from __future__ import annotations

import math

import numpy as np
import torch

import hellblast_b200 as hb

FWHM = 0.01  # beam of the smoothing cases, rad
EULER = (0.4, 1.1, -2.3)  # a general rotation, as galactic <-> equatorial frames need


def _case(name, kind, nside, lmax, nmaps=1, dtype="f32", mmax=None, weights="dz", wide=False, bf16=False):
    c = dict(kind=kind, nside=nside, lmax=lmax, mmax=lmax if mmax is None else mmax, nmaps=nmaps, dtype=dtype,
             weights=weights)
    if kind == "batched":
        c.update(wide=wide, bf16=bf16)
    return dict(c, name=name) if name else c


def listed():
    return [
        # the smallest grid people run in loops (likelihoods, unit checks): launch latency
        _case("roundtrip f64 64", "roundtrip", 64, 191, dtype="f64"),
        # masks and low-resolution data products: one small map, lmax = 3 nside - 1
        _case("anafast f32 128", "anafast", 128, 383),
        # one simulated sky, and one analysed sky, at the resolution most maps are published at
        _case("synth f32 1024", "synth", 1024, 2047),
        _case("anafast f32 1024", "anafast", 1024, 2047),
        # the same in double precision
        _case("roundtrip f64 1024", "roundtrip", 1024, 2047, dtype="f64"),
        # a handful of frequency maps with uniform pixel weights and an odd band limit
        _case("anafast f32 512 x5", "anafast", 512, 1301, nmaps=5, mmax=1200, weights="uniform"),
        # polarisation: one Q/U map analysed; a few low-resolution ones simulated in double precision
        _case("spin_anal f32 1024", "spin_anal", 1024, 2047),
        _case("spin_synth f64 256 x3", "spin_synth", 256, 700, nmaps=3, dtype="f64"),
        # map-making and inference: the gradient of a T/E/B spectrum loss to T, Q, U at full size
        _case("grad f32 2048", "grad", 2048, 4095),
        # 64 right-hand sides at full size, the batch the benchmark runs
        _case("batched 2048 x64", "batched", 2048, 4095, nmaps=64, wide=True, bf16=True),
        # Monte Carlo maps brought to a common beam
        _case("smooth f32 256 x16", "smooth", 256, 767, nmaps=16),
        # a change of frame of a full set of alm
        _case("rotate f64 767", "rotate", 0, 767, dtype="f64"),
    ]


def draw(rng):
    """One more case of the same ranges: any kind, sizes spread over their logarithm, band limits
    from nside to 3 nside (odd ones among them), sometimes a cut in m."""
    kind = rng.choice(["synth", "anafast", "roundtrip", "spin_synth", "spin_anal", "grad", "batched", "smooth",
                       "rotate"])
    if kind == "rotate":
        return _case(None, kind, 0, int(round(2 ** rng.uniform(5.0, 9.6))), nmaps=rng.choice([1, 1, 2]), dtype="f64")
    nside = 1 << rng.randint(4, 8 if kind in ("batched", "smooth") else 10)
    lmax = int(round(nside * 3.0 ** rng.random())) - rng.choice([0, 1])
    dtype = "f32" if kind in ("grad", "batched", "smooth") else rng.choice(["f32", "f32", "f64"])
    nmaps = 1
    if kind in ("batched", "smooth"):
        nmaps = int(round(2 ** rng.uniform(2.0, 6.5)))
    elif nside <= 512 and kind != "grad":
        nmaps = rng.choice([1, 1, 2, 3, 6])
    mmax = lmax if kind == "grad" or rng.random() < 0.75 else rng.randint(lmax // 2, lmax)
    return _case(None, kind, nside, lmax, nmaps=nmaps, dtype=dtype, mmax=mmax if kind != "smooth" else lmax,
                 weights=rng.choice(["dz", "dz", "uniform"]) if kind in ("anafast", "spin_anal") else "dz",
                 wide=rng.random() < 0.5, bf16=rng.random() < 0.5)


# --------------------------------------------------------------------------------------- inputs
def _types(case):
    return (torch.float32, torch.complex64) if case["dtype"] == "f32" else (torch.float64, torch.complex128)


def _generator(seed, salt):
    g = torch.Generator(device="cuda")
    g.manual_seed(1000003 * int(seed) + salt)
    return g


def _alm_sizes(lmax, mmax):
    """Index of (l = m, m) minus m for every m, and the number of alm (healpy m-major layout)."""
    m = np.arange(mmax + 1, dtype=np.int64)
    return m * (2 * lmax + 1 - m) // 2, mmax * (2 * lmax + 1 - mmax) // 2 + lmax + 1


def _lm(lmax, mmax):
    m = torch.arange(mmax + 1, device="cuda")
    m = torch.repeat_interleave(m, lmax + 1 - m)
    ofs, n = _alm_sizes(lmax, mmax)
    return torch.arange(n, device="cuda") - torch.from_numpy(ofs).cuda()[m], m


def _draw_alm(case, seed, salt, scale=1.0, lmin=0):
    """Gaussian alm with C_l = scale / (l + 10)^2, m = 0 real: [nmaps, nalm]."""
    l, m = _lm(case["lmax"], case["mmax"])
    sd = math.sqrt(scale) / (l.double() + 10.0) * (l >= lmin)
    re = torch.where(m > 0, sd * math.sqrt(0.5), sd)
    im = torch.where(m > 0, sd * math.sqrt(0.5), torch.zeros_like(sd))
    g = _generator(seed, salt)
    n = (case["nmaps"], l.numel())
    z = torch.complex(torch.randn(n, generator=g, device="cuda"), torch.randn(n, generator=g, device="cuda"))
    out = torch.empty(n, dtype=_types(case)[1], device="cuda")
    out.real = z.real * re
    out.imag = z.imag * im
    return out


def _rings(nside):
    """z, nphi, phi0 in units of pi/nphi and the dz weight of every HEALPix ring, north to south."""
    i = np.arange(1, 4 * nside, dtype=np.int64)
    ip = np.minimum(i, 4 * nside - i)
    cap = ip < nside
    z = np.where(cap, 1.0 - ip * ip / (3.0 * nside * nside), (2 * nside - ip) * 2.0 / (3.0 * nside))
    z = np.where(i > 2 * nside, -z, z)
    nphi = np.where(cap, 4 * ip, 4 * nside)
    half = np.where(cap, 1, 1 - ((i - nside) & 1))
    edge = np.concatenate([[1.0], 0.5 * (z[:-1] + z[1:]), [-1.0]])
    return z, nphi, half, edge[:-1] - edge[1:]


def _draw_maps(case, seed, salt, smooth=True):
    """White noise, as instrument noise is, on a large-scale signal: [nmaps, npix]."""
    nside = case["nside"]
    g = _generator(seed, salt)
    out = torch.randn(case["nmaps"], 12 * nside * nside, generator=g, device="cuda", dtype=_types(case)[0])
    if smooth:
        z, nphi, _, _ = _rings(nside)
        zr = torch.repeat_interleave(torch.from_numpy(z).cuda(), torch.from_numpy(nphi).cuda()).to(out.dtype)
        c = torch.randn(case["nmaps"], 3, 1, generator=g, device="cuda", dtype=out.dtype)
        out += c[:, 0] + c[:, 1] * zr + c[:, 2] * zr * zr
    return out


def _noise_cl(case):
    """Expected C_l of unit white noise, the level the loss of the gradient case compares with."""
    return 4.0 * math.pi / (12.0 * case["nside"] ** 2)


def _inputs(case, seed):
    k = case["kind"]
    if k in ("synth", "roundtrip", "batched", "rotate"):
        return {"alm": _draw_alm(case, seed, 1)}
    if k == "spin_synth":
        return {"E": _draw_alm(case, seed, 2, 0.1, 2), "B": _draw_alm(case, seed, 3, 0.01, 2)}
    if k == "spin_anal":
        return {"Q": _draw_maps(case, seed, 4), "U": _draw_maps(case, seed, 5)}
    if k == "grad":
        return {n: _draw_maps(case, seed, 6 + i, smooth=False) for i, n in enumerate("TQU")}
    return {"maps": _draw_maps(case, seed, 9)}


def prepare(case, seed):
    state = {"case": case, **_inputs(case, seed)}
    if case["kind"] == "batched":
        state["plan"] = hb.batched.plan(case["nside"], case["lmax"], case["nmaps"], mmax=case["mmax"],
                                        bf16=case["bf16"], wide=case["wide"])
    return state


# ----------------------------------------------------------------------------------------- runs
def run(state):
    c = state["case"]
    k, nside, lmax, mmax = c["kind"], c["nside"], c["lmax"], c["mmax"]
    if k == "synth":
        return {"map": hb.hp_compat.alm2map(state["alm"], nside, lmax=lmax, mmax=mmax)}
    if k == "anafast":
        a = hb.hp_compat.map2alm(state["maps"], lmax=lmax, mmax=mmax, weights=c["weights"])
        return {"alm": a, "cl": hb.alm2cl(a, lmax=lmax, mmax=mmax)}
    if k == "roundtrip":
        m = hb.hp_compat.alm2map(state["alm"], nside, lmax=lmax, mmax=mmax)
        a = hb.hp_compat.map2alm(m, lmax=lmax, mmax=mmax)
        return {"map": m, "alm": a, "cl": hb.alm2cl(a, lmax=lmax, mmax=mmax)}
    if k == "spin_synth":
        Q, U = hb.hp_compat.alm2map_spin(state["E"], state["B"], 2, nside=nside, lmax=lmax, mmax=mmax)
        return {"Q": Q, "U": U}
    if k == "spin_anal":
        E, B = hb.hp_compat.map2alm_spin(state["Q"], state["U"], 2, lmax=lmax, mmax=mmax, weights=c["weights"])
        return {"E": E, "B": B}
    if k == "grad":
        t, q, u = (state[n].detach().requires_grad_(True) for n in "TQU")
        e, b = hb.autograd.map2alm_spin(q, u, nside, lmax)
        cls = [hb.autograd.alm2cl(a, lmax) for a in (hb.autograd.map2alm(t, nside, lmax), e, b)]
        target = 1.1 * _noise_cl(c)
        loss = sum((((cl - target) / target)[:, 2:] ** 2).sum() for cl in cls)
        loss.backward()
        return {"loss": loss.detach(), "T": t.grad, "Q": q.grad, "U": u.grad}
    if k == "batched":
        m = state["plan"].alm2map(state["alm"])
        return {"map": m, "alm": state["plan"].map2alm(m)}
    if k == "smooth":
        return {"map": hb.smoothing.smooth_map(state["maps"], nside, lmax=lmax, fwhm=FWHM)}
    if k == "rotate":
        return {"alm": hb.rotate.rotate_alm_euler(state["alm"], *EULER, lmax=lmax)}
    raise ValueError(f"unknown kind {k}")


def work(case):
    """Each input read once and each output written once.  Flops of a scalar transform: 4 per
    (l, m, ring pair) for the recursion, shared by the maps, and 4 per map for the contraction; a
    spin-2 transform has two recursions of 6 and 16 per map."""
    k, lmax, mmax, nb = case["kind"], case["lmax"], case["mmax"], case["nmaps"]
    real = 4 if case["dtype"] == "f32" else 8
    nalm = _alm_sizes(lmax, mmax)[1]
    alm = 2 * real * nalm * nb
    if k == "rotate":  # a recursion step (5) and a complex product (4) per d^l_mm', m >= 0
        n = sum((l + 1) * (2 * l + 1) for l in range(lmax + 1))
        return {"bytes": 2 * alm, "flops": n * (5 + 4 * nb)}
    pix = real * 12 * case["nside"] ** 2 * nb
    n = nalm * 2 * case["nside"]
    scalar, spin = n * (4 + 4 * nb), n * (12 + 16 * nb)
    cl = 8 * nb * (lmax + 1)
    return {
        "synth": dict(bytes=alm + pix, flops=scalar),
        "anafast": dict(bytes=alm + pix + cl, flops=scalar),
        "roundtrip": dict(bytes=2 * alm + pix + cl, flops=2 * scalar),
        "spin_synth": dict(bytes=2 * (alm + pix), flops=spin),
        "spin_anal": dict(bytes=2 * (alm + pix), flops=spin),
        "grad": dict(bytes=6 * pix, flops=2 * (scalar + spin)),
        "batched": dict(bytes=2 * alm + pix, flops=2 * scalar),
        "smooth": dict(bytes=2 * pix, flops=2 * scalar),
    }[k]


# ------------------------------------------------------------------- the same results in 64 bits
BIG, UNIT = 2.0 ** 256, 2.0 ** 512  # values are kept as v * UNIT^e, e <= 0, while they are tiny


class _Grid:
    """Ring pairs of a HEALPix grid (north rings and the equator) and its ring FFTs."""

    def __init__(self, nside):
        self.nside = nside
        z, self.nphi, self.half, self.dz = _rings(nside)
        self.start = np.concatenate([[0], np.cumsum(self.nphi)])
        self.np = 2 * nside
        i = np.arange(1, 2 * nside + 1, dtype=np.float64)
        u = np.where(i < nside, i * i / (3.0 * nside * nside), 1.0 - (2 * nside - i) * 2.0 / (3.0 * nside))  # 1 - z
        dev = dict(dtype=torch.float64, device="cuda")
        self.x = torch.tensor(z[: self.np], **dev)
        self.log_sin = torch.tensor(0.5 * np.log2(u * (2.0 - u)), **dev)
        self.log_ch = torch.tensor(0.5 * np.log2(1.0 - 0.5 * u), **dev)
        self.log_sh = torch.tensor(0.5 * np.log2(0.5 * u), **dev)

    def _groups(self):
        """(pair slice, nphi) of the rings that share a length."""
        for p in range(self.nside - 1):
            yield slice(p, p + 1), 4 * (p + 1)
        yield slice(self.nside - 1, self.np), 4 * self.nside

    def _phase(self, ps, n, mmax):
        m = torch.arange(mmax + 1, device="cuda")[:, None]
        h = torch.from_numpy(self.half[ps].astype(np.int64)).cuda()[None, :]
        ang = ((m * h) % (2 * n)).double() * (math.pi / n)
        return torch.polar(torch.ones_like(ang), ang)  # [m, pair]

    def _pixels(self, ps, n, south):
        """First pixel of the group's rings (equal spacing n, southern rings in reverse order)."""
        r = np.arange(ps.start, ps.stop)
        first = self.start[4 * self.nside - 2 - r if south else r]
        return torch.from_numpy(first).cuda()[:, None] + torch.arange(n, device="cuda")[None, :]

    def synth(self, gn, gs):
        """G(m) of the north and south rings, [m, pair, map], m > 0 already doubled -> maps."""
        mmax, nb = gn.shape[0] - 1, gn.shape[2]
        out = torch.empty(nb, 12 * self.nside ** 2, dtype=torch.float64, device="cuda")
        for ps, n in self._groups():
            ph = self._phase(ps, n, mmax)[:, :, None]
            k = torch.arange(mmax + 1, device="cuda") % n
            for g, south in ((gn, False), (gs, True)):
                s = torch.zeros(n, ps.stop - ps.start, nb, dtype=torch.complex128, device="cuda")
                s.index_add_(0, k, g[:, ps] * ph)
                f = torch.fft.ifft(s, dim=0).real * n
                out[:, self._pixels(ps, n, south)] = f.permute(2, 1, 0)
        return out

    def anal(self, maps, mmax, weights):
        """F(m) = w_pix sum_j f_j exp(-i m phi_j) of north and south rings, [m, pair, map]; the
        equator has no south ring."""
        w = {"dz": 2.0 * math.pi * self.dz / self.nphi, "uniform": np.full(self.nphi.size, math.pi / 3 / self.nside ** 2),
             "one": np.ones(self.nphi.size)}[weights]
        f = [torch.zeros(mmax + 1, self.np, maps.shape[0], dtype=torch.complex128, device="cuda") for _ in range(2)]
        for ps, n in self._groups():
            ph = self._phase(ps, n, mmax).conj()[:, :, None]
            wr = torch.from_numpy(w[ps]).cuda()[:, None]
            k = torch.arange(mmax + 1, device="cuda") % n
            for side in range(2):
                s = torch.fft.fft(maps[:, self._pixels(ps, n, side == 1)].double() * wr, dim=2)
                f[side][:, ps] = s.permute(2, 1, 0)[k] * ph
        f[1][:, self.np - 1] = 0
        return f


class _Scaled:
    """Rows (order m, ring pair) of a three-term recursion in l whose early values underflow."""

    def __init__(self, shape):
        self.v1, self.v2, self.e = (torch.zeros(shape, dtype=torch.float64, device="cuda") for _ in range(3))
        self.live = torch.ones_like(self.e)

    def start(self, row, log2_value, sign):
        e = torch.floor((log2_value + 256.0) / 512.0).clamp(max=0.0)
        self.v1[row], self.v2[row], self.e[row] = sign * torch.exp2(log2_value - 512.0 * e), 0.0, e
        self.live[row] = (e == 0).double()

    def step(self, c1, c2):
        """v_l = c1 v_{l-1} - c2 v_{l-2}; c1 is overwritten."""
        self.v1, self.v2 = c1.mul_(self.v1).addcmul_(c2, self.v2, value=-1.0), self.v1

    def rescale(self):
        up = (self.e < 0) & (self.v1.abs() > BIG)
        self.v1 = torch.where(up, self.v1 / UNIT, self.v1)
        self.v2 = torch.where(up, self.v2 / UNIT, self.v2)
        self.e += up
        self.live = (self.e == 0).double()


def _scalar_tables(grid, lmax, ms):
    """lambda_lm [m in ms, l - ms[0], pair]."""
    m = torch.tensor(ms, dtype=torch.float64, device="cuda")[:, None]
    k = np.arange(1, ms[-1] + 1)
    c = 0.5 * (np.concatenate([[0.0], np.cumsum(np.log2((2 * k + 1) / (2.0 * k)))]) - math.log2(4 * math.pi))
    # x lambda_{l-1} = eps_l lambda_l + eps_{l-1} lambda_{l-2}, eps_l = sqrt((l^2-m^2)/(4l^2-1))
    l = torch.arange(ms[0], lmax + 1, dtype=torch.float64, device="cuda")[None, :]
    e1 = torch.sqrt(torch.clamp(l * l - m * m, min=1.0) / (4.0 * l * l - 1.0).abs())
    e0 = torch.sqrt(torch.clamp((l - 1.0) ** 2 - m * m, min=0.0) / (4.0 * (l - 1.0) ** 2 - 1.0).abs())
    c1, c2 = 1.0 / e1, e0 / e1
    s = _Scaled((len(ms), grid.np))
    out = torch.zeros(len(ms), lmax + 1 - ms[0], grid.np, dtype=torch.float64, device="cuda")
    for l in range(ms[0], lmax + 1):
        i = l - ms[0]
        s.step(grid.x * c1[:, i:i + 1], c2[:, i:i + 1])
        if l <= ms[-1]:
            s.start(i, c[l] + l * grid.log_sin, -1.0 if l & 1 else 1.0)
        if l % 16 == 0:
            s.rescale()
        torch.mul(s.v1, s.live, out=out[:, i])
    return out


def _spin_tables(grid, lmax, ms):
    """_{+2}lambda_lm and _{-2}lambda_lm of the north rings, [m in ms, l - ms[0], pair]."""
    m = torch.tensor(ms, dtype=torch.float64, device="cuda")[:, None]
    # log2 k!; the start at l0 = max(m, 2) is the edge element d^l0_{l0,o} or d^l0_{m,2}
    lf = np.concatenate([[0.0], np.cumsum(np.log2(np.arange(1, 2 * max(ms[-1], 2) + 3, dtype=np.longdouble)))])
    lp = torch.arange(ms[0], lmax + 1, dtype=torch.float64, device="cuda").clamp(min=3.0)[None, :]
    l = lp - 1.0
    r1 = torch.sqrt(torch.clamp(lp * lp - m * m, min=1.0) * (lp * lp - 4.0))
    r0 = torch.sqrt(torch.clamp((l * l - m * m) * (l * l - 4.0), min=0.0))
    n10, n1m = torch.sqrt((2 * l + 3) / (2 * l + 1)), torch.sqrt((2 * l + 3) / (2 * l - 1))
    a, b, c = n10 * (2 * l + 1) * lp / r1, n10 * (2 * l + 1) * 2.0 * m / (l * r1), n1m * lp * r0 / (l * r1)
    P, M = _Scaled((len(ms), grid.np)), _Scaled((len(ms), grid.np))
    outs = [torch.zeros(len(ms), lmax + 1 - ms[0], grid.np, dtype=torch.float64, device="cuda") for _ in range(2)]
    for lp in range(ms[0], lmax + 1):
        i = slice(lp - ms[0], lp - ms[0] + 1)
        P.step(torch.addcmul(b[:, i], a[:, i], grid.x), c[:, i])
        M.step(torch.addcmul(-b[:, i], a[:, i], grid.x), c[:, i])
        for mm in range(max(ms[0], 0 if lp == 2 else lp), min(lp, ms[-1]) + 1 if lp >= 2 else 0):
            o = min(mm, 2)
            k = 0.5 * (lf[2 * lp] - lf[lp + o] - lf[lp - o] + np.log2((2 * lp + 1) / (4 * np.pi)))
            sp = -1.0 if mm & 1 else 1.0
            P.start(mm - ms[0], float(k) + (lp - o) * grid.log_ch + (lp + o) * grid.log_sh, sp)
            M.start(mm - ms[0], float(k) + (lp + o) * grid.log_ch + (lp - o) * grid.log_sh, sp if mm >= 2 else 1.0)
        if lp % 16 == 0:
            P.rescale()
            M.rescale()
        for out, s in zip(outs, (P, M)):
            torch.mul(s.v1, s.live, out=out[:, lp - ms[0]])
    return outs


def _chunks(grid, lmax, mmax, tables):
    """Runs of consecutive orders whose tables stay within 64 GB."""
    m = 0
    while m <= mmax:
        n = max(1, min(mmax + 1 - m, 256, int(8e9 / (tables * grid.np * (lmax + 1 - m)))))
        yield list(range(m, m + n))
        m += n


def _rows(alm, lmax, ms):
    """alm [map, :] -> [m in ms, l - ms[0], map] (zero for l < m)."""
    ofs, _ = _alm_sizes(lmax, ms[-1])
    out = torch.zeros(len(ms), lmax + 1 - ms[0], alm.shape[0], dtype=torch.complex128, device="cuda")
    for i, m in enumerate(ms):
        out[i, m - ms[0]:] = alm[:, ofs[m] + m: ofs[m] + lmax + 1].T
    return out


def _unrows(rows, alm, lmax, ms):
    ofs, _ = _alm_sizes(lmax, ms[-1])
    for i, m in enumerate(ms):
        alm[:, ofs[m] + m: ofs[m] + lmax + 1] = rows[i, m - ms[0]:].T


def _mul(t, z):
    """Real [m, a, b] times complex [m, b, map]."""
    return torch.view_as_complex(torch.bmm(t, torch.view_as_real(z.contiguous()).flatten(2)).unflatten(2, (-1, 2)).contiguous())


def _eps(lmax, ms):
    """(-1)^(l - m), [m, l - ms[0], 1]."""
    l = torch.arange(ms[0], lmax + 1, device="cuda")[None, :]
    return (1.0 - 2.0 * ((l - torch.tensor(ms, device="cuda")[:, None]) & 1)).double()[:, :, None]


def _twice(mmax):
    c = torch.full((mmax + 1, 1, 1), 2.0, dtype=torch.float64, device="cuda")
    c[0] = 1.0
    return c


def _synth(alm, nside, lmax, mmax):
    grid = _Grid(nside)
    gn, gs = (torch.empty(mmax + 1, grid.np, alm.shape[0], dtype=torch.complex128, device="cuda") for _ in range(2))
    for ms in _chunks(grid, lmax, mmax, 1):
        t, a = _scalar_tables(grid, lmax, ms).transpose(1, 2), _rows(alm.to(torch.complex128), lmax, ms)
        gn[ms], gs[ms] = _mul(t, a), _mul(t, a * _eps(lmax, ms))
    c = _twice(mmax)
    return grid.synth(gn * c, gs * c)


def _anal(maps, nside, lmax, mmax, weights):
    grid = _Grid(nside)
    fn, fs = grid.anal(maps, mmax, weights)
    alm = torch.zeros(maps.shape[0], _alm_sizes(lmax, mmax)[1], dtype=torch.complex128, device="cuda")
    for ms in _chunks(grid, lmax, mmax, 1):
        t = _scalar_tables(grid, lmax, ms)
        _unrows(_mul(t, fn[ms]) + _eps(lmax, ms) * _mul(t, fs[ms]), alm, lmax, ms)
    return alm


def _spin_synth(E, B, nside, lmax, mmax):
    grid = _Grid(nside)
    g = [torch.empty(mmax + 1, grid.np, E.shape[0], dtype=torch.complex128, device="cuda") for _ in range(4)]
    for ms in _chunks(grid, lmax, mmax, 2):
        p, m = (t.transpose(1, 2) for t in _spin_tables(grid, lmax, ms))
        e, b = (_rows(a.to(torch.complex128), lmax, ms) for a in (E, B))
        ap, am, s = e + 1j * b, e - 1j * b, _eps(lmax, ms)
        x1, x2, x3, x4 = _mul(p, ap), _mul(m, am), _mul(p, s * am), _mul(m, s * ap)
        for out, v in zip(g, (-0.5 * (x1 + x2), -0.5 * (x3 + x4), -0.5j * (x2 - x1), -0.5j * (x3 - x4))):
            out[ms] = v
    c = _twice(mmax)
    return grid.synth(g[0] * c, g[1] * c), grid.synth(g[2] * c, g[3] * c)


def _spin_anal(Q, U, nside, lmax, mmax, weights):
    grid = _Grid(nside)
    (qn, qs), (un, us) = (grid.anal(x, mmax, weights) for x in (Q, U))
    E, B = (torch.zeros(Q.shape[0], _alm_sizes(lmax, mmax)[1], dtype=torch.complex128, device="cuda") for _ in range(2))
    for ms in _chunks(grid, lmax, mmax, 2):
        p, m = _spin_tables(grid, lmax, ms)
        s = _eps(lmax, ms)

        def both(t, n, sg):  # sum over the north rings, plus +-(-1)^(l-m) times the south ones
            return _mul(t, n[0][ms]) + sg * s * _mul(t, n[1][ms])
        q, u = (qn, qs), (un, us)
        _unrows(-0.5 * (both(p, q, 1) + 1j * both(p, u, -1) + both(m, q, 1) - 1j * both(m, u, -1)), E, lmax, ms)
        _unrows(-0.5 * (both(p, u, 1) - 1j * both(p, q, -1) + both(m, u, 1) + 1j * both(m, q, -1)), B, lmax, ms)
    return E, B


def _cl(alm, lmax, mmax):
    l, m = _lm(lmax, mmax)
    c = torch.zeros(alm.shape[0], lmax + 1, dtype=torch.float64, device="cuda")
    c.index_add_(1, l, alm.abs().square() * torch.where(m > 0, 2.0, 1.0))
    return c / (2.0 * torch.arange(lmax + 1, device="cuda") + 1.0)


def _grad(case, x):
    nside, lmax = case["nside"], case["lmax"]
    a = _anal(x["T"], nside, lmax, lmax, "dz"), *_spin_anal(x["Q"], x["U"], nside, lmax, lmax, "dz")
    l, _ = _lm(lmax, lmax)
    target, loss, g = 1.1 * _noise_cl(case), 0.0, []
    for alm in a:
        d = (_cl(alm, lmax, lmax) - target) / target
        d[:, :2] = 0
        loss = loss + d.square().sum()
        # dC_l/da = 2 c_m a / (2l + 1); the adjoint takes every m once, _synth m > 0 twice
        w = 2.0 * d / target * 2.0 / (2.0 * torch.arange(lmax + 1, device="cuda") + 1.0)
        g.append(alm * w[:, l])
    z, nphi, _, dz = _rings(nside)
    wr = torch.from_numpy(np.repeat(2.0 * math.pi * dz / nphi, nphi)).cuda()
    T = _synth(g[0], nside, lmax, lmax) * wr
    Q, U = _spin_synth(g[1], g[2], nside, lmax, lmax)
    return {"loss": loss, "T": T, "Q": Q * wr, "U": U * wr}


def _rotate(alm, lmax):
    """sum_m' exp(-i m alpha) d^l_mm'(beta) exp(-i m' gamma) a_lm', d^l by its recursion in l."""
    alpha, beta, gamma = EULER
    m = torch.arange(lmax + 1, dtype=torch.float64, device="cuda")[:, None]
    k = torch.arange(-lmax, lmax + 1, dtype=torch.float64, device="cuda")[None, :]
    lc, ls, x = math.log2(math.cos(beta / 2)), math.log2(math.sin(beta / 2)), math.cos(beta)
    lf = torch.from_numpy(np.concatenate([[0.0], np.cumsum(np.log2(np.arange(1, 2 * lmax + 2, dtype=np.longdouble)))]).astype(np.float64)).cuda()
    # edge l0 = max(m, |m'|): d_{j,k} with j = l0 up to sign; d_{a,b} = (-1)^(a-b) d_{b,a} = d_{-b,-a}
    big = m >= k.abs()
    j = torch.where(big, m + 0 * k, k.abs() + 0 * m)
    o = torch.where(big, k + 0 * m, torch.where(k > 0, m + 0 * k, -m + 0 * k))
    odd = torch.where(big | (k < 0), (j - o) % 2, torch.zeros_like(j))
    edge = 0.5 * (lf[(2 * j).long()] - lf[(j + o).long()] - lf[(j - o).long()]) + (j + o) * lc + (j - o) * ls
    sign = 1.0 - 2.0 * odd
    s = _Scaled((lmax + 1, 2 * lmax + 1))
    e0 = torch.floor((edge + 256.0) / 512.0).clamp(max=0.0)
    v0 = sign * torch.exp2(edge - 512.0 * e0)
    out = torch.zeros_like(alm)
    ofs, _ = _alm_sizes(lmax, lmax)
    ofs = torch.from_numpy(ofs).cuda()
    for l in range(lmax + 1):
        if l:
            q = l - 1.0
            r1 = torch.sqrt(torch.clamp((l * l - m * m) * (l * l - k * k), min=1.0))
            if q:
                r0 = torch.sqrt(torch.clamp(q * q - m * m, min=0.0) * torch.clamp(q * q - k * k, min=0.0))
                s.step((2 * q + 1) * (q * l * x - m * k) / (q * r1), l * r0 / (q * r1))
            else:
                s.step(torch.full_like(s.v1, x), torch.zeros_like(s.v1))
        at = j == l
        s.v1, s.v2, s.e = torch.where(at, v0, s.v1), torch.where(at, 0.0, s.v2), torch.where(at, e0, s.e)
        s.rescale()
        d = (s.v1 * s.live)[: l + 1, lmax - l: lmax + l + 1]
        a = alm[:, ofs[: l + 1] + l]
        full = torch.cat([(a.conj() * (1.0 - 2.0 * (torch.arange(l + 1, device="cuda") & 1)))[:, 1:].flip(1), a], 1)
        kk = k[0, lmax - l: lmax + l + 1]
        full = full * torch.polar(torch.ones_like(kk), -gamma * kk)
        r = torch.view_as_complex(torch.matmul(d, torch.view_as_real(full)).contiguous())
        mm = m[: l + 1, 0]
        out[:, ofs[: l + 1] + l] = r * torch.polar(torch.ones_like(mm), -alpha * mm)
    return out


def exact(case, seed):
    k, nside, lmax, mmax = case["kind"], case["nside"], case["lmax"], case["mmax"]
    if case["nmaps"] * case["nside"] ** 2 > 4 * 2048 ** 2:
        return None  # 64 maps at full size: minutes
    x = _inputs(case, seed)
    if k == "synth":
        return {"map": _synth(x["alm"], nside, lmax, mmax)}
    if k == "anafast":
        a = _anal(x["maps"], nside, lmax, mmax, case["weights"])
        return {"alm": a, "cl": _cl(a, lmax, mmax)}
    if k in ("roundtrip", "batched"):
        m = _synth(x["alm"], nside, lmax, mmax)
        a = _anal(m, nside, lmax, mmax, "dz")
        if k == "batched":
            return {"map": m.reshape(-1), "alm": a.reshape(-1)}
        return {"map": m, "alm": a, "cl": _cl(a, lmax, mmax)}
    if k == "spin_synth":
        Q, U = _spin_synth(x["E"], x["B"], nside, lmax, mmax)
        return {"Q": Q, "U": U}
    if k == "spin_anal":
        E, B = _spin_anal(x["Q"], x["U"], nside, lmax, mmax, case["weights"])
        return {"E": E, "B": B}
    if k == "grad":
        return _grad(case, x)
    if k == "smooth":
        l = torch.arange(lmax + 1, dtype=torch.float64, device="cuda")
        b = torch.exp(-0.5 * l * (l + 1.0) * FWHM ** 2 / (8.0 * math.log(2.0)))
        a = _anal(x["maps"], nside, lmax, mmax, "dz") * b[_lm(lmax, mmax)[0]]
        return {"map": _synth(a, nside, lmax, mmax)}
    return {"alm": _rotate(x["alm"].to(torch.complex128), lmax)}
