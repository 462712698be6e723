"""Cases of the estimator's public entry points: what a user of the framework has it compute.

Four kinds of work:

* ``box``: one particle box through a resident plan (``Estimator.run_device``): positions
  already in HBM, P(k) and B(k1,k2,k3) rows out.  The rows are returned as the columns of
  the record arrays that ``MEASUREMENTS.powerspectrum`` / ``bispectrum`` keep: float32,
  and float64 for the FP64 form, which a program picks for its extra digits.
* ``batch``: boxes that arrive on the host, through the captured form
  (``Estimator.graph_run_host``) as the serving loop runs it, results back on the host.
* ``cross``: two densities on the host through the f2py drop-ins ``measure_pk`` and
  ``measure_bk_cross``, the calls of a cross-spectrum session of the reference's script.
* ``catalog``: a catalogue's positions and velocities in HBM to the positions the
  assignment reads (``catalog.positions``).

One plan per configuration is kept between boxes, as a program that measures many boxes
does.  Positions, fields and catalogues come from the seed alone.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from pbi4_gb300 import bispectrumI4, catalog, powerI4, synthetic
from pbi4_gb300.estimator import Estimator, EstimatorConfig

BOX = 1000.0


# ------------------------------------------------------------------ cases ---
def _box(name, grid, npart, nintp, interlacing, multipoles, kbin, nbins, precision, clustered=True, iopen=True,
         weights=False, budget_mb=0, kind="box", batch=1):
    return dict(name=name, kind=kind, grid=grid, npart=npart, nintp=nintp, interlacing=interlacing,
                multipoles=multipoles, kbin=float(kbin), nbins=nbins, precision=precision, clustered=clustered,
                iopen=iopen, weights=weights, budget_mb=budget_mb, batch=batch)


def listed():
    return [
        # a quick look at a small mock: uniform points, CIC, real space, closed triangles, the default precision
        _box("cic_64", 64, 100_000, 2, False, False, 2, 8, "fp32", clustered=False, iopen=False),
        # P(k) alone of a sparse galaxy mock, the smallest request of a serving mix
        _box("pk_128", 128, 356_467, 3, True, False, 2, 0, "fp16split"),
        # four small clustered boxes of a serving queue, host to host in one launch
        _box("batch_192", 192, 300_007, 4, True, False, 2, 24, "fp16split", kind="batch", batch=4),
        # the redshift-space box of the benchmark, mixed precision
        _box("zeldovich_256", 256, 128 ** 3, 4, True, True, 3, 21, "fp16split"),
        # the same box by the default precision of the plan and of the drop-ins
        _box("zeldovich_256_fp32", 256, 128 ** 3, 4, True, True, 3, 21, "fp32"),
        # a weighted survey mock on a grid that no tile size divides
        _box("weighted_250_tf32", 250, 1_234_567, 3, True, True, 3, 17, "tf32split", weights=True),
        # the densest box of a serving mix
        _box("serving_384", 384, 10_000_000, 4, True, False, 2, 48, "fp16split"),
        # many shells of a simulation box on a fine grid
        _box("shells_512", 512, 256 ** 3, 4, True, True, 2, 40, "fp16split"),
        # the largest single box: its maps go through in slabs
        _box("large_1024", 1024, 512 ** 3, 4, True, True, 4, 25, "fp16split", budget_mb=4096),
        # a check run in double precision
        _box("check_128_fp64", 128, 64 ** 3, 4, True, True, 3, 10, "fp64"),
        # cross spectra of two tracers, from densities that the script keeps on the host
        dict(name="cross_128", kind="cross", grid=128, kbin=3.0, nbins=10, iopen=True),
        # a snapshot's catalogue into redshift space
        dict(name="catalog_1e7", kind="catalog", npart=10_000_000, double=False, velocities=True, mode=1),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["box", "box", "box", "box", "box", "batch", "cross", "catalog"])
    if kind == "catalog":
        return dict(kind=kind, npart=_log_int(rng, 10_000, 30_000_000), double=rng.random() < 0.3,
                    velocities=rng.random() < 0.7, mode=rng.choice([0, 1]))
    if kind == "cross":
        grid = 2 * rng.randint(32, 80)
        kbin = float(rng.choice([2, 3]))
        return dict(kind=kind, grid=grid, kbin=kbin, nbins=rng.randint(4, max(5, int(0.24 * grid / kbin))),
                    iopen=rng.random() < 0.7)
    if kind == "batch":
        grid = rng.choice([128, 192, 256])
        with_b = rng.random() < 0.6
        c = _box("", grid, _log_int(rng, 100_000, 3_000_000), rng.choice([2, 3, 4]), rng.random() < 0.5, False, 2,
                 grid // 8 if with_b else 0, "fp16split", clustered=rng.random() < 0.5, kind=kind,
                 batch=rng.randint(1, 4))
    else:
        grid = _log_int(rng, 64, 512)
        grid = grid // 16 * 16 if rng.random() < 0.5 else grid // 2 * 2
        multipoles = rng.random() < 0.5
        precision = rng.choice(["fp32", "fp32", "fp16split", "fp16split", "tf32split", "fp64"]
                               + ([] if multipoles else ["bf16"]))
        if precision == "fp64":
            grid = min(grid, 160)
        kbin = rng.choice([1, 2, 3, 4])
        most = {"fp32": 30, "fp64": 16}.get(precision, 44)
        nbins = min(most, rng.randint(3, max(4, int(0.24 * grid / kbin))))
        c = _box("", grid, _log_int(rng, 50_000, 20_000_000 if grid > 200 else 3_000_000), rng.choice([2, 3, 4]),
                 rng.random() < 0.7, multipoles, kbin, nbins if rng.random() < 0.75 else 0, precision,
                 clustered=rng.random() < 0.6, iopen=rng.random() < 0.7, weights=rng.random() < 0.25)
    del c["name"]
    return c


# ----------------------------------------------------------------- inputs ---
def _positions(case, seed):
    """(3, npart) float64 in [0, 1) on the GPU, in catalogue (lattice) or random order."""
    n = int(case["npart"])
    if case["clustered"]:
        side = max(8, math.ceil(n ** (1 / 3) - 1e-9))
        pos = synthetic.zeldovich_box_device(side, BOX, n_s=-1.5, rms_disp=5.0, f_growth=0.7, seed=int(seed))
        # a catalogue that is smaller than its lattice is an even thinning of it
        if side ** 3 > n:
            pos = pos[:, torch.div(torch.arange(n, device="cuda") * side ** 3, n, rounding_mode="floor")]
        return pos.contiguous()
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return torch.rand((3, n), generator=g, device="cuda", dtype=torch.float32).double()


def _weights(case, seed):
    if not case["weights"]:
        return None
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) + 1)
    return 0.5 + torch.rand(int(case["npart"]), generator=g, device="cuda", dtype=torch.float64)


def _batch_positions(case, seed):
    """The boxes of a batch: unequal particle counts, other particles each."""
    return [_positions(dict(case, npart=int(case["npart"]) - 1013 * b), int(seed) + 7919 * b)
            for b in range(int(case["batch"]))]


def _fields(case, seed):
    """Two correlated non-Gaussian densities: full complex spectra [z][y][x] on the GPU."""
    n = int(case["grid"])
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    k = torch.fft.fftfreq(n, 1.0 / n, dtype=torch.float64, device="cuda")
    k2 = k[:, None, None] ** 2 + k[None, :, None] ** 2 + k[None, None, :] ** 2
    amp = torch.where(k2 > 0, k2.clamp_min(1.0) ** -0.75, 0.0)
    out = []
    for _ in range(2):
        f = torch.randn((n, n, n), generator=g, dtype=torch.float64, device="cuda")
        if out:
            f = 0.8 * out[0] + 0.6 * f
        out.append(f)
    spectra = []
    for f, b in zip(out, (0.5, 0.3)):
        f = torch.fft.ifftn(torch.fft.fftn(f) * amp).real
        f = f / f.std()
        spectra.append(torch.fft.fftn(f + b * (f * f - 1)) * (BOX / n) ** 3)
    return spectra


def _catalogue(case, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    dt = torch.float64 if case["double"] else torch.float32
    n = int(case["npart"])
    pos = torch.rand((n, 3), generator=g, device="cuda", dtype=dt) * BOX
    vel = None
    if case["velocities"]:
        vel = 300.0 * torch.randn((n, 3), generator=g, device="cuda", dtype=dt)
        if int(case["mode"]) == 0:
            vel = vel / 100.0  # already a length
    return pos, vel


_HZ, _Z = 130.8, 0.5

_KEPT: dict = {}


def _plan(case):
    """The plan of this configuration, kept until another one is asked for."""
    key = tuple(sorted((k, v) for k, v in case.items() if k not in ("name", "clustered", "weights")))
    if key not in _KEPT:
        _KEPT.clear()
        stream = torch.cuda.Stream() if case["kind"] == "batch" else None
        cfg = EstimatorConfig(grid=int(case["grid"]), box=BOX, nintp=int(case["nintp"]),
                              interlacing=bool(case["interlacing"]), multipoles=bool(case["multipoles"]),
                              do_bispectrum=int(case["nbins"]) > 0, kbin_bs=case["kbin"], kcenter_bs=case["kbin"],
                              nbins_bs=max(1, int(case["nbins"])), iopen=bool(case["iopen"]),
                              precision=case["precision"], map_budget_mb=int(case["budget_mb"]))
        est = Estimator(cfg, stream=stream)
        if case["kind"] == "batch":
            est.graph_build(batch=int(case["batch"]), npart_cap=int(case["npart"]))
        _KEPT[key] = (est, stream)
    return _KEPT[key]


def prepare(case, seed):
    kind = case["kind"]
    if kind == "catalog":
        pos, vel = _catalogue(case, seed)
        return dict(case=case, pos=pos, vel=vel)
    if kind == "cross":
        # Fortran-ordered complex grids, as the script holds them; counts as count_triangles returns them
        d = [f.cpu().numpy().T for f in _fields(case, seed)]
        tri = _triangles(int(case["nbins"]), bool(case["iopen"]), True)
        counts = bispectrumI4.count_triangles(case["nbins"], case["grid"], case["kbin"], case["kbin"],
                                              case["iopen"], True, 1, len(tri))
        return dict(case=case, d=d, counts=counts, itot=len(tri))
    est, stream = _plan(case)
    if kind == "batch":
        pos = []
        for p in _batch_positions(case, seed):
            h = torch.empty(p.shape, dtype=torch.float64, pin_memory=True)
            h.copy_(p)
            pos.append(h)
        pout = [torch.empty((est.nbins_ps, 5), dtype=torch.float64, pin_memory=True) for _ in pos]
        bout = ([torch.empty((est.itot, est.brows), dtype=torch.float64, pin_memory=True) for _ in pos]
                if est.itot else None)
        return dict(case=case, est=est, stream=stream, pos=pos, pout=pout, bout=bout)
    pout, bout = est.alloc_outputs()
    return dict(case=case, est=est, pos=_positions(case, seed), weight=_weights(case, seed), pout=pout, bout=bout)


_P_ROWS = {True: ("avgk", "P0", "P2", "P4", "Nmodes"), False: ("avgk", "P0", "Nmodes")}
_B_ROWS = ("k1", "k2", "k3", "Pk1", "Pk2", "Pk3", "B0", "BSN", "Ntr", "B2", "B4")
_X_ROWS = ("k1", "k2", "k3", "B0", "Ntr")


def _record(case, pout, bout):
    out = {n: pout[i] for i, n in enumerate(_P_ROWS[bool(case["multipoles"])])}
    if bout is not None:
        out.update({n: bout[i] for i, n in enumerate(_B_ROWS[:bout.shape[0]])})
    return out


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "catalog":
        return catalog.positions(state["pos"], state["vel"], los=(0.0, 0.0, 1.0), hz=_HZ, z=_Z, box=BOX,
                                 rsd_mode=int(case["mode"]))
    if kind == "cross":
        g, kb, nb = case["grid"], case["kbin"], case["nbins"]
        pk = powerI4.measure_pk(g, BOX, 1.0, 1.0, g // 2, *state["d"])
        bk = bispectrumI4.measure_bk_cross(nb, g, kb, kb, case["iopen"], 2 * np.pi / BOX, 1, state["itot"], 1,
                                           state["counts"], *state["d"]).astype(np.float32)
        out = {n: pk[i] for i, n in enumerate(_P_ROWS[False])}
        out.update({"x" + n: bk[i] for i, n in enumerate(_X_ROWS)})
        return out
    est = state["est"]
    if kind == "batch":
        est.graph_run_host([p.numpy() for p in state["pos"]], [o.numpy() for o in state["pout"]],
                           [o.numpy() for o in state["bout"]] if state["bout"] else None)
        est.check()
        return [_record(case, p.numpy().T.astype(np.float32),
                        state["bout"][i].numpy().T.astype(np.float32) if state["bout"] else None)
                for i, p in enumerate(state["pout"])]
    est.run_device(state["pos"].shape[1], state["pos"], state["pout"], state["bout"], weight=state["weight"])
    pout, bout = state["pout"], state["bout"]
    if case["precision"] != "fp64":
        pout, bout = pout.float(), None if bout is None else bout.float()
    return _record(case, pout, bout)


# ------------------------------------------------------------------- work ---
def _triangles(nb, iopen, cross):
    """(l, j, i) of every triangle in the reference's order (kcenter = kbin)."""
    shift = 1 + (1 if iopen else 0)
    return [(l, j, i) for l in range(1, nb + 1) for j in range(1, l + 1)
            for i in range(max(1, l - j + 1 - shift), (min(nb, j + l - 1 + shift) if cross else j) + 1)]


def _kmax(case):
    return int(math.ceil((int(case["nbins"]) + 0.5) * case["kbin"]))


def work(case):
    kind = case["kind"]
    if kind == "catalog":
        n, s = int(case["npart"]), 8 if case["double"] else 4
        return dict(bytes=n * 3 * (s * (2 if case["velocities"] else 1) + 8), flops=n * 3 * 6)
    g, nb = int(case["grid"]), int(case["nbins"])
    if kind == "cross":
        tri, m = len(_triangles(nb, case["iopen"], True)), 3 * _kmax(case) + 1
        half = g * g * (g // 2 + 1)
        return dict(bytes=2 * 16 * half + 4 * tri + 8 * (5 * tri + 5 * (g // 2)),
                    flops=8 * half + 2 * nb * 2.5 * m ** 3 * 3 * math.log2(m) + 2 * m ** 3 * tri)
    npart, grids, sets = int(case["npart"]), 2 if case["interlacing"] else 1, 3 if case["multipoles"] else 1
    tri = len(_triangles(nb, case["iopen"], False)) if nb else 0
    by = npart * (32 if case["weights"] else 24) + 8 * (5 * (g // 2) + (11 if sets == 3 else 9) * tri)
    fl = grids * (npart * 2 * int(case["nintp"]) ** 3 + 2.5 * g ** 3 * 3 * math.log2(g)) + 12 * grids * g ** 3
    if nb:
        m = 3 * _kmax(case) + 1
        fl += sets * nb * 2.5 * m ** 3 * 3 * math.log2(m) + 2 * m ** 3 * tri * sets
    return dict(bytes=by * int(case["batch"]), flops=fl * int(case["batch"]))


# ------------------------------------------------------------------ exact ---
# The estimator in 64-bit torch, from its definition: direct assignment, full transforms,
# one matrix product over the grid points for the triangle sums.
_F64 = torch.float64
_TWOPI32 = float(np.float32(6.28319))  # the reference's constant


def _freq(n):
    k = torch.arange(n, device="cuda")
    return torch.where(k <= n // 2, k, k - n)


def _nint(t):
    a = t.abs()
    f = a.floor()
    return (torch.sign(t) * (f + (a - f >= 0.5).to(t.dtype))).long()


def _axis(p, n, nintp, shifted, single):
    """First cell and the stencil's weights on one axis."""
    v = n * p + 1.0
    if shifted:
        v = v - 0.5
    if nintp == 4:
        i = v.floor()
        h = v - i
        w0, w1, w3 = (1 - h) ** 3 / 6, 4 / 6 + (0.5 * h - 1) * h * h, h ** 3 / 6
        return i.long() - 2, [w0, w1, 1 - w0 - w1 - w3, w3]
    if nintp == 3:
        i = _nint(v)
        h = v - i
        w0, w1 = (0.5 - h) ** 2 / 2, 0.75 - h * h
        return i - 2, [w0, w1, 1 - w0 - w1]
    i = v.floor().long()
    h = v - _nint(v) if single else v - i
    return i, [1 - h, h]


def _assign(pos, weight, n, nintp, shifted, single):
    grid = torch.zeros(n ** 3, dtype=_F64, device="cuda")
    step = 1 << 23
    for s in range(0, pos.shape[1], step):
        ax = [_axis(pos[d, s:s + step], n, nintp, shifted, single) for d in range(3)]
        cell = [[torch.remainder(ax[d][0] + c, n) for c in range(nintp)] for d in range(3)]
        for z in range(nintp):
            for y in range(nintp):
                row = (cell[2][z] * n + cell[1][y]) * n
                wzy = ax[2][1][z] * ax[1][1][y]
                if weight is not None:
                    wzy = wzy * weight[s:s + step]
                for x in range(nintp):
                    grid.index_add_(0, row + cell[0][x], wzy * ax[0][1][x])
    return grid.view(n, n, n)


def _window(n, nintp):
    k = torch.arange(n // 2 + 1, dtype=_F64, device="cuda")
    r = (_TWOPI32 / n) * k / 2
    w = torch.where(k > 0, torch.sin(r) / r.clamp_min(1e-30), torch.ones_like(r))
    return w ** nintp


def _delta(case, pos, weight):
    """delta(k) on the kx >= 0 half: interlacing combine and window, [z][y][x]."""
    n, nintp, inter = int(case["grid"]), int(case["nintp"]), bool(case["interlacing"])
    t = np.float32(6.28319)
    kf3 = float(np.float32(np.float32(np.float32(np.float32(np.float32(t * t) * t) / np.float32(BOX))
                                      / np.float32(BOX)) / np.float32(BOX)))
    d = torch.fft.rfftn(_assign(pos, weight, n, nintp, False, not inter))
    w = _window(n, nintp)
    h, full = n // 2, torch.arange(n, device="cuda")
    wf = w[torch.minimum(full, n - full)]
    if inter:
        f2 = torch.fft.rfftn(_assign(pos, weight, n, nintp, True, False))
        # the phase signs: y, z as the signed frequency (the Nyquist planes as -N/2); on the kx = N/2
        # plane the reference's later writes mirror the half with the lower y (z) index
        ang = -(_TWOPI32 / n) / 2
        sg = torch.where((full > 0) & (full < h), 1.0, -1.0).to(_F64)
        mag = torch.minimum(full, n - full).to(_F64) * ang
        x = torch.arange(h + 1, dtype=_F64, device="cuda") * ang
        edge = (full == 0) | (full == h)
        for z in range(n):
            th = x[None, :] + (sg * mag)[:, None] + (sg * mag)[z]
            lo_z = 0 < z < h
            if z in (0, h):
                flip = (~edge) & (full < h)
                zs = torch.where(flip, 1.0, -1.0).to(_F64)
                ys = torch.where(flip, 1.0, -1.0).to(_F64)
            else:
                flip = torch.where(edge, torch.full_like(edge, lo_z), full < h)
                zs = torch.full_like(mag, 1.0 if lo_z else -1.0)
                ys = torch.where(edge, 1.0 if lo_z else -1.0, sg)
            xs = torch.where(flip, -1.0, 1.0).to(_F64)
            for e in (0, h):
                th[:, e] = xs * x[e] + ys * mag + zs * mag[z]
            d[z] = 0.5 * (d[z] + torch.polar(torch.ones_like(th), th) * f2[z])
        del f2
    d /= (wf[:, None, None] * wf[None, :, None] * w[None, None, :]) * (kf3 * pos.shape[1])
    return d


def _power(n, kbin, nbins, values, los_mu):
    """avgk, mode counts and the sums of `values(z)` (functions of a z plane) per P bin."""
    kf = float(np.float32(6.28319) / np.float32(BOX))
    h = n // 2
    ky, kx = _freq(n).to(_F64)[:, None], torch.arange(h + 1, dtype=_F64, device="cuda")[None, :]
    sums = [torch.zeros(nbins + 1, dtype=_F64, device="cuda") for _ in range(2 + len(los_mu))]
    for z in range(n):
        kz = float(z if z <= h else z - n)
        s = ((kf * kx) ** 2 + (kf * ky) ** 2) + (kf * kz) ** 2
        rk = torch.sqrt(s)
        b = _nint(rk / (kbin * kf) - 1.0 - 2.2250738585072014e-308) + 1
        keep = (kx > 0) | (ky > 0) | ((ky == 0) & torch.full_like(ky, kz > 0, dtype=torch.bool))
        b = torch.where(keep & (b >= 1) & (b <= nbins), b, 0).reshape(-1)
        p = values(z)
        k2 = kx * kx + ky * ky + kz * kz
        mu2 = kz * kz / k2.clamp_min(1.0)
        cols = [torch.ones_like(rk), rk] + [p * f(mu2) for f in los_mu]
        for a, c in zip(sums, cols):
            a.index_add_(0, b, c.reshape(-1))
    return [a[1:] for a in sums], kf ** 3


_LEG = (lambda m: torch.ones_like(m), lambda m: -0.5 + 1.5 * m, lambda m: 0.375 - 3.75 * m + 4.375 * m * m)


def _shell_of(k2, kbin, nb):
    b = _nint(torch.sqrt(k2.to(_F64)) / kbin - 1.0 - 1.1754943508222875e-38) + 1
    return torch.where((b >= 1) & (b <= nb), b, 0)


def _map_size(n, kmax):
    for m in range(2 * (3 * kmax // 2) + 2, n, 2):
        r = m
        for f in (2, 3, 5, 7):
            while r % f == 0:
                r //= f
        if r == 1:
            return m
    return n


def _shell_maps(n, kbin, nb, sources):
    """Real-space shell maps of each source (a half spectrum and a factor of mu^2) on the smallest
    alias-free grid, the shells' powers of the first source and the shells' mode counts."""
    kall = _freq(n)[:, None, None] ** 2 + _freq(n)[None, :, None] ** 2 + torch.arange(
        n // 2 + 1, device="cuda")[None, None, :] ** 2
    shell_n = _shell_of(kall, kbin, nb)
    two = torch.full((n // 2 + 1,), 2.0, dtype=_F64, device="cuda")
    two[0] = two[-1] = 1.0
    nmodes = torch.zeros(nb + 1, dtype=_F64, device="cuda").index_add_(
        0, shell_n.reshape(-1), two.expand(n, n, -1).reshape(-1))[1:]
    kmax = int(torch.sqrt(kall[shell_n > 0].max().to(_F64)).floor())
    del kall, shell_n
    m = _map_size(n, kmax)
    k = torch.cat([torch.arange(kmax + 1, device="cuda"), torch.arange(-kmax, 0, device="cuda")])
    kx = torch.arange(kmax + 1, device="cuda")
    k2 = k[:, None, None] ** 2 + k[None, :, None] ** 2 + kx[None, None, :] ** 2
    shell = _shell_of(k2, kbin, nb)
    mu2 = k[:, None, None].to(_F64) ** 2 / k2.clamp_min(1).to(_F64)
    wx = torch.where(kx > 0, 2.0, 1.0).to(_F64)
    im, jn = torch.remainder(k, m), torch.remainder(k, n)
    at_m = (im[:, None, None] * m + im[None, :, None]) * (m // 2 + 1) + kx
    neg = torch.remainder(-torch.arange(2 * kmax + 1, device="cuda"), 2 * kmax + 1)
    maps, power = torch.empty((len(sources) * nb, m ** 3), dtype=_F64, device="cuda"), None
    for s, (src, leg) in enumerate(sources):
        blk = src[jn][:, jn][:, :, kx].clone()
        p0 = blk[:, :, 0]
        blk[:, :, 0] = 0.5 * (p0 + p0[neg][:, neg].conj())
        blk *= leg(mu2)
        if power is None:
            power = torch.zeros(nb + 1, dtype=_F64, device="cuda").index_add_(
                0, shell.reshape(-1), (wx * (blk.real ** 2 + blk.imag ** 2)).reshape(-1))[1:]
        for b in range(nb):
            half = torch.zeros(m * m * (m // 2 + 1), dtype=torch.complex128, device="cuda")
            sel = shell == b + 1
            half[at_m[sel]] = blk[sel]
            maps[s * nb + b] = torch.fft.irfftn(half.view(m, m, -1), s=(m, m, m), norm="forward").reshape(-1)
    # indicator maps on one octant, weighted by its mirror images
    h = m // 2
    ind = torch.empty((nb, (h + 1) ** 3), dtype=_F64, device="cuda")
    for b in range(nb):
        half = torch.zeros(m * m * (m // 2 + 1), dtype=torch.complex128, device="cuda")
        half[at_m[shell == b + 1]] = 1.0
        full = torch.fft.irfftn(half.view(m, m, -1), s=(m, m, m), norm="forward")
        ind[b] = full[:h + 1, :h + 1, :h + 1].reshape(-1)
    o = torch.full((h + 1,), 2.0, dtype=_F64, device="cuda")
    o[0] = o[h] = 1.0
    wgt = (o[:, None, None] * o[None, :, None] * o[None, None, :]).reshape(-1)
    return maps, ind, wgt, power, nmodes, m


def _contract(pairs, left, right, weight=None):
    """sum over points of left[a] left[b] right[q], for every pair (a, b) and q."""
    a, b = pairs[:, 0], pairs[:, 1]
    out = torch.zeros((len(pairs), right.shape[0]), dtype=_F64, device="cuda")
    step = max(4096, (1 << 28) // max(1, len(pairs)))
    for s in range(0, right.shape[1], step):
        x = left[:, s:s + step]
        if weight is not None:
            x = x * torch.ones_like(x)
        f = x[a] * x[b]
        if weight is not None:
            f *= weight[s:s + step]
        out += f @ right[:, s:s + step].T
    return out


def _triangle_sums(tri, cross, sets, nb, maps, ind, wgt, m):
    """S[set][triangle] and the integer triangle counts."""
    t = torch.tensor(tri, device="cuda") - 1
    l, j, i = t[:, 0], t[:, 1], t[:, 2]
    first, second, third = (j, l, i) if cross else (i, j, l)
    pairs, inv = torch.unique(torch.stack([first, second], 1), dim=0, return_inverse=True)
    c = _contract(pairs, maps[:nb], maps[nb:] if cross else maps)
    s = [c[inv, third + k * nb] for k in range(sets)]
    cnt = torch.round(_contract(pairs, ind, ind, wgt)[inv, third] / m ** 3)
    return s, cnt


def _bispectrum(case, d, npart):
    n, nb, kbin = int(case["grid"]), int(case["nbins"]), float(case["kbin"])
    sets = 3 if case["multipoles"] else 1
    maps, ind, wgt, power, nmodes, m = _shell_maps(n, kbin, nb, [(d, _LEG[k]) for k in range(sets)])
    tri = _triangles(nb, bool(case["iopen"]), False)
    s, cnt = _triangle_sums(tri, False, sets, nb, maps, ind, wgt, m)
    kf = np.float32(2.0 * math.pi / BOX)
    kf3 = float(np.float32(np.float32(kf * kf) * kf))
    c = (float(n) ** 3 * cnt).float().double()
    psn = 1.0 / npart / kf3
    pw = kf3 * power / nmodes - psn
    t = torch.tensor(tri, device="cuda") - 1
    p = [pw[t[:, k]] for k in range(3)]
    bsn = (p[0] + p[1] + p[2]) * psn + psn * psn
    sf = (n / m) ** 3
    rows = [kbin + kbin * t[:, k].to(_F64) for k in range(3)] + p + [
        kf3 * sf * s[0] / c + bsn, bsn, (c / float(n) ** 3).float().double()]
    if sets == 3:
        rows += [5 * kf3 * sf * s[1] / c, 9 * kf3 * sf * s[2] / c]
    return rows


def _exact_box(case, pos, weight):
    n, mp = int(case["grid"]), bool(case["multipoles"])
    d = _delta(case, pos, weight)
    sums, kf3 = _power(n, 1.0, n // 2, lambda z: d[z].real ** 2 + d[z].imag ** 2, _LEG if mp else _LEG[:1])
    co, avgk = sums[0], sums[1] / sums[0]
    p = [(2 * 2 * k + 1) * s * kf3 / co for k, s in enumerate(sums[2:])]
    out = dict(zip(_P_ROWS[mp], [avgk] + p + [co]))
    if int(case["nbins"]):
        out.update(zip(_B_ROWS, _bispectrum(case, d, pos.shape[1])))
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind == "catalog":
        pos, vel = _catalogue(case, seed)
        p = pos.double()
        if vel is not None:
            los = torch.tensor([0.0, 0.0, 1.0], dtype=_F64, device="cuda")
            p = p + (vel.double() * los / _HZ * (1 + _Z) if int(case["mode"]) == 1 else vel.double() * los)
        return (torch.remainder(p + BOX, BOX) / BOX).clamp_max(1.0).T.contiguous()
    if kind == "cross":
        n, nb = int(case["grid"]), int(case["nbins"])
        d = [f[:, :, :n // 2 + 1] for f in _fields(case, seed)]
        sums, kf3 = _power(n, 1.0, n // 2, lambda z: d[0][z].real * d[1][z].real + d[0][z].imag * d[1][z].imag,
                           _LEG[:1])
        out = dict(avgk=sums[1] / sums[0], P0=sums[2] * kf3 / sums[0], Nmodes=sums[0])
        maps, ind, wgt, _, _, m = _shell_maps(n, float(case["kbin"]), nb, [(f, _LEG[0]) for f in d])
        tri = _triangles(nb, bool(case["iopen"]), True)
        s, cnt = _triangle_sums(tri, True, 1, nb, maps, ind, wgt, m)
        kf = np.float32(2.0 * math.pi / BOX)
        kf3 = float(np.float32(np.float32(kf * kf) * kf))
        c = (float(n) ** 3 * cnt).float().double()
        t = torch.tensor(tri, device="cuda") - 1
        rows = [float(case["kbin"]) * (1 + t[:, k].to(_F64)) for k in range(3)]
        rows += [kf3 * (n / m) ** 3 * s[0] / c, (c / float(n) ** 3).float().double()]
        out.update(("x" + k, v) for k, v in zip(_X_ROWS, rows))
        return out
    if kind == "batch":
        return [_exact_box(case, p, None) for p in _batch_positions(case, seed)]
    return _exact_box(case, _positions(case, seed), _weights(case, seed))
