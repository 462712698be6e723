"""The FP32 plan's tiled assignment on grids that are not a multiple of 16 (tiles of 10 to 16
cells), on both forms of its particle sort (up to 2048 tiles, and more), with particles on cell
edges, on the box's edges, outside the box and crowded into one cell, against the FP64 plan's
64-bit grid in global memory, for any particle order and where the records find no room."""
import numpy as np
import pytest

from pbi4_gb300._lib import lib
from pbi4_gb300.estimator import Estimator, EstimatorConfig

pytestmark = pytest.mark.gpu

# Modes up to a quarter of the grid an axis, where the window correction is at most 1.52^3 = 3.5
# (order 4).  Per particle, an FP32 axis weight is off by at most 4 2^-24 and the other two axes'
# weights sum to 1, so the summed error of its cells is at most 3 axes x 4 cells x 4 2^-24, and
# the mode's, divided by the particle number like the mode, 3.5 times that; 20 2^-24 for the FP32
# grid and transform.  Weights are at most 2.
TOL = (3.5 * 48 + 20) * 2.0 ** -24


def _particles(n, grid, seed):
    rng = np.random.default_rng(seed)
    pos = rng.random((3, n))
    edge = rng.integers(0, grid + 1, (3, n)) / grid
    half = (rng.integers(0, grid, (3, n)) + 0.5) / grid
    pick = rng.integers(0, 6, (3, n))
    pos = np.where(pick == 0, edge, np.where(pick == 1, half, pos))
    pos = np.where(pick == 2, np.nextafter(edge, rng.integers(0, 2, (3, n))), pos)
    pos[:, : n // 8] = pos[:, :1]  # one cell holds an eighth of them
    pos[:, -4:] = [[0.0, 1.0, -1e-3, 1.0 + 1e-3], [1.0, 0.0, -1e-3, 0.3], [1.0, 0.0, 0.7, 1.0 + 1e-3]]
    return np.ascontiguousarray(pos)


def _delta(pos, weight, precision="fp32", fail=0, **kw):
    import torch
    est = Estimator(EstimatorConfig(box=1000.0, do_bispectrum=False, precision=precision, **kw))
    p = torch.from_numpy(pos).cuda()
    w = None if weight is None else torch.from_numpy(weight).cuda()
    try:
        assert lib().pbi4g_debug_fail_alloc(fail) == 0
        est.density(pos.shape[1], p, w)
    finally:
        lib().pbi4g_debug_fail_alloc(0)
    d = est.delta_half()
    est.close()
    return d


def _low(d):
    n = d.shape[0]
    k = np.r_[0 : n // 4 + 1, n - n // 4 : n]
    return d[np.ix_(k, k, np.arange(n // 4 + 1))]


@pytest.mark.parametrize("grid,nintp,interlacing,weights,npart", [
    (32, 4, True, False, 700), (34, 4, True, False, 3001), (34, 1, False, True, 3001), (34, 3, True, True, 2000),
    (46, 2, False, False, 4000), (48, 2, True, True, 1), (50, 4, False, True, 5000), (62, 2, True, False, 9),
    (66, 1, True, False, 6000), (100, 3, False, False, 20000), (126, 4, True, True, 30000), (194, 4, True, False, 40000),
    (202, 3, True, True, 30000), (208, 2, False, False, 40000), (208, 4, True, False, 200000), (64, 1, True, False, 30000),
    (64, 2, True, True, 30000), (64, 3, False, True, 30000), (96, 3, True, False, 9000), (96, 4, False, False, 9000),
    (32, 2, True, False, 400000), (32, 4, True, True, 150000), (50, 4, True, False, 200000), (98, 3, False, True, 400000),
    (66, 1, True, True, 300000), (34, 2, True, False, 200000), (124, 4, True, True, 300000)])
def test_tiles_vs_global_grid(grid, nintp, interlacing, weights, npart):
    pos = _particles(max(npart, 8), grid, grid + nintp)[:, :npart].copy()
    w = np.random.default_rng(grid).uniform(-0.5, 2.0, npart) if weights else None
    kw = dict(grid=grid, nintp=nintp, interlacing=interlacing)
    a, b = _delta(pos, w, **kw), _delta(pos, w, precision="fp64", **kw)
    one = np.zeros((3, 1))
    unit = abs(_delta(one, None, precision="fp64", **kw)[0, 0, 0])  # all particles in phase
    assert np.abs(_low(a) - _low(b)).max() <= TOL * (2 if weights else 1) * unit
    order = np.random.default_rng(1).permutation(npart)
    c = _delta(np.ascontiguousarray(pos[:, order]), None if w is None else w[order].copy(), **kw)
    assert c.tobytes() == a.tobytes()


def test_no_room_for_records():
    pos = _particles(4000, 50, 2)
    kw = dict(grid=50, nintp=4, interlacing=True)
    a, b = _delta(pos, None, **kw), _delta(pos, None, fail=1, **kw)
    assert np.abs(_low(a) - _low(b)).max() <= 2 * TOL * abs(a[0, 0, 0])


@pytest.mark.parametrize("grid,nintp,interlacing", [(34, 4, True), (64, 4, True), (64, 3, False), (66, 2, True), (208, 1, False)])
def test_positions_far_outside(grid, nintp, interlacing):
    pos = _particles(3000, grid, 3)
    far = np.array([77.7, -3.2, 12.0 + 1 / 3, 2.0, 1.0 + 1.5 / grid, 1.0 + 2.5 / grid, 60.0, -0.5 / grid])
    rng = np.random.default_rng(4)
    pos[:, 500:540] = np.where(rng.random((3, 40)) < 0.5, rng.choice(far, (3, 40)), pos[:, 500:540])
    kw = dict(grid=grid, nintp=nintp, interlacing=interlacing)
    a, b = _delta(pos, None, **kw), _delta(pos, None, precision="fp64", **kw)
    # a negative offset (above -1) takes the weights to 4/3 at most
    assert np.abs(_low(a) - _low(b)).max() <= 4 * TOL * np.abs(_low(b)).max()
