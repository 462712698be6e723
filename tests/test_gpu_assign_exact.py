"""The tiled assignment's sums are integers: the same in every form that its kernels take, so
densities are compared byte for byte.

Grids that are not a multiple of 16 round their contributions as the 64-bit grid in global
memory does, which a box takes when its records find no room.  On the others, a particle whose
weight is negative sends its tile to the second pass (tiles of up to 65535 records) or to the
64-bit sums (more), and a weight of -1e-30 rounds to the same nothing as 1e-30."""
import numpy as np
import pytest

from pbi4_gb300._lib import lib
from pbi4_gb300.estimator import Estimator, EstimatorConfig

pytestmark = pytest.mark.gpu


def _delta(pos, weight, fail=0, **kw):
    import torch
    est = Estimator(EstimatorConfig(box=1000.0, do_bispectrum=False, **kw))
    p = torch.from_numpy(pos).cuda()
    w = None if weight is None else torch.from_numpy(weight).cuda()
    try:
        assert lib().pbi4g_debug_fail_alloc(fail) == 0
        est.density(pos.shape[1], p, w)
    finally:
        lib().pbi4g_debug_fail_alloc(0)
    d = est.delta_half()
    est.close()
    return d.tobytes()


def _positions(n, grid, seed):
    """Uniform, an eighth on cell edges or halves, a quarter crowded into one cell, a few outside."""
    rng = np.random.default_rng(seed)
    pos = rng.random((3, n))
    pos[:, : n // 8] = rng.integers(0, 2 * grid + 1, (3, n // 8)) / (2 * grid)
    pos[:, n // 8 : 3 * n // 8] = (grid // 3 + rng.random((3, 3 * n // 8 - n // 8))) / grid
    if n >= 100:
        pos[:, -6:] = rng.choice([-0.3, -1e-3, 1.0, 1.0 + 1e-3, 2.7], (3, 6))
    return np.ascontiguousarray(pos[:, rng.permutation(n)])


@pytest.mark.parametrize("grid,npart", [(34, 1), (50, 4000), (34, 60000), (66, 300000), (100, 20000), (202, 30000)])
@pytest.mark.parametrize("nintp,interlacing", [(1, False), (1, True), (2, False), (2, True), (3, False), (3, True),
                                               (4, False), (4, True)])
@pytest.mark.parametrize("weights", ["none", "positive", "both signs", "wide"])
def test_grids_not_a_multiple_of_16(grid, npart, nintp, interlacing, weights):
    rng = np.random.default_rng(npart)
    pos = _positions(npart, grid, grid + nintp)
    w = {"none": None, "positive": rng.uniform(0.1, 2.0, npart), "both signs": rng.uniform(-1.0, 2.0, npart),
         "wide": 10.0 ** rng.uniform(-6.0, 6.0, npart)}[weights]
    kw = dict(grid=grid, nintp=nintp, interlacing=interlacing)
    assert _delta(pos, w, **kw) == _delta(pos, w, fail=1, **kw)


@pytest.mark.parametrize("grid,npart", [(32, 60), (32, 300), (64, 3000), (48, 20000), (32, 64000), (32, 200000),
                                        (64, 1000000), (32, 900000), (208, 50000)])
@pytest.mark.parametrize("nintp,interlacing", [(1, False), (1, True), (2, True), (3, False), (3, True), (4, False),
                                               (4, True)])
@pytest.mark.parametrize("crowded", [False, True])
def test_second_pass_gives_the_same_sums(grid, npart, nintp, interlacing, crowded):
    pos = _positions(npart, grid, grid + nintp) if crowded else np.random.default_rng(grid).random((3, npart))
    w = np.random.default_rng(npart).uniform(0.2, 1.0, npart)
    mark = np.random.default_rng(7).random(npart) < 0.05
    w[mark] = 1e-30
    neg = np.where(mark, -w, w)
    kw = dict(grid=grid, nintp=nintp, interlacing=interlacing)
    assert _delta(pos, w, **kw) == _delta(pos, neg, **kw)
