"""CUDA-core triangle sums (csrc/trisum_simt.cu) at the sizes where their tiling can go
wrong: fewer shells than a tile is wide, runs of factor maps cut by the last shell, odd
shell counts, map grids whose point count leaves a ragged last stage (padded FP64 rows
among them), closed and open triangles, and tile lists of several groups and of more warps
than a CTA holds.

The FP64 sums through the drop-ins against the oracle: 1e-9 of the larger of |B| and the
rms of B over the triangles of its l shell (the fields are non-Gaussian, so B0 is no noise
sum); counts and k columns bit-exact.  The FP32 sums through the plan against the FP64
form: the FP32 form's 1e-5 of the larger of |B| and (2l+1)(P1 P2 + P1 P3 + P2 P3) with the
powers as measured, shot noise included: these boxes are nearly Poisson, and what is left
after the noise is subtracted can be far below the FP32 rounding of the density itself."""
import numpy as np
import pytest

from oracle import pbi4_oracle as O
from pbi4_gb300 import bispectrumI4 as B
from pbi4_gb300.estimator import Estimator, EstimatorConfig

pytestmark = pytest.mark.gpu

KF = 2 * np.pi / 1000.0


def _field(n, seed):
    """Full complex spectrum (Fortran order) of a real non-Gaussian field."""
    g = np.random.default_rng(seed).standard_normal((n, n, n))
    k = np.fft.fftfreq(n, 1.0 / n)
    k2 = k[:, None, None] ** 2 + k[None, :, None] ** 2 + k[None, None, :] ** 2
    f = np.fft.ifftn(np.fft.fftn(g) * np.where(k2 > 0, np.maximum(k2, 1.0) ** -0.5, 0.0)).real
    f /= f.std()
    return np.asfortranarray(np.fft.fftn(f + 0.5 * (f * f - 1)))


def _scale(ref, row):
    s = np.zeros(ref.shape[1])
    for kl in np.unique(ref[0]):
        sel = ref[0] == kl
        s[sel] = np.sqrt(np.mean(ref[row][sel] ** 2))
    return np.maximum(np.abs(ref[row]), s)


CASES = [  # grid, nb, kbin, iopen
    (16, 1, 1.0, True), (16, 2, 1.0, False), (16, 3, 1.0, True), (20, 5, 1.0, True), (22, 6, 1.0, False),
    (32, 4, 2.0, True), (34, 7, 1.0, True), (40, 11, 1.0, True), (50, 13, 1.0, False), (50, 16, 1.0, True),
]


@pytest.mark.parametrize("grid,nb,kbin,iopen", CASES)
def test_simt_sums_match_oracle(grid, nb, kbin, iopen, tol=1e-9):
    d = [_field(grid, s) for s in (1, 2, 3)]
    it, itx = O.itot(nb, kbin, kbin, iopen), O.itot(nb, kbin, kbin, iopen, True)
    counts = O.count_triangles(nb, grid, kbin, kbin, iopen, False, 1, it)
    countsx = O.count_triangles(nb, grid, kbin, kbin, iopen, True, 1, itx)
    got_counts = B.count_triangles(nb, grid, kbin, kbin, iopen, False, 1, it)
    np.testing.assert_array_equal(np.round(got_counts / grid ** 3), np.round(counts / grid ** 3))
    B.set_precision("fp64")
    try:
        a = (nb, grid, kbin, kbin, iopen, KF, 1)
        for got, ref, rows in (
                (B.measure_bk(*a, it, 1000, counts, d[0]), O.measure_bk(*a, it, 1000, counts, d[0]), (6,)),
                (B.measure_bk_multipoles(*a, it, 1000, counts, *d), O.measure_bk_multipoles(*a, it, 1000, counts, *d),
                 (6, 9, 10)),
                (B.measure_bk_cross(*a, itx, 1000, countsx, *d[:2]), O.measure_bk_cross(*a, itx, 1000, countsx, *d[:2]),
                 (3,))):
            np.testing.assert_array_equal(got[[0, 1, 2]], ref[[0, 1, 2]])
            for r in rows:
                ok = np.isfinite(ref[r])  # a closed triangle without modes has no B
                err = np.abs(got[r] - ref[r])[ok] / _scale(np.where(np.isfinite(ref), ref, 0.0), r)[ok]
                assert err.max() <= tol, (r, err.max())
    finally:
        B.set_precision("fp32")


@pytest.mark.parametrize("multipoles,nb,grid,iopen", [
    (True, 41, 192, True), (False, 58, 192, True), (True, 1, 32, True), (False, 1, 32, False), (True, 2, 32, True),
    (False, 3, 32, True), (True, 5, 50, False), (True, 7, 34, True), (False, 9, 48, True), (True, 13, 64, True)])
def test_simt_fp32_sums_match_fp64(multipoles, nb, grid, iopen):
    """The FP32 sums against the FP64 ones (tiles of another shape in other groups) on one
    box, whole and in z-slabs; the largest have tile lists of several groups."""
    pos = np.random.default_rng(4).random((3, 20000)) ** np.array([[1.0], [1.3], [0.8]])
    out = {}
    for name, prec, budget in (("fp64", "fp64", 0), ("fp32", "fp32", 0), ("slabs", "fp32", 4 * nb if grid == 192 else 0)):
        cfg = EstimatorConfig(grid=grid, box=1000.0, nintp=3, interlacing=True, multipoles=multipoles, kbin_bs=1.0,
                              kcenter_bs=1.0, nbins_bs=nb, iopen=iopen, precision=prec, map_budget_mb=budget)
        est = Estimator(cfg)
        out[name] = est.run_host(pos)[1]
        if budget:
            assert est.map_slabs()[1] > 1
        est.close()
    ref = out["fp64"]
    P = np.abs(ref[3:6] + 1.0 / pos.shape[1] / KF ** 3)
    den = P[0] * P[1] + P[0] * P[2] + P[1] * P[2]
    for name in ("fp32", "slabs"):
        for row, fac in ((6, 1.0), (9, 5.0), (10, 9.0)) if multipoles else ((6, 1.0),):
            err = np.abs(out[name][row] - ref[row]) / np.maximum(np.abs(ref[row]), fac * den)
            err = err[np.isfinite(err)]
            assert err.max() <= 1e-5, (name, row, err.max())
