"""P(k) sums over pairs of |k| (up to eight rows at once, runs of equal bins combined within a
warp): grids whose rows end anywhere in a warp, with and without rows at N/2, bins next to their
edges, wide and narrow bins, every mode of the kernel, twice in a row (the sums are cleared by
the launch before), against the oracle."""
import numpy as np
import pytest

from oracle import pbi4_oracle as O
from pbi4_gb300 import powerI4 as P
from pbi4_gb300.estimator import Estimator, EstimatorConfig

pytestmark = pytest.mark.gpu

GRIDS = [(4, 1.0, 1.0), (6, 1.0, 1.0), (10, 0.5, 0.5), (30, 1.5, 0.5), (32, 4.0, 4.0), (62, 1.0, 1.0), (64, 2.0, 2.5),
         (66, 1.0, 1.0), (94, 0.25, 1.0), (130, 1.0, 1.0)]


def _fields(grid):
    rng = np.random.default_rng(grid)
    d = np.asfortranarray(rng.standard_normal((grid,) * 3) + 1j * rng.standard_normal((grid,) * 3))
    return d, np.asfortranarray(d * rng.uniform(0, 1, d.shape)), np.asfortranarray(d * rng.uniform(0, 1, d.shape))


@pytest.mark.parametrize("grid,kbin,kcenter", GRIDS)
def test_drop_ins(grid, kbin, kcenter):
    d, d2, d4 = _fields(grid)
    nb = EstimatorConfig(grid=grid, box=1000.0, kbin_ps=kbin, kcenter_ps=kcenter).nbins_ps
    ref = O.measure_pk(grid, 1000.0, kbin, kcenter, nb, d, d2)
    got = P.measure_pk(grid, 1000.0, kbin, kcenter, nb, d, d2)
    np.testing.assert_array_equal(got[2], ref[2])
    # positive terms, fewer than 2^17 a bin, summed in any order
    np.testing.assert_allclose(got[:2], ref[:2], rtol=2e-11)
    ref = O.measure_pk_multipoles(grid, 1000.0, kbin, kcenter, nb, d, d2, d4)
    got = P.measure_pk_multipoles(grid, 1000.0, kbin, kcenter, nb, d, d2, d4)
    np.testing.assert_array_equal(got[4], ref[4])
    np.testing.assert_allclose(got[:4], ref[:4], rtol=2e-11)


@pytest.mark.parametrize("grid,kbin,kcenter", GRIDS)
@pytest.mark.parametrize("precision", ["fp32", "fp64"])
def test_plan(grid, kbin, kcenter, precision):
    import torch
    d = _fields(grid)[0]
    k = np.fft.fftfreq(grid, 1.0 / grid)
    k[grid // 2] = grid // 2
    kx, ky, kz = np.meshgrid(k, k, k, indexing="ij")
    los = (0.48, -0.6, 0.64)
    k2 = kx ** 2 + ky ** 2 + kz ** 2
    mu2 = (los[0] * kx + los[1] * ky + los[2] * kz) ** 2 / np.where(k2 > 0, k2, 1)
    l2, l4 = -0.5 + 1.5 * mu2, 0.375 - 3.75 * mu2 + 4.375 * mu2 ** 2
    for multipoles in (True, False):
        est = Estimator(EstimatorConfig(grid=grid, box=1000.0, kbin_ps=kbin, kcenter_ps=kcenter, los=los,
                                        multipoles=multipoles, precision=precision, do_bispectrum=False))
        est.set_delta_half(1, np.ascontiguousarray(d[: grid // 2 + 1].transpose(2, 1, 0)))
        ref = (O.measure_pk_multipoles(grid, 1000.0, kbin, kcenter, est.nbins_ps, d, d * l2, d * l4) if multipoles
               else O.measure_pk(grid, 1000.0, kbin, kcenter, est.nbins_ps, d, d))
        n = 4 if multipoles else 2
        # relative to P0: at most 64 roundings of a mode's terms and of the sums it goes through
        eps = 2e-11 if precision == "fp64" else 64 * 2.0 ** -24
        for _ in range(2):
            pout = torch.full((est.nbins_ps, 5), float("nan"), dtype=torch.float64, device="cuda")
            est.powerspectrum(pout)
            got = pout.cpu().numpy().T
            np.testing.assert_array_equal(got[n], ref[n])
            np.testing.assert_allclose(got[0], ref[0], rtol=2e-11)
            some = ref[n] > 0  # (a bin without modes is NaN on both sides)
            for row, factor in zip(range(1, n), (1, 5, 9)):
                assert np.max(np.abs(got[row] - ref[row])[some] / ref[1][some]) <= factor * eps
        est.close()
