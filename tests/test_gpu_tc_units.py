"""Unit layouts of the tensor-core triangle sums (TmPlan::build) where they can go wrong:
one and two shells (groups of fewer than four pairs, one warp of pairs), windows of every
width (16 to 64 plane rows), a tile whose rows need two windows (22 shells x 3 sets), pair
covers of one and two tiles for a single set.  Against the oracle, at the tolerance of the
forms (tests/test_gpu_tc.py)."""
import numpy as np
import pytest

from oracle import pbi4_oracle as O
from pbi4_gb300 import synthetic
from pbi4_gb300.estimator import Estimator, EstimatorConfig

from ._helpers import b_errors, oracle_density, ref_params

pytestmark = pytest.mark.gpu

TOL = {"fp16split": 1e-4, "tf32split": 1e-4, "bf16": 5e-2}


@pytest.fixture(scope="module")
def box_za():
    return synthetic.zeldovich_box(24, 1000.0, seed=12)


@pytest.mark.parametrize("nb,iopen,multipoles", [(1, True, True), (2, False, False), (3, True, True), (5, True, False),
                                                 (12, False, True), (17, True, True), (19, True, False),
                                                 (22, True, True), (25, True, False)])
def test_tensor_core_units(box_za, nb, iopen, multipoles):
    grid = 64
    p = ref_params(grid, 1000.0, 4, True, multipoles, iopen=iopen)
    p["nbins_bisp"] = nb
    npart, d, d2, d4 = oracle_density(box_za, p)
    it = O.itot(nb, 1.0, 1.0, iopen)
    counts = O.count_triangles(nb, grid, 1.0, 1.0, iopen, False, 1, it)
    a = (nb, grid, 1.0, 1.0, iopen, 2 * np.pi / 1000.0, 1, it, npart, counts)
    ref = O.measure_bk_multipoles(*a, d, d2, d4) if multipoles else O.measure_bk(*a, d)
    for precision, tol in TOL.items():
        if precision == "bf16" and nb <= 3:
            continue  # B4 of ten cancelling triangles: the 8-bit mantissas of the maps alone are 6% off
        est = Estimator(EstimatorConfig.from_params(p, precision=precision))
        bout = est.run_host(box_za)[1]
        est.close()
        np.testing.assert_array_equal(bout[[0, 1, 2, 8]], ref[[0, 1, 2, 8]])
        errs, pw = b_errors(bout, ref)
        assert max(errs) < tol and pw < 1e-5, (precision, errs, pw)
