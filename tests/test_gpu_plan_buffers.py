"""What a plan allocates: no tables of a form it does not use."""
import numpy as np
import pytest

from pbi4_gb300._lib import lib
from pbi4_gb300.estimator import Estimator, EstimatorConfig

pytestmark = pytest.mark.gpu


def _allocs():
    return int(lib().pbi4g_device_allocs())


def test_tensor_form_builds_its_own_tables_only():
    """The tensor-core form has units, pairs, slots, an error flag and exponents where the plain
    FP32 form has tiles, slots and groups: two buffers more."""
    made = {}
    for prec in ("fp32", "tf32split"):
        est = Estimator(EstimatorConfig(grid=64, box=1000.0, multipoles=True, kbin_bs=3.0, kcenter_bs=3.0, nbins_bs=6,
                                        precision=prec))
        est.triangle_counts()
        h = np.random.default_rng(1).standard_normal((64, 64, 33, 2)).view(complex)[..., 0]
        est.set_delta_half(1000, h)
        bout = est.alloc_outputs()[1]
        n = _allocs()
        est.bispectrum(bout)
        est.check()
        made[prec] = _allocs() - n
        est.close()
    assert made["tf32split"] == made["fp32"] + 2
