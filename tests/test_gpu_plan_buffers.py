"""What a plan allocates: no tables of a form it does not use, no more than its footprint says,
and on grids that are not a multiple of 16, whose assignment can do without its particle
records, no box that fails for the room they take."""
import numpy as np
import pytest

from pbi4_gb300._lib import Pbi4GpuError, lib
from pbi4_gb300.estimator import AssignScratch, Estimator, EstimatorConfig, footprint

pytestmark = pytest.mark.gpu


def _allocs():
    return int(lib().pbi4g_device_allocs())


def _free():
    import torch
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


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


def test_small_scratch_within_its_footprint():
    """Scratches for a few particles: 128 of them, so that the driver's pages (2 MiB) show only
    once.  (A scratch's buffers below 1 MiB share pages.)"""
    AssignScratch(32, 1).close()  # the context and the module
    free = _free()
    made = [AssignScratch(64, 1000) for _ in range(128)]
    held = free - _free()
    want = sum(s.bytes for s in made)
    for s in made:
        s.close()
    assert held <= want + (16 << 20), (held, want)


@pytest.mark.parametrize("grid,npart", [(32, 1), (32, 100), (32, 513), (256, 300), (48, 20000), (208, 20000), (256, 40)])
def test_scratch_serves_every_smaller_box(grid, npart):
    """A scratch of the largest grid and particle number holds the boxes of smaller ones."""
    import torch
    sc = AssignScratch(grid, npart)
    rng = np.random.default_rng(grid)
    for g in sorted({32, grid, max(32, grid // 32 * 16), min(grid, 192)}):
        for n in {1, max(1, npart // 3), npart}:
            est = Estimator(EstimatorConfig(grid=g, box=1000.0, do_bispectrum=False))
            pos = torch.from_numpy(rng.random((3, n))).cuda()
            est.density(n, pos)
            own = est.delta_half()
            est.use_scratch(sc)
            est.density(n, pos)
            assert est.delta_half().tobytes() == own.tobytes()
            est.close()
    sc.close()


@pytest.mark.parametrize("kw", [dict(grid=256, kbin_bs=8.0, kcenter_bs=8.0, nbins_bs=8, multipoles=True),
                                dict(grid=128, kbin_bs=1.0, kcenter_bs=1.0, nbins_bs=41, multipoles=True),
                                dict(grid=160, kbin_bs=1.0, kcenter_bs=1.0, nbins_bs=53, multipoles=False),
                                dict(grid=128, kbin_bs=1.0, kcenter_bs=1.0, nbins_bs=20, multipoles=True, map_budget_mb=16)])
@pytest.mark.parametrize("precision", ["fp32", "fp16split"])
def test_plan_within_its_footprint(kw, precision):
    import torch
    cfg = EstimatorConfig(box=1000.0, precision=precision, **kw)
    n = 20000
    pos = torch.rand((3, n), dtype=torch.float64, device="cuda")
    out = Estimator(cfg).alloc_outputs()
    warm = Estimator(cfg)  # loads the modules, counts the triangles
    warm.run_device(n, pos, *out)
    warm.check()
    warm.close()
    free = _free()
    est = Estimator(cfg)
    est.run_device(n, pos, *out)
    est.check()
    held = free - _free()
    est.close()
    assert held <= footprint(cfg, n), (held, footprint(cfg, n))


GEN = dict(grid=50, box=1000.0, nintp=4, interlacing=True, multipoles=True, kbin_bs=3.0, kcenter_bs=3.0, nbins_bs=4)


def _run(est, pos):
    import torch
    out = est.alloc_outputs()
    est.run_device(pos.shape[1], torch.from_numpy(pos).cuda(), *out)
    est.check()
    return [o.cpu().numpy() for o in out]


@pytest.mark.parametrize("precision", ["fp32", "fp16split"])
def test_records_give_way_to_later_stages(precision):
    """Whatever allocation of a box fails for want of room while the records are held: the
    records are given up and the box goes through, with the same density."""
    cfg = EstimatorConfig(precision=precision, **GEN)
    pos = np.random.default_rng(5).random((3, 5000))
    est = Estimator(cfg)
    est.triangle_counts()  # (counted once a process)
    n = _allocs()
    ref = _run(est, pos)
    n = _allocs() - n
    delta = est.delta_half().tobytes()
    est.close()
    for k in range(1, n + 1):
        est = Estimator(cfg)
        try:
            assert lib().pbi4g_debug_fail_alloc(k) == 0
            got = _run(est, pos)
        finally:
            lib().pbi4g_debug_fail_alloc(0)
        assert est.delta_half().tobytes() == delta, k
        for a, b in zip(got, ref):
            np.testing.assert_allclose(a, b, rtol=1e-5, atol=1e-6 * np.abs(b).max())
        _run(est, pos)
        made = _allocs()
        _run(est, pos)  # no second attempt at the same size
        assert _allocs() == made, k
        est.close()


def test_records_tried_again_for_fewer_particles():
    pos = np.random.default_rng(6).random((3, 6000))
    est = Estimator(EstimatorConfig(precision="fp32", **dict(GEN, multipoles=False)))
    try:
        assert lib().pbi4g_debug_fail_alloc(1) == 0
        _run(est, pos)
    finally:
        lib().pbi4g_debug_fail_alloc(0)
    made = _allocs()
    _run(est, pos)
    assert _allocs() == made
    _run(est, np.ascontiguousarray(pos[:, :3000]))
    assert _allocs() > made  # the records of half as many
    est.close()


def test_counts_without_room_are_counted_again():
    """A box whose triangle counts find no room on the device fails; the next one makes them."""
    import torch
    cfg = EstimatorConfig(grid=64, box=1000.0, kbin_bs=4.0, kcenter_bs=4.0, nbins_bs=4)
    pos = np.random.default_rng(8).random((3, 5000))
    est = Estimator(cfg)
    ref = _run(est, pos)  # (counted once a process)
    est.close()
    est = Estimator(cfg)
    est.density(5000, torch.from_numpy(pos).cuda())
    bout = est.alloc_outputs()[1]
    try:
        assert lib().pbi4g_debug_fail_alloc(1) == 0
        with pytest.raises(Pbi4GpuError):
            est.bispectrum(bout)
    finally:
        lib().pbi4g_debug_fail_alloc(0)
    est.bispectrum(bout)
    np.testing.assert_array_equal(bout.cpu().numpy()[8], ref[1][8])
    est.close()
