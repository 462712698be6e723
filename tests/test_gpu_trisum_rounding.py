"""Rounding of the plain FP32 triangle sums (csrc/trisum_simt.cu) beyond the sums of 64 points.

A thread adds its products of 64 points (a chunk) in FP32, two chains of 32, and then the
chunks' sums.  Maps streamed in slabs of one z-plane give each thread a single chunk a launch,
and the launches' sums are added in FP64: the same maps and the same chunks without the
additions between chunks, so the difference to the unstreamed sums is their rounding.

On smooth fields the products of neighbouring points have one sign and the chunks' sums add
up coherently.  The additions between the chunks may not round by more than one FP32 chain of
64 coherent points does (which is what chunks under a compensated sum leave): the j-th partial
sum of a chain of equal products p is rounded by 0.42 2^-24 j p rms (uniform within half an
ulp, over the binade), so a chain is off by 0.42 2^-24 p sqrt(sum j^2), and independent chains
of 64 points by TOL of the root of the summed squared products.  Each sum's own error is one
random draw: the rms over fields and multipoles is compared."""
import numpy as np
import pytest

from pbi4_gb300.estimator import Estimator, EstimatorConfig

pytestmark = pytest.mark.gpu

TOL = 0.42 * 2.0 ** -24 * np.sqrt(np.sum(np.arange(1, 65) ** 2.0)) / 8


LOW = np.r_[0:12, -12:0]  # the frequencies held: the first shell's


def _modes(seed, noise):
    """Modes 4 <= |k| < 12 (z, y, x frequencies LOW, LOW, 0..11) of a real field: waves along z of
    variance 1, and random modes of variance `noise`, which spread the products' low bits."""
    r = np.random.default_rng(seed)
    kz, ky, kx = np.meshgrid(LOW, LOW, np.arange(12), indexing="ij")
    k2 = kx ** 2 + ky ** 2 + kz ** 2
    a = np.where((k2 >= 16) & (k2 < 144), r.standard_normal(k2.shape) + 1j * r.standard_normal(k2.shape), 0)
    neg = -np.arange(24) % 24
    a[:, :, 0] = 0.5 * (a[:, :, 0] + np.conj(a[np.ix_(neg, neg)][:, :, 0]))
    a *= np.sqrt(noise / (2 * np.sum(np.abs(a) ** 2) - np.sum(np.abs(a[:, :, 0]) ** 2)))
    w = r.uniform(0.5, 1.5, 8) * np.exp(2j * np.pi * r.random(8))
    w /= np.sqrt(2 * np.sum(np.abs(w) ** 2))
    a[4:12, 0, 0] += w
    a[-4:-12:-1, 0, 0] += w.conj()
    return a


def _spectrum(a, n):
    h = np.zeros((n, n, n // 2 + 1), complex)
    h[np.ix_(LOW, LOW, np.arange(12))] = a
    return h


def _squared_products(a, fac, nm):
    """Root of the summed squared products M M M_fac of the maps on the grid nm."""
    kz, ky, kx = np.meshgrid(LOW, LOW, np.arange(12), indexing="ij")
    mu2 = kz ** 2 / np.maximum(kx ** 2 + ky ** 2 + kz ** 2, 1)
    leg = {0: 1.0, 2: -0.5 + 1.5 * mu2, 4: 0.375 + mu2 * (-3.75 + 4.375 * mu2)}[fac]
    m, q = (np.fft.irfftn(_spectrum(x, nm), (nm,) * 3, axes=(0, 1, 2)) * nm ** 3 for x in (a, a * leg))
    return np.sqrt(np.sum((m * m * q) ** 2))


@pytest.mark.parametrize("multipoles", [True, False])
def test_sums_of_smooth_fields(multipoles):
    grid, nb = 256, 8
    kf = np.float32(2 * np.pi / 1000.0)
    err = []
    ests = [Estimator(EstimatorConfig(grid=grid, box=1000.0, nintp=4, interlacing=True, multipoles=multipoles,
                                      los=(0.0, 0.0, 1.0), kbin_bs=8.0, kcenter_bs=8.0, nbins_bs=nb, iopen=True,
                                      precision="fp32", map_budget_mb=mb)) for mb in (0, 1)]
    nm = ests[0].map_grid
    for seed in range(6):
        a = _modes(seed, 0.05)
        out = []
        for est in ests:
            est.set_delta_half(10 ** 18, _spectrum(a, grid))  # (no shot noise beside B)
            bout = est.alloc_outputs()[1]
            est.bispectrum(bout)
            out.append(bout.cpu().numpy())
        assert ests[0].map_slabs()[1] == 1 and ests[1].map_slabs()[1] == nm  # whole; one plane a slab
        t = np.flatnonzero((out[0][:3] == 8.0).all(axis=0))[0]  # all sides in the first shell
        counts = float(np.float32(ests[0].triangle_counts()[t] * float(grid) ** 3))
        for row, fac in ((6, 0), (9, 2), (10, 4)) if multipoles else ((6, 0),):
            pre = float(kf * kf * kf) * {0: 1, 2: 5, 4: 9}[fac] * (grid / nm) ** 3 / counts
            err.append((out[0][row, t] - out[1][row, t]) / pre / _squared_products(a, fac, nm))
    for est in ests:
        est.close()
    assert np.sqrt(np.mean(np.square(err))) <= TOL, err
