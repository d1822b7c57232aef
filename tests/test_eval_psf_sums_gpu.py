"""EVAL's piston and the PSF's transforms against plain arithmetic, without the reference build: the
weighted mean of a tuple's OPD over its valid points is zero (the piston kernel sums 32 points at a
time), and PSF and MTF of asymmetric maps with holes equal numpy's transforms (padding 2, where the
first pass skips one stage, padding 4 and more, where it skips two, and MTF cuts that differ)."""

import numpy as np
import pytest
import torch

from mikroptim_b200 import _capi, engine, psf, workloads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("grid,half", [(1, False), (2, False), (6, False), (7, True), (8, False),
                                       (33, False), (33, True), (64, False)])
def test_the_piston_leaves_no_weighted_mean(grid, half):
    """|sum w OPD| / sum w is at most the rounding of two sums of n terms, (n + 3) 2^-53 of the
    path (below 500 mm here); leaving a point out would move it by OPD / n."""
    b, st, _, _ = workloads.objective(3, rings=3, spokes=6)
    got = engine.TraceEngine(0).evaluate(b, engine.EvalSettings(grid=grid, half_pupil=half))
    n = got.samples
    w = got.grid[:, 2]
    opd, ok = got.opd.reshape(-1, n), got.status.reshape(-1, n) == 0
    assert np.array_equal(np.isfinite(opd), ok & ok.any(axis=1, keepdims=True))
    if grid >= 33:
        assert (~ok).any() and n % 32 != 0
    for t in range(opd.shape[0]):
        if ok[t].any():
            mean = np.sum((w * opd[t])[ok[t]].astype(np.longdouble)) / np.sum(w[ok[t]])
            assert abs(mean) <= 2 * (n + 3) * 2.0 ** -53 * 500.0, t


def test_a_tuple_without_a_valid_ray_has_no_opd():
    b, st, _, _ = workloads.singlet(3)
    b.pupil_radius[1] = 100.0  # every point of the grid misses the first sphere
    got = engine.TraceEngine(0).evaluate(b, engine.EvalSettings(grid=2))
    opd, st = (a.reshape(3, -1) for a in (got.opd, got.status))
    assert np.isnan(opd[1]).all() and (st[1] != 0).all()
    assert np.isfinite(opd[[0, 2]]).all()


def _transforms(opd, lam, M, sign_x, sign_y, scale):
    N = opd.shape[0]
    field = np.zeros((M, M), dtype=complex)
    field[:N, :N] = np.where(np.isnan(opd), 0.0, np.exp(2j * np.pi * np.nan_to_num(opd) / lam))
    I = np.abs(np.fft.fft2(field)) ** 2 * scale
    o = np.arange(M)
    centred = np.empty_like(I)
    centred[np.ix_((M // 2 + sign_y * o) % M, (M // 2 + sign_x * o) % M)] = I
    otf = np.abs(np.fft.fft2(I)) / I.sum()
    k = np.arange(N + 1) % M
    return centred, np.stack([otf[0, k], otf[k, 0]])


@pytest.mark.parametrize("N,M", [(1, 2), (1, 4), (2, 4), (3, 8), (5, 16), (8, 16), (16, 64),
                                 (33, 128), (64, 128), (64, 256), (37, 256), (100, 512),
                                 (300, 2048)])
def test_psf_and_mtf_equal_plain_transforms(N, M):
    """Within 1e-13 of the unaberrated peak, the bar between two correct transforms."""
    rng = np.random.default_rng(N * M)
    y, x = np.mgrid[0:N, 0:N] / N - 0.4
    maps = np.stack([3e-4 * (x * x + 2 * y * y) + 4e-4 * y ** 3 * s + 5e-5 *
                     rng.standard_normal((N, N)) for s in (1.0, -2.0, 0.5)])
    if N > 2:
        maps[:, rng.integers(0, N, 3), rng.integers(0, N, 3)] = np.nan
        maps[1, :, : N // 3] = np.nan  # a lopsided pupil
    scale = 1.0 / (N * N) ** 2
    signs = [(1, 1), (-1, 1), (1, -1)]
    lam = [4.8e-4, 5.5e-4, 6.5e-4]
    params = [_capi.PsfPupilParams(lam[t], scale, *signs[t]) for t in range(3)]
    got, mtf = psf.psf_device(torch.from_numpy(maps).cuda(), params, N, M)
    for t in range(3):
        want, cuts = _transforms(maps[t], lam[t], M, *signs[t], scale)
        assert np.abs(got[t].cpu().numpy() - want).max() <= 1e-13
        assert np.abs(mtf[t].cpu().numpy() - cuts).max() <= 1e-13
        if N > 2:
            assert np.abs(cuts[0] - cuts[1]).max() > 1e-3
