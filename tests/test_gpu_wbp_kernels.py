"""GPU: the WBP back-projection onto the 2x grid and the shared-memory FFTs at the
sizes where they can go wrong, against the FP64 oracle.

Tolerance: an FFT of n points in FP32 has a relative error of about
log2(n) * 2^-24 and a voxel's mean over T tilts sqrt(T) * 2^-24, so 1e-6 to
2e-6; a prime factor above 13 adds two transforms of twice the length.  1e-5."""
import numpy as np
import pytest

from oracle_lib import rel_l2, wbp

pytestmark = pytest.mark.gpu

TOL = 1e-5


def _series(nx, ny, tilts, vol_z, seed):
    from aretomo3_b200 import synth
    ph = synth.Phantom(seed=seed, n_ellipsoids=30, axis_min=3, axis_max=14, n_beads=3, bead_radius=2)
    return synth.make_tilt_series(nx, ny, tilts, vol_z, ph)


def _run(frames, tilts, vol_z, **kw):
    from aretomo3_b200 import recon
    T, ny, nx = frames.shape
    plan = recon.Plan(nx, ny, tilts, vol_z, method=recon.WBP, **kw)
    try:
        vol = np.empty(plan.volume_shape, np.float32)
        plan.run_host([frames[t] for t in range(T)], [vol[y] for y in range(ny)])
        return vol, 1 if plan.c2r == recon.C2R_PACKED else 0
    finally:
        plan.close()


# widths and thicknesses whose transforms take every radix of the planner as first, middle and
# last stage (2 to 16, 7, 11, 13), single-stage lengths, and lengths with larger prime factors
@pytest.mark.parametrize("nx,nz", [(4, 2), (6, 3), (8, 5), (10, 9), (16, 8), (18, 15), (24, 12), (30, 45), (32, 16),
                                   (36, 25), (60, 81), (90, 54), (98, 77), (104, 143), (150, 100), (256, 135),
                                   (480, 240), (512, 75), (720, 162), (1024, 64), (34, 17), (158, 79), (718, 187),
                                   (2046, 31)])
def test_transform_lengths_vs_oracle(nx, nz):
    tilts = np.linspace(-60, 60, 9).astype(np.float32)
    f = _series(nx, 2, tilts, nz, seed=nx + nz)
    vol, mode = _run(f, tilts, nz)
    assert rel_l2(vol, wbp(f, tilts, nz, c2r_mode=mode)) < TOL


# tiles of 32 voxels and blocks of 2 x 2 with remainders; tilts whose windows leave the detector; more
# tilts than a chunk of 16 and a part-filled last chunk; 1 to 9 slices (groups of 4 and 8)
@pytest.mark.parametrize("nx,ny,nz,T,lim", [(64, 1, 16, 16, 60), (66, 4, 17, 17, 70), (34, 5, 48, 33, 80),
                                            (130, 8, 33, 41, 60), (100, 9, 31, 3, 50), (258, 3, 95, 21, 88)])
def test_back_projection_sizes_vs_oracle(nx, ny, nz, T, lim):
    tilts = np.linspace(-lim, lim, T).astype(np.float32)
    f = _series(nx, ny, tilts, nz, seed=nx + T)
    vol, mode = _run(f, tilts, nz)
    assert rel_l2(vol, wbp(f, tilts, nz, c2r_mode=mode)) < TOL


@pytest.mark.parametrize("storage", [0, 1, 2])
def test_slab_size_does_not_change_a_result(storage):
    tilts = np.linspace(-60, 60, 19).astype(np.float32)
    f = _series(96, 21, tilts, 40, seed=3)
    ref, _ = _run(f, tilts, 40, storage=storage)
    for slab in (1, 3, 4, 5, 8, 11):
        vol, _ = _run(f, tilts, 40, storage=storage, slab_slices=slab)
        assert np.array_equal(vol, ref), slab


@pytest.mark.parametrize("bad", [np.nan, np.inf, 1e36])
def test_an_unusual_row_leaves_the_others_alone(bad):
    tilts = np.linspace(-60, 60, 19).astype(np.float32)
    f = _series(96, 9, tilts, 40, seed=4)
    ref, _ = _run(f, tilts, 40)
    f[2, 5, 30] = bad
    vol, _ = _run(f, tilts, 40)
    same = [y for y in range(9) if y != 5]
    assert np.array_equal(vol[same], ref[same])
    assert not np.array_equal(vol[5], ref[5], equal_nan=True)


def _unusual(bad, ny):
    tilts = np.linspace(-60, 60, 19).astype(np.float32)
    f = _series(96, ny, tilts, 40, seed=4)
    f[2, ny - 1, 30] = bad
    f[7, ny - 1, 90] = bad
    return f, tilts


@pytest.mark.parametrize("ny", [3, 9])
@pytest.mark.parametrize("storage", [0, 1, 2])
@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
def test_a_pixel_that_is_not_finite_leaves_no_value_of_its_row(bad, storage, ny):
    """The R-weighting spreads it over its tilt's row and the crop over the slice: NaN, not a
    reconstruction without that tilt (a stored NaN is the 16-bit types' code of a missing value,
    but no value here is one)."""
    f, tilts = _unusual(bad, ny)
    vol, _ = _run(f, tilts, 40, storage=storage)
    assert np.isnan(vol[ny - 1]).all()
    assert np.isfinite(vol[:ny - 1]).all()


@pytest.mark.parametrize("ny", [3, 9])
@pytest.mark.parametrize("bad", [4e12, -4e12])
def test_an_unusual_row_equals_the_oracle(bad, ny):
    """The oracle's means of the samples above -1e10.  The filter makes samples of some 1e11 of the
    pixel, so that FP32 errors of 1e4 leave no sample on the other side of the test but one
    within 1e-6 of it: a voxel of the 2x grid, 1e-4 of the scale."""
    f, tilts = _unusual(bad, ny)
    vol, mode = _run(f, tilts, 40)
    y = ny - 1
    assert rel_l2(vol[y], wbp(f, tilts, 40, y0=y, y1=y + 1, c2r_mode=mode)[0]) < 1e-4
