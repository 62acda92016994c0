"""GPU: the SART kernels that stage volume rows, sinogram windows and voxel tiles by bulk
asynchronous copies (FP32 series whose rows fill groups of 16, 32 or 64 slices) against
the kernels that stage with loads (series of a few rows), on the same rows: windows that
reach past the detector edge, widths that are no multiple of 4, tilts about the steepest whose window
of a volume row fits the ring of copies (80 columns, about 77 degrees).

Both sum the same samples in FP32, in another order; a value is a few thousand
multiply-adds, sqrt(n) * 2^-24 ~ 4e-6 of the volume's scale: 2e-5 leaves room for
the iterations."""
import numpy as np
import pytest

from oracle_lib import rel_l2, sart

pytestmark = pytest.mark.gpu

TOL = 2e-5


def _series(nx, ny, tilts, vol_z, seed):
    from aretomo3_b200 import synth
    ph = synth.Phantom(seed=seed, n_ellipsoids=40, axis_min=3, axis_max=16, n_beads=4, bead_radius=3)
    return synth.make_tilt_series(nx, ny, tilts, vol_z, ph)


def _run(frames, tilts, vol_z, **kw):
    from aretomo3_b200 import recon
    T, ny, nx = frames.shape
    plan = recon.Plan(nx, ny, tilts, vol_z, method=recon.SART, **kw)
    try:
        vol = np.empty(plan.volume_shape, np.float32)
        plan.run_host([frames[t] for t in range(T)], [vol[y] for y in range(ny)])
        return vol, plan.flags_seen()
    finally:
        plan.close()


@pytest.mark.parametrize("nx,ny,lim", [(256, 32, 60), (512, 64, 72), (258, 50, 60), (131, 32, 81)])
def test_bulk_staging_equals_load_path(nx, ny, lim):
    tilts = np.linspace(-lim, lim, 37).astype(np.float32)
    f = _series(nx, ny, tilts, 64, seed=nx + lim)
    vol, seen = _run(f, tilts, 64, iterations=3, subsets=4)
    assert not seen & 16, "a wait for a bulk copy ran out"
    for y0 in (0, ny - 6):
        ref, _ = _run(np.ascontiguousarray(f[:, y0:y0 + 6]), tilts, 64, iterations=3, subsets=4)
        assert not np.array_equal(vol[y0:y0 + 6], ref), "both series ran the same kernels"
        assert rel_l2(vol[y0:y0 + 6], ref) < TOL


def test_tilts_about_the_ring_limit():
    """Tilts of 75 to 81 degrees and their mirror images, against the oracle: some walk the ring of
    copied rows, the others the volume sample by sample."""
    tilts = np.concatenate([np.linspace(-81, -75, 13), [0.0], np.linspace(75, 81, 13)]).astype(np.float32)
    f = _series(200, 32, tilts, 40, seed=7)
    vol, seen = _run(f, tilts, 40, iterations=2, subsets=3)
    assert not seen & 16
    assert rel_l2(vol, sart(f, tilts, 40, 0, tilts.size, 2, 3)) < TOL
