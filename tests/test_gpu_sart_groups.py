"""GPU: the SART kernels that put a slice group (16, 32 or 64 rows) on the lanes
(FP32 series whose rows fill the groups), at the sizes where they can go wrong,
against the FP64 oracle.

Tolerance: a value is a few thousand FP32 multiply-adds, so its relative error
is about sqrt(n) * 2^-24 ~ 4e-6 of the volume's scale; 2e-5 leaves the
few iterations' worth of room."""
import ctypes

import numpy as np
import pytest

from oracle_lib import rel_l2, sart

pytestmark = pytest.mark.gpu

TOL = 2e-5


def _series(nx, ny, tilts, vol_z, seed):
    from aretomo3_b200 import synth
    ph = synth.Phantom(seed=seed, n_ellipsoids=30, axis_min=3, axis_max=14, n_beads=3, bead_radius=2,
                       noise_kind=synth.NOISE_POISSON, noise_param=50.0)
    return synth.make_tilt_series(nx, ny, tilts, vol_z, ph)


def _run(frames, tilts, vol_z, **kw):
    from aretomo3_b200 import recon
    T, ny, nx = frames.shape
    plan = recon.Plan(nx, ny, tilts, vol_z, method=recon.SART, fill_seed=3, **kw)
    try:
        vol = np.empty(plan.volume_shape, np.float32)
        plan.run_host([frames[t] for t in range(T)], [vol[y] for y in range(ny)])
        return vol, plan.flags_seen()
    finally:
        plan.close()


# rows that fill and part-fill the groups, and rows that do not use them; widths that fill no
# ray block or voxel tile, down to the narrowest; odd thicknesses; tilts from flat to beyond the
# blocked windows (80+ degrees)
@pytest.mark.parametrize("nx,ny,nz,lim", [(64, 8, 24, 60), (65, 32, 31, 60), (34, 27, 17, 50), (130, 50, 40, 66),
                                          (48, 33, 2, 60), (4, 64, 9, 45), (6, 30, 5, 60), (97, 91, 50, 60),
                                          (250, 30, 75, 85), (40, 50, 200, 75)])
def test_sizes_vs_oracle(nx, ny, nz, lim):
    tilts = np.linspace(-lim, lim, 23).astype(np.float32)
    f = _series(nx, ny, tilts, nz, seed=nx + ny)
    vol, seen = _run(f, tilts, nz, iterations=3, subsets=4)
    assert not seen & 16, "a bulk copy did not arrive"
    assert rel_l2(vol, sart(f, tilts, nz, 0, tilts.size, 3, 4)) < TOL


# the narrowest widths at the least thickness that series of any size take the slice groups at (32), and
# thinner volumes, down to two rows, with enough rays (4 M in a subset) to take them
@pytest.mark.parametrize("nx,ny,nz,lim,subsets", [(4, 64, 33, 45, 4), (6, 30, 41, 60, 4), (34, 30, 35, 66, 5),
                                                  (65, 32, 32, 60, 4), (1024, 64, 2, 60, 1), (1024, 64, 4, 60, 1),
                                                  (1025, 64, 9, 70, 1)])
def test_narrow_and_thin_vs_oracle(nx, ny, nz, lim, subsets):
    tilts = np.linspace(-lim, lim, 65).astype(np.float32)
    f = _series(nx, ny, tilts, nz, seed=nx + nz)
    vol, seen = _run(f, tilts, nz, iterations=2, subsets=subsets)
    assert not seen & 16
    assert rel_l2(vol, sart(f, tilts, nz, 0, tilts.size, 2, subsets)) < TOL
    few, _ = _run(np.ascontiguousarray(f[:, :4]), tilts, nz, iterations=2, subsets=subsets)
    # (of two rows no ray has a sample: the volume stays what the first back-projection makes it)
    assert nz == 2 or not np.array_equal(vol[:4], few), "the four-slice kernels ran"


@pytest.mark.parametrize("storage", [0, 1, 2])
def test_slab_size_does_not_change_a_result(storage):
    """Groups of 16, 32 and 64 rows, whole and part-filled, give the same bits."""
    tilts = np.linspace(-60, 60, 21).astype(np.float32)
    f = _series(140, 64, tilts, 37, seed=5)
    ref, _ = _run(f, tilts, 37, iterations=2, subsets=3, storage=storage)
    for slab in (1, 5, 16, 20, 40, 63):
        vol, _ = _run(f, tilts, 37, iterations=2, subsets=3, storage=storage, slab_slices=slab)
        assert np.array_equal(vol, ref), slab


@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf, 1e35, -1e30, -3e9])
def test_an_unusual_row_leaves_the_others_alone(bad):
    """Rows with NaN, infinite, huge, missing or near-missing pixels take the
    per-sample paths; the other rows of their group keep their bits."""
    tilts = np.linspace(-60, 60, 21).astype(np.float32)
    f = _series(96, 30, tilts, 32, seed=11)
    ref, _ = _run(f, tilts, 32, iterations=2, subsets=4)
    g = f.copy()
    g[3, 5, 40:44] = bad
    g[10, 13, 7] = bad
    vol, _ = _run(g, tilts, 32, iterations=2, subsets=4)
    same = [y for y in range(30) if y not in (5, 13)]
    assert np.array_equal(vol[same], ref[same])
    assert not np.array_equal(vol[5], ref[5])
    if bad in (-1e30, -3e9):
        assert rel_l2(vol, sart(g, tilts, 32, 0, 21, 2, 4)) < 1e-4


def _same_values(vol, ref, tol):
    """NaN and infinities at the same voxels, the finite values within tol (relative L2)."""
    assert np.array_equal(np.isnan(vol), np.isnan(ref))
    assert np.array_equal(np.where(np.isinf(vol), np.sign(vol), 0), np.where(np.isinf(ref), np.sign(ref), 0))
    ok = np.isfinite(ref)
    assert rel_l2(vol[ok], ref[ok]) < tol


@pytest.mark.parametrize("ny", [30, 64])
@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf, 1e35, -1e30, -3e9])
def test_an_unusual_row_equals_the_four_slice_kernels(bad, ny):
    """A series of four rows takes other kernels, which sum a row with an infinite
    or NaN pixel as any other.  Both sum in FP32, in another order: 2e-5 as above; the
    fill takes the same voxels, so a voxel it fills agrees as its source does."""
    tilts = np.linspace(-60, 60, 21).astype(np.float32)
    f = _series(96, ny, tilts, 32, seed=11)
    f[3, 5, 40:44] = bad
    f[10, 13, 7] = bad
    vol, seen = _run(f, tilts, 32, iterations=2, subsets=4)
    for y0, y in ((4, 5), (12, 13)):
        ref, rseen = _run(np.ascontiguousarray(f[:, y0:y0 + 4]), tilts, 32, iterations=2, subsets=4)
        _same_values(vol[y], ref[y - y0], TOL)
        assert rseen & ~seen == 0, "a condition of the row was not seen"


@pytest.mark.parametrize("ny,nz", [(30, 40), (64, 90)])
def test_a_wait_that_runs_out_is_an_error(ny, nz):
    """With a limit of no polls every wait for a bulk copy gives up: the host form returns an
    error and the run is flagged.  With the limit back, the same plan gives the bits it gave
    before (no copy and no count of the failed run is left over)."""
    from aretomo3_b200 import recon
    tilts = np.linspace(-60, 60, 21).astype(np.float32)
    f = _series(140, ny, tilts, nz, seed=8)
    plan = recon.Plan(140, ny, tilts, nz, method=recon.SART, fill_seed=3, iterations=2, subsets=3)
    set_polls = recon.lib().at3r_plan_set_wait_polls
    set_polls.argtypes, set_polls.restype = [ctypes.c_void_p, ctypes.c_int], None
    try:
        def run():
            vol = np.empty(plan.volume_shape, np.float32)
            plan.run_host([f[t] for t in range(tilts.size)], [vol[y] for y in range(ny)])
            return vol
        ref = run()
        set_polls(plan._h, 0)
        with pytest.raises(recon.ReconError, match="bulk copy"):
            run()
        assert plan.flags_seen() & 16
        set_polls(plan._h, 1 << 22)
        assert np.array_equal(run(), ref)
        assert not plan.flags_seen() & 16
    finally:
        plan.close()


@pytest.mark.parametrize("nx,nz,T", [(8, 65535, 5), (8, 65537, 5), (4, 32, 65535), (4, 32, 65600)])
def test_sizes_around_the_grid_limits(nx, nz, T):
    """Thickness and tilt count at the largest y extent of a grid and past it, against the FP64
    oracle.  A serial FP32 sum of n nearly equal terms (the samples of a ray, the tilts
    of a voxel) can round the same way throughout: n * 2^-25 of itself."""
    tilts = np.linspace(-50, 50, T).astype(np.float32)
    f = np.random.default_rng(T).normal(50, 5, (T, 32, nx)).astype(np.float32)
    vol, seen = _run(f, tilts, nz, iterations=1, subsets=3)
    assert not seen & 16
    ref = sart(np.ascontiguousarray(f[:, 4:6]), tilts, nz, 0, T, 1, 3, threads=1)
    assert rel_l2(vol[4:6], ref) < max(nz, T) * 2.0 ** -25


# walks in one piece and in segments; tilts past the blocked windows; rows with NaN
@pytest.mark.parametrize("nx,ny,nz,lim,bad", [(140, 64, 37, 60, None), (250, 30, 75, 85, None), (97, 91, 200, 78, None),
                                              (140, 30, 130, 60, np.nan), (64, 32, 50, 60, np.inf)])
def test_slabs_of_a_few_slices_give_the_same_bits(nx, ny, nz, lim, bad):
    """Groups of 4 and 8 slices, which only slabs take, and their workspace."""
    from aretomo3_b200 import recon
    tilts = np.linspace(-lim, lim, 21).astype(np.float32)
    f = _series(nx, ny, tilts, nz, seed=6)
    if bad is not None:
        f[3, 5, 30:33] = bad
    ref, _ = _run(f, tilts, nz, iterations=2, subsets=3)
    for slab in (1, 3, 4, 6, 8, 9):
        vol, seen = _run(f, tilts, nz, iterations=2, subsets=3, slab_slices=slab)
        assert not seen & 16
        assert np.array_equal(vol, ref, equal_nan=True), slab
    ws = []
    for slab in (4, 16):
        plan = recon.Plan(nx, ny, tilts, nz, method=recon.SART, iterations=2, subsets=3, slab_slices=slab)
        ws.append(plan.workspace_bytes)
        assert plan.workspace_bytes <= recon.estimate_bytes(nx, ny, tilts, nz, method=recon.SART, iterations=2, subsets=3,
                                                            slab_slices=slab)
        plan.close()
    assert ws[0] < 0.3 * ws[1]


@pytest.mark.parametrize("nx,ny,nz,start,num,subsets", [(130, 32, 40, 3, 17, 4), (96, 64, 130, 0, 23, 5), (65, 30, 33, 7, 9, 9),
                                                        (48, 50, 32, 22, 1, 2)])
def test_tilt_range_and_rfactor(nx, ny, nz, start, num, subsets):
    """Subsets of a part of the tilts (all of them in the first back-projection; a subset may be
    empty), and the residual sums of each iteration: N * num * ny terms in FP32 warp sums
    added up in FP64, each with the error of its voxels."""
    from aretomo3_b200 import recon
    tilts = np.linspace(-60, 60, 23).astype(np.float32)
    f = _series(nx, ny, tilts, nz, seed=nx + ny)
    plan = recon.Plan(nx, ny, tilts, nz, method=recon.SART, start_tilt=start, num_tilts=num, iterations=3, subsets=subsets,
                      compute_rfactor=True, fill_seed=3)
    try:
        vol = np.empty(plan.volume_shape, np.float32)
        plan.run_host([f[t] for t in range(tilts.size)], [vol[y] for y in range(ny)])
        rf = plan.rfactor()
        assert not plan.flags_seen() & 16
    finally:
        plan.close()
    ref, rref = sart(f, tilts, nz, start, num, 3, subsets, rfactor=True)
    assert rel_l2(vol, ref) < TOL
    assert np.allclose(rf, rref, rtol=1e-4)


def test_same_bits_captured_served_tuned_and_side_by_side():
    """A graph of several plans replayed twice, the serving loop with slabs and a tail, a tuned
    slab, and two plans on two threads and streams: each as the plan alone."""
    import threading

    import torch
    from aretomo3_b200 import recon
    kw = dict(method=recon.SART, iterations=2, subsets=4, fill_seed=3)
    shapes = [(140, 64, 37, 21), (96, 32, 130, 25), (250, 91, 60, 19)]
    tl = [np.linspace(-60, 60, T).astype(np.float32) for *_, T in shapes]
    fr = [_series(nx, ny, t, nz, seed=nx) for (nx, ny, nz, _), t in zip(shapes, tl)]
    dev = [torch.from_numpy(f).cuda() for f in fr]
    plans = [recon.Plan(nx, ny, t, nz, **kw) for (nx, ny, nz, _), t in zip(shapes, tl)]
    vols = [torch.empty(p.volume_shape, device="cuda") for p in plans]
    ref = []
    for p, f, v in zip(plans, dev, vols):
        p.run_device(f.data_ptr(), v.data_ptr(), 0)
        torch.cuda.synchronize()
        ref.append(v.cpu().numpy())

    def check(what):
        torch.cuda.synchronize()
        for v, r in zip(vols, ref):
            assert np.array_equal(v.cpu().numpy(), r), what
            v.fill_(float("nan"))
        torch.cuda.synchronize()

    check("alone")
    batch = recon.Batch(plans, [f.data_ptr() for f in dev], [v.data_ptr() for v in vols], branches=2)
    for _ in range(2):
        batch.run(torch.cuda.current_stream().cuda_stream)
        check("captured")
    batch.close()

    def many(i, stream):
        for _ in range(4):
            plans[i].run_device(dev[i].data_ptr(), vols[i].data_ptr(), stream.cuda_stream)

    st = [torch.cuda.Stream() for _ in plans]
    th = [threading.Thread(target=many, args=(i, st[i])) for i in range(len(plans))]
    for t in th:
        t.start()
    for t in th:
        t.join()
    check("side by side")
    plans[2].autotune(dev[2].data_ptr(), vols[2].data_ptr(), 0)
    for p, f, v in zip(plans, dev, vols):
        p.run_device(f.data_ptr(), v.data_ptr(), 0)
    check("tuned")
    srv = recon.Server(max_inflight=3)
    try:
        ids = [srv.submit(f, t, nz, slab_slices=s, **kw)
               for f, t, (_, _, nz, _), s in list(zip(fr, tl, shapes, (0, 0, 0))) + list(zip(fr, tl, shapes, (20, 5, 33)))]
        for rid, r in zip(ids, ref + ref):
            assert np.array_equal(srv.wait(rid)[0], r), "served"
    finally:
        srv.close()
    assert not any(p.flags_seen() & 16 for p in plans)
    for p in plans:
        p.close()
