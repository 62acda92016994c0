"""The performance cases of this package: what its users have it do, through
its public entry points, over the range of sizes it is used at.

Kinds of case (``kind``):

* ``recon``  a device-resident tilt series reconstructed by a plan the program
             keeps (``recon.Plan.run_device``), WBP or SART, in FP32, FP16 or
             BF16 storage;
* ``doit``   the reference-shaped call on host frames (``CDoWbpRecon.DoIt`` /
             ``CDoSartRecon.DoIt``): plan set-up, copies, reconstruction and
             volume back in host memory;
* ``stack``  the input stage on device frames (``recon.Stack.run_device``):
             shift, rotation, random fill and Fourier-crop binning;
* ``bin``    the same entry point without the alignment: Fourier-crop binning.

Tilt series are seeded phantoms (spheres in ice, projected analytically) at an
electron-counting camera's level with counting noise.
"""
import math

import numpy as np
import torch

from aretomo3_b200 import recon

STORAGE = {"f32": recon.STORE_F32, "f16": recon.STORE_F16, "bf16": recon.STORE_BF16}


def _recon(name, method, nx, ny, tilts, vol_z, storage="f32", kind="recon", step=3.0, iterations=0, subsets=1,
           relax=0.0, skip=0):
    """skip: tilts left out of SART's subsets at either end of the series."""
    c = dict(kind=kind, method=method, nx=nx, ny=ny, tilts=tilts, step=step, vol_z=vol_z, storage=storage,
             iterations=iterations, subsets=subsets, relax=relax, skip=skip)
    if name:
        c["name"] = name
    return c


def _stack(name, kind, nx, ny, tilts, bin, axis):
    c = dict(kind=kind, nx=nx, ny=ny, tilts=tilts, bin=bin, axis=axis)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # a heavily binned preview while the series is still being collected:
        # launches and latency
        _recon("wbp_preview_128", "wbp", 128, 128, 41, 48),
        # the standard small WBP series (512 x 512 x 41, thickness 128)
        _recon("wbp_512", "wbp", 512, 512, 41, 128),
        # a cropped series whose sizes fit nothing: odd width, lengths with
        # large prime factors, uneven step
        _recon("wbp_ragged", "wbp", 719, 501, 37, 187, step=3.3),
        # an ordinary binned tomogram in FP16 storage
        _recon("wbp_1440_f16", "wbp", 1440, 512, 51, 400, storage="f16", step=2.4),
        # rows of an unbinned 4k series at thickness 1200 (one rank's or one
        # request's share of the series)
        _recon("wbp_4k_rows", "wbp", 4096, 128, 41, 1200),
        # a small SART tomogram
        _recon("sart_small", "sart", 256, 96, 41, 96, iterations=10, subsets=5),
        # rows of the standard SART series (1024 wide, 61 tilts, thickness
        # 300, 15 iterations, 5 subsets, relaxation 0.3)
        _recon("sart_1k", "sart", 1024, 256, 61, 300, step=2.0, iterations=15, subsets=5, relax=0.3),
        # a cropped series in BF16 storage, the outermost tilts left out of
        # the subsets, subsets that do not divide them
        _recon("sart_ragged_bf16", "sart", 925, 131, 53, 221, storage="bf16", step=2.3, iterations=8, subsets=7,
               skip=3),
        # a 2k series in FP16 storage
        _recon("sart_2k_f16", "sart", 2048, 96, 41, 600, storage="f16", iterations=10, subsets=5),
        # rows of the unbinned 4k series, 15 iterations
        _recon("sart_4k_rows", "sart", 4096, 64, 41, 1200, iterations=15, subsets=5),
        # the call a user of the reference makes: host frames in, host volume out
        _recon("doit_wbp_512", "wbp", 512, 512, 41, 128, kind="doit"),
        # the input stage on 4k frames, tilt axis near 86 degrees, binning 4
        _stack("stack_4k", "stack", 4096, 4096, 8, 4.0, 86.0),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _cost(case):
    """Rough device work, to keep drawn cases within the listed ones."""
    if case["kind"] in ("stack", "bin"):
        return 60.0 * case["nx"] * case["ny"] * case["tilts"]
    vox = float(case["nx"]) * case["ny"] * case["vol_z"] * case["tilts"]
    if case["method"] == "wbp":
        return 16.0 * vox
    return 100.0 * vox * (case["iterations"] + 1) / 15.0


def _smooth(n):
    for p in (2, 3, 5, 7, 11, 13):
        while n % p == 0:
            n //= p
    return n == 1


def draw(rng):
    while True:
        kind = rng.choice(["wbp", "wbp", "wbp", "sart", "sart", "sart", "doit", "stack", "bin"])
        if kind in ("stack", "bin"):
            case = _stack(None, kind, _log_int(rng, 700, 4096), _log_int(rng, 700, 4096), rng.randint(2, 8),
                          rng.choice([1.0, 1.7, 2.0, 3.0, 4.0, 6.5]) if kind == "stack" else
                          rng.choice([1.6, 2.0, 3.0, 4.0, 8.0]), rng.choice([-4.5, 1.2, 84.0, 86.0, 95.5]))
        else:
            method = kind if kind != "doit" else rng.choice(["wbp", "wbp", "sart"])
            tilts = rng.randint(21, 81)
            kw = dict(storage=rng.choice(["f32", "f32", "f16", "bf16"]), step=round(rng.uniform(100.0, 130.0) / tilts, 2))
            if method == "sart":
                kw.update(iterations=rng.randint(4, 20), subsets=rng.randint(3, 9), relax=rng.choice([0.0, 0.0, 0.3]),
                          skip=rng.choice([0, 0, 0, 2]))
            hi = 1024 if kind == "doit" else 4096
            case = _recon(None, method, _log_int(rng, 128, hi), _log_int(rng, 24, 512), tilts,
                          _log_int(rng, 40, 1200 if kind != "doit" else 300),
                          kind="doit" if kind == "doit" else "recon", **kw)
        if kind not in ("stack", "bin") and case["method"] == "wbp" and case["nx"] > 2048 and not _smooth(case["nx"] & ~1):
            continue   # refused: the 2x-grid row would not fit one block's shared memory
        if _cost(case) < max(_cost(c) for c in listed() if c["kind"] == case["kind"] or case["kind"] == "bin"
                             and c["kind"] == "stack"):
            return case


def _tilts(case):
    t = np.arange(case["tilts"], dtype=np.float64)
    return (case["step"] * (t - (case["tilts"] - 1) / 2)).astype(np.float32)


def _series(nx, ny, tilts, thick, seed):
    """frames[T][ny][nx] on the GPU: spheres of 1.5 % to 6 % of the width in a
    slab of ice, 50 counts per pixel, counting noise."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    pick = np.random.default_rng(seed)
    f = torch.randn((len(tilts), ny, nx), generator=g, device="cuda")
    u = torch.arange(nx, device="cuda", dtype=torch.float32) - 0.5 * nx
    v = torch.arange(ny, device="cuda", dtype=torch.float32)
    for t, deg in enumerate(tilts):
        c, s = math.cos(math.radians(float(deg))), math.sin(math.radians(float(deg)))
        p = torch.zeros((ny, nx), device="cuda")
        state = np.random.default_rng(seed + 1)
        for _ in range(12):
            r = nx * state.uniform(0.015, 0.06)
            x, y, z = state.uniform(-0.45, 0.45) * nx, state.uniform(0, ny), state.uniform(-0.5, 0.5) * thick
            d2 = (r * r - (v - y) ** 2)[:, None] - (u - (x * c + z * s))[None, :] ** 2
            p += state.uniform(0.2, 1.0) * 2.0 / r * torch.sqrt(d2.clamp_(min=0.0))
        mean = 50.0 * pick.uniform(0.8, 1.2) + 6.0 * p
        f[t] = (mean + torch.sqrt(mean) * f[t]).clamp_(min=0.0)
    return f


def _plan_args(case):
    kw = dict(method=recon.SART if case["method"] == "sart" else recon.WBP, storage=STORAGE[case["storage"]])
    if case["method"] == "sart":
        kw.update(start_tilt=case["skip"], num_tilts=case["tilts"] - 2 * case["skip"], iterations=case["iterations"],
                  subsets=case["subsets"], relax=case["relax"], fill_seed=1)
    return kw


def _inputs(case, seed):
    if case["kind"] in ("recon", "doit"):
        return _series(case["nx"], case["ny"], _tilts(case), case["vol_z"], seed)
    return _series(case["nx"], case["ny"], np.linspace(-30, 30, case["tilts"]), 0.2 * case["nx"], seed)


def prepare(case, seed):
    frames = _inputs(case, seed)
    state = dict(case=case)
    if case["kind"] == "recon":
        plan = recon.Plan(case["nx"], case["ny"], _tilts(case), case["vol_z"], **_plan_args(case))
        state.update(plan=plan, proj=frames, vol=torch.empty(plan.volume_shape, device="cuda"))
    elif case["kind"] == "doit":
        state.update(series=recon.TiltSeries(frames.cpu().numpy()), align=recon.AlignParam(_tilts(case)))
    else:
        T = case["tilts"]
        kw = dict(bin=case["bin"], seed=4242)
        if case["kind"] == "stack":
            rng = np.random.default_rng(seed)
            axes = (case["axis"] + rng.uniform(-1, 1, T)).astype(np.float32)
            kw.update(shifts=rng.uniform(-20, 20, (T, 2)).astype(np.float32), tilt_axes=axes, size_axis=float(axes[0]))
        else:
            kw.update(correct=False, rand_fill=False)
        st = recon.Stack(case["nx"], case["ny"], T, **kw)
        state.update(stack=st, raw=frames, out=torch.empty(st.binned_shape, device="cuda"))
    return state


def run(state):
    case = state["case"]
    if case["kind"] == "recon":
        state["plan"].run_device(state["proj"].data_ptr(), state["vol"].data_ptr(),
                                 torch.cuda.current_stream().cuda_stream)
        return state["vol"]
    if case["kind"] == "doit":
        kw = dict(storage=STORAGE[case["storage"]])
        if case["method"] == "wbp":
            return recon.CDoWbpRecon(**kw).DoIt(state["series"], state["align"], case["vol_z"])
        return recon.CDoSartRecon(fill_seed=1, relax=case["relax"], **kw).DoIt(
            state["series"], state["align"], case["skip"], case["tilts"] - 2 * case["skip"], case["vol_z"],
            case["iterations"], case["subsets"])
    state["stack"].run_device(state["raw"].data_ptr(), state["out"].data_ptr(),
                              torch.cuda.current_stream().cuda_stream)
    return state["out"]


def _binned(case):
    a = (case["nx"], case["ny"])
    if case["kind"] == "stack" and abs(math.sin(math.radians(case["axis"]))) > 0.707:
        a = a[::-1]
    return a, tuple(n if case["bin"] == 1.0 else int(n / case["bin"]) // 2 * 2 for n in a)


def work(case):
    """Bytes: frames in, volume (or binned frames) out.  Operations: WBP, the
    R-weight FFTs, two fused multiply-adds per voxel and tilt of the 2x grid
    and the crop's FFTs; SART, two fused multiply-adds per voxel and tilt of
    every back-projection and four per ray sample of every forward one."""
    if case["kind"] in ("stack", "bin"):
        (ax, ay), (bx, by) = _binned(case)
        T = case["tilts"]
        fl = 2.5 * ax * ay * math.log2(ax) + 5.0 * (bx // 2 + 1) * ay * math.log2(ay)
        fl += 5.0 * (bx // 2 + 1) * by * math.log2(by) + 2.5 * bx * by * math.log2(bx)
        return {"bytes": 4.0 * T * (case["nx"] * case["ny"] + bx * by), "flops": T * fl}
    Nx, Nz, ny, T = case["nx"] & ~1, case["vol_z"], case["ny"], case["tilts"]
    nbytes = 4.0 * ny * (T * case["nx"] + Nx * Nz)
    if case["method"] == "wbp":
        fl = 5.0 * T * Nx * math.log2(Nx) + 16.0 * Nx * Nz * T
        fl += 2.5 * 4 * Nx * Nz * math.log2(2 * Nx) + 5.0 * (Nx // 2 + 1) * 2 * Nz * math.log2(2 * Nz)
        fl += 5.0 * (Nx // 2 + 1) * Nz * math.log2(Nz) + 2.5 * Nx * Nz * math.log2(Nx)
    else:
        used = _tilts(case)[case["skip"]: T - case["skip"]]
        rays = float(np.sum(1.0 / np.cos(np.radians(used.astype(np.float64)))))
        fl = 4.0 * Nx * Nz * T + case["iterations"] * Nx * Nz * (4.0 * len(used) + 8.0 * rays)
    return {"bytes": nbytes, "flops": fl * ny}


def tolerance(case):
    """About four times the distance from exact() seen over listed and drawn
    cases: FP32 5e-7 to 3.6e-6, FP16 2.8e-4 to 4.4e-4, BF16 1.5e-3 to 2.4e-3."""
    if case["kind"] in ("stack", "bin"):
        return {"rel": 5e-6}
    if case["storage"] == "f32":
        return {"rel": 1.5e-5}
    return {"rel": 1.6e-3 if case["storage"] == "f16" else 1e-2}


# --- the same results in 64 bits, in plain torch ------------------------------
# Sample positions are part of the definition and are formed in FP32 with the
# reference's operation order; every value, weight and sum is FP64.

def _table(case):
    a = np.float32(0.017453) * _tilts(case)
    return np.cos(a.astype(np.float64)).astype(np.float32), np.sin(a.astype(np.float64)).astype(np.float32)


def _f32(x):
    """A product and sum formed in FP64 and rounded once is a fused FP32 operation."""
    return x.float().double()


def _lerp_at(xp, N):
    """Samples xp (FP32 values) of a row of N: cell, fraction, inside."""
    inside = (xp >= 0) & (xp <= N - 2)
    i = xp.clamp(0, max(N - 2, 0)).floor()
    return i.long(), torch.where(inside, xp - i, torch.zeros_like(xp)), inside


def _grid(n):
    return (torch.arange(n, device="cuda", dtype=torch.float64) - n / 2).float().double()


def _c2r_packed(nz, nx):
    """Whether cuFFT inverts an (nz, nx) C2R by half-length packing."""
    x = torch.zeros((1, nz, nx // 2 + 1), dtype=torch.complex64, device="cuda")
    x[0, 0, 0] = 1j
    return bool(torch.fft.irfft2(x, s=(nz, nx), dim=(1, 2), norm="forward")[0, 0, 0].abs() > 0.5)


def _wbp_exact(case, frames):
    cs, sn = _table(case)
    ny, T, Nz, N = case["ny"], case["tilts"], case["vol_z"], case["nx"] & ~1
    k = torch.arange(N // 2 + 1, device="cuda", dtype=torch.float64) / N
    h = 2.0 * k * (0.55 + 0.45 * torch.cos(float(np.float32(6.2831852)) * k))
    fX, fZ = _grid(2 * N)[None, :], _grid(2 * Nz)[:, None]
    packed = _c2r_packed(Nz, N)
    vol = torch.empty((ny, Nz, N), dtype=torch.float64, device="cuda")
    for y0 in range(0, ny, 8):
        rows = frames[:, y0:y0 + 8, :N].double().transpose(0, 1)               # [S][T][N]
        rows = rows * (torch.tensor(cs, device="cuda").double() / Nz)[None, :, None]
        rows = torch.fft.irfft(torch.fft.rfft(rows, dim=2) * h, n=N, dim=2)
        S = rows.shape[0]
        acc = torch.zeros((S, 4 * N * Nz), dtype=torch.float64, device="cuda")
        cnt = torch.zeros((4 * N * Nz,), dtype=torch.float64, device="cuda")
        for t in range(T):
            a = _f32(fX * float(cs[t]) + _f32(fZ * float(sn[t])))
            xp = _f32(_f32(a * 0.5 + float(N // 2)) + 0.5).reshape(-1)
            i, fr, ok = _lerp_at(xp, N)
            v = rows[:, t].contiguous()
            lo, hi = v.index_select(1, i), v.index_select(1, i + 1)
            acc += torch.where(ok, lo * (1.0 - fr) + hi * fr, torch.zeros_like(lo))
            cnt += ok
        acc = torch.where(cnt > 0, acc / cnt.clamp(min=1), torch.zeros_like(acc)).reshape(S, 2 * Nz, 2 * N)
        F = torch.fft.rfft2(acc) / (4.0 * N * Nz)
        F = F[:, :, :N // 2 + 1]
        F = torch.cat([F[:, :Nz // 2 + 1], F[:, Nz + Nz // 2 + 1:]], 1)
        W = torch.fft.ifft(F, dim=1, norm="forward")
        im0, imh = W[:, :, 0].imag, W[:, :, N // 2].imag
        out = torch.fft.irfft(W, n=N, dim=2, norm="forward")   # drops those imaginary parts
        if packed:
            out[:, :, 0::2] -= (im0 + imh)[:, :, None]
            out[:, :, 1::2] += (im0 - imh)[:, :, None]
        vol[y0:y0 + 8] = out.flip(1)
    return vol


def _csr(cols, vals, width):
    """Rows of equally many entries as a sparse matrix."""
    n, m = cols.shape
    crow = torch.arange(n + 1, device="cuda", dtype=torch.int32) * m
    return torch.sparse_csr_tensor(crow, cols.reshape(-1).int(), vals.reshape(-1), (n, width))


def _sart_exact(case, frames):
    cs, sn = _table(case)
    ny, T, Nz, N = case["ny"], case["tilts"], case["vol_z"], case["nx"] & ~1
    first, used = case["skip"], case["tilts"] - 2 * case["skip"]
    fX, fZ = _grid(N)[None, :], _grid(Nz)[:, None]

    def back(tilts):
        """sum over the tilts of the lerped rows [nt * N] -> voxels, and the counts"""
        cols, vals, cnt = [], [], torch.zeros((Nz * N,), dtype=torch.float64, device="cuda")
        for j, t in enumerate(tilts):
            a = _f32(fX * float(cs[t]) + _f32(fZ * float(sn[t])))
            i, fr, ok = _lerp_at(_f32(a + N / 2.0).reshape(-1), N)
            cols += [j * N + i, j * N + i + 1]
            vals += [torch.where(ok, 1.0 - fr, torch.zeros_like(fr)), torch.where(ok, fr, torch.zeros_like(fr))]
            cnt += ok
        return _csr(torch.stack(cols, 1), torch.stack(vals, 1), len(tilts) * N), cnt

    def forward(t):
        """mean of the bilinear samples of every ray of tilt t, and which rays have any"""
        c, s = float(cs[t]), float(sn[t])
        L = int(np.float32(np.float32(np.float32(Nz) / cs[t]) + np.float32(1.5)))
        u = torch.arange(N, device="cuda", dtype=torch.float64) - 0.5 * N
        tx = _f32(_f32(u / c) + N * 0.5)
        z0 = torch.arange(L, device="cuda", dtype=torch.float64) - 0.5 * L
        x = _f32(tx[:, None] - z0[None, :] * s)
        z = _f32(Nz * 0.5 + z0 * c)[None, :].expand(N, L)
        ok = (x >= 0) & (x <= N - 2) & (z >= 0) & (z <= Nz - 2)
        ix, iz = x.clamp(0, N - 2).floor(), z.clamp(0, Nz - 2).floor()
        wx, wz = x - ix, z - iz
        n = ok.sum(1)
        w = ok / n.clamp(min=1)[:, None]
        at = (iz * N + ix).long()
        cols = torch.stack([at, at + 1, at + N, at + N + 1], 2).reshape(N, -1)
        vals = torch.stack([(1 - wx) * (1 - wz) * w, wx * (1 - wz) * w, (1 - wx) * wz * w, wx * wz * w], 2)
        return _csr(cols, vals.reshape(N, -1), Nz * N), n > 0

    w = torch.tensor(cs, device="cuda").double() / Nz
    raw = frames[:, :, :N].double().transpose(1, 2) * w[:, None, None]          # [T][N][S]
    vol = torch.zeros((Nz * N, ny), dtype=torch.float64, device="cuda")

    def update(tilts, rows, relax):
        nonlocal vol
        B, cnt = back(tilts)
        new = (vol + (B @ rows.reshape(-1, ny)) * (relax / cnt.clamp(min=1))[:, None]).clamp(min=0)
        vol = torch.where((cnt > 0)[:, None], new, vol)

    update(list(range(T)), raw.contiguous(), 1.0)
    relax = case["relax"] if case["relax"] > 0 else 1.0 / case["subsets"]
    sizes = [used // case["subsets"] + (i < used % case["subsets"]) for i in range(case["subsets"])]
    rays = {t: forward(t) for t in range(first, first + used)}
    for _ in range(case["iterations"]):
        t0 = first
        for n in sizes:
            tilts = list(range(t0, t0 + n))
            t0 += n
            if not n:
                continue
            d = torch.stack([(raw[t] - rays[t][0] @ vol) * rays[t][1][:, None] for t in tilts])
            update(tilts, d, relax)
    return vol.t().reshape(ny, Nz, N).flip(1).contiguous()


def _bin_exact(case, frames):
    (ax, ay), (bx, by) = _binned(case)
    out = []
    for f in frames:
        F = torch.fft.rfft2(f.double()) / (ax * ay)
        F = torch.cat([F[:by // 2 + 1], F[ay - (by - by // 2 - 1):]], 0)[:, :bx // 2 + 1]
        W = torch.fft.ifft(F, dim=0, norm="forward")
        im0, imh = W[:, 0].imag, W[:, bx // 2].imag
        o = torch.fft.irfft(W, n=bx, dim=1, norm="forward")
        if _c2r_packed(by, bx):
            o[:, 0::2] -= (im0 + imh)[:, None]
            o[:, 1::2] += (im0 - imh)[:, None]
        out.append(o)
    return torch.stack(out)


def exact(case, seed):
    if case["kind"] == "stack":
        return None   # empty pixels take their values from a random table drawn by the library
    if case["kind"] == "recon" or case["kind"] == "doit":
        frames = _inputs(case, seed)
        vox = float(case["nx"]) * case["ny"] * case["vol_z"] * case["tilts"]
        if case["method"] == "sart":
            if vox * (case["iterations"] + 1) > 2.5e11:
                return None
            return _sart_exact(case, frames)
        return _wbp_exact(case, frames) if vox < 4e10 else None
    return _bin_exact(case, _inputs(case, seed))
