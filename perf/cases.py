"""The work that programs have this framework do, as cases to be timed and compared.

Each case is one call, or one short chain of calls, through the public entry points of
msbg_gpu, on seeded inputs of the kinds the tests and the benchmark use:

  mcf      mean-curvature-flow smoothing of a channel that stays on the GPU
  solve    MGPCG pressure solve of a prepared problem, the pressure copied to the host
  step     a FLIP pressure step: per-cell arrays in, prepare, solve, pressure out
  flip     the FLIP transfers around the solve, particles resident on the GPU
  g2p_mr   grid-to-particle velocities on a mixed-resolution grid
  splat    particles into the 16-bit density channel that the smoother reads
  cnn      the learned network: inference over tiles, or one training step
"""
import importlib
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "msbg-flip_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)
msbg_gpu = importlib.import_module("msbg_gpu")

STORAGE = {"f32": msbg_gpu.F32, "f16": msbg_gpu.F16, "bf16": msbg_gpu.BF16}


def listed():
    return [
        # the smoother on a small interactive grid: 16 short passes, launches count
        {"name": "mcf_f32_64_b16", "kind": "mcf", "dtype": "f32", "bsx": 16, "sx": 64, "sy": 64,
         "sz": 64, "spheres": 4, "rmin": 8.0, "rmax": 20.0, "iters": 2, "clamp": False},
        # the smoother on a production-size narrow band (the benchmark's smoothing workload)
        {"name": "mcf_f32_512_b16", "kind": "mcf", "dtype": "f32", "bsx": 16, "sx": 512, "sy": 512,
         "sz": 512, "spheres": 64, "rmin": 20.0, "rmax": 60.0, "iters": 20, "clamp": False},
        # 16-bit render density on a non-cubic grid, as a renderer smooths its splatted surface
        {"name": "mcf_u16_ragged_b16", "kind": "mcf", "dtype": "u16", "bsx": 16, "sx": 336,
         "sy": 208, "sz": 272, "spheres": 24, "rmin": 12.0, "rmax": 40.0, "iters": 8,
         "clamp": True},
        # the smallest solve in use: plain FP32 on a 64^3 adaptive grid, latency of one call
        {"name": "solve_f32_64_b16", "kind": "solve", "res": 64, "bsx0": 16, "levels": 2,
         "band": 4.0, "storage": "f32", "refine": 0},
        # an ordinary solve with FP16 vectors and FP64 refinement, 3 levels
        {"name": "solve_f16_256_b16", "kind": "solve", "res": 256, "bsx0": 16, "levels": 3,
         "band": 8.0, "storage": "f16", "refine": 30},
        # one pressure step of an ordinary simulation, a grid that is no power of two
        {"name": "step_f32_320_b32", "kind": "step", "res": 320, "bsx0": 32, "levels": 2,
         "band": 16.0, "storage": "f32", "refine": 30},
        # the benchmark's solve: 1024^3, 32^3 blocks, 2 levels, to a true FP64 residual of 1e-6
        {"name": "solve_f32_1024_b32", "kind": "solve", "res": 1024, "bsx0": 32, "levels": 2,
         "band": 64.0, "storage": "f32", "refine": 30},
        # particle-to-grid, gravity, pressure gradient, grid-to-particle of a 2-phase column
        {"name": "flip_160_b16", "kind": "flip", "res": 160, "bsx": 16, "ppv": 8, "z": 0.4,
         "channels": False},
        # grid-to-particle on a 3-level grid, particles in no order (the benchmark's transfer)
        {"name": "g2p_mr_512_b16", "kind": "g2p_mr", "res": 512, "bsx": 16, "levels": 3,
         "particles": 16000000},
        # the demo's particle cloud into the density channel (the benchmark's splat)
        {"name": "splat_1024_b16", "kind": "splat", "sx": 1024, "sy": 1024, "sz": 1024, "bsx": 16,
         "base": 4096},
        # inference of the learned guess over one chunk of tiles
        {"name": "cnn_forward_4096", "kind": "cnn", "tiles": 4096, "train": False},
        # a training step at the default batch
        {"name": "cnn_train_128", "kind": "cnn", "tiles": 128, "train": True},
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["mcf", "mcf", "mcf", "solve", "solve", "solve", "step", "flip", "flip",
                       "g2p_mr", "splat", "cnn"])
    if kind == "mcf":
        bsx = rng.choice([8, 16, 16, 32])
        d = [max(2, round(_log(rng, 48, 448) / bsx)) * bsx for _ in range(3)]
        rmin = 0.04 * max(d)
        return {"kind": kind, "dtype": rng.choice(["f32", "f32", "u16"]), "bsx": bsx, "sx": d[0],
                "sy": d[1], "sz": d[2], "spheres": rng.randint(3, 48), "rmin": rmin,
                "rmax": rmin * rng.uniform(1.5, 3.0), "iters": rng.choice([2, 4, 6, 10, 20]),
                "clamp": rng.random() < 0.3}
    if kind in ("solve", "step"):
        # grids that coarsen to the direct solve: a power of two times 2, 3, 5 or 7
        bsx0 = rng.choice([8, 16, 32, 32])
        top = 512 if kind == "solve" and bsx0 > 8 else 256
        sizes = sorted({m << k for m in (1, 3, 5, 7) for k in range(4, 10)
                        if 48 <= (m << k) <= top and (m << k) % bsx0 == 0 and (m << k) >= 2 * bsx0})
        res = min(sizes, key=lambda s: abs(math.log(s) - math.log(_log(rng, 48, top))))
        storage = rng.choice(["f32", "f32", "f16", "bf16"]) if bsx0 > 8 else "f32"
        return {"kind": kind, "res": res, "bsx0": bsx0,
                "levels": rng.randint(1, 2 if bsx0 == 8 else 3), "band": rng.choice([4.0, 8.0, 16.0]),
                "storage": storage, "refine": 30 if storage != "f32" else rng.choice([0, 30])}
    if kind == "flip":
        bsx = rng.choice([8, 16, 32])
        return {"kind": kind, "res": max(2, round(_log(rng, 32, 256) / bsx)) * bsx, "bsx": bsx,
                "ppv": rng.randint(2, 8), "z": round(rng.uniform(0.2, 0.6), 3),
                "channels": rng.random() < 0.5}
    if kind == "g2p_mr":
        bsx = rng.choice([8, 16, 32])
        return {"kind": kind, "res": max(8, round(_log(rng, 96, 512) / bsx)) * bsx, "bsx": bsx,
                "levels": rng.randint(2, 3), "particles": int(_log(rng, 1e4, 1.6e7))}
    if kind == "splat":
        bsx = rng.choice([8, 16, 32])
        d = [max(4, round(_log(rng, 96, 1024) / bsx)) * bsx for _ in range(3)]
        return {"kind": kind, "sx": d[0], "sy": d[1], "sz": d[2], "bsx": bsx,
                "base": int(_log(rng, 100, 2000))}
    train = rng.random() < 0.5
    return {"kind": "cnn", "tiles": int(_log(rng, 1, 512 if train else 4096)), "train": train}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
class _View:
    """Device memory of a context's channel, which lives as long as the context does."""

    def __init__(self, ctx, ptr, shape, typestr):
        self.ctx = ctx
        self.__cuda_array_interface__ = {"shape": shape, "typestr": typestr, "data": (ptr, False),
                                         "version": 3}


def _view(ctx, chan, shape, typestr):
    # the tensor holds the _View, and with it the context
    return torch.as_tensor(_View(ctx, ctx.device_ptr(chan), shape, typestr), device="cuda")


def _mcf_blocks(c, dev):
    """Block kinds of a union of spheres (value blocks where the surface is within 4 voxels),
    and the spheres.  One scene for all seeds: the seed moves the spheres inside it."""
    g = torch.Generator().manual_seed(2024)
    dims = torch.tensor([c["sx"], c["sy"], c["sz"]], dtype=torch.float64)
    cen = (torch.rand(c["spheres"], 3, generator=g, dtype=torch.float64) * dims).to(dev)
    rad = (c["rmin"] + torch.rand(c["spheres"], generator=g, dtype=torch.float64) *
           (c["rmax"] - c["rmin"])).to(dev)
    b = c["bsx"]
    nb = [c["sx"] // b, c["sy"] // b, c["sz"] // b]
    z, y, x = torch.meshgrid(*[(torch.arange(n, device=dev, dtype=torch.float64) + 0.5) * b
                               for n in nb[::-1]], indexing="ij")
    ctr = torch.stack([x.reshape(-1), y.reshape(-1), z.reshape(-1)], 1)
    d = (torch.cdist(ctr, cen) - rad).min(1).values
    near = d.abs() <= 4.0 + 0.5 * b * math.sqrt(3.0)
    kind = torch.where(near, 1, torch.where(d > 0, 2, 3)).to(torch.int8)
    return kind, cen, rad, nb


def _mcf_values(c, kind, cen, rad, nb, dev):
    b = c["bsx"]
    ids = torch.nonzero(kind == 1).reshape(-1)
    e = torch.arange(b ** 3, device=dev)
    vox = torch.stack([e % b, (e // b) % b, e // (b * b)], 1).float() + 0.5
    out = torch.empty(len(ids), b ** 3, device=dev)
    cen, rad = cen.float(), rad.float()
    step = max(1, (1 << 22) // b ** 3)
    for i in range(0, len(ids), step):
        q = ids[i:i + step]
        o = torch.stack([q % nb[0], (q // nb[0]) % nb[1], q // (nb[0] * nb[1])], 1).float() * b
        p = o[:, None, :] + vox[None]
        m = None
        for s in range(len(rad)):
            f = (p - cen[s]).square_().sum(-1).sqrt_() - rad[s]
            m = f if m is None else torch.minimum(m, f)
        out[i:i + step] = m
    if c["dtype"] == "u16" or c["clamp"]:  # the density of a surface 2 voxels in, 4 out
        out = 1.0 - ((out + 2.0) / 6.0).clamp(0.0, 1.0)
    return ids, out


def _mcf_consts(c):
    return (0.0, 1.0) if c["dtype"] == "u16" or c["clamp"] else (4.0, -4.0)


def _mcf_input(c, seed):
    kind, cen, rad, nb = _mcf_blocks(c, "cuda")
    g = torch.Generator().manual_seed(seed)
    cen = cen + (torch.rand(cen.shape, generator=g, dtype=torch.float64) - 0.5).to(cen.device)
    rad = rad + (torch.rand(rad.shape, generator=g, dtype=torch.float64) - 0.5).to(rad.device)
    ids, val = _mcf_values(c, kind, cen, rad, nb, "cuda")
    return kind, ids, val, nb


def _prepare_mcf(c, seed):
    kind, ids, val, _ = _mcf_input(c, seed)
    ctx = msbg_gpu.Context(0)
    ctx.set_topology(c["sx"], c["sy"], c["sz"], c["bsx"])
    empty, full = _mcf_consts(c)
    shape = (len(ids),) + (c["bsx"],) * 3
    if c["dtype"] == "u16":
        q = (val * 65535.0).round().to(torch.int32).cpu().numpy().astype(np.uint16)
        ctx.upload_channel_u16(1, 0, kind.cpu().numpy(), q, int(empty * 65535), int(full * 65535))
    else:
        ctx.upload_channel(1, 0, kind.cpu().numpy(), val.cpu().numpy(), empty, full)
    out = _view(ctx, 1, shape, "<i2" if c["dtype"] == "u16" else "<f4")
    return {"c": c, "ctx": ctx, "list": ids.to(torch.int32).cpu().numpy(), "out": out}


def _scene(c):
    # one geometry for all seeds; the seed makes the velocity field
    return msbg_gpu.PressureScene(c["res"], c["bsx0"], c["levels"], band=c["band"], n_modes=1)


def _rhs(c, seed, levels, flags):
    """The MAC divergence of 16 random Fourier modes (wave numbers up to 8) in liquid cells."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    g = torch.Generator().manual_seed(seed)
    res, b0 = c["res"], c["bsx0"]
    k = torch.randint(1, 9, (16, 3), generator=g) * (2 * torch.randint(0, 2, (16, 3), generator=g)
                                                     - 1)
    amp = torch.randn(16, 3, generator=g)
    coef = (2 * amp * torch.sin(math.pi * k / res)).sum(1).to(dev)
    phase = (2 * math.pi * torch.rand(16, 1, generator=g))
    x = (torch.arange(res) + 0.5) * (2 * math.pi / res)
    tab = [torch.polar(torch.ones(16, res), k[:, d:d + 1] * x + (phase if d == 0 else 0)).to(dev)
           for d in range(3)]
    lev = torch.from_numpy(levels.astype(np.int64)).to(dev)
    nb = res // b0
    out = np.empty(len(flags), np.float32)
    size = (b0 >> lev) ** 3
    end = torch.cumsum(size, 0)
    for i in range(0, len(flags), 1 << 24):
        e = torch.arange(i, min(i + (1 << 24), len(flags)), device=dev)
        blk = torch.searchsorted(end, e, right=True)
        L = lev[blk]
        bs = b0 >> L
        v = e - (end - size)[blk]
        X = (blk % nb) * b0 + ((v % bs) << L)
        Y = (blk // nb % nb) * b0 + ((v // bs % bs) << L)
        Z = (blk // (nb * nb)) * b0 + ((v // (bs * bs)) << L)
        s = torch.zeros(len(e), device=dev)
        for m in range(16):
            s += coef[m] * (tab[0][m][X] * tab[1][m][Y] * tab[2][m][Z]).real
        out[i:i + len(e)] = s.cpu().numpy()
    out[flags != 0] = 0.0
    return out


def _pressure_input(c, seed, pinned=False):
    scene = _scene(c)
    flags, face, rhs = scene.arrays(pinned=pinned)
    rhs[:] = _rhs(c, seed, scene.block_levels, flags)
    return scene, flags, face, rhs


def _prepare_solve(c, seed):
    scene, flags, face, rhs = _pressure_input(c, seed, c["kind"] == "step")
    s = {"c": c, "ctx": msbg_gpu.Context(0), "levels": scene.block_levels, "flags": flags,
         "face": face, "rhs": rhs, "out": msbg_gpu.pinned_empty(len(flags), np.float32),
         "prm": msbg_gpu.solve_params(tol=1e-6, maxRefine=c["refine"],
                                      storage=STORAGE[c["storage"]])}
    if c["kind"] == "solve":
        s["ctx"].pressure_prepare_arrays(c["res"], c["bsx0"], c["levels"], scene.block_levels,
                                         flags, face, rhs)
        for k in ("flags", "face", "rhs"):
            del s[k]
    return s


def _flip_particles(c, seed):
    """ppv particles per liquid cell below z, one per air cell in the 8 cells above, cell by
    cell; smooth velocities."""
    g = torch.Generator("cuda").manual_seed(seed)
    res, zl = c["res"], int(c["z"] * c["res"])
    parts = []
    for lo, hi, n, phase in ((0, zl, c["ppv"], 0), (zl, min(res, zl + 8), 1, 1)):
        z, y, x = torch.meshgrid(torch.arange(lo, hi, device="cuda"),
                                 torch.arange(res, device="cuda"),
                                 torch.arange(res, device="cuda"), indexing="ij")
        cell = torch.stack([x.reshape(-1), y.reshape(-1), z.reshape(-1)], 1).float()
        pos = cell.repeat_interleave(n, 0)
        pos = pos + torch.rand(pos.shape, generator=g, device="cuda")
        a = torch.randn(3, 3, generator=g, device="cuda")
        vel = torch.sin(2 * math.pi / res * (pos @ a.T))
        ph = torch.full((len(pos), 1), phase, dtype=torch.int32, device="cuda")
        parts.append(torch.cat([pos, vel, ph.view(torch.float32)], 1))
    p = torch.cat(parts).contiguous()
    pres = torch.rand(res ** 3, generator=g, device="cuda") * 10.0
    return p, pres


def _prepare_flip(c, seed):
    p, pres = _flip_particles(c, seed)
    ctx = msbg_gpu.Context(0)
    ctx.set_topology(c["res"], c["res"], c["res"], c["bsx"])
    host = msbg_gpu.pinned_empty(c["res"] ** 3, np.float32)
    host[:] = pres.cpu().numpy()
    return {"c": c, "ctx": ctx, "p": p, "pressure": host}


def _mr_levels(c):
    nb = c["res"] // c["bsx"]
    bz = np.arange(nb ** 3) // (nb * nb)
    lev = np.where(bz < nb * 3 // 8, 0, np.where(bz < nb * 6 // 8, 1, 2))
    return np.minimum(lev, c["levels"] - 1).astype(np.int32)


def _mr_input(c, seed):
    g = torch.Generator("cuda").manual_seed(seed)
    lev = _mr_levels(c)
    n = msbg_gpu.packed_voxels(c["bsx"], lev)
    vel = torch.randn(3 * n, generator=g, device="cuda")
    old = vel + 0.1 * torch.randn(3 * n, generator=g, device="cuda")
    p = torch.zeros(c["particles"], 7, device="cuda")
    p[:, :3] = torch.rand(c["particles"], 3, generator=g, device="cuda") * c["res"]
    p[:, 3:6] = torch.randn(c["particles"], 3, generator=g, device="cuda")
    return lev, vel, old, p


def _prepare_g2p_mr(c, seed):
    lev, vel, old, p = _mr_input(c, seed)
    ctx = msbg_gpu.Context(0)
    ctx.set_topology(c["res"], c["res"], c["res"], c["bsx"], c["levels"], lev)
    ctx.flip_mr_channel(msbg_gpu.FLIP_VEL, vel.cpu().numpy())
    ctx.flip_mr_channel(msbg_gpu.FLIP_VEL_OLD, old.cpu().numpy())
    ctx.flip_mr_dist(c["levels"])
    return {"c": c, "ctx": ctx, "p": p}


def _prepare_splat(c, seed):
    # one arrangement for all seeds (the blocks in use are part of the result): the seed moves
    # each particle within its cell
    pos = msbg_gpu.splat_demo_particles((c["sx"], c["sy"], c["sz"]), c["base"])
    jit = np.random.default_rng(seed).random(pos.shape, np.float32)
    pos = np.clip(np.floor(pos) + 0.01 + 0.98 * jit, 0.01, None).astype(np.float32)
    ctx = msbg_gpu.Context(0)
    ctx.set_topology(c["sx"], c["sy"], c["sz"], c["bsx"])
    return {"c": c, "ctx": ctx, "pos": torch.from_numpy(pos).cuda()}


def _cnn_input(c, seed):
    g = torch.Generator("cuda").manual_seed(seed)
    n = c["tiles"]
    shape = (n, 4, 18, 18, 18)
    feat = torch.zeros(shape, device="cuda")
    solid = torch.rand(n, 18, 18, 18, generator=g, device="cuda") < 0.03
    surf = 18 * torch.rand(n, 1, 1, 1, generator=g, device="cuda") + 6
    air = (torch.arange(18, device="cuda").reshape(1, 18, 1, 1) > surf) & ~solid
    liquid = ~solid & ~air
    k = 2 * math.pi * torch.rand(n, 3, generator=g, device="cuda") / 9
    ax = torch.arange(18, device="cuda")
    ph = (k[:, 0].reshape(n, 1, 1, 1) * ax.reshape(1, 18, 1, 1) +
          k[:, 1].reshape(n, 1, 1, 1) * ax.reshape(1, 1, 18, 1) +
          k[:, 2].reshape(n, 1, 1, 1) * ax.reshape(1, 1, 1, 18))
    feat[:, 0] = torch.cos(ph) * liquid
    feat[:, 1] = solid.float()
    feat[:, 2] = air.float()
    feat[:, 3] = (torch.rand(n, 1, 1, 1, generator=g, device="cuda") < 0.2).float()
    mask = liquid[:, 1:17, 1:17, 1:17].reshape(n, -1).float().contiguous()
    tgt = (torch.sin(ph[:, 1:17, 1:17, 1:17]).reshape(n, -1) * mask).contiguous()
    w = []
    gw = torch.Generator().manual_seed(seed)
    for ci, co in ((4, 16), (16, 16), (16, 16), (16, 1)):
        w.append(torch.randn(co, ci, 3, 3, 3, generator=gw) * math.sqrt(2.0 / (27 * ci)))
    return feat.reshape(n, -1).contiguous(), tgt, mask, w


def _prepare_cnn(c, seed):
    feat, tgt, mask, w = _cnn_input(c, seed)
    net = msbg_gpu.Cnn(0)
    net.set_weights(torch.cat([x.reshape(-1) for x in w]).numpy())
    s = {"c": c, "net": net, "feat": feat}
    if c["train"]:
        s.update(tgt=tgt, mask=mask, count=float(mask.sum().item()))
    return s


def prepare(case, seed):
    return {"mcf": _prepare_mcf, "solve": _prepare_solve, "step": _prepare_solve,
            "flip": _prepare_flip, "g2p_mr": _prepare_g2p_mr, "splat": _prepare_splat,
            "cnn": _prepare_cnn}[case["kind"]](case, seed)


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
DT, GRAVITY, ALPHA = 0.01, -9.81, 0.95


def run(s):
    c = s["c"]
    kind = c["kind"]
    if kind == "mcf":
        s["ctx"].apply_channel_pde_mcf(1, s["list"], c["iters"], 0.1, clamp01=c["clamp"])
        return s["out"]
    if kind == "solve":
        s["ctx"].pressure_solve(s["prm"])
        return s["ctx"].pressure_download(out=s["out"])
    if kind == "step":
        s["ctx"].pressure_prepare_arrays(c["res"], c["bsx0"], c["levels"], s["levels"],
                                         s["flags"], s["face"], s["rhs"])
        s["ctx"].pressure_solve(s["prm"])
        return s["ctx"].pressure_download(out=s["out"])
    if kind == "flip":
        ctx, p = s["ctx"], s["p"]
        ctx.flip_p2g_device(p.data_ptr(), len(p))
        out = [p[:, 3:6]]
        if c["channels"]:
            n = c["res"] ** 3
            out += [ctx.flip_channel(w, n) for w in (msbg_gpu.FLIP_VEL, msbg_gpu.FLIP_BETA,
                                                     msbg_gpu.FLIP_MASS)]
        ctx.flip_gravity(GRAVITY, DT)
        ctx.flip_pressure_gradient(s["pressure"], DT)
        ctx.flip_g2p_device(p.data_ptr(), len(p), ALPHA)
        return out
    if kind == "g2p_mr":
        s["ctx"].flip_g2p_mr_device(s["p"].data_ptr(), len(s["p"]), ALPHA)
        return s["p"][:, 3:6]
    if kind == "splat":
        ctx = s["ctx"]
        kinds = ctx.splat_device(7, s["pos"].data_ptr(), len(s["pos"]))
        n = ctx.num_value_blocks(7)
        return [kinds, _view(ctx, 7, (n,) + (c["bsx"],) * 3, "<i2")]
    if c["train"]:
        loss, grad = s["net"].loss_grad(s["feat"], s["tgt"], s["mask"], count=s["count"],
                                        want_grad=True)
        s["net"].adam_step(2e-3)
        return [loss, grad, s["net"].get_weights()]
    return s["net"].forward(s["feat"])


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def _packed_cells(c):
    return msbg_gpu.packed_voxels(c["bsx0"], _scene(c).block_levels)


def work(case):
    c, kind = case, case["kind"]
    if kind == "mcf":
        # every iteration needs the whole field of the one before it
        k = _mcf_blocks(c, "cuda" if torch.cuda.is_available() else "cpu")[0]
        n = int((k == 1).sum()) * c["bsx"] ** 3
        return {"bytes": 2.0 * n * c["iters"] * (2 if c["dtype"] == "u16" else 4),
                "flops": 60.0 * n * c["iters"]}
    if kind == "solve":  # operator (4 values a cell) and right-hand side in, pressure out
        n = _packed_cells(c)
        return {"bytes": 24.0 * n, "flops": 60.0 * n}
    if kind == "step":  # flags, 3 face values and right-hand side in, pressure out
        n = _packed_cells(c)
        return {"bytes": 22.0 * n, "flops": 80.0 * n}
    if kind == "flip":
        n, zl = c["res"] ** 3, int(c["z"] * c["res"])
        np_ = c["res"] ** 2 * (zl * c["ppv"] + min(8, c["res"] - zl))
        # particles twice in, velocities out; the grid's channels written and read once
        return {"bytes": np_ * (28.0 + 28.0 + 12.0) + n * (28.0 + 28.0 + 4.0),
                "flops": np_ * (24 * 8.0 + 48 * 4.0)}
    if kind == "g2p_mr":
        n = msbg_gpu.packed_voxels(c["bsx"], _mr_levels(c))
        return {"bytes": c["particles"] * 40.0 + n * 26.0, "flops": c["particles"] * 96 * 4.0}
    if kind == "splat":
        n = c["base"] ** 2
        # positions in; the density of about 3 voxels per particle out
        return {"bytes": n * 18.0, "flops": n * 268 * 6.0}
    macs = c["tiles"] * 4096.0 * 27 * (4 * 16 + 2 * 16 * 16 + 16)
    feat, cells = c["tiles"] * 4 * 18 ** 3 * 4.0, c["tiles"] * 4096 * 4.0
    if c["train"]:
        return {"bytes": feat + 2 * cells, "flops": 6 * macs}
    return {"bytes": feat + cells, "flops": 2 * macs}


# ---------------------------------------------------------------------------
# the same in 64 bits, in plain torch
# ---------------------------------------------------------------------------
def _exact_mcf(c, seed):
    if c["dtype"] == "u16":
        return None
    kind, ids, val, nb = _mcf_input(c, seed)
    b, dev = c["bsx"], val.device
    if len(ids) * b ** 3 * c["iters"] > 2_000_000_000:
        return None
    empty, full = _mcf_consts(c)
    n = len(ids)
    slot = torch.full((nb[0] * nb[1] * nb[2],), -1, dtype=torch.int64, device=dev)
    slot[ids] = torch.arange(n, device=dev)
    # one flat field: the value blocks, then the two constants
    f = torch.cat([val.double().reshape(-1), torch.tensor([empty, full], dtype=torch.float64,
                                                           device=dev)])
    e = torch.arange(-1, b + 1, device=dev)
    pz, py, px = [t.reshape(-1) for t in torch.meshgrid(e, e, e, indexing="ij")]
    bx, by, bz = ids % nb[0], (ids // nb[0]) % nb[1], ids // (nb[0] * nb[1])
    out_of = lambda v: torch.where(v < 0, -1, torch.where(v >= b, 1, 0))  # noqa: E731
    dx, dy, dz = out_of(px), out_of(py), out_of(pz)
    groups = []
    for col in range(8):
        q = torch.nonzero((bx & 1) + 2 * (by & 1) + 4 * (bz & 1) == col).reshape(-1)
        for i in range(0, len(q), max(1, (1 << 24) // (b + 2) ** 3)):
            s = q[i:i + max(1, (1 << 24) // (b + 2) ** 3)]
            groups.append((col, s))

    def tile_index(s):
        x = bx[s][:, None] + dx[None]
        y = by[s][:, None] + dy[None]
        z = bz[s][:, None] + dz[None]
        ok = (x >= 0) & (y >= 0) & (z >= 0) & (x < nb[0]) & (y < nb[1]) & (z < nb[2])
        nid = torch.where(ok, x + nb[0] * (y + nb[1] * z), ids[s][:, None])
        k = kind[nid]
        own = ~ok
        cx = torch.where(own, px.clamp(0, b - 1)[None], (px % b)[None])
        cy = torch.where(own, py.clamp(0, b - 1)[None], (py % b)[None])
        cz = torch.where(own, pz.clamp(0, b - 1)[None], (pz % b)[None])
        idx = slot[nid] * b ** 3 + cx + b * (cy + b * cz)
        idx = torch.where(k == 2, n * b ** 3, torch.where(k == 3, n * b ** 3 + 1, idx))
        return idx

    index = [tile_index(s) for _, s in groups] if n * (b + 2) ** 3 < 200_000_000 else None
    for _ in range(c["iters"] + c["iters"] % 2):
        for gi, (col, s) in enumerate(groups):
            t = f[index[gi] if index else tile_index(s)].reshape(-1, b + 2, b + 2, b + 2)
            sh = lambda i, j, k: t[:, 1 + k:b + 1 + k, 1 + j:b + 1 + j, 1 + i:b + 1 + i]  # noqa
            c0 = sh(0, 0, 0)
            fx = 0.5 * (sh(1, 0, 0) - sh(-1, 0, 0))
            fy = 0.5 * (sh(0, 1, 0) - sh(0, -1, 0))
            fz = 0.5 * (sh(0, 0, 1) - sh(0, 0, -1))
            fxx = sh(1, 0, 0) + sh(-1, 0, 0) - 2 * c0
            fyy = sh(0, 1, 0) + sh(0, -1, 0) - 2 * c0
            fzz = sh(0, 0, 1) + sh(0, 0, -1) - 2 * c0
            fxy = 0.25 * (sh(1, 1, 0) - sh(1, -1, 0) - sh(-1, 1, 0) + sh(-1, -1, 0))
            fxz = 0.25 * (sh(1, 0, 1) - sh(1, 0, -1) - sh(-1, 0, 1) + sh(-1, 0, -1))
            fyz = 0.25 * (sh(0, 1, 1) - sh(0, 1, -1) - sh(0, -1, 1) + sh(0, -1, -1))
            g2 = fx * fx + fy * fy + fz * fz
            h = ((fy * fy + fz * fz) * fxx + (fx * fx + fz * fz) * fyy + (fx * fx + fy * fy) * fzz
                 - 2 * (fx * fy * fxy + fx * fz * fxz + fy * fz * fyz))
            h = torch.where(g2 > 1e-7, h / g2.clamp_min(1e-300), 0.0)
            u = c0 + (0.1 * h).clamp(-0.1, 0.1)
            if c["clamp"]:
                u = u.clamp(0.0, 1.0)
            f[:-2].reshape(n, -1)[s] = u.reshape(len(s), -1)
    return f[:-2].reshape(n, b, b, b)


def _exact_solve(c, seed):
    """The finite-volume system of the packed cells, solved by Jacobi-preconditioned CG."""
    if c["res"] > 320:
        return None
    scene, flags, face, rhs = _pressure_input(c, seed)
    dev, b0 = "cuda" if torch.cuda.is_available() else "cpu", c["bsx0"]
    lev = torch.from_numpy(scene.block_levels.astype(np.int64)).to(dev)
    nb = c["res"] // b0
    size = (b0 >> lev) ** 3
    off = torch.cumsum(size, 0) - size
    n = int(size.sum())
    fluid = torch.from_numpy((flags & (0x1 | 0x2 | 0x1000)) == 0).to(dev)
    face = [torch.from_numpy(f).to(dev).double() for f in face]
    blk = torch.repeat_interleave(torch.arange(nb ** 3, device=dev), size)
    L = lev[blk]
    bs = b0 >> L
    v = torch.arange(n, device=dev) - off[blk]
    P = [(blk % nb) * bs + v % bs, ((blk // nb) % nb) * bs + (v // bs) % bs,
         (blk // (nb * nb)) * bs + v // (bs * bs)]
    h = (2.0 ** L.double())

    def cell_of(fv):  # the packed cell of a fine voxel, and its level
        b = (fv[0] // b0) + nb * ((fv[1] // b0) + nb * (fv[2] // b0))
        l2 = lev[b]
        q = [(t % b0) >> l2 for t in fv]
        return off[b] + q[0] + (b0 >> l2) * (q[1] + (b0 >> l2) * q[2]), l2

    diag = torch.zeros(n, dtype=torch.float64, device=dev)
    ri, ci, cv = [], [], []

    def couple(i, j, w):  # a face between cells i and j: both diagonals, the entries if liquid
        diag.index_add_(0, i, w)
        diag.index_add_(0, j, w)
        m = fluid[i] & fluid[j] & (w != 0)
        ri.extend([i[m], j[m]])
        ci.extend([j[m], i[m]])
        cv.extend([-w[m], -w[m]])

    for d in range(3):
        lo = [P[k] << L for k in range(3)]
        lo[d] = lo[d] - 1
        at_wall = lo[d] < 0
        diag += torch.where(at_wall, h * face[d], 0.0)
        i = torch.nonzero(~at_wall).reshape(-1)
        j, l2 = cell_of([t[i] for t in lo])
        same = l2 == L[i]
        couple(i[same], j[same], h[i[same]] * face[d][i[same]])
        up = l2 == L[i] + 1  # the lower neighbour is coarser: our own face
        couple(i[up], j[up], 2.0 / 3.0 * h[i[up]] * face[d][i[up]])
        hi = [P[k] << L for k in range(3)]
        hi[d] = (P[d] + 1) << L
        i = torch.nonzero(hi[d] < c["res"]).reshape(-1)
        j, l2 = cell_of([t[i] for t in hi])
        up = l2 == L[i] + 1  # the upper neighbour is coarser: the face it holds
        couple(i[up], j[up], 2.0 / 3.0 * h[i[up]] * face[d][j[up]])
    b = torch.where(fluid, torch.from_numpy(rhs).to(dev).double() * h ** 3, 0.0)
    live = fluid & (diag > 0)
    inv = torch.where(live, 1.0 / diag.clamp_min(1e-300), 0.0)
    row, col, w = torch.cat(ri), torch.cat(ci), torch.cat(cv)
    A = torch.sparse_coo_tensor(torch.stack([row, col]), w, (n, n)).coalesce().to_sparse_csr()
    dg = torch.where(live, diag, 0.0)
    x = torch.zeros(n, dtype=torch.float64, device=dev)
    r = torch.where(live, b, 0.0)
    z = inv * r
    p = z.clone()
    rz, bb = torch.dot(r, z), float(torch.dot(r, r))
    for it in range(6000):
        q = dg * p + A @ p
        a = rz / torch.dot(p, q)
        x += a * p
        r -= a * q
        if it % 25 == 24 and float(torch.dot(r, r)) <= 1e-20 * bb:
            break
        z = inv * r
        rz2 = torch.dot(r, z)
        p = z + (rz2 / rz) * p
        rz = rz2
    return x


_OFF = ((0.0, 0.5, 0.5), (0.5, 0.0, 0.5), (0.5, 0.5, 0.0))


def _corners(pos, d):
    g = pos - torch.tensor(_OFF[d], dtype=torch.float64, device=pos.device)
    i0 = torch.floor(g).long()
    f = g - i0
    for k in range(8):
        o = torch.tensor([k & 1, (k >> 1) & 1, k >> 2], device=pos.device)
        w = torch.where(o.bool(), f, 1 - f).prod(1)
        yield i0 + o, w


def _exact_flip(c, seed):
    p, pres = _flip_particles(c, seed)
    res, b = c["res"], c["bsx"]
    if len(p) > 20_000_000:
        return None
    n, nb = res ** 3, res // b
    pos, vel, phase = p[:, :3].double(), p[:, 3:6].double(), p.view(torch.int32)[:, 6]
    rl, rg, eps, bmin = 1000.0, 1.0, 1e-5, 1e-6

    def scatter(i, w):
        ok = ((i >= 0) & (i < res)).all(1)
        i = i[ok]
        return i[:, 0] + res * (i[:, 1] + res * i[:, 2]), ok

    zero = lambda: torch.zeros(n, dtype=torch.float64, device="cuda")  # noqa: E731
    mass, liq = zero(), zero()
    ci, ok = scatter(torch.floor(pos).long(), None)
    mass.index_add_(0, ci, torch.ones(len(ci), dtype=torch.float64, device="cuda"))
    liq.index_add_(0, ci, (phase[ok] == 0).double())
    mp = torch.where(phase == 0, rl, rg).double()
    cube = lambda t: t.reshape(res, res, res)  # noqa: E731
    ph = torch.where(mass > eps, torch.where(liq * 2 > torch.floor(mass + 0.5), 0, 1), -1)
    V, B = [], []
    rt0 = 8.0
    rmin, den = math.log(rl / rg) * rg * rt0, 1.0 * rt0 * rl

    def lower(t, d, fill):  # the value of the cell below in direction d
        t = cube(t)
        s = torch.full_like(t, fill)
        ax = 2 - d
        s.narrow(ax, 1, res - 1).copy_(t.narrow(ax, 0, res - 1))
        return s.reshape(-1)

    for d in range(3):
        v, w, r = zero(), zero(), zero()
        for i, wt in _corners(pos, d):
            k, ok = scatter(i, None)
            v.index_add_(0, k, vel[ok, d] * wt[ok])
            w.index_add_(0, k, wt[ok])
            r.index_add_(0, k, mp[ok] * wt[ok])
        V.append(torch.where(w > eps, v / w.clamp_min(1e-300), 0.0))
        phi = torch.where(r < rmin, 0.0, ((r - rmin).clamp_min(0) / den).sqrt().clamp_max(1.0))
        pa = lower(ph, d, -1)
        phi = torch.where((pa == 0) & (ph == 0), 1.0, phi)
        phi = torch.where((pa == 1) & (ph == 1), 0.0, phi)
        B.append((1.0 / (rg + phi * (rl - rg))).clamp_min(bmin))
    # block layout: bid order, x fastest inside a block
    def blocked(t):
        return t.reshape(nb, b, nb, b, nb, b).permute(0, 2, 4, 1, 3, 5).reshape(-1)

    chans = [torch.stack([blocked(t) for t in V], 1).reshape(-1),
             torch.stack([blocked(t) for t in B], 1).reshape(-1), blocked(mass)]
    old = [t.clone() for t in V]
    wet = mass > eps
    V[1] = torch.where(wet | lower(wet, 1, False), V[1] + GRAVITY * DT, V[1])
    for d, both in ((0, True), (1, False), (2, True)):
        t, ax = cube(V[d]), 2 - d
        t.select(ax, 0).zero_()
        if both:
            t.select(ax, res - 1).zero_()
    pr = pres.double().reshape(nb, nb, nb, b, b, b).permute(0, 3, 1, 4, 2, 5).reshape(-1)
    pr = torch.where(wet, pr, 0.0)
    for d in range(3):
        any_ = wet | lower(wet, d, False)
        t = torch.where(any_, V[d] - DT * B[d] * (pr - lower(pr, d, 0.0)), 0.0)
        cube(t).select(2 - d, 0).zero_()
        V[d] = t
    out = torch.empty(len(p), 3, dtype=torch.float64, device="cuda")
    for d in range(3):
        pic = torch.zeros(len(p), dtype=torch.float64, device="cuda")
        o = pic.clone()
        for i, wt in _corners(pos, d):
            k, ok = scatter(i, None)
            pic[ok] += wt[ok] * V[d][k]
            o[ok] += wt[ok] * old[d][k]
        out[:, d] = (1 - ALPHA) * pic + ALPHA * (vel[:, d] + pic - o)
    return [out] + (chans if c["channels"] else [])


def _exact_g2p_mr(c, seed):
    lev, vel, old, p = _mr_input(c, seed)
    res, b0, nl, dev = c["res"], c["bsx"], c["levels"], "cuda"
    nb = res // b0
    lev = torch.from_numpy(lev.astype(np.int64)).to(dev)
    size = (b0 >> lev) ** 3
    off = torch.cumsum(size, 0) - size
    cube = lev.reshape(1, 1, nb, nb, nb).double()
    coarse = torch.nn.functional.max_pool3d(cube, 3, 1, 1).reshape(-1) > lev  # next to coarser
    kind = []
    for l in range(nl):
        val = (lev == l) & coarse
        near = torch.nn.functional.max_pool3d(val.reshape(1, 1, nb, nb, nb).double(), 3, 1,
                                              1).reshape(-1) > 0
        kind.append(torch.where(val, 1, torch.where(near & ((lev == l) | (lev == l - 1)), 2, 0)))

    def dist_at(l, q):  # raw distance of level-l voxels q inside the grid
        bs = b0 >> l
        b = q // bs
        bid = b[:, 0] + nb * (b[:, 1] + nb * b[:, 2])
        k = kind[l][bid]
        d2 = torch.full((len(q),), 1e20, dtype=torch.float64, device=dev)
        for o in range(27):
            o3 = torch.tensor([o % 3 - 1, (o // 3) % 3 - 1, o // 9 - 1], device=dev)
            nbk = b + o3
            ok = ((nbk >= 0) & (nbk < nb)).all(1)
            nid = (nbk.clamp(0, nb - 1) * torch.tensor([1, nb, nb * nb], device=dev)).sum(1)
            ok &= lev[nid] > l
            ctr = q.double() + 0.5
            lo, hi = nbk.double() * bs, (nbk.double() + 1) * bs
            e = torch.maximum((lo - ctr).clamp_min(0), ctr - hi)
            d2 = torch.where(ok, torch.minimum(d2, e.square().sum(1)), d2)
        raw = torch.floor(d2.sqrt().clamp_max(6.0) * 1024.0)
        return torch.where(k == 1, raw, torch.where(k == 2, 6144.0, 0.0))

    def grid(l, q, ch, d):  # component d of the channels at level-l voxels q
        ok = ((q >= 0) & (q < (res >> l))).all(1)
        q = q.clamp(0, (res >> l) - 1)
        bs = b0 >> l
        b = q // bs
        bid = b[:, 0] + nb * (b[:, 1] + nb * b[:, 2])
        ok &= lev[bid] == l
        v = q % bs
        i = torch.where(ok, off[bid] + v[:, 0] + bs * (v[:, 1] + bs * v[:, 2]), 0)
        return [torch.where(ok, t[3 * i + d].double(), 0.0) for t in ch]

    sq3 = float(np.float32(1.73205080756887))
    la = float(np.float32(np.float32(sq3) * np.float32(1.01)))
    lb = float(np.float32(np.float32(0.99) * np.float32(8.0)) / np.float32(sq3))
    out = torch.empty(len(p), 3, dtype=torch.float64, device=dev)
    for i0 in range(0, len(p), 2_000_000):
        pp = p[i0:i0 + 2_000_000]
        pos = pp[:, :3].double()
        for d in range(3):
            # the sample's position as the call takes it, in FP32
            g = (pp[:, :3] - torch.tensor(_OFF[d], device=dev)).double()
            cell = torch.floor(g).long().clamp(0, res - 1) // b0
            lv = lev[cell[:, 0] + nb * (cell[:, 1] + nb * cell[:, 2])]

            def tri(l, q):
                c0 = torch.floor(q).long()
                f = q - c0
                s = [torch.zeros(len(q), dtype=torch.float64, device=dev) for _ in range(2)]
                for k in range(8):
                    o = torch.tensor([k & 1, (k >> 1) & 1, k >> 2], device=dev)
                    w = torch.where(o.bool(), f, 1 - f).prod(1)
                    for t, u in zip(s, grid(l, c0 + o, (vel, old), d)):
                        t += w * u
                return s

            pic, ol = tri(0, g)
            for l in range(1, nl):
                m = torch.nonzero(lv == l).reshape(-1)
                if not len(m):
                    continue
                q = g[m] / 2 ** l
                cp, co = tri(l, q)
                c0 = torch.floor(q - 0.5).long()
                f = q - 0.5 - c0
                dd = torch.zeros(len(m), dtype=torch.float64, device=dev)
                for k in range(8):
                    o = torch.tensor([k & 1, (k >> 1) & 1, k >> 2], device=dev)
                    w = torch.where(o.bool(), f, 1 - f).prod(1)
                    dd += w * dist_at(l, (c0 + o).clamp(0, (res >> l) - 1))
                af = ((dd / 1024.0 - la) / (lb - la)).clamp(0.0, 1.0)
                pic[m] = af * pic[m] + (1 - af) * cp
                ol[m] = af * ol[m] + (1 - af) * co
            out[i0:i0 + len(pp), d] = ((1 - ALPHA) * pic +
                                       ALPHA * (pp[:, 3 + d].double() + pic - ol))
    return out


def _exact_cnn(c, seed):
    feat, tgt, mask, w = _cnn_input(c, seed)
    w = [x.cuda().double().requires_grad_(c["train"]) for x in w]
    n, outs, loss = c["tiles"], [], 0.0
    count = float(mask.sum().item())
    cv = torch.nn.functional.conv3d
    with torch.backends.cudnn.flags(enabled=False):
        for i in range(0, n, 32):
            x = feat[i:i + 32].double().reshape(-1, 4, 18, 18, 18)
            y = torch.relu(cv(x, w[0]))
            for k in (1, 2):
                y = torch.relu(cv(y, w[k], padding=1))
            y = cv(y, w[3], padding=1).reshape(len(x), -1)
            if not c["train"]:
                outs.append(y)
                continue
            e = (mask[i:i + 32].double() * (y - tgt[i:i + 32].double()).square()).sum() / count
            e.backward()
            loss += float(e.detach())
    if not c["train"]:
        return torch.cat(outs)
    g = torch.cat([x.grad.reshape(-1) for x in w])
    return [loss, g, None]


def exact(case, seed):
    return {"mcf": _exact_mcf, "solve": _exact_solve, "step": _exact_solve, "flip": _exact_flip,
            "g2p_mr": _exact_g2p_mr, "splat": lambda c, s: None,
            "cnn": _exact_cnn}[case["kind"]](case, seed)
