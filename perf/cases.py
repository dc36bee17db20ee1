"""Performance cases of the water-surface path, each one pass through the
package's public entry points as a renderer, a simulation or a fit calls them.

The sizes are those of this repository's own configurations (workloads.py),
tests and benchmark; `draw` spreads the same kinds of work over their ranges.

Two things about what is returned.  The noise layer is sampled bilinearly, so
its slope, and with it the surface normal, jumps at texel edges: a last-bit
change of the sampled point moves a normal there by the whole jump, which
measures the texel cell and not the arithmetic.  So the patch cases that carry
the layer are position-only calls (`normals=False`, what a buoyancy query or a
depth pass asks for), the cases that return normals over regular patches have
no layer, and layer and normals come together on skewed patches and in the
frames.  NDC at height 0 divides by a w that passes through zero, and the
camera-facing normal changes sign, so `exact` has no value for those.
"""
import importlib
import math

import numpy as np
import torch

wt = importlib.import_module("wave-tool_gb300")

G = 9.81
STAGE = ("clip", "ndc0", "view", "facing", "nrm_yaw")


def listed():
    return [
        # the reference-sized call, four waves on one small grid: launch latency
        dict(name="grid_128x4", kind="grid", cols=128, rows=128, waves=4, extent=200.0, t=100.0, layer=False, flags=0),
        # one scene patch with a full spectrum
        dict(name="grid_1024x32", kind="grid", cols=1024, rows=1024, waves=32, extent=200.0, t=100.0, layer=False,
             flags=0),
        # the precision configuration: many waves, long run times, displacement
        # output in the vertex array's packed layout
        dict(name="grid_2048x128", kind="grid", cols=2048, rows=2048, waves=128, extent=409.4, t=1.0e4, layer=False,
             flags=wt.WT_OUT_DISPLACEMENT | wt.WT_LAYOUT_VEC3),
        # the batched ocean: 256 uneven patches, 8..64 waves, normals
        dict(name="ocean_256", kind="ocean", patches=256, lo=64, hi=1024, layer=False, flags=0),
        # the same with the 512^2 noise layer, positions only (buoyancy, depth pass)
        dict(name="ocean_256_noise", kind="ocean", patches=256, lo=64, hi=1024, layer=True, flags=0),
        # ragged skewed patches (no parallelograms), odd sizes, mirrored layer, normals
        dict(name="skewed_48_noise", kind="skewed", patches=48, lo=2, hi=400, tex=37, flags=wt.WT_OUT_DISPLACEMENT),
        # one training step of the wave fit: saving forward and adjoint under autograd
        dict(name="fit_512x16", kind="fit", cols=512, rows=512, waves=16, flags=wt.WT_OUT_DISPLACEMENT),
        # gradients of a batch without a saved forward
        dict(name="adjoint_64", kind="adjoint", patches=64, lo=64, hi=1024, flags=0),
        # the reference's own frame grid: 513^2, four waves, camera to vertex-stage outputs
        dict(name="frame_513x4", kind="frame", side=513, waves=4, pitch=-12.0, yaw=-90.0, height=4.0),
        # the benchmark's frame grid
        dict(name="frame_1024x32", kind="frame", side=1024, waves=32, pitch=-20.0, yaw=-90.0, height=4.0),
        # the water draw at 1080p: rasterisation and shading of that grid
        dict(name="draw_1080p", kind="draw", side=1024, waves=32, pitch=-20.0, yaw=-90.0, height=4.0, width=1920,
             rows=1080, depth=False),
        # the noise layer resynthesised at the frame time
        dict(name="noise_512x64", kind="noise", width=512, rows=512, terms=64, kmax=32, t=12.5),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _size(rng, lo, hi):
    return max(lo, min(hi, int(round(_log(rng, lo, hi)))))


def draw(rng):
    kind = rng.choice(["grid", "grid", "ocean", "ocean", "skewed", "fit", "adjoint", "frame", "draw", "noise"])
    if kind == "grid":
        return dict(kind=kind, cols=_size(rng, 16, 2048), rows=_size(rng, 16, 2048), waves=_size(rng, 1, 128),
                    extent=_log(rng, 20.0, 400.0), t=_log(rng, 1.0, 1.0e4), layer=rng.random() < 0.3,
                    flags=rng.choice([0, 1, 2, 3]))
    if kind == "ocean":
        return dict(kind=kind, patches=_size(rng, 4, 224), lo=64, hi=_size(rng, 128, 1024), layer=rng.random() < 0.4,
                    flags=rng.choice([0, 1, 2, 3]))
    if kind == "skewed":
        return dict(kind=kind, patches=_size(rng, 4, 64), lo=2, hi=_size(rng, 40, 512), tex=_size(rng, 3, 128),
                    flags=rng.choice([0, 1]))
    if kind == "fit":
        return dict(kind=kind, cols=_size(rng, 32, 1024), rows=_size(rng, 32, 1024), waves=_size(rng, 1, 64),
                    flags=rng.choice([1, 3]))
    if kind == "adjoint":
        return dict(kind=kind, patches=_size(rng, 1, 60), lo=64, hi=_size(rng, 128, 1024), flags=rng.choice([0, 2]))
    view = dict(pitch=rng.uniform(-30.0, -8.0), yaw=rng.uniform(-180.0, 180.0), height=rng.uniform(3.0, 12.0))
    if kind == "frame":
        return dict(kind=kind, side=_size(rng, 65, 1025), waves=_size(rng, 1, 64), **view)
    if kind == "draw":
        return dict(kind=kind, side=_size(rng, 129, 1025), waves=_size(rng, 4, 32), width=_size(rng, 320, 2560),
                    rows=_size(rng, 200, 1440), depth=rng.random() < 0.5, **view)
    return dict(kind=kind, width=_size(rng, 64, 2048), rows=_size(rng, 64, 2048), terms=_size(rng, 4, 128),
                kmax=rng.choice([4, 32]), t=_log(rng, 0.1, 1.0e4))


# ---- inputs ------------------------------------------------------------------

def _waves(rs, n, count=None, lam=(0.5, 60.0)):
    """n waves of the wide spectrum: lambda log-uniform, A = lambda / 100 *
    U[0.5, 1], within 90 degrees of the wind, deep-water speed."""
    l = np.exp(rs.uniform(math.log(lam[0]), math.log(lam[1]), n))
    a = l / 100.0 * rs.uniform(0.5, 1.0, n)
    ang = np.radians(rs.uniform(-90.0, 90.0, n))
    k = 2.0 * math.pi / l
    w = np.zeros(n, wt.WAVE_DTYPE)
    w["amplitude"], w["wavelength"] = a, l
    w["dir_x"], w["dir_z"] = np.cos(ang), np.sin(ang)
    w["steepness_q"] = 0.5 / (k * a * (count or n))
    w["speed"] = np.sqrt(G / k)
    w["phase"] = rs.uniform(0.0, 2.0 * math.pi, n)
    return w


def _patch(cx, cz, hx, hz, cols, rows, w0, n, t, out):
    p = np.zeros(1, wt.PATCH_DTYPE)
    p["bl"], p["br"], p["tl"], p["tr"] = (cx - hx, cz + hz), (cx + hx, cz + hz), (cx - hx, cz - hz), (cx + hx, cz - hz)
    p["cols"], p["rows"], p["wave_offset"], p["wave_count"] = cols, rows, w0, n
    p["time_s"], p["out_offset"] = t, out
    return p


def _terms(rs, n=64, kmax=32):
    t = np.zeros(n, wt.NOISE_TERM_DTYPE)
    for i in range(n):
        r2 = 0
        while r2 == 0 or r2 > kmax * kmax:
            kx, ky = rs.randint(-kmax, kmax + 1), rs.randint(-kmax, kmax + 1)
            r2 = kx * kx + ky * ky
        t[i] = (kx, ky, rs.uniform(0.5, 1.0) / math.sqrt(r2), rs.uniform(0.0, 2.0 * math.pi))
    return t


def _noise64(terms, width, height, rates=None, t=0.0):
    """The noise layer in 64 bits: the sum of sinusoids mapped to [0, 1]."""
    f = dict(dtype=torch.float64, device="cuda")
    i, j = torch.arange(width, **f)[None, :], torch.arange(height, **f)[:, None]
    h = torch.zeros((height, width), **f)
    for m in range(len(terms)):
        kx, ky, a, ph = (float(v) for v in terms[m])
        turn = 2.0 * math.pi * ((kx * i / width) % 1.0 + (ky * j / height) % 1.0)
        shift = ph + (float(rates[m]) * t if rates is not None else 0.0)
        h += a * torch.sin(turn + math.fmod(shift, 2.0 * math.pi))
    return (h - h.min()) / (h.max() - h.min())


def _layer(texels, sample_scale, disp_scale, wrap=0):
    return wt.DeviceHeightmap(texels.cuda(), sample_scale, disp_scale, wrap)


def _inputs(case, seed):
    """Host tables (patches, waves) and the layer (texels, scales, wrap) of a
    patch case."""
    rs = np.random.RandomState(seed % (1 << 32))
    kind = case["kind"]
    hm = None
    if kind in ("grid", "fit"):
        n = case["waves"]
        extent, t, lam = (case["extent"], case["t"], (0.5, 60.0)) if kind == "grid" else (100.0, 10.0, (1.0, 30.0))
        waves = _waves(rs, n, lam=lam)
        cx, cz = (rs.uniform(-50.0, 50.0), rs.uniform(-50.0, 50.0)) if kind == "grid" else (0.0, 0.0)
        hz = 0.5 * extent * case["rows"] / max(case["cols"], case["rows"])
        hx = 0.5 * extent * case["cols"] / max(case["cols"], case["rows"])
        patches = _patch(cx, cz, hx, hz, case["cols"], case["rows"], 0, n, t, 0)
    elif kind in ("ocean", "adjoint"):
        per_row = int(math.ceil(math.sqrt(case["patches"])))
        rows, ws, out, w0 = [], [], 0, 0
        # the batch's sizes do not depend on the seed, so that every state of a case is the same work
        sizes = np.random.RandomState(case["patches"] * 1031 + case["hi"])
        for i in range(case["patches"]):
            side = int(round(math.exp(sizes.uniform(math.log(case["lo"]), math.log(case["hi"])))))
            n = sizes.randint(8, 65)
            half = 0.5 * (side - 1) * 0.2
            rows.append(_patch((i % per_row) * 256.0, (i // per_row) * 256.0, half, half, side, side, w0, n,
                               rs.uniform(0.0, 1.0e3), out))
            ws.append(_waves(rs, n))
            out, w0 = out + side * side, w0 + n
        patches, waves = np.concatenate(rows), np.concatenate(ws)
    else:  # skewed
        sizes = np.random.RandomState(case["patches"] * 1031 + case["hi"])
        rows, ws, out, w0 = [], [], 0, 0
        for i in range(case["patches"]):
            cols, rws = (int(sizes.randint(case["lo"], case["hi"] + 1)) for _ in range(2))
            n = int(sizes.randint(0, 41))
            hx, hz = 0.5 * (cols - 1) * 0.37, 0.5 * (rws - 1) * 0.37
            p = _patch(rs.uniform(-3000, 3000), rs.uniform(-3000, 3000), hx, hz, cols, rws, w0, n,
                       rs.uniform(0.0, 5.0e3), out)
            for c in ("bl", "br", "tl", "tr"):
                p[c] += rs.uniform(-0.2, 0.2, (1, 2)) * hx
            p["y_offset"] = rs.uniform(-0.1, 0.1)
            rows.append(p)
            ws.append(_waves(rs, n, max(n, 1)))
            out, w0 = out + cols * rws, w0 + n
        patches, waves = np.concatenate(rows), np.concatenate(ws + [_waves(rs, 1)])
        tex = torch.from_numpy(rs.uniform(0.0, 1.0, (case["tex"], case["tex"])).astype(np.float32))
        hm = (tex, rs.uniform(0.01, 0.3), rs.uniform(0.05, 0.5), wt.WT_WRAP_MIRRORED_REPEAT)
    if case.get("layer"):
        hm = (_noise64(_terms(rs), 512, 512).float(), 0.02, 0.2, wt.WT_WRAP_REPEAT)
    return patches, waves, hm


def _vertices(p):
    return int(p["cols"]) * int(p["rows"])


def _residual(case, seed, patches, waves):
    """Upstream gradients of an L2 height + normal loss, as the wave fit has
    them: the difference of the surface to that of a perturbed wave set."""
    rs = np.random.RandomState((seed + 77) % (1 << 32))
    other = waves.copy()
    for f in ("amplitude", "wavelength", "steepness_q"):
        other[f] *= rs.uniform(0.9, 1.1, len(waves)).astype(np.float32)
    other["phase"] += rs.uniform(-0.5, 0.5, len(waves)).astype(np.float32)
    n = sum(_vertices(p) for p in patches)
    width = 3 if case["flags"] & wt.WT_LAYOUT_VEC3 else 4
    gpos = torch.zeros((n, width), device="cuda")
    gnrm = torch.zeros((n, width), device="cuda")
    for p in patches:
        o, m = int(p["out_offset"]), _vertices(p)
        a = _surface(p, _fields(waves, p, torch.float32), None, torch.float32)
        b = _surface(p, _fields(other, p, torch.float32), None, torch.float32)
        gpos[o:o + m, 1] = (2.0 / n) * (a[0][:, 1] - b[0][:, 1])
        gnrm[o:o + m, :3] = (2.0 / n) * (a[1] - b[1])
    return gpos, gnrm


def _camera_args(case, amp):
    return dict(position=(0.0, case["height"], 70.0), yaw_deg=case["yaw"], pitch_deg=case["pitch"], aspect=16.0 / 9.0,
                displaceable_amplitude=amp)


def _frame_inputs(case, seed):
    rs = np.random.RandomState(seed % (1 << 32))
    n = case["waves"]
    waves = _waves(rs, n)
    side = case["side"]
    patches = _patch(0.0, 0.0, 100.0, 100.0, side, side, 0, n, rs.uniform(0.0, 1.0e3), 0)
    tex = _noise64(_terms(rs), 512, 512).float()
    amp = float(np.sum(waves["amplitude"].astype(np.float64))) + 0.2
    return patches, waves, (tex, 0.02, 0.2, wt.WT_WRAP_REPEAT), _camera_args(case, amp)


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("grid", "ocean", "skewed"):
        patches, waves, hm = _inputs(case, seed)
        surf = wt.Surface(patches, waves, _layer(*hm) if hm else None)
        pos, nrm = surf.alloc_outputs(case["flags"], normals=not case.get("layer"))
        return dict(kind=kind, surf=surf, pos=pos, nrm=nrm, flags=case["flags"])
    if kind in ("fit", "adjoint"):
        patches, waves, _ = _inputs(case, seed)
        surf = wt.Surface(patches, waves)
        gpos, gnrm = _residual(case, seed, patches, waves)
        fit = importlib.import_module("wave-tool_gb300.fit")
        fields = fit.waves_to_fields(waves).requires_grad_(kind == "fit")
        return dict(kind=kind, surf=surf, gpos=gpos, gnrm=gnrm, flags=case["flags"], fields=fields,
                    fn=fit.GerstnerFunction)
    if kind == "frame":
        patches, waves, hm, cam = _frame_inputs(case, seed)
        c = wt.camera(**cam)
        _, view, _ = wt.projected_grid(c, patches)
        surf = wt.Surface(patches, waves, _layer(*hm))
        out = {k: torch.empty((surf.n_vertices, 2 if k == "ndc0" else 4), device="cuda") for k in STAGE}
        return dict(kind=kind, surf=surf, cam=wt.to_device(c), view=wt.to_device(view), out=out)
    if kind == "draw":
        W, H, side = case["width"], case["rows"], case["side"]
        stage = {k: v.float().contiguous() for k, v in _frame64(case, seed).items()}
        g = torch.Generator(device="cuda").manual_seed(seed)
        byte = lambda *s: torch.randint(0, 256, s, dtype=torch.uint8, device="cuda", generator=g)  # noqa: E731
        idx = wt.grid_indices(side, side)
        n = side * side
        return dict(kind=kind, stage=stage, idx=idx, W=W, H=H, sky=byte(6, 256, 256, 4), refl=byte(H, W, 4),
                    refr=byte(H, W, 4),
                    depth=torch.rand((H, W), device="cuda", generator=g) * 0.015 + 0.985 if case["depth"] else None,
                    frags=torch.empty((H, W), dtype=torch.int64, device="cuda"),
                    ws=wt.empty_bytes(wt.water_raster_workspace_bytes(n, idx.numel() // 3)),
                    colour=torch.empty((H, W, 4), device="cuda"),
                    shading=wt.water_shading(sun_position=(0.6, 0.8, 0.0)))
    rs = np.random.RandomState(seed % (1 << 32))
    terms = _terms(rs, case["terms"], case["kmax"])
    rates = rs.uniform(-2.0, 2.0, len(terms)).astype(np.float32)
    return dict(kind=kind, terms=wt.to_device(terms), rates=torch.from_numpy(rates).cuda(), t=case["t"],
                W=case["width"], H=case["rows"], out=torch.empty((case["rows"], case["width"]), device="cuda"),
                ws=wt.empty_bytes(wt.noise_workspace_bytes(len(terms), case["width"], case["rows"])))


def run(s):
    kind = s["kind"]
    if kind in ("grid", "ocean", "skewed"):
        pos, nrm = s["surf"].displace(s["pos"], s["nrm"], flags=s["flags"])
        return {"pos": pos} if nrm is None else {"pos": pos, "nrm": nrm}
    if kind == "fit":
        pos, nrm = s["fn"].apply(s["fields"], s["surf"], s["flags"])
        grad, = torch.autograd.grad([pos, nrm], [s["fields"]], [s["gpos"], s["gnrm"]])
        return {"pos": pos, "nrm": nrm, "grad": grad}
    if kind == "adjoint":
        return {"grad": s["surf"].adjoint(s["gpos"], s["gnrm"], flags=s["flags"])}
    if kind == "frame":
        wt.projected_grid_async(s["cam"], s["surf"].patches, s["view"])
        return dict(s["surf"].displace_stage(s["view"], out=s["out"]))
    if kind == "draw":
        st = s["stage"]
        wt.water_raster(st["clip"], s["idx"], s["W"], s["H"], scene_depth=s["depth"], fragments=s["frags"],
                        workspace=s["ws"])
        wt.water_shade(s["frags"], st["clip"], s["idx"], st, s["W"], s["H"], s["shading"], s["sky"],
                       scene_depth=s["depth"], local_reflections=s["refl"], local_refractions=s["refr"],
                       colour=s["colour"])
        return {"fragments": s["frags"], "colour": s["colour"]}
    return {"texels": wt.noise_synth(s["terms"], s["W"], s["H"], rates=s["rates"], time_s=s["t"], out=s["out"],
                                     workspace=s["ws"])}


# ---- the work a pass cannot do without ------------------------------------------

def work(case):
    kind = case["kind"]
    if kind == "noise":
        px = case["width"] * case["rows"]
        return {"bytes": 4 * px + 20 * case["terms"], "flops": 4 * px * case["terms"]}
    if kind in ("frame", "draw"):
        n = case["side"] ** 2
        if kind == "frame":  # a term: 2 FMA of recurrence and 8 of sums
            return {"bytes": 72 * n + 4 * 512 * 512, "flops": n * (20 * case["waves"] + 150)}
        px = case["width"] * case["rows"]
        tri = 2 * (case["side"] - 1) ** 2
        return {"bytes": 72 * n + 12 * tri + px * (8 + 16 + 8), "flops": 60 * tri + 300 * px}
    patches, waves, hm = _inputs(dict(case, layer=False), 0)
    terms = sum(_vertices(p) * int(p["wave_count"]) for p in patches)
    n = sum(_vertices(p) for p in patches)
    table = patches.nbytes + waves.nbytes
    width = 12 if case["flags"] & wt.WT_LAYOUT_VEC3 else 16
    if kind == "adjoint":
        return {"bytes": table + 2 * width * n + waves.nbytes, "flops": 64 * terms + 150 * n}
    if kind == "fit":
        return {"bytes": table + 4 * width * n + waves.nbytes, "flops": 64 * terms + 250 * n}
    outs = 1 if case.get("layer") else 2
    return {"bytes": table + outs * width * n + (4 * 512 * 512 if case.get("layer") else 0),
            "flops": 20 * terms + 100 * n}


# ---- the same in 64 bits ---------------------------------------------------------

def _fields(waves, p, dtype):
    o, n = int(p["wave_offset"]), int(p["wave_count"])
    f = np.ascontiguousarray(waves[o:o + n]).view(np.float32).reshape(n, 8)
    return torch.from_numpy(f.copy()).to("cuda", dtype)


def _grid(p, dtype, r0=0, r1=None):
    cols, rows = int(p["cols"]), int(p["rows"])
    r1 = rows if r1 is None else r1
    u = torch.arange(cols, dtype=dtype, device="cuda")[None, :] / (cols - 1)
    v = torch.arange(r0, r1, dtype=dtype, device="cuda")[:, None] / (rows - 1)
    bl, br, tl, tr = ([float(x) for x in p[k]] for k in ("bl", "br", "tl", "tr"))
    return [((1 - v) * ((1 - u) * bl[i] + u * br[i]) + v * ((1 - u) * tl[i] + u * tr[i])).reshape(-1) for i in (0, 1)]


def _wrap(i, n, wrap):
    if wrap == wt.WT_WRAP_MIRRORED_REPEAT:
        a = i % (2 * n) - n
        return n - 1 - torch.where(a >= 0, a, -(1 + a))
    return i % n


def _surface(p, f, hm, dtype, r0=0, r1=None):
    """Displacement (n, 3), unit normal (n, 3) and grid x, z of a patch's rows
    r0..r1: the Gerstner sum, the bilinear layer at the displaced point, the
    bounce, normalize(dP/dz x dP/dx)."""
    x, z = _grid(p, dtype, r0, r1)
    dx, dy, dz, jx, jz, sxx, sxz, szz = (torch.zeros_like(x) for _ in range(8))
    for i in range(f.shape[0]):
        A, lam, Dx, Dz, Q, speed, phase = (f[i, j] for j in range(7))
        k = 2.0 * math.pi / lam
        th = k * (Dx * x + Dz * z) + (speed * k * float(p["time_s"]) + phase)
        c, s = torch.cos(th), torch.sin(th)
        qa, ak = Q * A, A * k
        dx, dy, dz = dx + (qa * Dx) * c, dy + A * s, dz + (qa * Dz) * c
        jx, jz = jx + (ak * Dx) * c, jz + (ak * Dz) * c
        sxx, sxz, szz = sxx + (Q * ak * Dx * Dx) * s, sxz + (Q * ak * Dx * Dz) * s, szz + (Q * ak * Dz * Dz) * s
    px, pz = [1 - sxx, jx, -sxz], [-sxz, jz, 1 - szz]
    if hm is not None:
        tex, scale, disp, wrap = hm
        H, W = tex.shape
        t = tex.to("cuda", dtype).reshape(-1)
        ut, vt = scale * W * (x + dx) - 0.5, -scale * H * (z + dz) - 0.5
        fu, fv = torch.floor(ut), torch.floor(vt)
        a, b = ut - fu, vt - fv
        i0, i1 = _wrap(fu.long(), W, wrap), _wrap(fu.long() + 1, W, wrap)
        j0, j1 = _wrap(fv.long(), H, wrap), _wrap(fv.long() + 1, H, wrap)
        t00, t10, t01, t11 = t[j0 * W + i0], t[j0 * W + i1], t[j1 * W + i0], t[j1 * W + i1]
        r0_, r1_ = t00 + a * (t10 - t00), t01 + a * (t11 - t01)
        dy = dy + 2.0 * disp * (r0_ + b * (r1_ - r0_) - 0.5)
        hx = 2.0 * disp * ((t10 - t00) + b * ((t11 - t01) - (t10 - t00))) * (scale * W)
        hz = -2.0 * disp * (r1_ - r0_) * (scale * H)
        px[1], pz[1] = px[1] + hx * px[0] + hz * px[2], pz[1] + hx * pz[0] + hz * pz[2]
    dy = dy + float(p["y_offset"])
    n = torch.stack([pz[1] * px[2] - pz[2] * px[1], pz[2] * px[0] - pz[0] * px[2], pz[0] * px[1] - pz[1] * px[0]], 1)
    n = n / n.norm(dim=1, keepdim=True)
    return torch.stack([dx, dy, dz], 1), n, x, z


def _lay_out(parts, flags):
    """Per-patch displacements, normals and grid points as the call lays them out."""
    pos, nrm = [], []
    for d, n, x, z in parts:
        world = not flags & wt.WT_OUT_DISPLACEMENT
        q = d + torch.stack([x, torch.zeros_like(x), z], 1) if world else d
        if not flags & wt.WT_LAYOUT_VEC3:
            q = torch.cat([q, torch.full_like(q[:, :1], 1.0 if world else 0.0)], 1)
            n = torch.cat([n, torch.zeros_like(n[:, :1])], 1)
        pos.append(q)
        nrm.append(n)
    return torch.cat(pos), torch.cat(nrm)


def _gradient(p, fields, gpos, gnrm):
    """dL/d(wave fields) of one patch, a few rows at a time."""
    f = fields.detach().clone().requires_grad_(True)
    total = torch.zeros_like(f)
    cols, rows, o = int(p["cols"]), int(p["rows"]), int(p["out_offset"])
    step = max(1, (1 << 18) // cols)
    for r0 in range(0, rows, step):
        r1 = min(rows, r0 + step)
        d, n, _, _ = _surface(p, f, None, torch.float64, r0, r1)
        a, b = o + r0 * cols, o + r1 * cols
        loss = (d * gpos[a:b, :3].double()).sum() + (n * gnrm[a:b, :3].double()).sum()
        total += torch.autograd.grad(loss, f)[0]
    return total


def _unit(v):
    return v / np.linalg.norm(v)


def _projected_grid64(cam):
    """The projected grid (render-engine.cpp:797-1042): corners BL BR TL TR
    (x, z), the view-projection and the yaw-only view matrix, row-major."""
    eye = np.array(cam["position"], np.float64)
    amp, aspect, zn, zf, fov = cam["displaceable_amplitude"], cam["aspect"], 0.1, 100.0, math.radians(72.0)
    yaw, pitch = math.radians(cam["yaw_deg"]), math.radians(cam["pitch_deg"])
    ty = math.tan(fov / 2)
    tx = ty * aspect

    def basis(yaw, sp, cp):
        fwd = _unit(np.array([math.cos(yaw) * cp, sp, math.sin(yaw) * cp]))
        right = np.array([-math.sin(yaw), 0.0, math.cos(yaw)])
        return fwd, right, _unit(np.cross(right, fwd))

    fwd, right, up = basis(yaw, math.sin(pitch), math.cos(pitch))
    ppos = eye.copy()
    if eye[1] < amp + 1.0:
        ppos[1] = amp + 1.0 - eye[1] if eye[1] < 0 else amp + 1.0
    fs = fwd.copy()
    if abs(fs[1]) < 0.001:
        fs[1] = 0.001 if fs[1] >= 0 else -0.001
    ray = fs if (fs[1] < 0) != (eye[1] < 0) else fs * np.array([1.0, -1.0, 1.0])
    aim1 = eye - (eye[1] / ray[1]) * ray
    aim2 = (eye + fwd) * np.array([1.0, 0.0, 1.0])
    d = (1 - abs(fs[1])) * aim2 + abs(fs[1]) * aim1 - ppos
    hz = math.hypot(d[0], d[2])
    r = math.hypot(hz, d[1])
    sp, cp = -abs(d[1]) / r, hz / r
    if cp < math.cos(math.radians(89.0)):
        sp, cp = -math.sin(math.radians(89.0)), math.cos(math.radians(89.0))
    pf, pr, pu = basis(yaw, sp, cp)
    corner = [eye + (1.2 if i & 4 else -1.2) * tx * dep * right + (1.2 if i & 2 else -1.2) * ty * dep * up + dep * fwd
              for i in range(8) for dep in [zf if i & 1 else zn]]
    pts = [c for c in corner if -amp <= c[1] <= amp]
    for i in range(8):
        for bit in (1, 2, 4):
            if not i & bit:
                a, b = corner[i], corner[i | bit]
                for h in (amp, -amp):
                    if a[1] != b[1] and min(a[1], b[1]) <= h <= max(a[1], b[1]):
                        pts.append(a + (h - a[1]) / (b[1] - a[1]) * (b - a))
    q = [np.array([p[0], 0.0, p[2]]) - ppos for p in pts]
    X = [pr.dot(v) / tx / pf.dot(v) for v in q]
    Y = [pu.dot(v) / ty / pf.dot(v) for v in q]
    out = []
    for y in (min(Y), max(Y)):
        for x in (min(X), max(X)):
            v = x * tx * pr + y * ty * pu + pf
            c = ppos - ppos[1] / v[1] * v
            out.append((c[0], c[2]))

    def look(f, s, u):
        m = np.eye(4)
        m[0, :3], m[1, :3], m[2, :3] = s, u, -f
        m[:3, 3] = -m[:3, :3].dot(eye)
        return m

    P = np.zeros((4, 4))
    P[0, 0], P[1, 1], P[2, 2], P[2, 3], P[3, 2] = 1 / tx, 1 / ty, -(zf + zn) / (zf - zn), -2 * zf * zn / (zf - zn), -1.0
    level = look(np.array([math.cos(yaw), 0.0, math.sin(yaw)]), right, np.array([0.0, 1.0, 0.0]))
    return out, P.dot(look(fwd, right, up)), level, eye


def _frame64(case, seed):
    """The vertex-stage outputs of a frame (water-grid.vert:150-193)."""
    patches, waves, hm, cam = _frame_inputs(case, seed)
    corners, vp, level, eye = _projected_grid64(cam)
    for k, c in zip(("bl", "br", "tl", "tr"), corners):
        patches[k] = c
    p = patches[0]
    d, n, x, z = _surface(p, _fields(waves, p, torch.float64), hm, torch.float64)
    f = dict(dtype=torch.float64, device="cuda")
    M, Y = torch.tensor(vp, **f), torch.tensor(level[:3, :3].copy(), **f)
    one = torch.ones_like(x)
    pos = torch.stack([x + d[:, 0], d[:, 1], z + d[:, 2]], 1)
    h0 = torch.stack([pos[:, 0], 0 * one, pos[:, 2], one], 1) @ M.T
    v = torch.tensor(eye, **f)[None, :] - pos
    facing = torch.where((n * v).sum(1, keepdim=True) < 0, -n, n)
    yaw = facing @ Y.T
    pad = lambda a: torch.cat([a, 0 * one[:, None]], 1)  # noqa: E731
    return {"clip": torch.cat([pos, one[:, None]], 1) @ M.T, "ndc0": h0[:, :2] / h0[:, 3:], "view": pad(v),
            "facing": pad(facing), "nrm_yaw": pad(yaw / yaw.norm(dim=1, keepdim=True))}


def exact(case, seed):
    kind = case["kind"]
    if kind in ("grid", "ocean", "skewed"):
        patches, waves, hm = _inputs(case, seed)
        pos, nrm = _lay_out((_surface(p, _fields(waves, p, torch.float64), hm, torch.float64) for p in patches),
                            case["flags"])
        # positions only with the layer on regular patches; on skewed ones its slope jumps at texel edges
        return {"pos": pos} if case.get("layer") else {"pos": pos, "nrm": nrm if kind != "skewed" else None}
    if kind in ("fit", "adjoint"):
        patches, waves, _ = _inputs(case, seed)
        gpos, gnrm = _residual(case, seed, patches, waves)
        if kind == "fit":
            p = patches[0]
            f = _fields(waves, p, torch.float64)
            pos, nrm = _lay_out([_surface(p, f, None, torch.float64)], case["flags"])
            return {"pos": pos, "nrm": nrm, "grad": _gradient(p, f, gpos, gnrm)}
        out = []
        for p in patches:
            f = _fields(waves, p, torch.float64)
            g = _gradient(p, f, gpos, gnrm)
            ang = -f[:, 3] * g[:, 2] + f[:, 2] * g[:, 3]  # with respect to the direction's angle
            out.append(torch.stack([g[:, 0], g[:, 1], ang, g[:, 4], g[:, 6], g[:, 5], g[:, 2], g[:, 3]], 1))
        return {"grad": torch.cat(out)}
    if kind == "frame":
        r = _frame64(case, seed)
        return {k: r[k] if k in ("clip", "view") else None for k in STAGE}
    if kind == "draw":
        return None  # the visibility buffer is whole numbers, and the colours follow from it
    rs = np.random.RandomState(seed % (1 << 32))
    terms = _terms(rs, case["terms"], case["kmax"])
    rates = rs.uniform(-2.0, 2.0, len(terms)).astype(np.float32)
    return {"texels": _noise64(terms, case["width"], case["rows"], rates, case["t"])}
