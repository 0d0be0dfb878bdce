"""Workloads of fastqsl_gb300 by its public entry points, for timing and for
comparing outputs between two versions of the library.

Each case stands for something a user of the package does: the drop-in tracer
kernels the reference's notebooks launch (with the Q assembly and the curl
around them), the field-line polylines their plots draw, and the native Q maps
on resident fields, as single planes, cubes, batches of requests and series of
host fields.  Fields are potential fields of seeded sub-surface charges.

    listed()            the cases
    draw(rng)           one more case of the same ranges
    prepare(case, seed) what the program has in hand before the call
    run(state)          one pass through the public entry points
    work(case)          bytes and flops the pass cannot do without
    exact(case, seed)   the outputs in 64 bits, by plain torch
"""
import math
import time

import numpy as np
import torch

from fastqsl_gb300 import api, params
from fastqsl_gb300.fastqslpy import FastQSL, MagTool, kernels

F32_OUT = ["start_x", "start_y", "start_z", "end_x", "end_y", "end_z", "B_this_x", "B_this_y", "B_this_z",
           "B_start_x", "B_start_y", "B_start_z", "B_end_x", "B_end_y", "B_end_z"]
I32_OUT = ["flag_start", "flag_end", "B_flag"]
FEET = ["start_x", "start_y", "start_z", "end_x", "end_y", "end_z"]


def listed():
    return [
        # the reference's fixed-step tracer as its RK4 notebook runs it: one
        # bottom-plane map of a small box (64^3, 128 x 128 seeds, h = 0.1)
        dict(name="rk4_plane", kind="rk4", nx=64, ny=64, nz=64, n0=128, n1=128, planes=1, z=0.0, s_len=0.1,
             twist=False),
        # the whole 2-D notebook workflow with the adaptive drop-in: trace the
        # bottom plane at twice the grid's resolution, Q, pseudo-lines of the
        # near-in-plane pixels, their trace, their Q, the merge
        dict(name="map_rkf45", kind="map", nx=256, ny=256, nz=128, n0=256, n1=512, tol_coef=0.5),
        # the twist notebook: curl B, then the adaptive drop-in with the twist
        # integral over a few planes inside an odd-sized box
        dict(name="twist_planes", kind="rkf45", nx=251, ny=253, nz=127, n0=201, n1=203, planes=4, z=12.0, s_len=0.25,
             tol_coef=10.0, twist=True),
        # the deviation-vector (Scott) notebook's drop-in kernel on a plane
        dict(name="scott_plane", kind="scott", nx=256, ny=256, nz=128, n0=200, n1=300, tol_coef=1.0),
        # the stretched-grid notebook's drop-in kernel (cells by search)
        dict(name="stretch_plane", kind="stretch", nx=192, ny=160, nz=128, n0=250, n1=300, tol_coef=1.0, uni=False,
             native=False),
        # field lines for a plot: 300 polylines of up to 10^4 points
        dict(name="polylines", kind="lines", nx=160, ny=144, nz=96, n=300, maxstep=10000),
        # a quick look: a 100 x 100 map in a small box on the native path
        dict(name="q_small", kind="qmap", layout="h4b", nx=64, ny=64, nz=64, n0=100, n1=100, planes=1, tol=1e-4,
             twist=False, hybrid=False),
        # a production 2-D map: one plane at twice the grid's resolution
        dict(name="q_plane", kind="qmap", layout="h4b", nx=256, ny=256, nz=128, n0=258, n1=514, planes=1, tol=1e-4,
             twist=False, hybrid=False),
        # Q and twist together on the float32 store, odd ragged sizes
        dict(name="q_twist_f4", kind="qmap", layout="f4", nx=201, ny=173, nz=97, n0=131, n1=147, planes=12, tol=1e-4,
             twist=True, hybrid=False),
        # the Q cube: every cell of a 256 x 256 x 128 sub-box of a 512 x 512 x
        # 256 field on the fp16 brick store
        dict(name="q_cube", kind="qmap", layout="h4b", nx=512, ny=512, nz=256, n0=258, n1=258, planes=128, tol=1e-4,
             twist=False, hybrid=False),
        # two small requests of a server as one native batch, built per pass
        # because each batch holds newly arrived requests
        dict(name="requests", kind="requests", nx=384, ny=384, nz=256, n=2, seeds=17000, tol=1e-4),
        # a series of host fields (time steps of a simulation): upload, pack,
        # Q map of one plane each, Q back to the host
        dict(name="series", kind="series", nx=256, ny=256, nz=128, n0=130, n1=258, planes=1, fields=2, tol=1e-4),
    ]


def _size(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _box(rng, lo, hi):
    nx = _size(rng, lo, hi)
    return dict(nx=nx, ny=max(lo // 2, int(nx * rng.uniform(0.7, 1.2))), nz=max(lo // 2, int(nx * rng.uniform(0.45, 1.0))))


def draw(rng):
    kind = rng.choice(["rk4", "map", "rkf45", "scott", "stretch", "lines", "qmap", "qmap", "qmap", "requests", "series"])
    tol = rng.choice([1e-3, 1e-4, 1e-5])
    if kind == "rk4":
        return dict(kind=kind, **_box(rng, 48, 160), n0=_size(rng, 40, 200), n1=_size(rng, 40, 200), planes=1,
                    z=rng.choice([0.0, 8.5]), s_len=rng.choice([0.1, 0.25, 1.0]), twist=rng.choice([False, True]))
    if kind == "map":
        return dict(kind=kind, **_box(rng, 64, 320), n0=_size(rng, 60, 600), n1=_size(rng, 60, 600),
                    tol_coef=rng.choice([0.5, 1.0, 10.0]))
    if kind == "rkf45":
        return dict(kind=kind, **_box(rng, 64, 300), n0=_size(rng, 60, 400), n1=_size(rng, 60, 400),
                    planes=rng.randint(1, 8), z=rng.uniform(4.0, 14.0), s_len=0.25, tol_coef=rng.choice([1.0, 10.0]),
                    twist=rng.choice([False, True]))
    if kind == "scott":
        return dict(kind=kind, **_box(rng, 64, 256), n0=_size(rng, 60, 300), n1=_size(rng, 60, 300),
                    tol_coef=rng.choice([1.0, 10.0]))
    if kind == "stretch":
        return dict(kind=kind, **_box(rng, 48, 240), n0=_size(rng, 60, 400), n1=_size(rng, 60, 400), tol_coef=1.0,
                    uni=rng.choice([False, True]), native=rng.choice([False, True]))
    if kind == "lines":
        return dict(kind=kind, **_box(rng, 64, 240), n=_size(rng, 10, 2000), maxstep=_size(rng, 1000, 10000))
    if kind == "qmap":
        twist = rng.choice([False, False, True])
        return dict(kind=kind, layout=rng.choice(["h4b", "h4b", "f4", "h8c", "soa"]), **_box(rng, 64, 320),
                    n0=_size(rng, 60, 400), n1=_size(rng, 60, 400), planes=_size(rng, 1, 24), tol=tol, twist=twist,
                    hybrid=(not twist) and rng.random() < 0.2)
    if kind == "requests":
        return dict(kind=kind, **_box(rng, 128, 384), n=rng.randint(1, 4), seeds=_size(rng, 10000, 60000), tol=tol)
    return dict(kind="series", **_box(rng, 96, 256), n0=_size(rng, 80, 300), n1=_size(rng, 80, 300),
                planes=rng.randint(1, 3), fields=rng.randint(1, 3), tol=tol)


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------

def _charges(seed, nx, ny, m):
    """m charges below the bottom plane, positions as fractions of the box."""
    g = np.random.default_rng(seed)
    pos = np.column_stack([g.uniform(0.02, 0.98, m) * (nx - 1), g.uniform(0.02, 0.98, m) * (ny - 1),
                           -g.uniform(5.0, 18.0, m)])
    q = g.uniform(0.3, 1.8, m) * np.where(np.arange(m) % 2 == 0, 1.0, -1.0)
    return pos, q - q.mean()


def _potential(seed, nx, ny, nz, coords=None, scale=1.0):
    """(Bx, By, Bz) on the grid, float32 CUDA tensors of shape (nx, ny, nz)
    with x fastest in memory.  coords: node coordinates (default: indices)."""
    m = max(4, min(32, nx // 16))
    pos, q = _charges(seed, nx, ny, m)
    d = dict(dtype=torch.float64, device="cuda")
    if coords is None:
        coords = [np.arange(n, dtype=np.float64) for n in (nx, ny, nz)]
    else:
        pos = np.column_stack([coords[0][0] + pos[:, 0] / (nx - 1) * (coords[0][-1] - coords[0][0]),
                               coords[1][0] + pos[:, 1] / (ny - 1) * (coords[1][-1] - coords[1][0]), pos[:, 2] * scale])
    x, y, z = (torch.as_tensor(np.asarray(c, np.float64), **d) for c in coords)
    out = [torch.empty((nz, ny, nx), dtype=torch.float32, device="cuda") for _ in range(3)]
    step = max(1, (1 << 23) // (nx * ny))
    for k in range(0, nz, step):
        zz = z[k:k + step].view(-1, 1, 1)
        acc = [0.0, 0.0, 0.0]
        for (cx, cy, cz), s in zip(pos.tolist(), q.tolist()):
            r = [(x - cx).view(1, 1, -1), (y - cy).view(1, -1, 1), zz - cz]
            r2 = r[0] * r[0] + r[1] * r[1] + r[2] * r[2]
            w = s / (r2 * torch.sqrt(r2))
            acc = [a + w * c for a, c in zip(acc, r)]
        for o, a in zip(out, acc):
            o[k:k + step] = a.float()
    return tuple(o.permute(2, 1, 0) for o in out)


def _plane(nx, ny, n0, n1, zs, edge=0.06, scale=(1.0, 1.0), origin=(0.0, 0.0)):
    """Stacked (n0, n1) seed planes over the central part of the box (columns
    along x), float32 CUDA vectors."""
    d = dict(dtype=torch.float32, device="cuda")
    xi = torch.linspace(edge * (nx - 1) * scale[0] + origin[0], (1 - edge) * (nx - 1) * scale[0] + origin[0], n1, **d)
    yi = torch.linspace(edge * (ny - 1) * scale[1] + origin[1], (1 - edge) * (ny - 1) * scale[1] + origin[1], n0, **d)
    zt = torch.as_tensor(zs, **d).view(-1, 1, 1)
    shape = (zt.shape[0], n0, n1)
    return tuple(t.expand(shape).reshape(-1).contiguous() for t in (xi.view(1, 1, -1), yi.view(1, -1, 1), zt))


def _heights(c):
    """Seed heights of a case: one plane at its z, or `planes` one cell apart."""
    return [c["z"] + k for k in range(c["planes"])]


def _axes(c):
    """Stretched-grid coordinates: x, y uniform, z growing 2 % per cell."""
    nx, ny, nz = c["nx"], c["ny"], c["nz"]
    za = np.concatenate([[0.0], np.cumsum(1.02 ** np.arange(nz - 1))])
    return [np.linspace(-6.0, 6.0, nx).astype(np.float32), np.linspace(-5.0, 5.0, ny).astype(np.float32),
            (za * (10.0 / za[-1])).astype(np.float32)]


def _scalar(v, dtype):
    return torch.tensor([v], dtype=dtype, device="cuda")


def _buffers(n, f32=F32_OUT, i32=I32_OUT):
    o = {k: torch.zeros(n, dtype=torch.float32, device="cuda") for k in f32}
    o.update({k: torch.zeros(n, dtype=torch.int32, device="cuda") for k in i32})
    o["LineLen"] = torch.zeros(n, dtype=torch.float64, device="cuda")
    o["twist"] = torch.zeros(n, dtype=torch.float64, device="cuda")
    return o


def _tail(o, seeds, normal, s_len, tol_coef, n):
    """The part of the 35-argument list from inp_x on."""
    return (*seeds, normal, o["start_x"], o["start_y"], o["start_z"], o["flag_start"], o["end_x"], o["end_y"],
            o["end_z"], o["flag_end"], o["B_this_x"], o["B_this_y"], o["B_this_z"], o["B_flag"], o["B_start_x"],
            o["B_start_y"], o["B_start_z"], o["B_end_x"], o["B_end_y"], o["B_end_z"], s_len, n, o["LineLen"], tol_coef)


def _qparams(c):
    return params.absolute_rkf45(tol=c["tol"])


def _qseeds(c):
    """Seeds of a native Q map: unit spacing where the planes fit the box
    (then every pixel is a grid cell), else the box's central part."""
    nx, ny, nz, npl = c["nx"], c["ny"], c["nz"], c["planes"]
    z0 = 0.0 if npl == 1 else 0.25 * nz
    dz = 1.0 if z0 + npl <= nz - 4 else (nz - 4 - z0) / npl
    zs = [z0 + dz * k for k in range(npl)]
    if c["n1"] <= nx - 4 and c["n0"] <= ny - 4 and npl > 1:
        x0, y0 = (nx - c["n1"]) // 2, (ny - c["n0"]) // 2
        return api.plane_seed_grid(float(x0), float(x0 + c["n1"] - 1), c["n1"], float(y0), float(y0 + c["n0"] - 1),
                                   c["n0"], zs), 1.0
    s = 0.88 * min((nx - 1) / (c["n1"] - 1), (ny - 1) / (c["n0"] - 1))
    xc, yc = 0.5 * (nx - 1), 0.5 * (ny - 1)
    hx, hy = 0.5 * s * (c["n1"] - 1), 0.5 * s * (c["n0"] - 1)
    return api.plane_seed_grid(xc - hx, xc + hx, c["n1"], yc - hy, yc + hy, c["n0"], zs), s


def _request_list(c, seed):
    """c["n"] requests: horizontal planes of different shapes, and heights
    from the seed."""
    g = np.random.default_rng(seed)
    out = []
    for k in range(c["n"]):
        n = c["seeds"] * (0.6 + 0.4 * ((5 * k + 3) % 7) / 6)
        n1 = int(math.sqrt(n * (0.8 + 0.8 * ((3 * k + 1) % 5) / 4)))
        n0 = max(20, int(n / n1))
        s = 0.8 * min((c["nx"] - 1) / (n1 - 1), (c["ny"] - 1) / (n0 - 1))
        out.append(dict(n0=n0, n1=n1, spacing=s, height=float(g.uniform(0.0, 0.3) * c["nz"])))
    return out


def prepare(case, seed):
    c, kind = case, case["kind"]
    nx, ny, nz = c["nx"], c["ny"], c["nz"]
    f32, i64 = torch.float32, torch.int64
    st = dict(case=c)
    if kind == "stretch":
        ax = _axes(c)
        st["B"] = B = _potential(seed, nx, ny, nz, ax, scale=10.0 / nx)
        st["axes_h"] = ax
        st["seeds"] = seeds = _plane(nx, ny, c["n0"], c["n1"], [1e-3], scale=(12.0 / (nx - 1), 10.0 / (ny - 1)),
                                     origin=(-6.0, -5.0))
    elif kind in ("requests", "series"):
        pass
    else:
        st["B"] = B = _potential(seed, nx, ny, nz)
    if kind in ("rk4", "map", "rkf45", "scott", "stretch"):
        # as the notebooks allocate once and launch many times
        dummy = torch.zeros((1, 1), dtype=f32, device="cuda")
        normal = torch.tensor([0.0, 0.0, 1.0], device="cuda")
        if kind in ("map", "scott"):
            st["seeds"] = seeds = _plane(nx, ny, c["n0"], c["n1"], [0.0])
        elif kind != "stretch":
            st["seeds"] = seeds = _plane(nx, ny, c["n0"], c["n1"], _heights(c))
        n = seeds[0].numel()
        st["shape"] = torch.tensor([nx, ny, nz], dtype=torch.int32, device="cuda")
        st["normal"], st["dummy"] = normal, dummy
        s_len = c.get("s_len", {"map": 0.125, "scott": 0.25, "stretch": 0.01}.get(kind, 0.25))
        st["s_len"], st["tol_coef"] = _scalar(s_len, f32), _scalar(c.get("tol_coef", 1.0), f32)
        st["N"] = _scalar(n, i64)
        st["twist_on"] = _scalar(bool(c.get("twist", False)), torch.bool)
        st["off"] = _scalar(False, torch.bool)
        if kind == "scott":
            st["out"] = o = _buffers(n, FEET + ["B_this_x", "B_this_y", "B_this_z", "q_0", "q_perp"],
                                     ["flag_start", "flag_end"])
            st["kernel"] = kernels.compileTraceBlineScott()
            st["args"] = (*B, st["shape"], dummy, dummy, dummy, o["twist"], st["off"], *seeds, normal, o["start_x"],
                          o["start_y"], o["start_z"], o["flag_start"], o["end_x"], o["end_y"], o["end_z"],
                          o["flag_end"], o["B_this_x"], o["B_this_y"], o["B_this_z"], o["q_0"], o["q_perp"],
                          st["s_len"], st["N"], o["LineLen"], st["tol_coef"])
        elif kind == "stretch":
            if c["native"]:
                st["order"] = api.tile_order(1, c["n0"], c["n1"], 8, 8)
                st["prm"] = params.reference_stretch(arith=params.ARITH_FAST)
                st["out"] = api.alloc_trace_outputs(n)
            else:
                st["out"] = o = _buffers(n)
                st["kernel"] = kernels.compileTraceBlineAdaptiveStretch()
                ax = [torch.from_numpy(a).cuda() for a in st["axes_h"]]
                st["args"] = (*B, st["shape"], *ax, _scalar(c["uni"], torch.bool), dummy, dummy, dummy, o["twist"],
                              st["off"], *_tail(o, seeds, normal, st["s_len"], st["tol_coef"], st["N"]))
        else:
            st["out"] = _buffers(n)
            st["kernel"] = kernels.compileTraceBlineRK4() if kind == "rk4" else kernels.compileTraceBlineAdaptive()
            st["axes"] = [torch.arange(k, dtype=f32, device="cuda") for k in (nx, ny, nz)]
    elif kind == "lines":
        g = np.random.default_rng(seed + 77)
        st["pts"] = g.uniform(0.08, 0.92, (c["n"], 3)) * np.array([nx - 1, ny - 1, 0.4 * (nz - 1)])
    elif kind == "qmap":
        st["store"] = api.FieldStore(*B, layout=c["layout"])
        st["xyz"], st["stride"] = _qseeds(c)
        st["plan"] = api.QMapPlan(c["n0"], c["n1"], c["planes"], hybrid=c["hybrid"])
        st["cur"] = None
        if c["twist"]:
            J = FastQSL.curl_of_B_grid(*B, *[np.arange(k, dtype=np.float32) for k in (nx, ny, nz)])
            st["cur"] = api.FieldStore(*[j.float() for j in J], layout=c["layout"])
        if c["layout"] != "soa":
            del st["B"]
    elif kind == "requests":
        st["stores"] = [api.FieldStore(*_potential(seed + 1000 * k, nx, ny, nz), layout="h4b") for k in range(2)]
        st["requests"] = _request_list(c, seed)
        st["flying"] = []
    elif kind == "series":
        st["xyz"], st["stride"] = _qseeds(c)
        st["host"] = [[b.permute(2, 1, 0).cpu().pin_memory() for b in _potential(seed + 1000 * k, nx, ny, nz)]
                      for k in range(c["fields"])]
        st["q"] = [torch.zeros((c["planes"], c["n0"] - 2, c["n1"] - 2), dtype=torch.float64).pin_memory()
                   for _ in range(c["fields"])]
        st["series"] = api.QSeries((nx, ny, nz), c["n0"], c["n1"], c["planes"])
    return st


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------

def _trace_dropin(st, out, seeds, N, cur=None):
    c = st["case"]
    cur = cur if cur is not None else (st["dummy"],) * 3
    args = (*st["B"], st["shape"], *cur, out["twist"], st["twist_on"], *_tail(out, seeds, st["normal"], st["s_len"],
                                                                             st["tol_coef"], N))
    st["kernel"]((128, 1, 1), (28, 1), args[:34] if c["kind"] == "rk4" else args)


def _run_map(st):
    c = st["case"]
    o = st["out"]
    _trace_dropin(st, o, st["seeds"], st["N"])
    g = dict(zip(F32_OUT + I32_OUT, FastQSL.ResReshape((c["n0"], c["n1"]), *[o[k] for k in F32_OUT + I32_OUT])))
    feet = [g[k] for k in ("end_x", "end_y", "end_z", "flag_end", "start_x", "start_y", "start_z", "flag_start",
                           "B_start_x", "B_start_y", "B_start_z", "B_end_x", "B_end_y", "B_end_z")]
    stride = 0.88 * (c["nx"] - 1) / (c["n1"] - 1)
    Q = FastQSL.QCalcPlane(*feet, g["B_this_x"], g["B_this_y"], g["B_this_z"], g["B_flag"], stride)
    (ix, iy, iz, sx, sy, sz, fs, ex, ey, ez, fe, tx, ty, tz, bf, bsx, bsy, bsz, bex, bey, bez, N, length, bz0,
     bz1) = FastQSL.CookPseudoLine(*feet, g["B_this_z"], g["B_flag"], stride)
    cut = dict(start_x=sx, start_y=sy, start_z=sz, flag_start=fs, end_x=ex, end_y=ey, end_z=ez, flag_end=fe,
               B_this_x=tx, B_this_y=ty, B_this_z=tz, B_flag=bf, B_start_x=bsx, B_start_y=bsy, B_start_z=bsz,
               B_end_x=bex, B_end_y=bey, B_end_z=bez, LineLen=length, twist=st["dummy"])
    Q_final = Q
    if ix.numel():
        _trace_dropin(st, cut, (ix, iy, iz), N)
        Qcut = FastQSL.QCalcCut(sx, sy, sz, fs, ex, ey, ez, fe, bz0, bz1, stride)
        _, Q_final = FastQSL.QMerge(Q, Qcut, g["B_flag"])
    return {**{k: o[k] for k in FEET + I32_OUT + ["LineLen"]}, "Q": Q_final}


def run(st):
    c, kind = st["case"], st["case"]["kind"]
    if kind in ("rk4", "rkf45"):
        cur = None
        if c["twist"]:
            cur = [j.float() for j in FastQSL.curl_of_B_grid(*st["B"], *st["axes"])]
        _trace_dropin(st, st["out"], st["seeds"], st["N"], cur)
        return st["out"] if cur is None else {**st["out"], "J": cur}
    if kind == "map":
        return _run_map(st)
    if kind == "scott":
        st["kernel"]((128, 1, 1), (28, 1), st["args"])
        return st["out"]
    if kind == "stretch":
        if c["native"]:
            api.trace_stretch(*st["B"], st["axes_h"], *st["seeds"], st["prm"], s_len=0.01, tol_coef=c["tol_coef"],
                              uni=c["uni"], out=st["out"], order=st["order"])
            return {k: v for k, v in st["out"].items() if v is not None}
        st["kernel"]((128, 1, 1), (28, 1), st["args"])
        return st["out"]
    if kind == "lines":
        return MagTool.TraceBlines(*st["B"], st["pts"], maxstep=c["maxstep"])
    if kind == "qmap":
        plan = st["plan"]
        Q = plan.run(st["store"], *st["xyz"], _qparams(c), s_len=0.25, stride=st["stride"], curB=st["cur"])
        out = {k: plan.main[k] for k in FEET + I32_OUT}
        if st["cur"] is not None:
            out["twist"] = plan.twist_map
        return {**out, "Q": Q}
    if kind == "requests":
        # batches in flight are kept until their work is done, at most 12
        fly = st["flying"]
        while fly and (fly[0][1].query() or len(fly) >= 12):
            fly[0][1].synchronize()
            fly.pop(0)
        jobs = [dict(field=st["stores"][k % 2], params=_qparams(c), center=((c["nx"] - 1) / 2, (c["ny"] - 1) / 2, r["height"]),
                     normal=(0.0, 0.0, 1.0), u=(1.0, 0.0, 0.0), v=(0.0, 1.0, 0.0), spacing=r["spacing"], n0=r["n0"],
                     n1=r["n1"], nplanes=1) for k, r in enumerate(st["requests"])]
        batch = api.PlaneQBatch(jobs)
        Q = batch.run()
        done = torch.cuda.Event()
        done.record()
        fly.append((batch, done))
        return list(Q)
    for host, q in zip(st["host"], st["q"]):
        st["series"].push(*host, *st["xyz"], _qparams(c), q, s_len=0.25, stride=st["stride"])
    st["series"].wait()
    return list(st["q"])


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------

def work(case):
    """Field, seeds and outputs once each; flops: trilinear samples (75 each,
    and an integrator's share of 22) for lines about as long as the box's
    larger side takes, from the step each integrator settles on."""
    c, kind = case, case["kind"]
    nodes = c["nx"] * c["ny"] * c["nz"]
    if kind == "lines":
        pts = c["n"] * c["maxstep"]
        return dict(bytes=12 * nodes + 24 * c["n"] + 12 * pts, flops=100.0 * 4 * c["n"] * min(c["maxstep"], 8 * c["nx"]))
    if kind == "requests":
        lines, q = c["n"] * 0.8 * c["seeds"], 1
        bytes_ = 20 * nodes * min(2, c["n"]) + lines * 20
    elif kind == "series":
        lines = c["fields"] * c["planes"] * c["n0"] * c["n1"]
        bytes_ = c["fields"] * 12 * nodes + lines * 20
    else:
        lines = c.get("planes", 1) * c["n0"] * c["n1"]
        per_node = {"h4b": 20, "h8c": 64, "f4": 16}.get(c.get("layout"), 12)
        bytes_ = per_node * nodes * (2 if c.get("twist") else 1) + lines * (12 + 80)
    size = max(c["nx"], c["ny"])
    samples = {"rk4": 4 * 1.2 * size / c.get("s_len", 1.0), "map": 2.0 * size, "rkf45": 2.0 * size,
               "scott": 42 * 0.5 * size, "stretch": 2.0 * size}.get(kind, 3.4 * size)
    return dict(bytes=bytes_, flops=97.0 * lines * samples)


# ---------------------------------------------------------------------------
# the outputs in 64 bits
# ---------------------------------------------------------------------------

class _Late(Exception):
    pass


class _Grid:
    """Trilinear sampling in float64 of float32 nodes, by index or by node
    coordinates (the reference's interval search or its uniform formula)."""

    def __init__(self, B, ax=None, uni=False):
        self.n = tuple(int(v) for v in B[0].shape)
        nx, ny, nz = self.n
        self.B = torch.stack([b.permute(2, 1, 0).reshape(-1) for b in B], 1).double()
        self.corner = torch.tensor([dx + nx * (dy + ny * dz) for dz in (0, 1) for dy in (0, 1) for dx in (0, 1)],
                                   device="cuda")
        self.ax = None
        if ax is not None:
            self.ax = [torch.as_tensor(a.astype(np.float64), device="cuda") for a in ax]
            self.tab = [self._table(a, uni) for a in ax]
        self.uni = uni
        self.lo = [0.0] * 3 if ax is None else [float(a[0]) for a in ax]
        self.hi = [float(v - 1) for v in self.n] if ax is None else [float(a[-1]) for a in ax]

    @staticmethod
    def _table(a, uni):
        """The cell the reference's bisection gives for each interval."""
        n, out = len(a), []
        for j in range(n - 1):
            i0, i1, mid = 0, n - 1, n // 2
            while i1 - i0 > 3:
                if j >= mid:
                    i0 = mid
                else:
                    i1 = mid
                mid = (i0 + i1) // 2
            r = mid if j >= mid else mid - 1
            out.append(min(max(r, 0), n - 2))
        return torch.tensor(out, device="cuda")

    def _cell(self, k, c):
        n = self.n[k]
        if self.ax is None:
            i = torch.clamp(torch.floor(c), 0, n - 2).nan_to_num().long()
            return i, torch.clamp(c - i, 0.0, 1.0)
        a, lo, hi = self.ax[k], self.lo[k], self.hi[k]
        c = torch.where(c > lo, c, torch.full_like(c, lo + 1e-6))
        c = torch.where(c < hi, c, torch.full_like(c, hi - 1e-6))
        if self.uni:
            i = torch.clamp(torch.floor((c - lo) / ((hi - lo) / n)), 0, n - 2).long()
        else:
            i = self.tab[k][torch.clamp(torch.searchsorted(a, c.contiguous()) - 1, 0, n - 2)]
        return i, (c - a[i]) / (a[i + 1] - a[i])

    def raw(self, p):
        nx, ny, _ = self.n
        (ix, rx), (iy, ry), (iz, rz) = (self._cell(k, p[:, k]) for k in range(3))
        o = (ix + nx * (iy + ny * iz))[:, None] + self.corner
        f = torch.stack([rx, ry, rz], 1)
        w = torch.stack([1 - f, f], 2)
        w = w[:, 2, :, None, None] * w[:, 1, None, :, None] * w[:, 0, None, None, :]
        return (self.B[o] * w.reshape(-1, 8, 1)).sum(1)

    def unit(self, p):
        b = self.raw(p)
        return b / b.norm(dim=1, keepdim=True)

    def flag(self, p):
        lo, hi = p.new_tensor(self.lo), p.new_tensor(self.hi)
        inside = ((p >= lo) & (p <= hi)).all(1) & (p[:, 1] > lo[1])
        below, above = p < lo, p >= hi
        f = torch.full((len(p),), 42, device=p.device)
        for d in range(3):
            rest = [k for k in range(3) if k != d]
            ok = ~(below[:, rest] | above[:, rest]).any(1)
            f = torch.where(below[:, d] & ok, torch.full_like(f, 2 * d + 1), f)
            f = torch.where(above[:, d] & ok, torch.full_like(f, 2 * d + 2), f)
        return torch.where(inside, torch.zeros_like(f), f)


_A = [[], [1 / 4], [3 / 32, 9 / 32], [1932 / 2197, -7200 / 2197, 7296 / 2197], [439 / 216, -8.0, 3680 / 513, -845 / 4104],
      [-8 / 27, 2.0, -3544 / 2565, 1859 / 4104, -11 / 40]]
_B5 = [16 / 135, 0.0, 6656 / 12825, 28561 / 56430, -9 / 50, 2 / 55]
_E = [1 / 360, 0.0, -128 / 4275, -2197 / 75240, 1 / 50, 2 / 55]


def _fehlberg(g, p, h):
    k = []
    for row in _A:
        q = p
        for a, b in zip(row, k):
            q = q + (a * h)[:, None] * b
        k.append(g.unit(q))
    inc = h[:, None] * sum(b * v for b, v in zip(_B5, k))
    err = h.abs() * sum(e * v for e, v in zip(_E, k)).norm(dim=1)
    return inc, err


def _rk4(g, p, h):
    hh = h[:, None]
    k1 = g.unit(p)
    k2 = g.unit(p + hh * k1 / 2)
    k3 = g.unit(p + hh * k2 / 2)
    k4 = g.unit(p + hh * k3)
    return hh / 6 * (k1 + 2 * k2 + 2 * k3 + k4)


def _to_face(g, p, h, d):
    """RK4 in the coordinate along axis d (a tensor of axes) over h."""
    def rhs(q):
        b = g.unit(q)
        return b / b.gather(1, d[:, None])
    hh = h[:, None]
    k1 = rhs(p)
    k2 = rhs(p + hh * k1 / 2)
    k3 = rhs(p + hh * k2 / 2)
    k4 = rhs(p + hh * k3)
    return p + hh / 6 * (k1 + 2 * k2 + 2 * k3 + k4)


def _integrate(g, p0, sign, s_len, tol, h_min, h_max, limit, fixed, until):
    """Every line in the direction of its sign: (footpoint, length)."""
    n = len(p0)
    foot, length = p0.clone(), p0.new_zeros(n)
    idx = torch.arange(n, device=p0.device)
    p, h, ln = p0.clone(), p0.new_full((n,), s_len), p0.new_zeros(n)
    while idx.numel():
        if time.monotonic() > until:
            raise _Late()
        if fixed:
            inc, ok = _rk4(g, p, sign[idx] * h), torch.ones_like(h, dtype=torch.bool)
        else:
            inc, err = _fehlberg(g, p, sign[idx] * h)
            scale = (tol[idx] / err / 11.09) ** 0.2
            ok = ~(scale < 0.618)
            h = torch.where(ok, torch.clamp(h * scale, h_min, h_max), h * 0.618)
        p2 = torch.where(ok[:, None], p + inc, p)
        dl = (p2 - p).norm(dim=1)
        flag = torch.where(ok, g.flag(p2), torch.zeros_like(idx))
        out = flag > 0
        done = out.clone()
        if out.any():
            j = out.nonzero()[:, 0]
            face, a, b = flag[j], p[j], p2[j]
            d = torch.clamp((face - 1) // 2, 0, 2)
            q1, q2 = a.gather(1, d[:, None])[:, 0], b.gather(1, d[:, None])[:, 0]
            top = torch.tensor([float(v) for v in g.n], dtype=p.dtype, device=p.device)[d]
            qm = torch.where(face % 2 == 1, torch.zeros_like(top), top)
            lin = (a * (q2 - qm)[:, None] + b * (qm - q1)[:, None]) / (q2 - q1)[:, None]
            ua, ub = g.unit(a), g.unit(b)
            na, nb = (u.gather(1, d[:, None])[:, 0].abs() for u in (ua, ub))
            e = torch.where(((na < 0.2) | (nb < 0.2))[:, None], lin, _to_face(g, a, qm - q1, d))
            far = (q1 - q2).abs() > 1e-3
            e = torch.where(far[:, None], e, a)
            more = torch.where(far, (qm - q1).abs() / (1e-4 + na), torch.zeros_like(na))
            corner = face > 6
            e = torch.where(corner[:, None], b, e)
            foot[idx[j]] = e
            length[idx[j]] = ln[j] + torch.where(corner, torch.zeros_like(more), more)
        ln = torch.where(ok & ~out, ln + dl, ln)
        stop = ~out & (ln >= limit)
        if stop.any():
            foot[idx[stop]], length[idx[stop]] = p2[stop], ln[stop]
            done |= stop
        keep = ~done
        idx, p, h, ln = idx[keep], p2[keep], h[keep], ln[keep]
    return foot, length


def _exact_feet(g, seeds, s_len, tol, h_min, h_max, ratio, fixed=False, limit=18.0):
    """Both footpoints and the line length of every seed, or None when it
    would take too long."""
    until = time.monotonic() + limit
    p0 = torch.stack(seeds, 1).double()
    t = torch.full((len(p0),), float(tol), dtype=torch.float64, device="cuda")
    lim = ratio * (sum(g.n) if g.ax is None else sum(g.hi) - sum(g.lo))
    try:
        sign = torch.cat([torch.ones_like(t), -torch.ones_like(t)])
        foot, length = _integrate(g, torch.cat([p0, p0]), sign, s_len, torch.cat([t, t]), h_min, h_max, lim, fixed,
                                  until)
    except _Late:
        return None
    e, s = foot.chunk(2)
    le, ls = length.chunk(2)
    names = dict(zip(FEET, [s[:, 0], s[:, 1], s[:, 2], e[:, 0], e[:, 1], e[:, 2]]))
    names["LineLen"] = ls + le
    return names


def _b_at(g, seeds):
    b = g.raw(torch.stack(seeds, 1).double())
    return {"B_this_x": b[:, 0], "B_this_y": b[:, 1], "B_this_z": b[:, 2]}


def _exact_lines(B, pts, maxstep, limit=18.0):
    """The polylines: fixed RK4 steps of 0.25 from every seed, both ways, the
    clamps of the module kept."""
    until = time.monotonic() + limit
    n = torch.tensor([float(v) for v in B[0].shape], dtype=torch.float64, device="cuda")
    g = _Grid(B)
    top = n - 1

    def unit(q):
        q = torch.where(q < 0, torch.full_like(q, 1e-8), torch.where(q > n, n - 1e-8, q))
        return g.unit(torch.minimum(q, top))

    out = torch.full((3, len(pts), maxstep), float("nan"), dtype=torch.float64, device="cuda")
    mid = maxstep // 2
    for dr, rng in ((0.25, range(mid, maxstep)), (-0.25, range(mid, 0, -1))):
        idx = torch.arange(len(pts), device="cuda")
        p = torch.as_tensor(pts, dtype=torch.float64, device="cuda")
        for k in rng:
            live = ((p >= 0) & (p <= n[0])).all(1)
            idx, p = idx[live], p[live]
            if not idx.numel():
                break
            if time.monotonic() > until:
                return None
            p = torch.where(p > n, n - 1e-8, p)
            f1 = unit(p)
            f2 = unit(p + dr * f1 * 0.5)
            f3 = unit(p + dr * f2 * 0.5)
            f4 = unit(p + dr * f3)
            out[:, idx, k] = p.T
            p = p + dr * (f1 + 2 * f2 + 2 * f3 + f4) / 6
    return tuple(v.cpu().numpy() for v in out)


def _exact_curl(B):
    """Three-point curl on the unit grid, boundary planes copied inward."""
    b = [v.double() for v in B]

    def diff(f, axis):
        s = [slice(1, -1)] * 3
        hi, lo = list(s), list(s)
        hi[axis], lo[axis] = slice(2, None), slice(None, -2)
        return (f[tuple(hi)] - f[tuple(lo)]) / 2

    inner = (diff(b[2], 1) - diff(b[1], 2), diff(b[0], 2) - diff(b[2], 0), diff(b[1], 0) - diff(b[0], 1))
    return [torch.nn.functional.pad(v[None, None], (1,) * 6, mode="replicate")[0, 0] for v in inner]


def exact(case, seed):
    """Footpoints where the line is integrated at a set step or a tight
    tolerance, field values, the curl and the polylines.  The adaptive
    drop-ins run at the reference's loose tolerances: their step sequences,
    and with them footpoints and lengths, move with the last bit of the error
    estimate, so a 64-bit run says nothing of them.  Nor has Q (its norm is
    that of its few largest pixels, which move with the last bit of a
    footpoint), nor the deviation vectors' q, nor the twist (one term per
    step) a usable 64-bit value."""
    c, kind = case, case["kind"]
    if kind in ("requests", "series") or c["nx"] * c["ny"] * c["nz"] > 3e7:
        return None
    st = prepare(case, seed)
    B = st.get("B") or _potential(seed, c["nx"], c["ny"], c["nz"])
    if kind == "lines":
        return _exact_lines(B, st["pts"], c["maxstep"])
    g = _Grid(B, st.get("axes_h"), c.get("uni", False))
    if kind == "qmap":
        feet = _exact_feet(g, st["xyz"], 0.25, c["tol"], 1e-3, 1.0, 3.0)
        if feet is None:
            return None
        return {k: feet.get(k) for k in FEET + I32_OUT + (["twist"] if c["twist"] else []) + ["Q"]}
    if kind == "map":
        return None
    res = {}
    if kind == "rk4":
        res = _exact_feet(g, st["seeds"], float(st["s_len"]), 1e-3, 0.1, 100.0, 2.0, fixed=True) or {}
        res.pop("LineLen", None)
    res.update(_b_at(g, st["seeds"]))
    res = {k: res.get(k) for k in st["out"] if st["out"][k] is not None}
    if c.get("twist"):
        res["J"] = _exact_curl(B)
    return res
