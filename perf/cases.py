"""What this framework is used for, as cases that can be timed and compared.

A case is one call sequence of a user's program through the package's public
entry points: a height field in (device memory, or host memory where the
server takes it), the complex out in host memory, whole.  Height fields follow
``mscomplex_gb300.synth``: sums of Gaussian bumps (smooth, with a little
noise, or quantised to 1/256 of the range) and white noise, made here on the
GPU from the seed alone.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import mscomplex_gb300 as M
from mscomplex_gb300 import primitives

DEV = "cuda"


def listed():
    return [
        # the smallest whole-grid call: a field of a few thousand vertices from
        # heights to its simplified complex; launches and host latency count
        dict(name="grid_65x63", kind="grid", nx=65, ny=63, field="smooth", halo=0, ocl=False, tresh=0.05, discs=False),
        # the 256x256 noisy-bumps field at 5% with its manifold discs
        dict(name="grid_256_bumps", kind="grid", nx=256, ny=256, field="bumps", halo=0, ocl=False, tresh=0.05,
             discs=True),
        # one piece of a larger white-noise grid with a halo on every side: an
        # odd-sized, unaligned window of a field in device memory
        dict(name="piece_1023x771", kind="grid", nx=1023, ny=771, field="noise", halo=1, ocl=False, tresh=0.0,
             discs=False),
        # an ordinary ragged field with the -ocl gradient, simplified at 2%, with discs
        dict(name="grid_2047x1365_ocl", kind="grid", nx=2047, ny=1365, field="smooth", halo=0, ocl=True, tresh=0.02,
             discs=True),
        # the 4096x4096 quantised field: gradient, owners, connectivity and all
        # discs, dataset and complex kept from field to field
        dict(name="grid_4096_quantised", kind="stream", nx=4096, ny=4096, field="quantised"),
        # exact persistence cancellation where many values tie: a field of the
        # mixed-size workloads quantised to 256 steps, at 1%
        dict(name="simplify_288_steps", kind="grid", nx=288, ny=288, field="steps", halo=0, ocl=False,
             tresh=0.01, discs=True),
        # the piece pipeline over white noise in 16 blocks (2D splits, no threshold)
        dict(name="pipeline_2048_noise", kind="pipeline", nx=2048, ny=2048, field="noise", levels=4, split2d=True,
             tresh=0.0),
        # the command line's usual run: y-splits of a ragged smooth field,
        # simplified at the root, discs of every piece
        dict(name="pipeline_1025x769", kind="pipeline", nx=1025, ny=769, field="smooth", levels=3, split2d=False,
             tresh=0.05),
        # many grids of mixed sizes in shared launches, simplified at 2%
        dict(name="batch_1000", kind="batch", count=1000, lo=64, hi=2048, tresh=0.02),
        # a burst of requests to the server, each its own size and threshold
        dict(name="serve_32", kind="serve", count=32, lo=64, hi=512, tresh=0.05),
        # the scan and sort primitives at an ordinary and a large odd size
        dict(name="scan_16777259", kind="scan", n=16777259),
        dict(name="sort_3000017", kind="sort", n=3000017, batch=1, ascending=True),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["grid", "grid", "grid", "stream", "simplify", "pipeline", "batch", "serve", "scan", "sort"])
    if kind == "grid":
        field = rng.choice(["smooth", "noise", "quantised"])
        halo = rng.choice([0, 0, 1, 2])
        return dict(kind="grid", nx=_log_int(rng, 48, 3000), ny=_log_int(rng, 48, 3000), field=field, halo=halo,
                    ocl=rng.random() < 0.3, tresh=rng.choice([0.0, 0.01, 0.05]) if field == "smooth" and not halo else 0.0,
                    discs=not halo and rng.random() < 0.7)  # a piece's discs come after the merges
    if kind == "stream":
        return dict(kind="stream", nx=_log_int(rng, 512, 4096), ny=_log_int(rng, 512, 4096),
                    field=rng.choice(["smooth", "quantised"]))
    if kind == "simplify":
        n = rng.randint(96, 256)
        return dict(kind="grid", nx=n, ny=n, field=rng.choice(["bumps", "steps"]), halo=0, ocl=False,
                    tresh=rng.choice([0.01, 0.02]), discs=rng.random() < 0.5)
    if kind == "pipeline":
        field = rng.choice(["smooth", "noise"])
        return dict(kind="pipeline", nx=rng.randint(300, 1600), ny=rng.randint(300, 1600), field=field,
                    levels=rng.randint(1, 4), split2d=rng.random() < 0.5,
                    tresh=rng.choice([0.01, 0.05]) if field == "smooth" else 0.0)
    if kind == "batch":
        lo = _log_int(rng, 16, 256)
        return dict(kind="batch", count=_log_int(rng, 8, 600), lo=lo, hi=lo * rng.randint(1, 7),
                    tresh=rng.choice([0.0, 0.02, 0.05]))
    if kind == "serve":
        lo = _log_int(rng, 16, 128)
        return dict(kind="serve", count=rng.randint(1, 48), lo=lo, hi=lo * rng.randint(1, 4), tresh=0.05)
    if kind == "scan":
        return dict(kind="scan", n=_log_int(rng, 100, 30000000) | 1)
    batch = rng.choice([1, 1, 3, 17])
    return dict(kind="sort", n=_log_int(rng, 100, 4000000 // batch), batch=batch, ascending=rng.random() < 0.7)


# ---- inputs -----------------------------------------------------------------
def _bumps(nx, ny, nb, lo, hi, gen, windowed):
    """A sum of nb Gaussians on the GPU in double precision (separable: one
    matrix product), windowed at 4 sigma or evaluated everywhere."""
    u = torch.rand(4, nb, generator=gen, device=DEV, dtype=torch.float64)
    sg = lo + (hi - lo) * u[2]
    amp = 2.0 * u[3] - 1.0

    def axis(n, c):
        t = (torch.arange(n, device=DEV, dtype=torch.float64)[None, :] - c[:, None]) / sg[:, None]
        g = torch.exp(-0.5 * t * t)
        return torch.where(t.abs() <= 4.0, g, torch.zeros_like(g)) if windowed else g

    return (axis(ny, u[1] * (ny - 1)) * amp[:, None]).T @ axis(nx, u[0] * (nx - 1))


def _steps(f):
    """f in 256 steps of its range."""
    lo, hi = f.min(), f.max()
    step = torch.clamp_min(hi - lo, 1e-300) / 256
    return lo + torch.round((f - lo) / step) * step


def _field(kind, nx, ny, seed):
    gen = torch.Generator(device=DEV)
    gen.manual_seed(seed)
    if kind == "noise":  # white noise U[0, 1)
        return torch.rand(ny, nx, generator=gen, device=DEV, dtype=torch.float32)
    if kind == "bumps":  # 16 bumps and a little noise
        f = _bumps(nx, ny, 16, nx / 32.0, nx / 8.0, gen, True)
        return (f + 1e-3 * torch.rand(ny, nx, generator=gen, device=DEV, dtype=torch.float64)).float()
    if kind == "quantised":  # the 4096^2 workload's bump density and sizes, scaled, in 256 steps of the range
        k = math.sqrt(nx * ny) / 4096.0
        f = _bumps(nx, ny, max(4, round(512 * k * k)), max(1.0, 4.0 * k), max(2.0, 64.0 * k), gen, True)
        return _steps(f).float()
    # smooth: the mixed-size batch's fields, a Gaussian per 8192 vertices; steps: those, quantised
    f = _bumps(nx, ny, max(1, round(nx * ny / 8192)), 4.0, 32.0, gen, False)
    return (_steps(f) if kind == "steps" else f).float()


def _sides(case):
    """The sides of a batch's or burst's square grids: log-uniform, the same for every seed."""
    rng = np.random.default_rng(case["count"])
    return [int(n) for n in np.exp(rng.uniform(math.log(case["lo"]), math.log(case["hi"]), case["count"]))]


# Room in the host buffers a program keeps for its results, per vertex of the
# field: critical points, arcs of each kind, disc cells of each kind.  A field
# that needs more gets larger buffers in its pass.
ROOM = {"smooth": (0.08, 0.5, 3.0), "bumps": (0.5, 3.0, 16.0), "quantised": (0.2, 0.8, 10.0),
        "steps": (0.5, 4.0, 24.0), "noise": (0.97, 2.0, 2.8)}


def _room(n, dt):
    """A host buffer of n elements, pinned where it is large."""
    dt = np.dtype(dt)
    n = int(n)
    if n * dt.itemsize < 65536:
        return np.zeros(n, dt)
    return torch.zeros(n * dt.itemsize, dtype=torch.uint8, pin_memory=True).numpy().view(dt)


def _rooms(field, nv, nodes, levels, discs):
    c, a, d = ROOM[field]
    cps = c * nv * levels + 1000 * nodes
    arcs = a * nv * levels + 2000 * nodes
    cells = d * nv + 2000 * nodes if discs else 0
    n = dict(rect_ext=8 * nodes, cellid=2 * cps, fn=cps, pair_idx=cps, flags=cps, asc_off=cps + nodes, asc=arcs,
             des_off=cps + nodes, des=arcs, adisc_off=cps + nodes, adisc=2 * cells, ddisc_off=cps + nodes,
             ddisc=2 * cells)
    types = dict(cellid=np.int16, rect_ext=np.int16, fn=np.float32, flags=np.uint8, adisc=np.int16, ddisc=np.int16)
    return {k: _room(v, types.get(k, np.uint32)) for k, v in n.items()}


def prepare(case, seed):
    s = dict(case)
    kind = case["kind"]
    if kind in ("grid", "pipeline"):
        # a window of a larger field: its rows are not aligned and not adjacent
        s["heights"] = _field(case["field"], case["nx"] + 3, case["ny"], seed)[:, 1:1 + case["nx"]]
        if kind == "grid":
            s["out"] = _rooms(case["field"], case["nx"] * case["ny"], 1, 1, case["discs"])
        else:  # every node of the piece tree, whose boundaries hold further critical points
            s["out"] = _rooms(case["field"], case["nx"] * case["ny"] + 64 * (case["nx"] + case["ny"]),
                              2 ** (case["levels"] + 1), case["levels"] + 1, True)
    elif kind == "stream":
        s["heights"] = _field(case["field"], case["nx"], case["ny"], seed)
        r = (0, 0, 2 * (case["nx"] - 1), 2 * (case["ny"] - 1))
        s["dataset"], s["complex"] = M.GridDataset(r, r), None
        s["stream"] = torch.cuda.Stream()
        s["out"] = _rooms(case["field"], case["nx"] * case["ny"], 1, 1, True)
    elif kind == "batch":
        sides = _sides(case)
        s["sizes"] = np.array([[n, n] for n in sides], np.int32).reshape(-1)
        s["packed"] = torch.cat([_field("smooth", n, n, seed * 1000003 + i).reshape(-1) for i, n in enumerate(sides)])
        s["batch"] = M.GridBatch()
        r = _rooms("smooth", sum(n * n for n in sides), case["count"], 1, False)
        s["out"] = {k: _room(case["count"] + 1, np.uint32) for k in ("cp_base", "asc_base", "des_base")}
        s["out"].update({k: r[k] for k in ("fn", "pair_idx", "flags", "asc_off", "asc", "des_off", "des")})
        s["out"]["cellid"] = _room(r["fn"].size, np.uint32)
    elif kind == "serve":
        rng = np.random.default_rng(seed + 1)
        s["fields"] = [_field("smooth", int(n), int(n), seed * 1000003 + i).cpu().numpy()
                       for i, n in enumerate(_sides(case))]
        s["treshs"] = rng.uniform(0.0, case["tresh"], case["count"])
        s["server"] = M.GridServer()
        r = _rooms("smooth", sum(n * n for n in _sides(case)), case["count"], 1, False)
        s["out"] = {k: r[k] for k in ("cellid", "fn", "pair_idx", "flags", "asc_off", "asc", "des_off", "des")}
    else:  # scan, sort
        gen = torch.Generator(device=DEV)
        gen.manual_seed(seed)
        n = case["n"] * case.get("batch", 1)
        s["x"] = torch.randint(-2**31, 2**31 - 1, (n,), generator=gen, device=DEV, dtype=torch.int32)
        if kind == "scan":
            s["x"] &= 255  # counts, as the collation scans them
        else:
            s["v"] = torch.arange(n, device=DEV, dtype=torch.int32)
    return s


# ---- passes -----------------------------------------------------------------
def _whole(out, sizes):
    """The result buffers with the counts that say how much of each is filled."""
    out = {k: v.view(np.int32) if v.dtype == np.uint32 else v for k, v in out.items()}
    out["sizes"] = np.asarray(sizes, np.int64)
    return out


def _export(s, complexes, stream=None):
    """The complexes' flat arrays one behind the other in the state's host buffers."""
    out = s["out"]
    shapes = [m.export_shapes() for m in complexes]
    at = dict.fromkeys(out, 0)
    for k, buf in out.items():
        n = sum(math.prod(sh[k][0]) for sh in shapes)
        if n > buf.size:
            out[k] = _room(n + n // 4, buf.dtype)
    for m, sh in zip(complexes, shapes):
        part = {}
        for k in out:
            n = math.prod(sh[k][0])
            part[k] = out[k][at[k]:at[k] + n]
            at[k] += n
        m.export(part, stream=stream)
    return _whole(out, [m.sizes() for m in complexes])


def _run_grid(s):
    nx, ny, h = s["nx"], s["ny"], s["halo"]
    ext = (0, 0, 2 * (nx - 1), 2 * (ny - 1))
    rect = (2 * h, 2 * h, 2 * (nx - 1 - h), 2 * (ny - 1 - h))
    ds = M.GridDataset(rect, ext).init(s["heights"])
    if s["ocl"]:
        msc = ds.work_ocl().writeout_connectivity_ocl()
    else:
        msc = ds.work().writeout_connectivity()
    if s["tresh"] > 0:
        msc.simplify_un_simplify(s["tresh"])
    if s["discs"]:
        ds.post_merge_fill_discs(msc)
    return _export(s, [msc])


def _run_stream(s):
    st = s["stream"]
    st.wait_stream(torch.cuda.current_stream())
    h = st.cuda_stream
    ds = s["dataset"].init(s["heights"], stream=h).work(stream=h)
    s["complex"] = ds.writeout_connectivity(s["complex"], stream=h)
    ds.post_merge_fill_discs(s["complex"], stream=h)
    return _export(s, [s["complex"]], stream=h)


def _run_pipeline(s):
    p = M.GridDataManager(s["heights"], levels=s["levels"], tresh=s["tresh"], split2d=s["split2d"])
    return _export(s, [p.piece(i) for i in range(2 * p.num_pieces - 1)])


def _run_batch(s):
    b = s["batch"].run(packed=s["packed"], sizes=s["sizes"], tresh=s["tresh"])
    ncp, na, nd = b.totals()
    out = s["out"]
    for k, n in dict(cellid=ncp, fn=ncp, pair_idx=ncp, flags=ncp, asc_off=ncp + 1, asc=na, des_off=ncp + 1,
                     des=nd).items():
        if n > out[k].size:
            out[k] = _room(n + n // 4, out[k].dtype)
    b.export_all(out)
    return _whole(out, [ncp, na, nd])


def _run_serve(s):
    ids = [s["server"].submit(f, t) for f, t in zip(s["fields"], s["treshs"])]
    out, at = s["out"], dict.fromkeys(s["out"], 0)
    sizes = []
    for i in ids:
        got = s["server"].result(i)
        for k in out:
            v = got[k].reshape(-1)
            if at[k] + v.size > out[k].size:
                out[k] = np.concatenate([out[k], _room(out[k].size + v.size, out[k].dtype)])
            out[k][at[k]:at[k] + v.size] = v
            at[k] += v.size
        sizes.append([got["fn"].size, got["asc"].size, got["des"].size])
    return _whole(out, sizes)


def run(s):
    kind = s["kind"]
    if kind == "grid":
        return _run_grid(s)
    if kind == "stream":
        return _run_stream(s)
    if kind == "pipeline":
        return _run_pipeline(s)
    if kind == "batch":
        return _run_batch(s)
    if kind == "serve":
        return _run_serve(s)
    if kind == "scan":
        return primitives.prefix_scan(s["x"])
    return primitives.sort_pairs(s["x"], s["v"], batch=s["batch"], ascending=s["ascending"])


def exact(case, seed):
    """The primitives' outputs.  A complex holds no computed numbers: its cells,
    lists and discs are whole numbers, its values copies of input heights."""
    if case["kind"] == "scan":
        x = prepare(case, seed)["x"].to(torch.int64)
        return (torch.cumsum(x, 0) - x).to(torch.int32)
    if case["kind"] == "sort":
        s = prepare(case, seed)
        key = (s["x"].to(torch.int64) & 0xFFFFFFFF).reshape(case["batch"], case["n"])
        key, at = torch.sort(key, dim=1, stable=True, descending=not case["ascending"])
        val = torch.gather(s["v"].reshape(case["batch"], case["n"]), 1, at)
        return key.to(torch.int32).reshape(-1), val.reshape(-1)
    return None


# Bytes of a complex per vertex of its field: (critical points and arcs, discs),
# measured on these generators at the listed sizes.
OUT_BYTES = {"smooth": (0.08, 8.2), "bumps": (1.1, 8.6), "quantised": (2.7, 48.0),
             "steps": (2.7, 20.0), "noise": (31.4, 16.0)}


def work(case):
    kind = case["kind"]
    if kind == "scan":
        return {"bytes": 8.0 * case["n"], "flops": 0.0}
    if kind == "sort":
        return {"bytes": 16.0 * case["n"] * case["batch"], "flops": 0.0}
    if kind in ("batch", "serve"):
        lo, hi = float(case["lo"]), float(case["hi"])
        area = (hi * hi - lo * lo) / (2.0 * math.log(hi / lo)) if hi > lo else lo * lo  # mean of side^2
        return {"bytes": case["count"] * area * (4.0 + OUT_BYTES["smooth"][0]), "flops": 0.0}
    graph, discs = OUT_BYTES[case["field"]]
    if kind == "grid" and not case["discs"]:
        discs = 0.0
    if kind == "pipeline":
        graph *= case["levels"] + 1  # every node of the piece tree is written out
    return {"bytes": case["nx"] * case["ny"] * (4.0 + graph + discs), "flops": 0.0}
