"""The timed cases: what a program that uses this package has it do, through the public entry
points, over the sizes, shapes, storage types and options of the repository's own tests, studies
and benchmark.

Kinds of case (the "kind" of a case's dict):
  sweep   one brickSweep of a resident field (the plain drop-in; also FP32 / BF16 storage, the
          float-float and compensated accumulation modes, other brick dims and folds)
  steps   timeSteps: ping-pong sweeps with the periodic ghost fill before each (the time loop of
          the weak-scaling driver and of the precision study)
  batch   Batch.run: many uneven periodic domains, one launch per step and stencil, replayed
          from a captured graph
  serve   a Server that takes a burst of mixed jobs with host inputs and outputs
  sweep4  one sweep of 4-D bricks (the 4-D weak-scaling driver)
  move    array -> bricks, periodic ghost fill, bricks -> array on the device: what a time loop
          in array-based code does around its sweeps
"""
import math

import numpy as np
import torch

from bricklib_gb300 import batch as BT
from bricklib_gb300 import bricks as B
from bricklib_gb300 import bricks4 as B4
from bricklib_gb300 import serving as SV
from bricklib_gb300 import stencils

TORCH = {"f64": torch.float64, "f32": torch.float32, "bf16": torch.bfloat16}
SIZE = {"f64": 8, "f32": 4, "bf16": 2}
ACC = {"native": 0, "compensated": 1, "floatfloat": 2}
DEV = "cuda"


# ---------------------------------------------------------------- the cases

def listed():
    return [
        # the smallest call: one sweep of a 32^3 block, as a strong-scaling rank's share or a unit
        # test has it -- launch and host time
        sweep("f64-star7-32", "star7", (32, 32, 32), "f64"),
        # the reference driver's own size: 128^3 interior, one ghost brick, the 7-point Laplacian
        sweep("f64-lap7-128", "lap7", (128, 128, 128), "f64"),
        # a box that is no cube and fills no round number of blocks, in single precision
        sweep("f32-star13-ragged", "star13", (136, 408, 200), "f32"),
        # the plain drop-in at the benchmark's size: widest star, plain cube, symmetric cube
        sweep("f64-star25-512", "star25", (512, 512, 512), "f64"),
        sweep("f64-cube27-256", "cube27", (256, 256, 256), "f64"),
        sweep("f64-cube125-512", "cube125", (512, 512, 512), "f64"),
        # time steps of an explicit heat solve in double precision, ghost zone refreshed each step
        steps("f64-heat7-steps", "heat7", (256, 256, 256), "f64", 10),
        # the precision study: the same heat solve stored in bfloat16 at the study's size
        steps("bf16-heat7-steps", "heat7", (512, 512, 512), "bf16", 10),
        # ... and its 125-point cube in single precision with compensated sums
        steps("f32-cube125-comp-steps", "cube125", (256, 256, 256), "f32", 4, acc="compensated"),
        # many small independent problems at once: the batched form's own workload
        {"name": "f32-batch-256", "kind": "batch", "dtype": "f32", "domains": 256, "mix": 4, "lo": 16, "hi": 192,
         "steps": 10},
        # a burst of requests to the server: mixed sizes, shapes, step counts and storage types
        {"name": "serve-24", "kind": "serve", "jobs": 24, "mix": 11, "lo": 16, "hi": 128, "max_steps": 60,
         "f64_share": 0.5},
        # the 4-D driver's star on 64^4
        {"name": "f64-4d-64", "kind": "sweep4", "dtype": "f64", "n0": 64, "n1": 64, "n2": 64, "n3": 64},
    ]


def sweep(name, shape, n, dtype, acc="native", layout="8x8x8"):
    return {"name": name, "kind": "sweep", "shape": shape, "nk": n[0], "nj": n[1], "ni": n[2], "dtype": dtype,
            "acc": acc, "layout": layout}


def steps(name, shape, n, dtype, count, acc="native"):
    return {"name": name, "kind": "steps", "shape": shape, "nk": n[0], "nj": n[1], "ni": n[2], "dtype": dtype,
            "acc": acc, "layout": "8x8x8", "steps": count}


# brick dims and folds (k, j, i) in use besides the default: the small brick of the autotuner,
# the long ones, and a fold that is not row-major
LAYOUTS = {
    "8x8x8": B.Layout((8, 8, 8), (1, 4, 8)),
    "4x4x4": B.Layout((4, 4, 4), (1, 4, 4)),
    "16x8x8": B.Layout((16, 8, 8), (1, 4, 8)),
    "8x8x32": B.Layout((8, 8, 32), (1, 1, 32)),
    "8x8x8 fold 2x4x4": B.Layout((8, 8, 8), (2, 4, 4)),
}


def draw(rng):
    kind = rng.choices(["sweep", "steps", "batch", "serve", "sweep4", "move"], [8, 3, 2, 1, 1, 1])[0]
    log = lambda lo, hi: math.exp(rng.uniform(math.log(lo), math.log(hi)))  # noqa: E731
    shapes = ["star7", "star13", "star25", "cube27", "cube125", "heat7"]

    def box(unit, most):
        while True:
            n = [max(unit[a], int(round(log(16, 512) / unit[a])) * unit[a]) for a in range(3)]
            if n[0] * n[1] * n[2] <= most:
                return n

    if kind == "sweep":
        dtype = rng.choices(["f64", "f32", "bf16"], [3, 2, 1])[0]
        layout = rng.choices(list(LAYOUTS), [12, 1, 1, 1, 1])[0]
        acc = "native"
        if layout == "8x8x8" and rng.random() < 0.2:
            acc = "floatfloat" if dtype == "f64" else "compensated"
        shape = rng.choice(shapes)
        if layout != "8x8x8":
            shape = rng.choice(["star7", "star13", "cube27"])
        n = box([max(8, b) for b in LAYOUTS[layout].bdim], 512 ** 3 if layout == "8x8x8" else 200 ** 3)
        c = sweep("", shape, n, dtype, acc, layout)
    elif kind == "steps":
        dtype = rng.choice(["f64", "f32", "bf16"])
        c = steps("", rng.choice(shapes), box([8, 8, 8], 256 ** 3), dtype, rng.randint(1, 8))
    elif kind == "batch":
        c = {"kind": "batch", "dtype": rng.choice(["f32", "f32", "f64"]), "domains": int(log(4, 160)),
             "mix": rng.randint(1, 999), "lo": 16, "hi": rng.choice([64, 96, 128]), "steps": 2 * rng.randint(1, 5)}
    elif kind == "serve":
        c = {"kind": "serve", "jobs": rng.randint(4, 24), "mix": rng.randint(1, 999), "lo": 16,
             "hi": rng.choice([48, 64, 96]), "max_steps": rng.randint(10, 60), "f64_share": rng.choice([0.0, 0.5, 1.0])}
    elif kind == "sweep4":
        n = [4 * rng.randint(4, 16) for _ in range(4)]
        c = {"kind": "sweep4", "dtype": rng.choice(["f64", "f32"]), "n0": n[0], "n1": n[1], "n2": n[2], "n3": n[3]}
    else:
        n = box([8, 8, 8], 384 ** 3)
        c = {"kind": "move", "nk": n[0], "nj": n[1], "ni": n[2], "dtype": rng.choice(["f64", "f32"]),
             "layout": "8x8x8"}
    c.pop("name", None)
    return c


# ---------------------------------------------------------------- helpers

class _View:
    def __init__(self, owner, ptr, count, typestr):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": (count,), "typestr": typestr, "data": (ptr, False), "version": 3,
                                         "strides": None}


def as_tensor(storage, dtype):
    """The storage's device memory as a torch tensor [chunks, step] (no copy)."""
    typestr = {"f64": "<f8", "f32": "<f4", "bf16": "<i2"}[dtype]
    t = torch.as_tensor(_View(storage, storage.ptr, storage.chunks * storage.step, typestr), device=DEV)
    t = t.view(torch.bfloat16) if dtype == "bf16" else t
    return t.view(storage.chunks, storage.step)


def generator(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    return g


def uniform_array(n, dtype, seed):
    """Uniform [-1, 1) values in the storage type."""
    a = torch.rand(tuple(n), dtype=torch.float64, device=DEV, generator=generator(seed))
    return a.mul_(2.0).sub_(1.0).to(TORCH[dtype])


def sines_array(n, dtype, seed):
    """A sum of eight random-phase sines and uniform noise of amplitude 1e-3."""
    r = np.random.RandomState(seed % (1 << 31))
    a = torch.zeros(tuple(n), dtype=torch.float64, device=DEV)
    x = [torch.arange(m, dtype=torch.float64, device=DEV) / m for m in n]
    for _ in range(8):
        f, ph = r.randint(1, 5, 3), r.uniform(0, 2 * math.pi)
        a += torch.sin(2 * math.pi * (f[0] * x[0][:, None, None] + f[1] * x[1][:, None] + f[2] * x[2]) + ph)
    a += 1e-3 * (2 * torch.rand(tuple(n), dtype=torch.float64, device=DEV, generator=generator(seed)) - 1)
    return a.to(TORCH[dtype])


def layout_of(case):
    return LAYOUTS[case["layout"]]


def ghost_of(lay):
    return tuple(max(8, b) for b in lay.bdim)


def interior_of(case):
    return (case["nk"], case["nj"], case["ni"])


def to_bricks(arr, lay):
    """A (k, j, i) array of whole bricks as [bricks, elements in storage order]."""
    bd = lay.bdim
    nb = [arr.shape[a] // bd[a] for a in range(3)]
    t = arr.reshape(nb[0], bd[0], nb[1], bd[1], nb[2], bd[2]).permute(0, 2, 4, 1, 3, 5)
    t = t.reshape(nb[0] * nb[1] * nb[2], bd[0] * bd[1] * bd[2])
    fk, fj, fi = lay.fold
    k, j, i = np.meshgrid(*[np.arange(b) for b in bd], indexing="ij")
    vec = ((k // fk) * (bd[1] // fj) + j // fj) * (bd[2] // fi) + i // fi
    off = (vec * (fk * fj * fi) + ((k % fk) * fj + j % fj) * fi + i % fi).reshape(-1)
    out = torch.empty_like(t)
    out[:, torch.from_numpy(off).to(t.device)] = t
    return out


def taps_of(shape):
    st = stencils.make(shape, 5)
    return list(zip(st.taps, [float(c) for c in st.coeff]))


def sum_of_taps(views, coeffs, careful):
    """sum of c * view in 64 bits; careful: with the rounding errors of products and sums carried
    along, so that the value is the sum's own and not that of one order of summation."""
    s = None
    if not careful:
        for v, c in zip(views, coeffs):
            s = v * c if s is None else s.add_(v, alpha=c)
        return s
    e = None
    for (v, vh, vl), c in zip(views, coeffs):
        t = c * 134217729.0
        ch = t - (t - c)
        cl = c - ch
        p = v * c
        pe = (vh * ch).sub_(p).add_(vl, alpha=ch).add_(vh, alpha=cl).add_(vl, alpha=cl)
        if s is None:
            s, e = p, pe
            continue
        n = s + p
        b = n - s
        e.add_(pe).add_(p.sub_(b)).add_(s.sub_(n.sub(b)))
        s = n
    return s.add_(e)


def split(x):
    t = x * 134217729.0
    h = t - (t - x)
    return x, h, x - h


def apply_box(arr, taps, org, n, careful):
    """The stencil at every point of the box [org, org + n) of a 64-bit array."""
    parts = split(arr) if careful else (arr,)

    def at(p, t):
        return p[tuple(slice(org[a] + t[a], org[a] + t[a] + n[a]) for a in range(len(n)))]

    views = [tuple(at(p, t) for p in parts) if careful else at(parts[0], t) for t, _ in taps]
    return sum_of_taps(views, [c for _, c in taps], careful)


def apply_periodic(arr, taps, careful=False):
    r = max(max(abs(a) for a in t) for t, _ in taps)
    big = arr
    for a in range(arr.dim()):
        m = arr.shape[a]
        idx = torch.arange(-r, m + r, device=arr.device) % m
        big = big.index_select(a, idx)
    return apply_box(big, taps, (r,) * arr.dim(), tuple(arr.shape), careful)


def domain(case, dtype):
    """The device side of one block: adjacency, interior list and grid of interior + ghost."""
    lay, n = layout_of(case), interior_of(case)
    ghost = ghost_of(lay)
    g = tuple((n[a] + 2 * ghost[a]) // lay.bdim[a] for a in range(3))
    grid, info = B.init_grid(list(reversed(g)))
    gb = tuple(ghost[a] // lay.bdim[a] for a in range(3))
    nb = tuple(n[a] // lay.bdim[a] for a in range(3))
    inner = grid.reshape(g)[gb[0]:gb[0] + nb[0], gb[1]:gb[1] + nb[1], gb[2]:gb[2] + nb[2]].reshape(-1)
    return {"lay": lay, "n": n, "ghost": ghost, "g": g, "grid": grid, "info": B.movBrickInfo(info), "nb": nb, "gb": gb,
            "nbricks": info.nbricks, "blist": B.BrickList(np.ascontiguousarray(inner))}


def interior_slices(n, ghost):
    return tuple(slice(ghost[a], ghost[a] + n[a]) for a in range(3))


# ---------------------------------------------------------------- sweep, steps, move

def prepare_block(case, seed):
    kind, dtype = case["kind"], case["dtype"]
    d = domain(case, dtype)
    lay, n, ghost = d["lay"], d["n"], d["ghost"]
    a = B.BrickStorage.allocate_device(d["nbricks"], lay.size, dtype)
    b = B.BrickStorage.allocate_device(d["nbricks"], lay.size, dtype)
    d["a"], d["b"] = B.Brick(d["info"], a, 0, lay), B.Brick(d["info"], b, 0, lay)
    d["ta"], d["tb"] = as_tensor(a, dtype), as_tensor(b, dtype)
    full = tuple(n[x] + 2 * ghost[x] for x in range(3))
    if kind == "sweep":
        d["ta"].copy_(to_bricks(uniform_array(full, dtype, seed), lay))
        d["st"] = B.to_c_stencil(stencils.make(case["shape"], 5))
        d["acc"] = ACC[case["acc"]]
        return d
    d["plan"] = B.GhostPlan.periodic(d["grid"], d["nb"], d["gb"])
    if kind == "steps":
        arr = torch.zeros(full, dtype=TORCH[dtype], device=DEV)
        arr[interior_slices(n, ghost)] = sines_array(n, dtype, seed)
        d["ta"].copy_(to_bricks(arr, lay))
        d["st"] = B.to_c_stencil(stencils.make(case["shape"], 5))
        d["acc"], d["steps"] = ACC[case["acc"]], case["steps"]
        return d
    d["arr"] = uniform_array(full, dtype, seed)
    d["back"] = torch.zeros_like(d["arr"])
    d["grid_dev"] = B.BrickList(d["grid"])
    return d


def run_sweep(s):
    B.brickSweep(s["a"], s["b"], s["blist"], s["st"], s["acc"])
    return s["tb"]


def run_steps(s):
    new = B.timeSteps(s["a"], s["b"], s["blist"], s["st"], s["steps"], plan=s["plan"], acc=s["acc"])
    return s["ta"] if new is s["a"] else s["tb"]


def run_move(s):
    n, gh = s["n"], s["ghost"]
    inner = [n[2], n[1], n[0]]
    whole = [n[2] + 2 * gh[2], n[1] + 2 * gh[1], n[0] + 2 * gh[0]]
    g = [gh[2], gh[1], gh[0]]
    B.copyToBrickDevice(inner, [0, 0, 0], g, s["arr"].data_ptr(), s["grid_dev"].ptr, s["a"])
    B.ghostFill(s["plan"], s["a"])
    B.copyFromBrickDevice(whole, [0, 0, 0], [0, 0, 0], s["back"].data_ptr(), s["grid_dev"].ptr, s["a"])
    return s["ta"], s["back"]


def exact_block(case, seed):
    kind, dtype = case["kind"], case["dtype"]
    lay, n = layout_of(case), interior_of(case)
    ghost = ghost_of(lay)
    full = tuple(n[x] + 2 * ghost[x] for x in range(3))
    out = torch.zeros(full, dtype=torch.float64, device=DEV)
    inner = interior_slices(n, ghost)
    if kind == "sweep":
        arr = uniform_array(full, dtype, seed).double()
        out[inner] = apply_box(arr, taps_of(case["shape"]), ghost, n, dtype == "f64")
        return to_bricks(out, lay)
    if kind == "steps":
        # the ghost bricks of the returned field hold the fill of an earlier step or nothing:
        # what the last fill of this buffer put there
        cur = sines_array(n, dtype, seed).double()
        taps = taps_of(case["shape"])
        fill = None
        for t in range(case["steps"]):
            if t % 2 == case["steps"] % 2:
                fill = cur
            cur = apply_periodic(cur, taps, dtype == "f64")
        if fill is not None:
            out.copy_(wrap(fill, n, ghost))
        out[inner] = cur
        return to_bricks(out, lay)
    arr = uniform_array(full, dtype, seed).double()
    w = wrap(arr[inner], n, ghost)
    return to_bricks(w, lay), w


def wrap(arr, n, ghost):
    for a in range(3):
        arr = arr.index_select(a, torch.arange(-ghost[a], n[a] + ghost[a], device=arr.device) % n[a])
    return arr


# ---------------------------------------------------------------- batch

def workload(case):
    return BT.make_workload(case["domains"], case["mix"], case["lo"], case["hi"])


def domain_array(n, dtype, seed, q):
    return uniform_array(n, dtype, seed * 1009 + q)


def prepare_batch(case, seed):
    lay = B.DEFAULT_LAYOUT
    w = workload(case)
    b = BT.Batch(w, lay, B.dtype_of(case["dtype"]), init=False)
    nbricks = sum(ds.nbricks for ds in b.doms)
    arena = B.BrickStorage(nbricks, 2 * lay.size, case["dtype"], device=b.arena)
    t = as_tensor(arena, case["dtype"])
    first = 0
    for q, ds in enumerate(b.doms):
        inner = torch.from_numpy(ds.interior.astype(np.int64) + first).to(DEV)
        t[inner, :lay.size] = to_bricks(domain_array(ds.spec.n, case["dtype"], seed, q), lay)
        first += ds.nbricks
    return {"batch": b, "arena": t, "steps": case["steps"]}


def run_batch(s):
    s["batch"].run(s["steps"])
    return s["arena"]


def exact_batch(case, seed):
    lay = B.DEFAULT_LAYOUT
    w = workload(case)
    out = []
    for q, d in enumerate(w.domains):
        st = w.stencils[d.stencil]
        taps = list(zip(st.taps, [float(c) for c in st.coeff]))
        cur = domain_array(d.n, case["dtype"], seed, q).double()
        last = cur
        for _ in range(case["steps"]):
            last, cur = cur, apply_periodic(cur, taps)
        nb = [x // 8 + 2 for x in d.n]
        part = torch.zeros(nb + [2 * lay.size], dtype=torch.float64, device=DEV)
        part[1:-1, 1:-1, 1:-1, :lay.size] = to_bricks(cur, lay).reshape([x // 8 for x in d.n] + [lay.size])
        part[1:-1, 1:-1, 1:-1, lay.size:] = to_bricks(last, lay).reshape([x // 8 for x in d.n] + [lay.size])
        out.append(part.reshape(-1, 2 * lay.size))
    return torch.cat(out)


# ---------------------------------------------------------------- serve

def jobs_of(case):
    return SV.make_jobs(case["jobs"], case["mix"], case["lo"], case["hi"], case["max_steps"],
                        fp64_frac=case["f64_share"])


def job_input(job, seed, q):
    a = np.random.default_rng([seed, q]).random(job.n, dtype=np.float64)
    a *= 2.0
    a -= 1.0
    return a.astype(np.float64 if job.dtype == 0 else np.float32)


def prepare_serve(case, seed):
    jobs = jobs_of(case)
    sizes = [j.points * (8 if j.dtype == 0 else 4) for j in jobs]
    bytes_ = torch.empty(2 * sum(sizes), dtype=torch.uint8, pin_memory=True).numpy()
    off, ins, outs = 0, [], []
    for q, (j, size) in enumerate(zip(jobs, sizes)):
        dt = np.float64 if j.dtype == 0 else np.float32
        ins.append(bytes_[off:off + size].view(dt).reshape(j.n))
        outs.append(bytes_[off + size:off + 2 * size].view(dt).reshape(j.n))
        ins[-1][...] = job_input(j, seed, q)
        off += 2 * size
    sts = [B.to_c_stencil(stencils.make(j.shape, 5)) for j in jobs]
    return {"server": SV.Server(), "jobs": jobs, "sts": sts, "ins": ins, "outs": outs}


def run_serve(s):
    ids = [s["server"].submit(j.n, st, j.steps, j.dtype, 0, a, o)
           for j, st, a, o in zip(s["jobs"], s["sts"], s["ins"], s["outs"])]
    for i in ids:
        s["server"].wait(i)
    return s["outs"]


def exact_serve(case, seed):
    jobs = jobs_of(case)
    if sum(j.points * j.steps * len(taps_of(j.shape)) for j in jobs) > 1.5e11:
        return None
    out = []
    for q, j in enumerate(jobs):
        cur = torch.from_numpy(job_input(j, seed, q)).to(DEV).double()
        taps = taps_of(j.shape)
        for _ in range(j.steps):
            cur = apply_periodic(cur, taps)
        out.append(cur.cpu().numpy())
    return out


# ---------------------------------------------------------------- sweep4

def dims4(case):
    return (case["n0"], case["n1"], case["n2"], case["n3"])


def fold4():
    """Storage position of every element of a 4^4 brick in row-major order, fold (1, 1, 2, 4)."""
    l, k, j, i = np.indices((4, 4, 4, 4)).reshape(4, -1)
    return torch.from_numpy(((l * 4 + k) * 2 + j // 2) * 8 + (j % 2) * 4 + i).to(DEV)


def prepare_sweep4(case, seed):
    lay = B4.Layout4()
    g = [x // 4 + 2 for x in dims4(case)]
    grid, adj = B4.init_grid(list(reversed(g)))
    inner = grid.reshape(g)[1:-1, 1:-1, 1:-1, 1:-1].reshape(-1)
    dev = B.DeviceBuffer(adj.nbytes)
    dev.upload(adj)
    a = B.BrickStorage.allocate_device(len(grid), lay.size, case["dtype"])
    b = B.BrickStorage.allocate_device(len(grid), lay.size, case["dtype"])
    as_tensor(a, case["dtype"]).copy_(uniform_array((len(grid), lay.size), case["dtype"], seed))
    return {"adj": dev, "nbricks": len(grid), "a": a, "b": b, "tb": as_tensor(b, case["dtype"]),
            "blist": B.BrickList(np.ascontiguousarray(inner)), "st": B4.to_c_stencil4(B4.mpi9pt()), "lay": lay}


def run_sweep4(s):
    B4.sweep4(s["adj"], s["nbricks"], s["a"], 0, 0, s["blist"], s["st"], s["lay"], out_storage=s["b"])
    return s["tb"]


def exact_sweep4(case, seed):
    g = [x // 4 + 2 for x in dims4(case)]
    pos = fold4()
    t = uniform_array((g[0] * g[1] * g[2] * g[3], 256), case["dtype"], seed).double()[:, pos]
    arr = t.reshape(g + [4, 4, 4, 4]).permute(0, 4, 1, 5, 2, 6, 3, 7).reshape([4 * x for x in g])
    n = dims4(case)
    taps = [((0, 0, 0, 0), 0.2)]
    for a in (3, 2, 1, 0):
        for s in (1, -1):
            taps.append((tuple(s if d == a else 0 for d in range(4)), 0.1))
    out = torch.zeros_like(arr)
    out[tuple(slice(4, 4 + x) for x in n)] = apply_box(arr, taps, (4,) * 4, n, case["dtype"] == "f64")
    t = out.reshape(g[0], 4, g[1], 4, g[2], 4, g[3], 4).permute(0, 2, 4, 6, 1, 3, 5, 7).reshape(-1, 256)
    r = torch.empty_like(t)
    r[:, pos] = t
    return r


# ---------------------------------------------------------------- the interface

PREPARE = {"sweep": prepare_block, "steps": prepare_block, "move": prepare_block, "batch": prepare_batch,
           "serve": prepare_serve, "sweep4": prepare_sweep4}
RUN = {"sweep": run_sweep, "steps": run_steps, "move": run_move, "batch": run_batch, "serve": run_serve,
       "sweep4": run_sweep4}
EXACT = {"sweep": exact_block, "steps": exact_block, "move": exact_block, "batch": exact_batch, "serve": exact_serve,
         "sweep4": exact_sweep4}


def prepare(case, seed):
    s = PREPARE[case["kind"]](case, seed)
    s["run"] = RUN[case["kind"]]
    return s


def run(state):
    return state["run"](state)


def exact(case, seed):
    return EXACT[case["kind"]](case, seed)


def work(case):
    """Bytes: every point read and written once per sweep (what one step needs of the field),
    copies likewise.  Flops: two per tap and point."""
    kind = case["kind"]
    if kind == "batch":
        w = workload(case)
        p = sum(math.prod(d.n) for d in w.domains)
        f = sum(math.prod(d.n) * 2 * w.stencils[d.stencil].npoints for d in w.domains)
        return {"bytes": 2 * SIZE[case["dtype"]] * p * case["steps"], "flops": f * case["steps"]}
    if kind == "serve":
        jobs = jobs_of(case)
        return {"bytes": sum(2 * (8 if j.dtype == 0 else 4) * j.points * j.steps for j in jobs),
                "flops": sum(2 * len(taps_of(j.shape)) * j.points * j.steps for j in jobs)}
    if kind == "sweep4":
        p = math.prod(dims4(case))
        return {"bytes": 2 * SIZE[case["dtype"]] * p, "flops": 18 * p}
    p = math.prod(interior_of(case))
    es = SIZE[case["dtype"]]
    if kind == "move":
        full = math.prod(x + 16 for x in interior_of(case))
        # array in and bricks out; ghost bricks read and written; bricks in and array out
        return {"bytes": 2 * es * (p + (full - p) + full), "flops": 0}
    t = case.get("steps", 1)
    return {"bytes": 2 * es * p * t, "flops": 2 * len(taps_of(case["shape"])) * p * t}
