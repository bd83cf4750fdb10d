"""The work that a program using abhsf_b200 has it do, as cases to be timed.

A case is a dict of plain values.  "do" names the path:

spmv   y += A x with the matrix resident on the GPU
spmm   Y += A X, X and Y with k columns
batch  y_i += A_i x_i for many matrices of different sizes, one call
cg     solves A x = b (a Laplacian) to 1e-10: FP64 CG, or the mixed-precision
       CG on an f32 / bf16 copy of the matrix
build  the format built from COO triplets on the GPU and one y += A x with it
       (a program whose matrix changes pays for both)
stats  the block histograms of all 64 block sizes

and "shape" the kind of matrix: "mixture" (64 x 64 tiles of the densities that
every storage scheme serves), "rmat" (power-law graph), "banded", "laplacian2d"
and "laplacian3d" (5- and 7-point stencils).
"""
import math

import numpy as np
import torch

from abhsf_b200 import AbhsfBatch, AbhsfMatrix, block_histograms_all, cg, cg_mixed
from abhsf_b200 import workloads as W

TILE = 64
# mean elements of an occupied mixture tile: 20% hold 0.9 of 64 x 64, 30% a
# share U[0.15, 0.5], 50% 1 to 8 elements
MIX_MEAN = 0.2 * 0.9 * 4096 + 0.3 * 0.325 * 4096 + 0.5 * 4.5
MIX_BITMAP = 0.5


def listed():
    return [
        # the smallest matrix of a set of many: the call itself is what counts
        {"name": "spmv_banded_1k", "do": "spmv", "shape": "banded", "n": 1000, "band": 5, "values": "f64", "block": 64},
        # the large mixed-scheme matrix: the product that ABHSF is for
        {"name": "spmv_mixture", "do": "spmv", "shape": "mixture", "n": 4194304, "tiles": 0.8, "values": "f64",
         "block": 64},
        # its f32-stored copy, for solvers and learning code that work in f32
        {"name": "spmv_mixture_f32", "do": "spmv", "shape": "mixture", "n": 4194304, "tiles": 0.8, "values": "f32",
         "block": 64},
        # a power-law graph with rows of a few and of 100,000 elements
        {"name": "spmv_rmat22", "do": "spmv", "shape": "rmat", "scale": 22, "edge": 16, "values": "f64", "block": 64},
        # block Krylov and multi-vector programs: many right-hand sides
        {"name": "spmm_mixture_k32", "do": "spmm", "shape": "mixture", "n": 4194304, "tiles": 0.8, "k": 32, "block": 64},
        # an odd number of right-hand sides on a graph
        {"name": "spmm_rmat18_k7", "do": "spmm", "shape": "rmat", "scale": 18, "edge": 8, "k": 7, "block": 64},
        # 256 matrices, n log-uniform in [1k, 200k], half banded, half R-MAT
        {"name": "batch_256", "do": "batch", "count": 256, "n_min": 1000, "n_max": 200000, "block": 64},
        # a solve whose iteration is a few microseconds of small kernels
        {"name": "cg_laplacian2d_512", "do": "cg", "shape": "laplacian2d", "g": 512, "low": "none", "block": 64},
        # the large solve: bf16 copy inside, FP64 outside
        {"name": "cg_mixed_laplacian3d_256", "do": "cg", "shape": "laplacian3d", "g": 256, "low": "bf16", "block": 32},
        # the format of the large mixed-scheme matrix, from sorted triplets
        {"name": "build_mixture", "do": "build", "shape": "mixture", "n": 4194304, "tiles": 0.8, "values": "f64",
         "block": 64, "auto": False, "shuffled": False},
        # a graph's format, the block size picked by least storage, triplets in no order
        {"name": "build_auto_rmat17", "do": "build", "shape": "rmat", "scale": 17, "edge": 8, "values": "f64",
         "block": 64, "auto": True, "shuffled": True},
        # the block statistics that the choice of a block size is studied with
        {"name": "stats_mixture", "do": "stats", "shape": "mixture", "n": 4194304, "tiles": 0.8},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_shape(rng, kinds):
    shape = rng.choice(kinds)
    if shape == "mixture":
        n = _log(rng, 20_000, 4_000_000)
        # up to about as many elements as the listed mixture
        most = 40_000 / (n / TILE)
        return {"shape": shape, "n": n, "tiles": round(min(math.exp(rng.uniform(math.log(0.5), math.log(12.0))), most), 2)}
    if shape == "rmat":
        return {"shape": shape, "scale": rng.randint(12, 21), "edge": rng.randint(4, 16)}
    if shape == "banded":
        n = _log(rng, 1000, 1_000_000)
        return {"shape": shape, "n": n, "band": max(1, min(_log(rng, 1, 100), 15_000_000 // n))}
    return {"shape": shape, "g": rng.randint(100, 1500) if shape == "laplacian2d" else rng.randint(20, 180)}


def draw(rng):
    do = rng.choice(["spmv", "spmv", "spmv", "spmm", "spmm", "batch", "cg", "build", "build", "stats"])
    every = ["mixture", "rmat", "banded", "laplacian2d", "laplacian3d"]
    if do == "spmv":
        return {"do": do, **_draw_shape(rng, every), "values": rng.choice(["f64", "f64", "f32", "bf16"]),
                "block": rng.choice([64, 64, 32, 16, 128, 256])}
    if do == "spmm":
        c = {"do": do, **_draw_shape(rng, every), "block": rng.choice([64, 64, 32])}
        return {**c, "k": rng.choice([2, 3, 4, 5, 8, 11, 16, 20, 32])}
    if do == "batch":
        lo = _log(rng, 500, 5000)
        return {"do": do, "count": rng.randint(8, 120), "n_min": lo, "n_max": lo * rng.randint(2, 40), "block":
                rng.choice([64, 64, 32])}
    if do == "cg":
        shape = rng.choice(["laplacian2d", "laplacian3d"])
        return {"do": do, "shape": shape, "g": rng.randint(60, 700) if shape == "laplacian2d" else rng.randint(16, 160),
                "low": rng.choice(["none", "f32", "bf16"]), "block": rng.choice([64, 32])}
    if do == "build":
        auto = rng.random() < 0.3
        return {"do": do, **_draw_shape(rng, every), "values": rng.choice(["f64", "f64", "f32", "bf16"]),
                "block": rng.choice([64, 64, 32, 16, 128, 256]), "auto": auto, "shuffled": rng.random() < 0.5}
    return {"do": do, **_draw_shape(rng, ["mixture", "rmat"])}


# ------------------------------------------------------------------ matrices
def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _mixture(n, tiles, seed):
    """n x n in 64 x 64 tiles, on average `tiles` occupied ones a block row:
    20% hold each entry with probability 0.9, 30% with a probability
    U[0.15, 0.5], 50% hold 1 to 8 entries.  (row, column) sorted by row."""
    g = _generator(seed)
    nb = -(-n // TILE)
    at = torch.unique(torch.randint(0, nb * nb, (max(1, int(tiles * nb)),), device="cuda", generator=g))
    kind = torch.rand(at.numel(), device="cuda", generator=g)
    dens = torch.rand(at.numel(), device="cuda", generator=g) * 0.35 + 0.15
    dens = torch.where(kind < 0.2, torch.full_like(dens, 0.9), dens)
    few = kind >= 0.5
    keys = []

    def add(tile, loc):
        r = torch.div(tile, nb, rounding_mode="floor") * TILE + torch.div(loc, TILE, rounding_mode="floor")
        c = tile % nb * TILE + loc % TILE
        ok = (r < n) & (c < n)
        keys.append(r[ok] * n + c[ok])

    full = torch.nonzero(~few).squeeze(1)
    for part in torch.split(full, 4096):
        hit = torch.rand((part.numel(), TILE * TILE), device="cuda", generator=g) < dens[part][:, None]
        t, loc = torch.nonzero(hit, as_tuple=True)
        add(at[part][t], loc)
    some = torch.nonzero(few).squeeze(1)
    count = torch.randint(1, 9, (some.numel(),), device="cuda", generator=g)
    t = torch.repeat_interleave(at[some], count)
    add(t, torch.randint(0, TILE * TILE, (t.numel(),), device="cuda", generator=g))
    key = torch.unique(torch.cat(keys))
    rows = torch.div(key, n, rounding_mode="floor")
    return rows, key - rows * n, n


def _banded(n, w):
    offs = torch.arange(-w, w + 1, device="cuda")
    rows = torch.arange(n, device="cuda").repeat_interleave(offs.numel())
    cols = rows + offs.repeat(n)
    ok = (cols >= 0) & (cols < n)
    return rows[ok], cols[ok], n


def _coordinates(case, seed):
    """(rows, cols, n) of the case's matrix, sorted by row, then column."""
    shape = case["shape"]
    if shape == "mixture":
        return _mixture(case["n"], case["tiles"], seed)
    if shape == "rmat":
        rows, cols, _, n = W.rmat_device(case["scale"], case["edge"], seed=seed, device="cuda")
        return rows, cols, n
    if shape == "banded":
        return _banded(case["n"], case["band"])
    g = case["g"]
    d = 2 if shape == "laplacian2d" else 3
    n = g ** d
    i = torch.arange(n, device="cuda")
    steps, inside = [0], [None]
    for k in range(d):
        x = torch.div(i, g ** k, rounding_mode="floor") % g
        steps = [-g ** k] + steps + [g ** k]
        inside = [x > 0] + inside + [x < g - 1]
    ok = torch.stack([torch.ones_like(i, dtype=torch.bool) if m is None else m for m in inside], 1)
    at = torch.nonzero(ok)
    rows = at[:, 0].contiguous()
    return rows, rows + torch.tensor(steps, device="cuda")[at[:, 1]], n


def _triplets(case, seed):
    rows, cols, n = _coordinates(case, seed)
    if case["shape"].startswith("laplacian"):
        vals = torch.where(rows == cols, 4.0 if case["shape"] == "laplacian2d" else 6.0, -1.0).double()
    else:
        vals = torch.randn(rows.numel(), dtype=torch.float64, device="cuda", generator=_generator(seed + 1))
    return rows, cols, vals, n


def _vector(seed, *shape, dtype=torch.float64):
    return torch.rand(shape, dtype=torch.float64, device="cuda", generator=_generator(seed)).mul_(2).sub_(1).to(dtype)


def _vectors(case, seed, n):
    dtype = torch.float64 if case.get("values", "f64") == "f64" else torch.float32
    shape = (n, case["k"]) if "k" in case else (n,)
    return _vector(seed + 2, *shape, dtype=dtype), _vector(seed + 3, *shape, dtype=dtype)


def _batch(case, seed):
    """The matrices of the batch, one after another: sizes log-uniform (the
    case's own, whatever the seed), every other one banded (3 to 64 entries to
    each side), the others R-MAT of edge factor 8."""
    rng = np.random.default_rng([case["count"], case["n_min"], case["n_max"]])
    sizes = np.exp(rng.uniform(math.log(case["n_min"]), math.log(case["n_max"]), case["count"])).astype(int)
    bands = rng.integers(3, 65, case["count"])
    g = _generator(seed)
    for i in range(case["count"]):
        n = int(sizes[i])
        if i % 2 == 0:
            rows, cols, _ = _banded(n, int(bands[i]))
        else:
            r = torch.zeros(8 * n, dtype=torch.int64, device="cuda")
            c = torch.zeros_like(r)
            for _ in range((n - 1).bit_length()):
                u = torch.rand(8 * n, device="cuda", generator=g)
                r = 2 * r + (u >= 0.76)
                c = 2 * c + (((u >= 0.57) & (u < 0.76)) | (u >= 0.95))
            ok = (r < n) & (c < n)
            key = torch.unique(r[ok] * n + c[ok])
            rows = torch.div(key, n, rounding_mode="floor")
            cols = key - rows * n
        yield rows, cols, torch.randn(rows.numel(), dtype=torch.float64, device="cuda", generator=g), n


def _views(flat, sizes):
    """A vector of each size in one buffer, each from a 512-byte boundary."""
    out, at = [], 0
    for n in sizes:
        out.append(flat[at:at + n])
        at += -(-n // 64) * 64
    return out


def _padded(sizes):
    return sum(-(-n // 64) * 64 for n in sizes)


# ------------------------------------------------------------------ the calls
def prepare(case, seed):
    do, s = case["do"], {"case": case}
    if do == "batch":
        mats, sizes = [], []
        for rows, cols, vals, n in _batch(case, seed):
            mats.append(AbhsfMatrix.from_elements(rows, cols, vals, n, n, block_size=case["block"]))
            sizes.append(n)
        x, s["y"] = _vector(seed + 2, _padded(sizes)), _vector(seed + 3, _padded(sizes))
        s["batch"] = AbhsfBatch(mats)
        s["tables"] = s["batch"].pointer_tables(_views(x, sizes), _views(s["y"], sizes))
        s["x"] = x
        return s
    rows, cols, vals, n = _triplets(case, seed)
    if do == "stats":
        s["rows"], s["cols"], s["n"] = rows, cols, n
        return s
    if do == "cg":
        s["A"] = AbhsfMatrix.from_elements(rows, cols, vals, n, n, block_size=case["block"])
        if case["low"] != "none":
            s["low"] = AbhsfMatrix.from_elements(rows, cols, vals, n, n, block_size=case["block"],
                                                 value_type=case["low"])
        s["b"], s["x"] = _vector(seed + 2, n), torch.zeros(n, dtype=torch.float64, device="cuda")
        return s
    s["x"], s["y"] = _vectors(case, seed, n)
    if do == "build":
        if case["shuffled"]:
            order = torch.randperm(rows.numel(), device="cuda", generator=_generator(seed + 4))
            rows, cols, vals = rows[order], cols[order], vals[order]
        s["coo"], s["n"] = (rows, cols, vals), n
        return s
    s["A"] = AbhsfMatrix.from_elements(rows, cols, vals, n, n, block_size=case["block"],
                                       value_type=case.get("values", "f64"))
    return s


def _product(A, case, x, y):
    if case.get("values", "f64") == "f64":
        A.spmv(x, y)
    else:
        A.spmv_f32(x, y)


def _counts(hists):
    """Per block size, the number of blocks of 0, 1, ... r s elements."""
    out = []
    for size, h in hists.items():
        r, s = size.split("x")
        count = np.zeros(int(r) * int(s) + 1, np.int64)
        count[list(h.keys())] = list(h.values())
        out.append(count)
    return out


def run(state):
    case = state["case"]
    do = case["do"]
    if do == "spmv":
        _product(state["A"], case, state["x"], state["y"])
        return state["y"]
    if do == "spmm":
        state["A"].spmm(state["x"], state["y"])
        return state["y"]
    if do == "batch":
        state["batch"].spmv_tables(*state["tables"])
        return state["y"]
    if do == "cg":
        state["x"].zero_()
        if case["low"] == "none":
            info = cg(state["A"], state["b"], state["x"], rtol=1e-10)
        else:
            info = cg_mixed(state["A"], state["low"], state["b"], state["x"], rtol=1e-10)
        return [state["x"], info["converged"]]
    if do == "build":
        n = state["n"]
        A = AbhsfMatrix.from_elements(*state["coo"], n, n, block_size="auto" if case["auto"] else case["block"],
                                      value_type=case["values"])
        _product(A, case, state["x"], state["y"])
        st = A.stats()
        out = [state["y"], st["block_size"], list(st["tiles_per_scheme"].values()),
               list(st["nnz_per_scheme"].values()), st["msmf_bits"]]
        A.release()
        return out
    return _counts(block_histograms_all(state["rows"], state["cols"], state["n"], state["n"]))


# ------------------------------------------------------- floors and 64 bits
def _sizes(case):
    """(n, elements, bytes of the index arrays) of the case's matrix, expected."""
    shape = case["shape"]
    if shape == "mixture":
        n = case["n"]
        t = case["tiles"] * (-(-n // TILE))
        return n, t * MIX_MEAN, t * (MIX_BITMAP * TILE * TILE / 8 + (1 - MIX_BITMAP) * 4.5 * 2 + 8)
    if shape == "rmat":
        n = 1 << case["scale"]
        z = 0.96 * n * case["edge"]
    elif shape == "banded":
        n = case["n"]
        z = n * (2 * case["band"] + 1)
    else:
        d = 2 if shape == "laplacian2d" else 3
        n = case["g"] ** d
        z = n * (2 * d + 1) - 2 * d * case["g"] ** (d - 1)
    return n, z, 4 * z


def work(case):
    do = case["do"]
    if do == "batch":
        # n log-uniform: the mean of n, half with 67 elements a row, half with 8
        lo, hi = case["n_min"], case["n_max"]
        n = case["count"] * (hi - lo) / math.log(hi / lo)
        z = n * (67 + 7.9) / 2
        return {"bytes": z * (8 + 2) + 24 * n, "flops": 2 * z}
    n, z, index = _sizes(case)
    v = {"f64": 8, "f32": 4, "bf16": 2}[case.get("values", "f64")]
    vec = 24 * n if v == 8 else 12 * n
    once = z * v + index + vec * case.get("k", 1)
    if do in ("spmv", "spmm"):
        return {"bytes": once, "flops": 2 * z * case.get("k", 1)}
    if do == "stats":
        return {"bytes": 16 * z, "flops": 0}
    if do == "build":
        return {"bytes": 24 * z + z * v + index + once, "flops": 2 * z}
    # CG: about as many iterations as the grid's side times 2.9 (2D) or 4.1 (3D),
    # each one product and eleven vectors read or written
    its = case["g"] * (2.9 if case["shape"] == "laplacian2d" else 4.1)
    lv, w = {"none": (8, 8), "f32": (4, 4), "bf16": (2, 4)}[case["low"]]
    return {"bytes": its * (z * lv + index + 3 * w * n + 11 * w * n), "flops": its * (2 * z + 12 * n)}


def exact(case, seed):
    do = case["do"]
    if do == "stats":
        return None
    if do == "batch":
        mats = [(r, c, v, n) for r, c, v, n in _batch(case, seed)]
        sizes = [m[3] for m in mats]
        x, y = _vector(seed + 2, _padded(sizes)), _vector(seed + 3, _padded(sizes))
        for (r, c, v, _), xi, yi in zip(mats, _views(x, sizes), _views(y, sizes)):
            yi.index_add_(0, r, v * xi[c])
        return y
    if do == "cg":
        # the Laplacian's eigenvectors are products of sines
        g, d = case["g"], 2 if case["shape"] == "laplacian2d" else 3
        j = torch.arange(1, g + 1, dtype=torch.float64, device="cuda")
        S = torch.sin(j[:, None] * j[None, :] * (math.pi / (g + 1))) * math.sqrt(2 / (g + 1))
        lam = 2 - 2 * torch.cos(j * (math.pi / (g + 1)))
        t = _vector(seed + 2, *([g] * d))
        for k in range(d):
            t = torch.tensordot(t, S, dims=([0], [0]))
        if d == 2:
            t = t / (lam[:, None] + lam[None, :])
        else:
            t = t / (lam[:, None, None] + lam[None, :, None] + lam[None, None, :])
        for k in range(d):
            t = torch.tensordot(t, S, dims=([0], [0]))
        return [t.reshape(-1), None]
    rows, cols, vals, n = _triplets(case, seed)
    x, y = (t.double() for t in _vectors(case, seed, n))
    if case.get("values") == "f32":
        vals = vals.float().double()
    elif case.get("values") == "bf16":
        vals = vals.float().bfloat16().double()
    if "k" in case:
        for h in range(case["k"]):
            col = y[:, h].contiguous()
            y[:, h] = col.index_add_(0, rows, vals * x[:, h].contiguous()[cols])
    else:
        y.index_add_(0, rows, vals * x[cols])
    return [y, None, None, None, None] if do == "build" else y
