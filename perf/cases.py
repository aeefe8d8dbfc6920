"""The work a user of this library has it do, as measurable cases.

Four kinds of call through the public entry points: one product y = A x on
device data (block rows of any block size, or CSR), one product on host
buffers, one BiCGStab solve, and many solves at once (the batch, the server).

Every case's inputs come from its seed: the matrices' values, the patterns of
the synthetic matrices, the material constants of the elasticity operators and
the right-hand sides.
"""
import ctypes
import math

import numpy as np
import torch

import block_matrix_format_performance_gb300 as bm

DTYPES = {"f32": torch.float32, "f64": torch.float64}

# Relative residuals asked for: tight enough that two correct solves agree in x
# to well below 1e-9 on these operators.
TOLERANCE = {"fp64": 1e-12, "mixed": 1e-11}


def listed():
    return [
        # The smallest call: the elasticity operator of a 200x50-node grid
        # (20 000 rows, block size 2), one product through its handle. What an
        # outside Krylov loop calls thousands of times; launch latency counts.
        {"name": "spmv q4 200x50 f64", "kind": "spmv", "pattern": "q4", "nx": 200, "ny": 50, "bs": 2, "dtype": "f64",
         "api": "handle"},
        # The CSR entry point on the arrays of the 1000x250 elasticity operator
        # (500 000 rows, 18 entries each): a caller that never blocked its matrix.
        {"name": "spmv csr 1000x250 f64", "kind": "spmv", "pattern": "q4", "nx": 1000, "ny": 250, "bs": 0,
         "dtype": "f64", "api": "arrays"},
        # The block-size sweep's 100 000 block rows x 8 blocks in a +-64 band at
        # block size 4, FP32, through a handle.
        {"name": "spmv band bs4 f32", "kind": "spmv", "pattern": "band", "rows": 100000, "blocks": 8, "bs": 4,
         "dtype": "f32", "api": "handle"},
        # Block size 3 (three degrees of freedom per node), uneven rows with
        # empty ones among them, on the caller's device arrays.
        {"name": "spmv ragged bs3 f64", "kind": "spmv", "pattern": "ragged", "rows": 150001, "blocks": 8, "bs": 3,
         "dtype": "f64", "api": "arrays"},
        # One of the odd sizes of the reference's sweep over block sizes 2..32:
        # 50 000 block rows of 6 neighbouring blocks, FP32, on device arrays.
        {"name": "spmv ndiag bs12 f32", "kind": "spmv", "pattern": "ndiag", "rows": 50000, "blocks": 6, "bs": 12,
         "dtype": "f32", "api": "arrays"},
        # The largest product of the sweep: block size 32, FP64, 6.6 GB.
        {"name": "spmv band bs32 f64", "kind": "spmv", "pattern": "band", "rows": 100000, "blocks": 8, "bs": 32,
         "dtype": "f64", "api": "handle"},
        # The reference's calling convention: every array in (page-locked) host
        # memory, one call that uploads, multiplies and downloads.
        {"name": "host spmv bs8 f64", "kind": "host", "pattern": "band", "rows": 50000, "blocks": 8, "bs": 8,
         "dtype": "f64"},
        # One implicit time step (K + shift I) on the small grid: latency of a
        # whole solve.
        {"name": "solve 200x50 fp64", "kind": "solve", "nx": 200, "ny": 50, "shift": 1e-2, "precision": "fp64",
         "precond": "none", "format": "bcsr"},
        # The same step at half a million rows with FP32 inner solves.
        {"name": "solve 1000x250 mixed", "kind": "solve", "nx": 1000, "ny": 250, "shift": 1e-2, "precision": "mixed",
         "precond": "none", "format": "bcsr"},
        # The large grid (2 million rows) in plain FP64.
        {"name": "solve 2000x500 fp64", "kind": "solve", "nx": 2000, "ny": 500, "shift": 1e-2, "precision": "fp64",
         "precond": "none", "format": "bcsr"},
        # 256 uneven systems (grids 20x5 to 400x100) in one launch, mixed
        # precision.
        {"name": "batch 256 mixed", "kind": "batch", "systems": 256, "nx_max": 400, "shift": 1e-2,
         "precision": "mixed"},
        # A burst of requests to the server: uneven small grids and a few
        # 1000x250 ones, submitted together, each waited for.
        {"name": "serve 40+2 mixed", "kind": "serve", "systems": 40, "nx_max": 400, "large": 2, "shift": 1e-2,
         "precision": "mixed"},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["spmv", "spmv", "spmv", "spmv", "host", "solve", "solve", "batch", "serve"])
    if kind in ("spmv", "host"):
        pattern = rng.choice(["band", "ragged", "ndiag", "q4"]) if kind == "spmv" else "band"
        dtype = rng.choice(["f32", "f64"])
        if pattern == "q4":
            nx = _log_int(rng, 40, 1200)
            return {"kind": kind, "pattern": "q4", "nx": nx, "ny": max(2, nx // rng.choice([3, 4, 5])),
                    "bs": rng.choice([0, 2]), "dtype": dtype, "api": rng.choice(["arrays", "handle"])}
        bs = rng.choice([1, 2, 3, 4, 5, 6, 7, 8, 9, 11, 12, 13, 16, 17, 24, 27, 32])
        blocks = rng.choice([5, 6, 8, 9])
        most = min(150000, int(2e9 / (blocks * bs * bs * 8)))
        rows = _log_int(rng, 2000, most if kind == "spmv" else max(2001, most // 8))
        case = {"kind": kind, "pattern": pattern, "rows": rows, "blocks": blocks, "bs": bs, "dtype": dtype}
        if kind == "spmv":
            case["api"] = rng.choice(["arrays", "handle"])
        return case
    shift = 10.0 ** rng.uniform(-2.2, -1.0)
    precision = rng.choice(["fp64", "mixed"])
    if kind == "solve":
        nx = _log_int(rng, 40, 1400)
        return {"kind": "solve", "nx": nx, "ny": max(4, nx // rng.choice([3, 4, 5])), "shift": shift,
                "precision": precision, "precond": rng.choice(["none", "none", "jacobi", "block_jacobi"]),
                "format": rng.choice(["bcsr", "bcsr", "csr"])}
    case = {"kind": kind, "systems": _log_int(rng, 8, 128), "nx_max": rng.choice([100, 200, 400]), "shift": shift,
            "precision": precision}
    if kind == "serve":
        case["systems"] = min(case["systems"], 48)
        case["large"] = rng.choice([0, 1, 2])
    return case


# ------------------------------------------------------------------ matrices

def _gen(seed, salt):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) * 1000003 + salt)
    return g


def _synthetic(case, seed):
    """Block row offsets, sorted distinct block columns and uniform values in
    [-1, 1), on the GPU. band: `blocks` columns at random within +-64 of the
    diagonal; ragged: as band, 0 to 2 `blocks` - 1 of them per row; ndiag:
    `blocks` neighbouring columns."""
    n, k, bs = case["rows"], case["blocks"], case["bs"]
    dev, g = "cuda", _gen(seed, 1)
    i = torch.arange(n, device=dev)
    if case["pattern"] == "ndiag":
        first = (i - k // 2).clamp(0, n - k)
        cols = first[:, None] + torch.arange(k, device=dev)
        keep = torch.ones_like(cols, dtype=torch.bool)
    else:
        window = 129
        count = torch.full((n,), k, device=dev)
        if case["pattern"] == "ragged":
            count = torch.randint(0, 2 * k, (n,), device=dev, generator=g)
        most = int(count.max())
        offset = torch.rand(n, window, device=dev, generator=g).topk(most, dim=1).indices
        keep = torch.arange(most, device=dev)[None, :] < count[:, None]
        offset = torch.where(keep, offset, window).sort(dim=1).values
        keep = offset < window
        cols = (i - 64).clamp(0, n - window)[:, None] + offset
    row_ptr = torch.zeros(n + 1, dtype=torch.int32, device=dev)
    row_ptr[1:] = keep.sum(1).cumsum(0)
    cols = cols[keep].to(torch.int32)
    vals = torch.empty(cols.numel() * bs * bs, dtype=DTYPES[case["dtype"]], device=dev)
    vals.uniform_(-1.0, 1.0, generator=g)
    return row_ptr, cols, vals, n


def _elasticity(nx, ny, seed, shift=0.0):
    """Plane-stress stiffness of an nx x ny node grid (BCSR, block size 2, host
    arrays) for a seeded material; shift > 0 adds shift * E on the diagonal (the
    mass term of an implicit time step)."""
    r = np.random.RandomState(int(seed) % (1 << 31))
    young, poisson = r.uniform(0.5, 2.0), r.uniform(0.25, 0.35)
    rp, c, v, _ = bm.gen_q4_elasticity(nx, ny, np.float64, young, poisson)
    if shift:
        rows = np.repeat(np.arange(rp.size - 1, dtype=np.int32), np.diff(rp))
        v.reshape(-1, 2, 2)[c == rows] += shift * young * np.eye(2)
    return rp, c, v


def _grids(case, seed):
    """Uneven grids, nx log-uniform from 20 to nx_max, ny = nx / 4 (the same
    sizes for every seed: the seed makes materials and loads)."""
    r = np.random.RandomState(7)
    nx = np.exp(r.uniform(math.log(20), math.log(case["nx_max"]), case["systems"])).round().astype(int)
    grids = [(int(a), max(5, int(round(a / 4)))) for a in nx]
    return grids + [(1000, 250)] * case.get("large", 0)


def _systems(case, seed):
    if case["kind"] == "solve":
        grids = [(case["nx"], case["ny"])]
    else:
        grids = _grids(case, seed)
    return [_elasticity(nx, ny, seed * 1009 + k, case["shift"]) for k, (nx, ny) in enumerate(grids)]


def _loads(systems, seed):
    """Random loads uniform in [-1, 1)."""
    r = np.random.RandomState((int(seed) + 17) % (1 << 31))
    return [r.uniform(-1.0, 1.0, 2 * (s[0].size - 1)) for s in systems]


def _device_matrix(row_ptr, cols, vals, bs, n_block_cols):
    """A matrix handle from device arrays."""
    h = ctypes.c_void_p()
    dt = bm.dtype_enum(vals.dtype)
    bm.check(bm.load().bmfp_matrix_create_bcsr_device(
        ctypes.byref(h), dt, row_ptr.numel() - 1, n_block_cols, bs, cols.numel(), row_ptr.data_ptr(), cols.data_ptr(),
        vals.data_ptr(), torch.cuda.current_stream().cuda_stream))
    return bm.Matrix(h, dt, row_ptr.numel() - 1, n_block_cols, bs, cols.numel())


def _arrays(case, seed):
    """(row_ptr, cols, vals, n_block_cols) on the GPU."""
    if case["pattern"] != "q4":
        return _synthetic(case, seed)
    rp, c, v = _elasticity(case["nx"], case["ny"], seed)
    n = rp.size - 1
    if case["bs"] == 0:
        rp, c, v = bm.bcsr_to_csr(rp, c, v, 2)
        n *= 2
    return (torch.from_numpy(rp).cuda(), torch.from_numpy(c).cuda(),
            torch.from_numpy(v).cuda().to(DTYPES[case["dtype"]]), n)


# --------------------------------------------------------------------- cases

def prepare(case, seed):
    kind = case["kind"]
    if kind in ("spmv", "host"):
        rp, c, v, n = _arrays(case, seed)
        b = case["bs"] or 1
        x = torch.empty(n * b, dtype=v.dtype, device="cuda").uniform_(-1.0, 1.0, generator=_gen(seed, 2))
        if kind == "host":
            def pinned(t):
                return torch.empty(t.shape, dtype=t.dtype, pin_memory=True).copy_(t).numpy()
            y = torch.empty(n * b, dtype=v.dtype, pin_memory=True).numpy()
            return {"kind": kind, "bs": b, "rp": pinned(rp), "c": pinned(c), "v": pinned(v), "x": pinned(x), "y": y}
        y = torch.empty(n * b, dtype=v.dtype, device="cuda")
        if case["api"] == "arrays":
            return {"kind": "csr" if case["bs"] == 0 else "bcsr", "bs": b, "rp": rp, "c": c, "v": v, "x": x, "y": y}
        if case["bs"]:
            m = _device_matrix(rp, c, v, b, n)
        else:
            m = bm.Matrix.from_csr(rp.cpu().numpy(), c.cpu().numpy(), v.cpu().numpy(), n)
        return {"kind": "handle", "m": m, "x": x, "y": y}
    systems = _systems(case, seed)
    loads = _loads(systems, seed)
    if case.get("format") == "csr":
        mats = [bm.Matrix.from_csr(*bm.bcsr_to_csr(*s, 2), 2 * (s[0].size - 1)) for s in systems]
    else:
        mats = [bm.Matrix.from_bcsr(*s, 2) for s in systems]
    state = {"kind": kind, "mats": mats}
    if kind == "serve":
        state["server"] = bm.Server(precision=case["precision"], tol=TOLERANCE[case["precision"]])
        state["b"] = loads
        state["x"] = [np.zeros_like(b) for b in loads]
        return state
    state["b"] = [torch.from_numpy(b).cuda() for b in loads]
    state["x"] = [torch.empty_like(b) for b in state["b"]]
    if kind == "solve":
        precond = case["precond"] if case["format"] == "bcsr" or case["precond"] != "block_jacobi" else "jacobi"
        state["solver"] = bm.Solver(mats[0], case["precision"], tol=TOLERANCE[case["precision"]], preconditioner=precond)
    else:
        state["batch"] = bm.Batch(mats, case["precision"], tol=TOLERANCE[case["precision"]])
    return state


def run(state):
    kind = state["kind"]
    if kind == "handle":
        return state["m"].spmv(state["x"], state["y"])
    if kind == "bcsr":
        return bm.bcsr_spmv(bm.BCSR_NATIVE, state["rp"], state["c"], state["v"], state["x"], state["y"], state["bs"])
    if kind == "csr":
        return bm.csr_spmv(bm.CSR_NATIVE, state["rp"], state["c"], state["v"], state["x"], state["y"])
    if kind == "host":
        return bm.bcsr_spmv_host(state["rp"], state["c"], state["v"], state["x"], state["bs"], y=state["y"])
    if kind == "solve":
        state["solver"].solve(state["b"][0], state["x"][0])
        return state["x"][0]
    if kind == "batch":
        state["batch"].solve(state["b"], state["x"])
        return torch.cat(state["x"])
    tickets = [state["server"].submit(m, b, x) for m, b, x in zip(state["mats"], state["b"], state["x"])]
    for t in tickets:
        state["server"].wait(t)
    return np.concatenate(state["x"])


# ---------------------------------------------------------------------- work

def _q4_blocks(nx, ny):
    return (3 * nx - 2) * (3 * ny - 2)


def work(case):
    """Bytes: every input read once, every output written once. Operations: two
    per stored entry and product; a solve on K + shift I takes about
    15 / sqrt(shift) iterations of two products and 12 operations per row."""
    if case["kind"] in ("spmv", "host"):
        s = 8 if case["dtype"] == "f64" else 4
        if case["pattern"] == "q4":
            blocks, n = _q4_blocks(case["nx"], case["ny"]), case["nx"] * case["ny"]
            entries = 4 * blocks
            index = 4 * (entries + 2 * n) if case["bs"] == 0 else 4 * (blocks + n)
            rows = 2 * n
        else:
            blocks = case["rows"] * (case["blocks"] - 0.5 if case["pattern"] == "ragged" else case["blocks"])
            entries, rows = blocks * case["bs"] ** 2, case["rows"] * case["bs"]
            index = 4 * (blocks + case["rows"])
        return {"bytes": entries * s + index + 2 * rows * s, "flops": 2 * entries}
    grids = [(case["nx"], case["ny"])] if case["kind"] == "solve" else _grids(case, 0)
    iterations = 15 / math.sqrt(case["shift"])
    entries = sum(4 * _q4_blocks(*g) for g in grids)
    rows = sum(2 * a * b for a, b in grids)
    return {"bytes": 8 * entries + entries + 16 * rows, "flops": iterations * (4 * entries + 12 * 2 * rows)}


# --------------------------------------------------------------------- exact

def _product(rp, c, v, x, bs):
    """y = A x in 64 bits, some block rows at a time."""
    n = rp.numel() - 1
    y = torch.zeros(n, bs, dtype=torch.float64, device="cuda")
    counts = (rp[1:] - rp[:-1]).long()
    rows = torch.repeat_interleave(torch.arange(n, device="cuda"), counts)
    v, x = v.view(-1, bs, bs), x.double().view(-1, bs)
    step = max(1, (1 << 27) // (bs * bs))
    for k in range(0, c.numel(), step):
        part = torch.bmm(v[k:k + step].double(), x[c[k:k + step].long()].unsqueeze(2)).squeeze(2)
        y.index_add_(0, rows[k:k + step], part)
    return y.view(-1)


def _solution(systems, loads):
    """Conjugate gradients in 64 bits on the systems side by side (they are
    symmetric positive definite), from x = 0 until the residual stops falling."""
    width, first = 9, 0
    cols, vals = [], []
    for rp, c, v in systems:
        rp, c, v = torch.from_numpy(rp).cuda().long(), torch.from_numpy(c).cuda().long(), torch.from_numpy(v).cuda()
        n = rp.numel() - 1
        rows = torch.repeat_interleave(torch.arange(n, device="cuda"), rp[1:] - rp[:-1])
        place = torch.arange(c.numel(), device="cuda") - rp[rows]
        cc = torch.zeros(n, width, dtype=torch.int64, device="cuda")
        vv = torch.zeros(n, width, 2, 2, dtype=torch.float64, device="cuda")
        cc[rows, place] = c + first
        vv[rows, place] = v.view(-1, 2, 2)
        cols.append(cc)
        vals.append(vv)
        first += n
    cols, vals = torch.cat(cols), torch.cat(vals)
    flat = vals.permute(0, 2, 1, 3).reshape(first, 2, 2 * width).contiguous()

    def matvec(p):
        return torch.bmm(flat, p.view(-1, 2)[cols].reshape(first, 2 * width, 1)).view(-1)

    b = torch.from_numpy(np.concatenate(loads)).cuda()
    x = torch.zeros_like(b)
    for _ in range(3):  # from the true residual again, for the last digits
        r = b - matvec(x)
        p, d, rr = r.clone(), torch.zeros_like(b), torch.dot(r, r)
        stop = 1e-24 * rr.item()
        for it in range(4000):
            q = matvec(p)
            a = rr / torch.dot(p, q)
            d += a * p
            r -= a * q
            new = torch.dot(r, r)
            p = r + (new / rr) * p
            rr = new
            if it % 16 == 15 and rr.item() < stop:
                break
        x += d
    return x


def exact(case, seed):
    if case["kind"] in ("spmv", "host"):
        rp, c, v, n = _arrays(case, seed)
        b = case["bs"] or 1
        x = torch.empty(n * b, dtype=v.dtype, device="cuda").uniform_(-1.0, 1.0, generator=_gen(seed, 2))
        y = _product(rp, c, v, x, b)
        return y.cpu().numpy() if case["kind"] == "host" else y
    systems = _systems(case, seed)
    x = _solution(systems, _loads(systems, seed))
    return x.cpu().numpy() if case["kind"] == "serve" else x
