"""Performance cases of the sparse tile products: what is timed, on which sizes.

Each case is one call (or the pair of calls) that a program makes in its inner
loop, on tiles that are already resident on the GPU:

* ``spgemm``   C = A * B over tile grids through ``gemm``: sizes the output,
               allocates it and computes it.
* ``numeric``  the values of a product whose plan and output arrays the
               program keeps, because only the values of A and B change.
* ``spmm``     C += A * B with a dense B, in place, through ``gemm``.
* ``retile``   a CSR matrix on the device cut into tiles and gathered back.

Inputs are seeded and made on the GPU: power-law graphs (R-MAT, a=.57,
b=c=.19), uniformly random matrices and the 27-point stencil, as the
benchmark's workloads use them.
"""
import math
import random

import torch

from bcl_b200.containers import BlockCustom, DMatrix, SPMatrix, gemm, spgemm_numeric, spgemm_symbolic

F32, I32, BF16 = "f32", "i32", "bf16"


def listed():
    return [
        # a small system inside a larger loop: launches and host work count
        dict(name="spgemm_er1k", kind="spgemm", pattern="er", n=1024, deg=8, grid=4, dtype=F32),
        # the benchmark's headline: two-hop neighbourhoods of a power-law graph
        dict(name="spgemm_rmat16", kind="spgemm", pattern="rmat", n=65536, deg=16, grid=8, dtype=F32),
        # integer values (path counting), sizes that divide nothing evenly
        dict(name="spgemm_ragged_i32", kind="spgemm", pattern="rmat", n=30011, deg=9, grid=5, dtype=I32),
        # the same product on a graph and tile grid four times as large
        dict(name="spgemm_rmat18", kind="spgemm", pattern="rmat", n=262144, deg=16, grid=16, dtype=F32),
        # a discretised operator squared (multigrid set-up) on a fine tile grid
        dict(name="spgemm_stencil128", kind="spgemm", pattern="stencil", n=128 ** 3, deg=27, grid=128, dtype=F32),
        # graph times sparse features: structure fixed, new values every epoch
        dict(name="numeric_features", kind="numeric", pattern="rmat", n=65536, deg=12, grid=6, dtype=F32, cols=3001,
             cols_deg=20),
        # the benchmark's small sparse x dense product: fits in L2
        dict(name="spmm_er16k", kind="spmm", pattern="er", n=16384, deg=16, grid=4, dtype=F32, width=128),
        # graph neural network aggregation over hidden features, both storage types
        dict(name="spmm_rmat21", kind="spmm", pattern="rmat", n=2097152, deg=16, grid=8, dtype=F32, width=256),
        dict(name="spmm_rmat21_bf16", kind="spmm", pattern="rmat", n=2097152, deg=16, grid=8, dtype=BF16, width=256),
        # the last layer: as many columns as there are classes, rows off 16 bytes
        dict(name="spmm_classes47", kind="spmm", pattern="rmat", n=169343, deg=14, grid=4, dtype=F32, width=47),
        # a narrow block of vectors (block Krylov, small hidden layers)
        dict(name="spmm_narrow16", kind="spmm", pattern="rmat", n=400001, deg=16, grid=2, dtype=F32, width=16),
        # loading a matrix and handing the result back
        dict(name="retile_rmat19", kind="retile", pattern="rmat", n=524288, deg=16, grid=8, dtype=F32),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["spgemm", "spgemm", "spgemm", "numeric", "spmm", "spmm", "spmm", "retile"])
    pattern = rng.choice(["rmat", "rmat", "er", "stencil"])
    c = dict(kind=kind, pattern=pattern, deg=rng.randint(4, 16))
    if kind == "spgemm":
        c["n"] = _log_int(rng, 1000, 200000)
        c["dtype"] = rng.choice([F32, F32, I32])
    elif kind == "numeric":
        c["n"] = _log_int(rng, 1000, 100000)
        c["dtype"] = rng.choice([F32, F32, I32])
        c["cols"] = _log_int(rng, 200, 20000)
        c["cols_deg"] = rng.randint(2, 24)
    elif kind == "spmm":
        c["n"] = _log_int(rng, 2000, 1500000)
        c["dtype"] = rng.choice([F32, BF16])
        c["width"] = rng.choice([_log_int(rng, 4, 256), 8 * rng.randint(1, 32)])
    else:
        c["n"] = _log_int(rng, 1000, 1000000)
        c["dtype"] = rng.choice([F32, I32])
    if pattern == "stencil":
        c["deg"] = 27
        c["n"] = max(6, round(c["n"] ** (1 / 3))) ** 3
    # tiles of at most 16384 columns for the sparse products, a few thousand rows where there are that many
    least = -(-c["n"] // 16384) if kind in ("spgemm", "numeric") else 1
    c["grid"] = rng.randint(max(1, least), max(8, least + 4))
    return c


# ---- inputs ----------------------------------------------------------------------


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _keys(pattern, m, n, deg, g):
    """Sorted distinct row * n + column of the entries."""
    if pattern == "stencil":
        s = round(m ** (1 / 3))
        idx = torch.arange(m, device="cuda")
        x, y, z = idx % s, idx // s % s, idx // (s * s)
        parts = []
        for dz in (-1, 0, 1):
            for dy in (-1, 0, 1):
                for dx in (-1, 0, 1):
                    ok = (x + dx >= 0) & (x + dx < s) & (y + dy >= 0) & (y + dy < s) & (z + dz >= 0) & (z + dz < s)
                    i = idx[ok]
                    parts.append(i * n + i + dx + s * dy + s * s * dz)
        return torch.cat(parts).sort().values
    count = m * deg
    if pattern == "er":
        rows = torch.arange(m, device="cuda").repeat_interleave(deg)
        cols = torch.randint(0, n, (count,), generator=g, device="cuda")
    else:  # R-MAT on the next power of two, scaled onto m x n
        scale = max(1, (max(m, n) - 1).bit_length())
        rows = torch.zeros(count, dtype=torch.int64, device="cuda")
        cols = torch.zeros(count, dtype=torch.int64, device="cuda")
        for _ in range(scale):
            r = torch.rand(count, generator=g, device="cuda")
            down = r >= 0.76
            right = ((r >= 0.57) & ~down) | (r >= 0.95)
            rows = rows * 2 + down
            cols = cols * 2 + right
        rows, cols = rows * m >> scale, cols * n >> scale
    return torch.unique(rows * n + cols)


def _values(keys, pattern, n, dtype, g):
    if dtype == I32:
        return torch.randint(-8, 9, keys.shape, generator=g, device="cuda", dtype=torch.int32)
    v = torch.rand(keys.shape, generator=g, device="cuda") * 2 - 1
    if pattern == "stencil":  # a variable-coefficient operator: a strong diagonal, negative neighbours
        v = torch.where(keys // n == keys % n, 26 + v, -1 + 0.1 * v)
    return v


def _csr(pattern, m, n, deg, dtype, g, shift=(0, 0)):
    """row_ptr, col_ind (int32) and values of one matrix, on the GPU.  The
    entries' places are the sizes' own, moved cyclically by `shift` (rows,
    columns); the values are the generator's."""
    keys = _keys(pattern, m, n, deg, _gen(m + deg))
    if shift != (0, 0):
        keys = ((keys // n + shift[0]) % m * n + (keys % n + shift[1]) % n).sort().values
    rp = torch.searchsorted(keys, torch.arange(m + 1, device="cuda") * n).to(torch.int32)
    return rp, (keys % n).to(torch.int32), _values(keys, pattern, n, dtype, g)


def _operands(c, seed):
    """A's CSR arrays, and B's (A's own for a square product).  Another seed
    numbers a graph's vertices from another one on (the hubs lie in other
    tiles, the output has as many entries) and draws other values."""
    g = _gen(seed)
    s = 0 if c["pattern"] == "stencil" else random.Random(seed).randrange(c["n"])
    a = _csr(c["pattern"], c["n"], c["n"], c["deg"], F32 if c["dtype"] == BF16 else c["dtype"], g, (s, s))
    if c["kind"] == "numeric":
        return a, _csr("er", c["n"], c["cols"], c["cols_deg"], c["dtype"], g, (s, 0)), g
    return a, a, g


def _tile(n, grid):
    return -(-n // grid)


def _shapes(c):
    """A's tile shape, B's tile shape."""
    t = _tile(c["n"], c["grid"])
    if c["kind"] == "numeric":
        return (t, t), (t, _tile(c["cols"], max(_tile(c["cols"], 16384), c["grid"] // 4)))
    return (t, t), (t, c.get("width", t))


def _dense(c, g):
    dt = torch.bfloat16 if c["dtype"] == BF16 else torch.float32
    b = torch.randn((c["n"], c["width"]), generator=g, device="cuda").to(dt)
    c0 = torch.randn((c["n"], c["width"]), generator=g, device="cuda").to(dt)
    return b, c0, dt


def prepare(case, seed):
    c = case
    a, b, g = _operands(c, seed)
    ta, tb = _shapes(c)
    if c["kind"] == "retile":
        return dict(case=c, csr=a, tile=ta)
    A = SPMatrix.from_device_csr(c["n"], c["n"], *a, ta)
    if c["kind"] == "spgemm":
        return dict(case=c, A=A, B=A)
    if c["kind"] == "numeric":
        B = SPMatrix.from_device_csr(c["n"], c["cols"], *b, tb)
        plan, out, trp, toff, nnz = spgemm_symbolic(A, B)
        ci = torch.empty(max(nnz, 1), dtype=torch.int32, device="cuda")
        v = torch.empty(max(nnz, 1), dtype=a[2].dtype, device="cuda")
        out.col_ind, out.vals = ci.data_ptr(), v.data_ptr()
        return dict(case=c, A=A, B=B, plan=plan, out=out, arrays=(trp, toff, ci, v))
    b, c0, dt = _dense(c, g)
    return dict(case=c, A=A, B=DMatrix.from_array(b, BlockCustom(tb), dtype=dt),
                C=DMatrix.from_array(c0, BlockCustom((ta[0], tb[1])), dtype=dt))


def _packed(s):
    return dict(tile_row_ptr=s.tile_row_ptr, tile_offset=s.tile_offset, col_ind=s.col_ind, vals=s.vals)


def run(state):
    kind = state["case"]["kind"]
    if kind == "spgemm":
        return _packed(gemm(state["A"], state["B"]))
    if kind == "numeric":
        spgemm_numeric(state["plan"], state["A"], state["B"], state["out"])
        return dict(zip(("tile_row_ptr", "tile_offset", "col_ind", "vals"), state["arrays"]))
    if kind == "spmm":
        return gemm(state["A"], state["B"], state["C"]).tiles
    n = state["case"]["n"]
    S = SPMatrix.from_device_csr(n, n, *state["csr"], state["tile"])
    rp, ci, v = S.get_device()
    return dict(_packed(S), row_ptr=rp, global_col_ind=ci, global_vals=v)


# ---- what a pass cannot do without -------------------------------------------------


def _sparse_bytes(nnz, rows):
    return 8 * nnz + 4 * (rows + 1)


def work(case):
    c = case
    a, b, _ = _operands(c, 0)
    nnz_a, nnz_b, n = a[1].numel(), b[1].numel(), c["n"]
    if c["kind"] == "retile":  # in, tiles out; tiles in, CSR out
        slots = c["grid"] * n
        return dict(bytes=2 * (_sparse_bytes(nnz_a, n) + _sparse_bytes(nnz_a, slots)), flops=0)
    if c["kind"] == "spmm":
        es = 2 if c["dtype"] == BF16 else 4
        return dict(bytes=_sparse_bytes(nnz_a, c["grid"] * n) + 3 * es * n * c["width"], flops=2 * nnz_a * c["width"])
    lens = (b[0][1:] - b[0][:-1]).to(torch.int64)
    products = int(lens[a[1].to(torch.int64)].sum())
    ta, tb = _shapes(c)
    A = SPMatrix.from_device_csr(n, n, *a, ta)
    B = SPMatrix.from_device_csr(n, c["cols"], *b, tb) if c["kind"] == "numeric" else A
    plan, _, _, _, nnz_c = spgemm_symbolic(A, B)
    plan.close()
    read = _sparse_bytes(nnz_a, n * A.gn) + (_sparse_bytes(nnz_b, n * B.gn) if B is not A else 0)
    return dict(bytes=read + _sparse_bytes(nnz_c, n * B.gn), flops=2 * products)


# ---- the same results in 64 bits ----------------------------------------------------


def _in_tiles(full, tm, tn):
    m, n = full.shape
    gm, gn = -(-m // tm), -(-n // tn)
    pad = torch.zeros((gm * tm, gn * tn), dtype=full.dtype, device=full.device)
    pad[:m, :n] = full
    return pad.view(gm, tm, gn, tn).permute(0, 2, 1, 3).reshape(gm * gn, tm, tn)


def _product_rows(a, b, n_cols, r0, r1):
    """Columns and values of rows [r0, r1) of A * B, by row and column."""
    (arp, aci, av), (brp, bci, bv) = a, b
    p0, p1 = int(arp[r0]), int(arp[r1])
    k = aci[p0:p1].to(torch.int64)
    rows = torch.repeat_interleave(torch.arange(r1 - r0, device="cuda"), (arp[r0 + 1:r1 + 1] - arp[r0:r1]).to(torch.int64))
    start, lens = brp[k].to(torch.int64), (brp[k + 1] - brp[k]).to(torch.int64)
    first = lens.cumsum(0) - lens
    e = torch.repeat_interleave(torch.arange(p1 - p0, device="cuda"), lens)
    at = torch.arange(e.numel(), device="cuda") - first[e] + start[e]
    keys = rows[e] * n_cols + bci[at]
    vals = av[p0:p1].double()[e] * bv[at].double()
    keys, order = keys.sort()
    uniq, inv = torch.unique_consecutive(keys, return_inverse=True)
    return uniq % n_cols, torch.zeros(uniq.numel(), dtype=torch.float64, device="cuda").index_add_(0, inv, vals[order])


def _product_vals(a, b, m, n_cols, tm, tn):
    """The values of A * B in the order of the packed tiles."""
    lens = (b[0][1:] - b[0][:-1]).to(torch.int64)
    per_entry = lens[a[1].to(torch.int64)]
    ends = torch.cat([torch.zeros(1, dtype=torch.int64, device="cuda"), per_entry.cumsum(0)])[a[0].to(torch.int64)]
    ends = ends.cpu().numpy()  # products before each row
    out = []
    for t0 in range(0, m, tm):
        t1 = min(m, t0 + tm)
        cols, vals, r = [], [], t0
        while r < t1:  # as many rows at once as make about 6e7 products
            q = int(ends.searchsorted(ends[r] + 60_000_000, side="right")) - 1
            q = min(t1, max(r + 1, q))
            col, val = _product_rows(a, b, n_cols, r, q)
            cols.append((col // tn).to(torch.int16))
            vals.append(val)
            r = q
        order = torch.cat(cols).sort(stable=True).indices
        out.append(torch.cat(vals)[order])
    return torch.cat(out)


def exact(case, seed):
    c = case
    if c["dtype"] == I32:  # whole numbers
        return None
    a, b, g = _operands(c, seed)
    ta, tb = _shapes(c)
    if c["kind"] == "retile":
        return dict(tile_row_ptr=None, tile_offset=None, col_ind=None, vals=None, row_ptr=None, global_col_ind=None,
                    global_vals=a[2].double())
    if c["kind"] == "spmm":
        dense, c0, _ = _dense(c, g)
        A = torch.sparse_csr_tensor(a[0].to(torch.int64), a[1].to(torch.int64), a[2].double(), (c["n"], c["n"]))
        return _in_tiles(c0.double() + A @ dense.double(), ta[0], tb[1])
    vals = _product_vals(a, b, c["n"], c.get("cols", c["n"]), ta[0], tb[1])
    return dict(tile_row_ptr=None, tile_offset=None, col_ind=None, vals=vals)
