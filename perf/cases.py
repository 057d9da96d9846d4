"""The operator calls whose speed this package is judged by: sparse sums, products and reductions of
operands that already lie in device memory, through the operators of ``nacho_b200.nacho``.

A case names an operator and the shape of its operands:
  matrices   ``rows`` x ``cols`` with about ``entries`` stored positions per operand; row lengths
             follow lognormal(0, ``skew``) weights and columns are uniform. The second and third
             operand share a fraction ``overlap`` of the first one's positions.
  tensors    ``d0`` x ``d1`` x ``d2``; slice sizes follow a power law (rank ** -1.5 over a random
             permutation of the first mode), (j, k) is uniform.
  graphs     an R-MAT pattern (0.57, 0.19, 0.19, 0.05) of ``n`` vertices and about ``entries`` edges.
  meshes     a 5-point stencil on an ``nx`` x ``ny`` grid with a coefficient of its own at every point.
Values are U(-1, 1) float32, indices int32. A case stands for one shape of result, so a seed draws the
values and where along every mode the case's pattern begins (a cyclic shift per mode): positions and
values differ from seed to seed, while the lengths of operands and results do not.
"""
import math
import zlib

import torch

from nacho_b200 import nacho

DEVICE = "cuda"
RMAT = (0.57, 0.19, 0.19, 0.05)


# ------------------------------------------------------------------------------------- cases ----

def listed():
    return [
        # the smallest calls: a test-suite sized sum, where only latency counts
        {"name": "csr_add_200", "op": "csr_add", "rows": 200, "cols": 180, "entries": 1800, "skew": 0.0, "overlap": 0.05},
        # a matrix that fits the L2: 40 entries per row, independent operands
        {"name": "csr_add_4k", "op": "csr_add", "rows": 4096, "cols": 4096, "entries": 163840, "skew": 0.0, "overlap": 0.0},
        # the largest sum: 64 M entries per operand, bound by device memory
        {"name": "csr_add_64M", "op": "csr_add", "rows": 1 << 20, "cols": 1 << 20, "entries": 1 << 26, "skew": 0.0, "overlap": 0.0},
        # intersection of two patterns that share half their positions; short rows with a long tail
        {"name": "csr_mul_16M", "op": "csr_mul", "rows": 1 << 20, "cols": 1 << 20, "entries": 1 << 24, "skew": 1.5, "overlap": 0.5},
        # three-operand sum on ragged sizes with a strong row skew
        {"name": "csr_add_3_9M", "op": "csr_add_3", "rows": 300007, "cols": 1000003, "entries": 9000001, "skew": 2.0, "overlap": 0.1},
        # an operator on a mesh squared: millions of rows of 13 entries
        {"name": "spgemm_mesh", "op": "spgemm", "nx": 512, "ny": 512},
        # a graph times its transpose: hub rows with millions of products
        {"name": "spgemm_rmat", "op": "spgemm", "n": 1 << 16, "entries": 1 << 20},
        # product of a graph with itself on the graph's own positions (triangle counting)
        {"name": "sssmm_rmat", "op": "sssmm", "n": 50021, "entries": 800003},
        # coordinate-list sum of a large 3-mode tensor
        {"name": "coo3d_add_100M", "op": "coo3d_add", "d0": 1 << 17, "d1": 1 << 16, "d2": 1 << 12, "entries": 100_000_000, "overlap": 0.3},
        # the same operation on compressed trees, ragged extents
        {"name": "csf_add_25M", "op": "csf_add", "d0": 100003, "d1": 50021, "d2": 4001, "entries": 25_000_003, "overlap": 0.3},
        # hypersparse rows: most of the four million rows are empty
        {"name": "dcsr_add_3M", "op": "dcsr_add", "rows": 1 << 22, "cols": 1 << 20, "entries": 3_000_017, "skew": 3.0, "overlap": 0.3},
        # full reduction of two coordinate lists
        {"name": "inner_prod_coo_4M", "op": "inner_prod_coo", "d0": 20011, "d1": 8009, "d2": 3001, "entries": 4_000_037, "overlap": 0.5},
    ]


def _log(rng, lo, hi):
    """A whole number between lo and hi, spread over the logarithm."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["csr_add", "csr_add", "csr_add", "csr_mul", "csr_mul", "csr_add_3", "spgemm_mesh", "spgemm_rmat", "sssmm",
                     "coo3d_add", "csf_add", "dcsr_add", "inner_prod_coo"])
    overlap = round(rng.uniform(0.0, 0.6), 2)
    if op == "spgemm_mesh":
        return {"op": "spgemm", "nx": _log(rng, 20, 512), "ny": _log(rng, 20, 512)}
    if op in ("spgemm_rmat", "sssmm"):
        n = _log(rng, 500, 1 << 16)
        return {"op": op.split("_")[0], "n": n, "entries": n * rng.randint(4, 16) + rng.randint(0, n)}
    if op in ("coo3d_add", "csf_add", "inner_prod_coo"):
        return {"op": op, "d0": _log(rng, 1000, 1 << 17), "d1": _log(rng, 5000, 1 << 16), "d2": _log(rng, 1000, 1 << 12),
                "entries": _log(rng, 2000, 60_000_000), "overlap": overlap}
    if op == "dcsr_add":
        return {"op": op, "rows": _log(rng, 1 << 14, 1 << 22), "cols": _log(rng, 1 << 12, 1 << 20), "entries": _log(rng, 2000, 8_000_000),
                "skew": rng.choice([2.0, 3.0]), "overlap": overlap}
    rows = _log(rng, 100, 1 << 20)
    per_row = _log(rng, 4, 64)
    return {"op": op, "rows": rows, "cols": _log(rng, 8 * per_row, 1 << 20), "entries": rows * per_row + rng.randint(0, rows),
            "skew": rng.choice([0.0, 1.0, 2.0, 3.0]), "overlap": overlap}


# ------------------------------------------------------------------------------------ inputs ----

def _values(n, g):
    return torch.rand(n, generator=g, device=DEVICE) * 2.0 - 1.0


def _i32(t):
    return t.to(torch.int32).contiguous()


def _positions(weights, width, entries, g):
    """About ``entries`` distinct positions ``row * width + column`` in order: rows by weight, columns uniform."""
    cdf = torch.cumsum(weights.double(), 0)
    r = torch.searchsorted(cdf, torch.rand(entries, generator=g, device=DEVICE, dtype=torch.float64) * cdf[-1])
    r.clamp_(max=weights.numel() - 1)
    return torch.unique(r * width + torch.randint(0, width, (entries,), generator=g, device=DEVICE))


def _shifted(keys, sizes, shifts):
    """The same positions with every mode's numbering moved round by its shift, in order again."""
    out, stride = torch.zeros_like(keys), 1
    for size, shift in zip(reversed(sizes), reversed(shifts)):
        out += (keys + shift) % size * stride
        keys = torch.div(keys, size, rounding_mode="floor")
        stride *= size
    return torch.sort(out)[0]


def _operand_positions(count, weights, width, entries, overlap, g):
    first = _positions(weights, width, entries, g)
    out = [first]
    for _ in range(count - 1):
        kept = first[torch.rand(first.numel(), generator=g, device=DEVICE) < overlap]
        fresh = _positions(weights, width, max(1, int(entries * (1.0 - overlap))), g)
        out.append(torch.unique(torch.cat([kept, fresh])))
    return out


def _offsets(row_of_entry, rows):
    rp = torch.zeros(rows + 1, dtype=torch.int64, device=DEVICE)
    torch.cumsum(torch.bincount(row_of_entry, minlength=rows), 0, out=rp[1:])
    return _i32(rp)


def _csr(keys, rows, cols, g):
    r = torch.div(keys, cols, rounding_mode="floor")
    return nacho.CSR_gpu(_offsets(r, rows), _i32(keys - r * cols), _values(keys.numel(), g), torch.tensor([rows, cols], dtype=torch.int32))


def _dcsr(keys, rows, cols, g):
    r = torch.div(keys, cols, rounding_mode="floor")
    present, lengths = torch.unique_consecutive(r, return_counts=True)
    jp = torch.zeros(present.numel() + 1, dtype=torch.int64, device=DEVICE)
    torch.cumsum(lengths, 0, out=jp[1:])
    return nacho.DCSR_gpu(_i32(present), _i32(jp), _i32(keys - r * cols), _values(keys.numel(), g), torch.tensor([rows, cols], dtype=torch.int32))


def _coo3(keys, dims, g):
    ij, k = torch.div(keys, dims[2], rounding_mode="floor"), keys % dims[2]
    return nacho.COO3_gpu(_i32(torch.div(ij, dims[1], rounding_mode="floor")), _i32(ij % dims[1]), _i32(k), _values(keys.numel(), g),
                          torch.tensor(dims, dtype=torch.int32))


def _csf3(keys, dims, g):
    ij, k = torch.div(keys, dims[2], rounding_mode="floor"), keys % dims[2]
    fibres, per_fibre = torch.unique_consecutive(ij, return_counts=True)
    slices, per_slice = torch.unique_consecutive(torch.div(fibres, dims[1], rounding_mode="floor"), return_counts=True)
    zero = torch.zeros(1, dtype=torch.int64, device=DEVICE)
    return nacho.CSF3_gpu(_i32(slices), _i32(torch.cat([zero, torch.cumsum(per_slice, 0)])), _i32(fibres % dims[1]),
                          _i32(torch.cat([zero, torch.cumsum(per_fibre, 0)])), _i32(k), _values(keys.numel(), g), torch.tensor(dims, dtype=torch.int32))


def _rmat_keys(n, entries, g):
    """Distinct positions of an R-MAT graph cut down to its first ``n`` vertices (the last ones of a power of two are nearly empty)."""
    a, b, c, _ = RMAT
    r = torch.zeros(entries, dtype=torch.int64, device=DEVICE)
    k = torch.zeros(entries, dtype=torch.int64, device=DEVICE)
    for bit in range(_rmat_scale(n)):
        u = torch.rand(entries, generator=g, device=DEVICE)
        r |= (u >= a + b).to(torch.int64) << bit
        k |= (((u >= a) & (u < a + b)) | (u >= a + b + c)).to(torch.int64) << bit
    inside = (r < n) & (k < n)
    return torch.unique(r[inside] * n + k[inside])


def _rmat_scale(n):
    return max(1, (n - 1).bit_length())


def _transposed(keys, n):
    return torch.sort((keys % n) * n + torch.div(keys, n, rounding_mode="floor"))[0]


def _mesh_keys(nx, ny):
    n = nx * ny
    p = torch.arange(n, device=DEVICE)
    x, y = p % nx, torch.div(p, nx, rounding_mode="floor")
    parts = [p * n + p] + [p[ok] * n + p[ok] + step for ok, step in ((y > 0, -nx), (x > 0, -1), (x < nx - 1, 1), (y < ny - 1, nx))]
    return torch.sort(torch.cat(parts))[0]


def prepare(case, seed):
    op = case["op"]
    pattern = torch.Generator(device=DEVICE)
    pattern.manual_seed(zlib.crc32(repr(sorted((k, v) for k, v in case.items() if k != "name")).encode()))
    g = torch.Generator(device=DEVICE)
    g.manual_seed(int(seed))

    def shifts(sizes):
        return [int(torch.randint(0, size, (1,), generator=g, device=DEVICE)) for size in sizes]

    if "nx" in case:  # the mesh itself is what it is: only its coefficients are drawn
        n = case["nx"] * case["ny"]
        keys = _mesh_keys(case["nx"], case["ny"])
        operands = [_csr(keys, n, n, g), _csr(keys, n, n, g)]
    elif "n" in case:
        n = case["n"]
        keys = _shifted(_rmat_keys(n, case["entries"], pattern), (n, n), shifts((n,)) * 2)  # vertices renamed: the same shift for both modes
        a = _csr(keys, n, n, g)
        operands = [a, a, a] if op == "sssmm" else [a, _csr(_transposed(keys, n), n, n, g)]
    elif "d0" in case:
        dims = [case["d0"], case["d1"], case["d2"]]
        ranks = torch.arange(1, dims[0] + 1, device=DEVICE, dtype=torch.float64)
        weights = ranks[torch.randperm(dims[0], generator=pattern, device=DEVICE)] ** -1.5
        build, by = _csf3 if op == "csf_add" else _coo3, shifts(dims)
        operands = [build(_shifted(k, dims, by), dims, g)
                    for k in _operand_positions(2, weights, dims[1] * dims[2], case["entries"], case["overlap"], pattern)]
    else:
        rows, cols = case["rows"], case["cols"]
        weights = torch.exp(case["skew"] * torch.randn(rows, generator=pattern, device=DEVICE, dtype=torch.float64))
        build, by = _dcsr if op == "dcsr_add" else _csr, shifts((rows, cols))
        operands = [build(_shifted(k, (rows, cols), by), rows, cols, g)
                    for k in _operand_positions(3 if op == "csr_add_3" else 2, weights, cols, case["entries"], case["overlap"], pattern)]
    return {"operator": getattr(nacho, "gpu_%s_f32" % op), "operands": operands}


# ---------------------------------------------------------------------------------- one call ----

_ARRAYS = {
    nacho.CSR_gpu: ("dim_j_offsets", "dim_j_indices", "values"),
    nacho.DCSR_gpu: ("dim_i_indices", "dim_j_offsets", "dim_j_indices", "values"),
    nacho.COO3_gpu: ("dim_i_indices", "dim_j_indices", "dim_k_indices", "values"),
    nacho.CSF3_gpu: ("dim_i_indices", "dim_j_offsets", "dim_j_indices", "dim_k_offsets", "dim_k_indices", "values"),
    nacho.Scalar_gpu: ("values",),
}


def run(state):
    z = state["operator"](*state["operands"])
    return [getattr(z, name) for name in _ARRAYS[type(z)]]


# ------------------------------------------------------------------------- what a call needs ----

def _rmat_counts(n, m):
    """Expected (stored entries, products of two such matrices, entries of the product) of R-MAT graphs with m edges, from the
    counts of the bit patterns that two vertices share: every bit of an edge is drawn on its own."""
    a, b, c, d = RMAT
    s = _rmat_scale(n)
    lam = [a * a + b * b, a * c + b * d, c * c + d * d]  # two rows meeting in a column: bits (0, 0), (0, 1) or (1, 0), (1, 1)
    stored = result = products = 0.0
    for p in range(s + 1):
        column = 0.0  # entries of a column whose number has s - p set bits
        for q in range(s - p + 1):
            ways = math.comb(s, p) * math.comb(s - p, q) * 2.0 ** q
            stored += ways * -math.expm1(-m * a ** p * b ** q * d ** (s - p - q))
            result += ways * -math.expm1(-float(m) * m * lam[0] ** p * lam[1] ** q * lam[2] ** (s - p - q))
        for q in range(p + 1):
            for r in range(s - p + 1):
                ways = math.comb(p, q) * math.comb(s - p, r)
                column += ways * -math.expm1(-m * a ** q * c ** (p - q) * b ** r * d ** (s - p - r))
        products += math.comb(s, p) * column * column
    return stored, products, min(result, products)


def work(case):
    op = case["op"]
    if "nx" in case:
        n = case["nx"] * case["ny"]
        nnz = 5 * n - 2 * (case["nx"] + case["ny"])
        return {"bytes": 2 * (4 * (n + 1) + 8 * nnz) + 4 * (n + 1) + 8 * 13 * n, "flops": 2 * 25 * n}
    if "n" in case:
        n = case["n"]
        nnz, products, result = _rmat_counts(n, case["entries"])
        operand = 4 * (n + 1) + 8 * nnz
        if op == "sssmm":  # one matrix in all three places; nearly every position of the mask is reached
            return {"bytes": operand + 4 * (n + 1) + 8 * nnz, "flops": 3 * products}
        return {"bytes": 2 * operand + 4 * (n + 1) + 8 * result, "flops": 2 * products}
    nnz, shared = case["entries"], case["entries"] * case["overlap"]
    if op == "csr_mul":
        return {"bytes": 3 * 4 * (case["rows"] + 1) + 8 * (2 * nnz + shared), "flops": shared}
    if op == "csr_add":
        return {"bytes": 3 * 4 * (case["rows"] + 1) + 8 * (4 * nnz - shared), "flops": shared}
    if op == "csr_add_3":
        return {"bytes": 4 * 4 * (case["rows"] + 1) + 8 * (6 * nnz - 2 * shared), "flops": 2 * shared}
    if op == "dcsr_add":  # about as many stored rows as the weights and the entries allow; 8 bytes each
        return {"bytes": 3 * 8 * min(case["rows"], nnz) * 0.25 + 8 * (4 * nnz - shared), "flops": shared}
    if op == "coo3d_add":
        return {"bytes": 16 * (4 * nnz - shared), "flops": shared}
    if op == "csf_add":  # k and value of every entry; the levels above are a fraction of that
        return {"bytes": 8 * (4 * nnz - shared), "flops": shared}
    return {"bytes": 16 * 2 * nnz, "flops": 2 * shared}  # inner_prod_coo


def tolerance(case):
    if case["op"] in ("spgemm", "sssmm", "inner_prod_coo"):
        return {"rel": 1e-5}  # float32 sums in any order; the structure is exact
    return "exact"  # one IEEE addition or multiplication per value
