"""GPU suite: the routes of the sparse products by the width of the result, the number of long rows and the number of products,
in one call and in two, with operands that are row blocks of larger arrays."""
import ctypes as C

import numpy as np
import pytest

from helpers import csr_to_gpu, synth_csr
from oracle.cpu_oracle import CSR
from test_tile_edges_gpu import check_masked

pytestmark = pytest.mark.gpu

REL_TOL = 1e-5  # float32 sums in any order, relative to the sum of the terms' magnitudes


@pytest.fixture(scope="module")
def nacho():
    import torch
    assert torch.cuda.is_available(), "GPU suite needs a CUDA device"
    from nacho_b200 import nacho as mod
    return mod


def csr_of_rows(rows_of_columns, cols, rng):
    """A matrix whose row r stores the sorted columns rows_of_columns[r]."""
    rp = np.zeros(len(rows_of_columns) + 1, np.int32)
    np.cumsum([len(r) for r in rows_of_columns], out=rp[1:])
    col = np.concatenate(rows_of_columns).astype(np.int32)
    return CSR(len(rows_of_columns), cols, rp, col, rng.uniform(-1, 1, len(col)).astype(np.float32))


def scattered(cols, n, rng):
    return np.sort(rng.choice(cols, n, replace=False))


class Block:
    """A matrix on the GPU as a row block: `shift` entries of another block lie in front of its own."""

    def __init__(self, m, shift):
        import torch
        from nacho_b200._capi import CsrStruct
        pad = lambda x, fill: torch.from_numpy(np.concatenate([np.full(shift, fill, x.dtype), x])).cuda()
        self.rp = torch.from_numpy(np.ascontiguousarray(m.row_ptr + shift, np.int32)).cuda()
        self.col, self.val = pad(m.col, 7), pad(m.val, np.float32(np.nan))
        self.struct = CsrStruct(m.rows, m.cols, len(m.col), self.rp.data_ptr(), self.col.data_ptr(), self.val.data_ptr())


class Result:
    def __init__(self, rows):
        import torch
        from nacho_b200._capi import CsrStruct
        self.rp = torch.empty(rows + 1, dtype=torch.int32, device="cuda")
        self.struct = CsrStruct(0, 0, 0, self.rp.data_ptr(), None, None)

    def take(self, nnz):
        import torch
        self.col, self.val = torch.full((nnz,), -1, dtype=torch.int32, device="cuda"), torch.full((nnz,), float("nan"), device="cuda")
        self.struct.col, self.struct.val, self.struct.nnz = self.col.data_ptr(), self.val.data_ptr(), nnz

    def holds(self, want, v64, abs64):
        import torch
        torch.cuda.synchronize()
        assert np.array_equal(self.rp.cpu().numpy(), want.row_ptr), "row offsets"
        assert np.array_equal(self.col.cpu().numpy(), want.col), "columns"
        assert np.all(np.abs(self.val.cpu().numpy().astype(np.float64) - v64) <= REL_TOL * abs64 + 1e-30)


def two_passes(oracle, a, b, shift):
    """The numeric pass on offsets from elsewhere; then both passes, and the numeric one again with other values in A and B."""
    import torch
    from nacho_b200._capi import check, lib
    want, v64, abs64, products = oracle.spgemm(a, b, 8, extras=True)
    ga, gb = Block(a, shift), Block(b, shift)
    ref = lambda x: C.byref(x.struct)
    z = Result(a.rows)
    z.rp.copy_(torch.from_numpy(want.row_ptr.astype(np.int32)))
    z.struct.rows, z.struct.cols = a.rows, b.cols
    z.take(len(want.col))
    check(lib.nb200_release_workspaces(), "release")
    check(lib.nb200_spgemm_f32_numeric(ref(ga), ref(gb), ref(z), None), "numeric alone")
    z.holds(want, v64, abs64)
    z = Result(a.rows)
    p = C.c_int64(0)
    check(lib.nb200_spgemm_f32_symbolic(ref(ga), ref(gb), ref(z), C.byref(p), None), "symbolic")
    assert p.value == products and z.struct.nnz == len(want.col)
    z.take(len(want.col))
    check(lib.nb200_spgemm_f32_numeric(ref(ga), ref(gb), ref(z), None), "numeric")
    z.holds(want, v64, abs64)
    ga.val.mul_(2.0)
    gb.val.mul_(-0.5)
    z.take(len(want.col))
    check(lib.nb200_spgemm_f32_numeric(ref(ga), ref(gb), ref(z), None), "numeric again")
    z.holds(want, -v64, abs64)
    return products


@pytest.mark.parametrize("rows", [300, 8200])
@pytest.mark.parametrize("cols", [131000, 131073, 262145, 600000])
def test_wide_results(nacho, oracle, cols, rows):
    """Windows of 4096 bitmap words and more, one and several of them, for few rows and for many; rows from 260 to 2300 entries, rows of B
    without entries among those they select."""
    from test_spgemm_gpu import check
    rng = np.random.default_rng(cols + rows)
    inner = 500
    b = csr_of_rows([scattered(cols, n, rng) for n in rng.choice([0, 40, 130, 500], inner, p=[0.2, 0.4, 0.3, 0.1])], cols, rng)
    lengths = np.diff(b.row_ptr)
    long_rows = np.flatnonzero(lengths >= 130)
    a_rows = [np.unique(np.concatenate([scattered(inner, 3, rng), rng.choice(long_rows, 3, replace=False)])) for _ in range(rows)]
    a_rows[7] = np.arange(inner)  # every row of B
    a = csr_of_rows(a_rows, inner, rng)
    check(nacho, oracle, a, b)
    two_passes(oracle, a, b, 5)


@pytest.mark.parametrize("rows", [600, 8300])
def test_many_products_in_two_passes(nacho, oracle, rows):
    """More than 32 M products of a clustered B that is read often: its rows as bitmap words in the symbolic pass, as pairs in the numeric one
    where there are many rows. B and A begin in the middle of their arrays, and some rows of B are empty."""
    rng = np.random.default_rng(rows)
    cols, inner = 50000, 320
    starts = rng.integers(0, cols - 4000, inner)
    b = csr_of_rows([np.arange(0) if r % 9 == 4 else np.sort(rng.choice(np.arange(s, s + 4000), 2400, replace=False)) for r, s in enumerate(starts)], cols, rng)
    per_row = 2 if rows > 8192 else 40
    a = csr_of_rows([scattered(inner, per_row + (r % 50 == 3), rng) for r in range(rows)], inner, rng)
    assert two_passes(oracle, a, b, 5) >= 32 << 20


def test_forms_of_b_give_way_to_the_result(nacho, oracle):
    """Where the result's arrays are refused while other forms of B are held, the call gives those back and asks again; a second refusal
    ends it."""
    import torch
    from nacho_b200 import _capi
    from nacho_b200._capi import TakeFn, lib
    rng = np.random.default_rng(5)
    b = csr_of_rows([np.arange(s, s + 2000) for s in rng.integers(0, 30000, 300)], 32000, rng)
    a = csr_of_rows([scattered(300, 2, rng) for _ in range(8400)], 300, rng)
    want, v64, abs64, products = oracle.spgemm(a, b, 8, extras=True)
    assert products >= 32 << 20
    ga, gb = Block(a, 0), Block(b, 0)
    for refusals in (1, 2):
        z, free = Result(a.rows), []

        def take(ctx, entries, p_col, p_val):
            free.append(torch.cuda.mem_get_info()[0])
            if len(free) <= refusals:
                return _capi.E_NOMEM
            z.take(entries)
            p_col[0], p_val[0] = z.col.data_ptr(), z.val.data_ptr()
            return _capi.OK

        status = lib.nb200_spgemm_f32_with(C.byref(ga.struct), C.byref(gb.struct), C.byref(z.struct), TakeFn(take), None, None)
        torch.cuda.synchronize()
        assert len(free) == 2 and free[1] >= free[0] + 16 * len(b.col)
        assert status == (_capi.E_NOMEM if refusals == 2 else _capi.OK)
        if refusals == 1:
            z.holds(want, v64, abs64)


def profile(run):
    """The names of the kernels that `run` launches."""
    import torch
    from nacho_b200 import _capi
    _capi.profile_reset()
    _capi.profile_enable(True)
    try:
        run()
        torch.cuda.synchronize()
    finally:
        _capi.profile_enable(False)
    return {n for n in _capi.profile_names() if _capi.profile_read(n)[0] > 0}


def test_masked_product_of_a_few_rows_with_a_large_matrix(nacho, oracle):
    """What 50 rows select of a matrix of 6 M entries: no kernel reads the rest of it, and the scratch is that of the mask."""
    import torch
    from nacho_b200._capi import lib
    rng = np.random.default_rng(3)
    inner, cols, per_row = 60000, 40000, 100
    b = CSR(inner, cols, (per_row * np.arange(inner + 1)).astype(np.int32),
            (np.sort(rng.integers(0, cols // per_row, (inner, per_row)), axis=1) + np.arange(per_row) * (cols // per_row)).ravel().astype(np.int32),
            rng.uniform(-1, 1, inner * per_row).astype(np.float32))
    a = csr_of_rows([scattered(inner, 40 + 90 * (r % 2), rng) for r in range(50)], inner, rng)
    c = csr_of_rows([scattered(cols, n, rng) for n in rng.choice([30, 900, 3000], 50)], cols, rng)
    ga, gb, gc = csr_to_gpu(a), csr_to_gpu(b), csr_to_gpu(c)
    lib.nb200_release_workspaces()
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    names = profile(lambda: nacho.gpu_sssmm_f32(ga, gb, gc))
    assert before - torch.cuda.mem_get_info()[0] < 32 << 20  # an eighth of a byte per entry of B would be 0.75 MB, 8 bytes 60 MB
    assert not [n for n in names if not n.startswith("sssmm_")]
    check_masked(nacho, oracle, a, b, c)


@pytest.mark.parametrize("width", [3, 40, 130])
def test_masked_product_of_a_band(nacho, oracle, width):
    """A band squared on its own positions: nearly every product reaches the mask, neighbours in neighbouring positions."""
    rng = np.random.default_rng(width)
    n = 1500
    a = csr_of_rows([np.arange(max(r - width, 0), min(r + width + 1, n)) for r in range(n)], n, rng)
    check_masked(nacho, oracle, a, a, a)


def test_masked_product_of_row_blocks(nacho, oracle):
    """Operands that begin in the middle of their arrays, on every list of the masked product."""
    import torch
    from nacho_b200._capi import CsrStruct, check, lib
    from test_family_gpu import mask_classes_case
    a, b, c = (synth_csr(t) for t in mask_classes_case())
    full, v64, abs64, _ = oracle.spgemm(a, b, 8, extras=True)
    key = lambda m: np.repeat(np.arange(m.rows, dtype=np.int64), np.diff(m.row_ptr)) * m.cols + m.col
    common, i_f, i_c = np.intersect1d(key(full), key(c), return_indices=True)
    ga, gb, gc = Block(a, 5), Block(b, 3), Block(c, 6)
    rp = torch.empty(a.rows + 1, dtype=torch.int32, device="cuda")
    col, val = torch.empty(len(c.col), dtype=torch.int32, device="cuda"), torch.empty(len(c.col), device="cuda")
    z = CsrStruct(0, 0, 0, rp.data_ptr(), col.data_ptr(), val.data_ptr())
    check(lib.nb200_sssmm_f32_into(C.byref(ga.struct), C.byref(gb.struct), C.byref(gc.struct), C.byref(z), len(c.col), None), "sssmm")
    torch.cuda.synchronize()
    got = CSR(a.rows, b.cols, rp.cpu().numpy(), col.cpu().numpy()[:z.nnz], val.cpu().numpy()[:z.nnz])
    assert np.array_equal(key(got), common)
    bound = REL_TOL * abs64[i_f] * np.abs(c.val[i_c]) + 1e-30
    assert np.all(np.abs(got.val.astype(np.float64) - v64[i_f] * c.val[i_c].astype(np.float64)) <= bound)
