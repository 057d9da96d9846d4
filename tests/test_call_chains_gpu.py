"""GPU suite: calls whose operands are the results of calls that may still be running, held to the CPU oracle."""
import numpy as np
import pytest

from helpers import assert_same, csr_from_gpu, csr_to_gpu
from oracle.cpu_oracle import CSR
from test_tile_edges_gpu import csr_of_keys, key_pair, nacho  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("total", [300, 60_000, 1_500_000, 7_000_000])
def test_results_as_operands(nacho, oracle, total):
    """Every call of a chain takes what the one before it has just returned, in storage that earlier rounds have used."""
    rng = np.random.default_rng(total)
    rows, cols = total // 12 + 1, 5000
    ka, kb = key_pair(total, rows * cols, 0.4, rng)
    a, b = csr_of_keys(ka, rows, cols, rng), csr_of_keys(kb, rows, cols, rng)
    ga, gb = csr_to_gpu(a), csr_to_gpu(b)
    want = oracle.csr_add(a, b, 8)
    want = oracle.csr_mul(want, a, 8)
    want = oracle.csr_add_3(want, b, a, 8)
    want = oracle.csr_add(want, want, 8)
    for _ in range(5):
        z = nacho.gpu_csr_add_f32(ga, gb)
        z = nacho.gpu_csr_mul_f32(z, ga)
        z = nacho.gpu_csr_add_3_f32(z, gb, ga)
        z = nacho.gpu_csr_add_f32(z, z)
        assert_same(csr_from_gpu(z), want, "chain")


def test_product_of_a_fresh_sum(nacho, oracle):
    """Products, plain and masked, of a sum that has just been returned: same structure, sums within float32 rounding."""
    rng = np.random.default_rng(4)
    n = 3000
    ka, kb = key_pair(60_000, n * n, 0.3, rng)
    a, b = csr_of_keys(ka, n, n, rng), csr_of_keys(kb, n, n, rng)
    s = oracle.csr_add(a, b, 8)
    full, v64, abs64, _ = oracle.spgemm(s, s, 8, extras=True)
    ga, gb = csr_to_gpu(a), csr_to_gpu(b)
    for _ in range(3):
        gs = nacho.gpu_csr_add_f32(ga, gb)
        p, m = nacho.gpu_spgemm_f32(gs, gs), nacho.gpu_sssmm_f32(gs, gs, gs)
        z = csr_from_gpu(p)
        assert np.array_equal(z.row_ptr, full.row_ptr) and np.array_equal(z.col, full.col)
        assert np.all(np.abs(z.val - v64) <= 1e-5 * abs64 + 1e-30)
        key = lambda t: np.repeat(np.arange(t.rows, dtype=np.int64), np.diff(t.row_ptr)) * t.cols + t.col
        common, i_f, i_s = np.intersect1d(key(full), key(s), return_indices=True)
        z = csr_from_gpu(m)
        assert np.array_equal(key(z), common)
        assert np.all(np.abs(z.val - v64[i_f] * s.val[i_s].astype(np.float64)) <= 1e-5 * abs64[i_f] * np.abs(s.val[i_s]) + 1e-30)


@pytest.mark.parametrize("total", [24_000, 700_000, 6_100_000])
def test_a_merge_that_gives_up_ends_its_chain(nacho, oracle, total):
    """A three-operand add whose first union runs without its first tile, with few and with many tiles: the second
    union follows none of its offsets, which are what the scratch held, and so writes no row; the call reports the wait,
    and the same call works afterwards."""
    import ctypes as C
    import torch
    from nacho_b200 import _capi
    from nacho_b200._capi import CsrStruct, lib
    rng = np.random.default_rng(total)
    rows, cols = total // 9, 30000
    ka, kb = key_pair(total, rows * cols, 0.2, rng)
    a, b = csr_of_keys(ka, rows, cols, rng), csr_of_keys(kb, rows, cols, rng)
    ga, gb = csr_to_gpu(a), csr_to_gpu(b)
    cap = 2 * len(a.col) + len(b.col)
    want = oracle.csr_add_3(a, b, a, 8)
    for _ in range(2):
        assert_same(csr_from_gpu(nacho.gpu_csr_add_3_f32(ga, gb, ga)), want, "add_3")
        rp = torch.full((rows + 1,), -1, dtype=torch.int32, device="cuda")
        col = torch.empty(cap, dtype=torch.int32, device="cuda")
        val = torch.empty(cap, dtype=torch.float32, device="cuda")
        z = CsrStruct(rows, cols, 0, rp.data_ptr(), col.data_ptr(), val.data_ptr())
        sa, sb = ga._struct(), gb._struct()
        status = lib.nb200_selftest_chain_timeout(C.byref(sa), C.byref(sb), C.byref(sa), C.byref(z), cap, 50, None)
        torch.cuda.synchronize()
        assert status == _capi.E_TIMEOUT and "look-back" in lib.nb200_last_cuda_error().decode()
        assert bool((rp[1:] == -1).all())
    assert_same(csr_from_gpu(nacho.gpu_csr_add_3_f32(ga, gb, ga)), want, "add_3 after a give-up")
    sa.nnz = 10
    assert lib.nb200_selftest_chain_timeout(C.byref(sa), C.byref(sa), C.byref(sa), C.byref(z), cap, 50, None) == _capi.E_BADARG


def test_levels_behind_one_that_gave_up(nacho, oracle):
    """A CSF3 add whose slice lists give up: neither the fibres nor the entries are merged, and the call says why."""
    import ctypes as C
    import torch
    from nacho_b200 import _capi
    from nacho_b200._capi import Csf3Struct, lib
    from helpers import csf3_levels
    from oracle.cpu_oracle import CSF3
    from test_tensor3_gpu import _seeded, csf3_from_gpu
    dims = (60_000, 500, 400)
    (ca, va), (cb, vb) = _seeded(dims, 90_000, 5)
    ga, gb = nacho.to_csf3(ca, va, dims, "cuda"), nacho.to_csf3(cb, vb, dims, "cuda")
    want = oracle.csf3_add(CSF3(dims, *csf3_levels(ca), va), CSF3(dims, *csf3_levels(cb), vb))
    n_i, n_j, n_k = (len(getattr(ga, f)) + len(getattr(gb, f)) for f in ("dim_i_indices", "dim_j_indices", "dim_k_indices"))
    assert n_i >= 24_000
    for _ in range(2):
        assert_same(csf3_from_gpu(nacho.gpu_csf_add_f32(ga, gb)), want, "csf3")
        i, jp, j, kp, k = (torch.full((n,), -1, dtype=torch.int32, device="cuda") for n in (n_i, n_i + 1, n_j, n_j + 1, n_k))
        v = torch.empty(n_k, dtype=torch.float32, device="cuda")
        z = Csf3Struct((C.c_int32 * 3)(), 0, 0, 0, *(t.data_ptr() for t in (i, jp, j, kp, k, v)))
        sa, sb = ga._struct(), gb._struct()
        status = lib.nb200_selftest_levels_timeout(C.byref(sa), C.byref(sb), C.byref(z), n_i, n_j, n_k, 50, None)
        torch.cuda.synchronize()
        assert status == _capi.E_TIMEOUT and "look-back" in lib.nb200_last_cuda_error().decode()
        assert bool((jp[1:] == -1).all()) and bool((kp[1:] == -1).all()) and bool((k == -1).all())
    assert_same(csf3_from_gpu(nacho.gpu_csf_add_f32(ga, gb)), want, "csf3 after a give-up")


@pytest.mark.parametrize("total", [24_000, 400_000, 1_500_000, 6_100_000])
def test_a_late_give_up_is_reported(nacho, oracle, total):
    """A first tile that takes a millisecond, for the two million empty rows it begins with, and others that wait for its
    count for some polls only: a call either says that they gave up or its result is whole. Few tiles, which all
    find their cuts themselves, and many, whose cuts come from the CTAs in front of them."""
    import ctypes as C
    import torch
    from nacho_b200 import _capi
    from nacho_b200._capi import CsrStruct, lib
    rng = np.random.default_rng(total)
    empty, cols = 2_000_000, 30000
    rows = empty + total // 9
    ka, kb = key_pair(total, (total // 9) * cols, 0.2, rng)
    a, b = csr_of_keys(ka + empty * cols, rows, cols, rng), csr_of_keys(kb + empty * cols, rows, cols, rng)
    ga, gb = csr_to_gpu(a), csr_to_gpu(b)
    want = oracle.csr_add(a, b, 8)
    seen = []
    for polls in [1, 8, 64, 200, 500, 1000, 1500, 2000, 1 << 20]:
        rp = torch.full((rows + 1,), -1, dtype=torch.int32, device="cuda")
        col = torch.full((total,), -1, dtype=torch.int32, device="cuda")
        val = torch.full((total,), float("nan"), dtype=torch.float32, device="cuda")
        z = CsrStruct(rows, cols, 0, rp.data_ptr(), col.data_ptr(), val.data_ptr())
        sa, sb = ga._struct(), gb._struct()
        status = lib.nb200_selftest_late_give_up(C.byref(sa), C.byref(sb), C.byref(z), total, polls, None)
        torch.cuda.synchronize()
        assert status in (_capi.OK, _capi.E_TIMEOUT)
        seen.append(status)
        if status == _capi.OK:
            assert_same(CSR(rows, cols, rp.cpu().numpy(), col[:z.nnz].cpu().numpy(), val[:z.nnz].cpu().numpy()), want, f"{polls} polls")
    assert seen[0] == _capi.E_TIMEOUT and seen[-1] == _capi.OK, seen
    assert_same(csr_from_gpu(nacho.gpu_csr_add_f32(ga, gb)), want, "add after a give-up")


@pytest.mark.parametrize("total", [2000, 200_000])
@pytest.mark.parametrize("before", ["nothing", "kernel", "copy", "other stream"])
def test_asynchronous_calls_in_a_graph(nacho, oracle, total, before):
    """Two asynchronous sums captured behind nothing, a kernel, a copy or the work of another stream, and replayed."""
    import ctypes as C
    import torch
    from nacho_b200 import _capi
    from nacho_b200._capi import CsrStruct, check, lib
    rng = np.random.default_rng(total)
    rows, cols = total // 10, 3000
    ka, kb = key_pair(total, rows * cols, 0.3, rng)
    a, b = csr_of_keys(ka, rows, cols, rng), csr_of_keys(kb, rows, cols, rng)
    want = oracle.csr_add(a, b, 8)
    ga, gb = csr_to_gpu(a), csr_to_gpu(b)
    rp, col = (torch.empty(n, dtype=torch.int32, device="cuda") for n in (rows + 1, total))
    val, x, y = (torch.zeros(n, device="cuda") for n in (total, 1000, 1000))
    res = torch.empty(3, dtype=torch.int64, device="cuda")
    z, sa, sb = CsrStruct(rows, cols, 0, rp.data_ptr(), col.data_ptr(), val.data_ptr()), ga._struct(), gb._struct()
    stream, side = torch.cuda.Stream(), torch.cuda.Stream()

    def call():
        check(lib.nb200_csr_add_f32_async(C.byref(sa), C.byref(sb), C.byref(z), total, res.data_ptr(), stream.cuda_stream), "async")

    torch.cuda.synchronize()
    with torch.cuda.stream(stream):
        call()  # takes the stream's scratch before the capture begins
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        if before == "kernel":
            x.add_(1)
        elif before == "copy":
            x.copy_(y)
        elif before == "other stream":
            side.wait_stream(stream)
            with torch.cuda.stream(side):
                y.add_(1)
            stream.wait_stream(side)
        call()
        call()
        x.add_(1)
    for _ in range(3):
        for t in (rp, col, val, res):
            t.fill_(-1)
        graph.replay()
        torch.cuda.synchronize()
        n = len(want.col)
        assert res.tolist() == [n, _capi.OK, rows]
        assert_same(CSR(rows, cols, rp.cpu().numpy(), col[:n].cpu().numpy(), val[:n].cpu().numpy()), want, before)
