"""GPU suite: calls whose operands are the results of calls that may still be running, held to the CPU oracle."""
import numpy as np
import pytest

from helpers import assert_same, csr_from_gpu, csr_to_gpu
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
