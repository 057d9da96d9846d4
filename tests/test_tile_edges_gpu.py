"""GPU suite: the sizes at which the merge tiles, the row classes and the routes of a call change, held to the
CPU oracle. Merged values are one float32 addition or product, so everything there is compared bit for bit;
sums of products are held to a bound in the magnitude that was summed."""
import threading

import numpy as np
import pytest

from helpers import assert_same, csf3_levels, csr_from_gpu, csr_to_gpu
from oracle.cpu_oracle import COO3, CSF3, CSR, DCSR

pytestmark = pytest.mark.gpu

SMALL_STEP = 256 * 15 - 1  # entries of a small CSR tile
LARGE_FROM = 6_000_000     # a tile holds 256 * 31 from here whatever its rows and columns (from SWITCH on where they allow it)
COO_STEP = 256 * 7 - 1     # entries of a small coordinate tile of a reduction (of a sum: SUM_STEP)
DIRECT_TILES = 128         # a few of the windows in which a tile reads the counts in front of it


@pytest.fixture(scope="module")
def nacho():
    import torch
    assert torch.cuda.is_available(), "GPU suite needs a CUDA device"
    from nacho_b200 import nacho as mod
    return mod


def csr_of_keys(key, rows, cols, rng):
    row = key // cols
    val = rng.uniform(-1, 1, len(key)).astype(np.float32)
    val[rng.random(len(key)) < 0.01] = -0.0
    return CSR(rows, cols, np.searchsorted(row, np.arange(rows + 1)).astype(np.int32), (key % cols).astype(np.int32), val)


def key_pair(total, space, shared, rng):
    """Two sorted lists of distinct keys below `space`, exactly `total` keys together, `shared` of the second in both."""
    n_a, n_b = total - total // 2, total // 2
    both = int(n_b * shared)
    n = total - both
    every = np.cumsum(1 + rng.integers(0, max((space - n) // n, 1), n)) - 1
    in_a = rng.permutation(n) < n_a
    in_b = ~in_a
    in_b[rng.permutation(np.flatnonzero(in_a))[:both]] = True
    assert in_a.sum() + in_b.sum() == total and every[-1] < space
    return every[in_a], every[in_b]


EDGES = [1, SMALL_STEP - 1, SMALL_STEP, SMALL_STEP + 1, 2 * SMALL_STEP, 2 * SMALL_STEP + 1, DIRECT_TILES * SMALL_STEP,
         DIRECT_TILES * SMALL_STEP + 1, (DIRECT_TILES + 1) * SMALL_STEP + 7]


@pytest.mark.parametrize("shape", ["one row", "rows of an entry", "rows of ten", "wide rows", "equal operands"])
@pytest.mark.parametrize("total", EDGES + [LARGE_FROM - 1, LARGE_FROM + 2])
def test_csr_tiles(nacho, oracle, total, shape):
    """Tiles of one entry more or less, more row starts than a tile keeps, columns too wide for keys of 32 bits,
    and operands with equal columns only, so that twins fall on every share and tile boundary."""
    rows, cols = {"one row": (1, 1 << 28), "rows of an entry": (total + 1, 300), "rows of ten": (total // 10 + 1, 4000),
                  "wide rows": (1 << 12, (1 << 31) - 1), "equal operands": (total // 30 + 1, 1 << 16)}[shape]
    rng = np.random.default_rng(total)
    ka, kb = key_pair(total, rows * cols, 1.0 if shape == "equal operands" else 0.3, rng)
    a, b = csr_of_keys(ka, rows, cols, rng), csr_of_keys(kb, rows, cols, rng)
    ga, gb = csr_to_gpu(a), csr_to_gpu(b)
    assert_same(csr_from_gpu(nacho.gpu_csr_add_f32(ga, gb)), oracle.csr_add(a, b, 8), "add")
    assert_same(csr_from_gpu(nacho.gpu_csr_mul_f32(ga, gb)), oracle.csr_mul(a, b, 8), "mul")
    c = csr_of_keys(np.union1d(ka[::2], kb[1::3]), rows, cols, rng)
    assert_same(csr_from_gpu(nacho.gpu_csr_add_3_f32(ga, gb, csr_to_gpu(c))), oracle.csr_add_3(a, b, c, 8), "add_3")


@pytest.mark.parametrize("total", [9, SMALL_STEP - 2, 2 * SMALL_STEP + 5, LARGE_FROM + 3])
@pytest.mark.parametrize("shift", [(0, 1), (1, 0), (2, 3)])
def test_csr_values_off_alignment(nacho, oracle, total, shift):
    """Values whose place in memory sits differently on 16-byte boundaries than their columns': no bulk copy can bring them to the
    columns' words."""
    import torch
    rows, cols = total // 20 + 1, 5000
    rng = np.random.default_rng(total)
    ka, kb = key_pair(total, rows * cols, 0.3, rng)

    def moved(x, by):
        t = torch.empty(len(x) + by, dtype=torch.from_numpy(x).dtype, device="cuda")[by:]
        return t.copy_(torch.from_numpy(x))

    def matrices(key, by):
        m = csr_of_keys(key, rows, cols, rng)
        return m, nacho.CSR_gpu(torch.from_numpy(m.row_ptr).cuda(), moved(m.col, by[0]), moved(m.val, by[1]), torch.tensor([rows, cols], dtype=torch.int32))

    (a, ga), (b, gb) = matrices(ka, shift), matrices(kb, shift[::-1])
    assert_same(csr_from_gpu(nacho.gpu_csr_add_f32(ga, gb)), oracle.csr_add(a, b, 8), "add")
    assert_same(csr_from_gpu(nacho.gpu_csr_mul_f32(ga, gb)), oracle.csr_mul(a, b, 8), "mul")


RESIDENT, OWN_CUTS_UP_TO = 592, 8192  # tiles that all find their cuts themselves; tiles beyond which a launch in front of the merge makes them
LARGE_STEP = 256 * 31 - 1


@pytest.mark.parametrize("total", [RESIDENT * SMALL_STEP, RESIDENT * SMALL_STEP + 1, 5_999_999, OWN_CUTS_UP_TO * LARGE_STEP, OWN_CUTS_UP_TO * LARGE_STEP + 1])
def test_cuts_of_many_tiles(nacho, oracle, total):
    """As many tiles as are at work at once and one more, and as many as have no launch in front of them and one more, on a stream of their
    own each: what the calls there keep starts with the smallest, and has to grow inside the chain of a three-operand sum."""
    import torch
    rows, cols = total // 50 + 1, 1 << 16
    rng = np.random.default_rng(total)
    ka, kb = key_pair(total, rows * cols, 0.3, rng)
    a, b = csr_of_keys(ka, rows, cols, rng), csr_of_keys(kb, rows, cols, rng)
    with torch.cuda.stream(torch.cuda.Stream()):
        ga, gb = csr_to_gpu(a), csr_to_gpu(b)
        if total < 6_000_000:
            assert_same(csr_from_gpu(nacho.gpu_csr_add_3_f32(ga, gb, ga)), oracle.csr_add_3(a, b, a, 8), "add_3")
        assert_same(csr_from_gpu(nacho.gpu_csr_add_f32(ga, gb)), oracle.csr_add(a, b, 8), "add")
        assert_same(csr_from_gpu(nacho.gpu_csr_mul_f32(ga, gb)), oracle.csr_mul(a, b, 8), "mul")


@pytest.mark.parametrize("total,rows,cols", [(t, (waves * 1856 * t) // LARGE_STEP + more, 1 << 13) for t, waves in ((RESIDENT * SMALL_STEP + 1, 2), (RESIDENT * LARGE_STEP, 2),
                                                                                                                  (RESIDENT * LARGE_STEP + 1, 1)) for more in (0, 1)]
                         + [(RESIDENT * LARGE_STEP + more, 1 << 12, (1 << 30) + wide) for more, wide in ((0, 1), (1, 0), (1, 1))])
def test_rows_and_columns_that_keep_tiles_small(nacho, oracle, total, rows, cols):
    """Merges on either side of the lines up to which many rows, and columns beyond 2^30, are merged in small tiles, more of them than are at
    work at once."""
    rng = np.random.default_rng(total + rows)
    ka, kb = key_pair(total, rows * cols, 0.3, rng)
    a, b = csr_of_keys(ka, rows, cols, rng), csr_of_keys(kb, rows, cols, rng)
    ga, gb = csr_to_gpu(a), csr_to_gpu(b)
    assert_same(csr_from_gpu(nacho.gpu_csr_add_f32(ga, gb)), oracle.csr_add(a, b, 8), "add")
    assert_same(csr_from_gpu(nacho.gpu_csr_mul_f32(ga, gb)), oracle.csr_mul(a, b, 8), "mul")
    assert_same(csr_from_gpu(nacho.gpu_csr_add_3_f32(ga, gb, ga)), oracle.csr_add_3(a, b, a, 8), "add_3")


def test_pieces_of_many_calls(nacho):
    """More reductions than control blocks are kept for, of one tile, of few and of many: each begins from nothing."""
    import torch
    rng = np.random.default_rng(3)
    dims = (2000, 300, 200)

    def tensor(n):
        key = np.unique(rng.integers(0, dims[0] * dims[1] * dims[2], n))
        c = np.stack([key // 60000, key // 200 % 300, key % 200], axis=1).astype(np.int32)
        return nacho.to_coo3(c, np.ones(len(key), np.float32), dims, "cuda"), len(key)

    operands = [tensor(n) for n in (500, 20_000, 400_000, 3_000_000)]
    got = [nacho.gpu_inner_prod_coo_f32(t, t).values for _ in range(6) for t, _ in operands]
    torch.cuda.synchronize()
    assert [float(v.cpu()[0]) for v in got] == [float(n) for _ in range(6) for _, n in operands]  # sums of ones: exact in double, and below 2^24


@pytest.mark.parametrize("gap", [3000, 1_200_000])
def test_runs_of_empty_rows(nacho, oracle, gap):
    """More tiles than fit the chip at once, with more rows between two of them than a tile keeps offsets of, empty but for a few: what a tile
    asks for ahead of time ends there."""
    rng = np.random.default_rng(gap)
    clusters, entries, cols = 16, 160_000, 5000
    rows = clusters * (gap + 1000)
    key = [np.sort(rng.choice(1000 * cols, entries, replace=False)) + c * (gap + 1000) * cols for c in range(clusters)]
    ka = np.concatenate(key)
    kb = np.sort(np.unique(np.concatenate([ka[::3], ka[1::4] + 1])))
    a, b = csr_of_keys(ka, rows, cols, rng), csr_of_keys(kb[kb < rows * cols], rows, cols, rng)
    assert len(a.col) + len(b.col) > 700 * SMALL_STEP
    ga, gb = csr_to_gpu(a), csr_to_gpu(b)
    assert_same(csr_from_gpu(nacho.gpu_csr_add_f32(ga, gb)), oracle.csr_add(a, b, 8), "add")
    assert_same(csr_from_gpu(nacho.gpu_csr_mul_f32(ga, gb)), oracle.csr_mul(a, b, 8), "mul")


@pytest.mark.parametrize("dims", [(3, 4, 1 << 28), (1 << 26, 9, 5), (1 << 20, 1 << 21, 1 << 22)])
@pytest.mark.parametrize("total", [1, COO_STEP, COO_STEP + 1, DIRECT_TILES * COO_STEP + 1, 3_000_000, 4096 * (256 * 17 - 1) + 1])
def test_coordinate_tiles(nacho, oracle, total, dims):
    """Coordinates whose differences within a tile fit 32 bits, and such that do not; the cuts of few and of many tiles."""
    from test_tensor3_gpu import coo3_from_gpu, coo3_to_gpu
    space = min(dims[0] * dims[1] * dims[2], 1 << 62)
    rng = np.random.default_rng(total)
    ka, kb = key_pair(total, space, 0.3, rng)

    def tensor(key):
        ij, k = np.divmod(key, dims[2])
        i, j = np.divmod(ij, dims[1])
        return COO3(dims, i.astype(np.int32), j.astype(np.int32), k.astype(np.int32), rng.uniform(-1, 1, len(key)).astype(np.float32))

    a, b = tensor(ka), tensor(kb)
    ga, gb = coo3_to_gpu(nacho, a), coo3_to_gpu(nacho, b)
    assert_same(coo3_from_gpu(nacho.gpu_coo3d_add_f32(ga, gb)), oracle.coo3_add(a, b, 8), "coo3 add")
    _, at_a, at_b = np.intersect1d(ka, kb, assume_unique=True, return_indices=True)
    terms = a.val[at_a].astype(np.float64) * b.val[at_b]
    got = float(nacho.gpu_inner_prod_coo_f32(ga, gb).values.cpu()[0])
    assert abs(got - terms.sum()) <= 1e-5 * np.abs(terms).sum() + 1e-30  # float32 products, 2^-24 each, summed wider


@pytest.mark.parametrize("total", [592 * (256 * v - 1) + more for v in (7, 11, 17) for more in (0, 1)])
def test_coordinate_tiles_of_one_wave(nacho, oracle, total):
    """As many tiles of every size as are at work at once, and one entry more: there reductions, then sums, take larger ones, and then a launch for their cuts."""
    test_coordinate_tiles(nacho, oracle, total, (1 << 9, 1 << 10, 1 << 11))


@pytest.mark.parametrize("total", [9, COO_STEP - 2, 2 * COO_STEP + 5, 3_000_011])
@pytest.mark.parametrize("shift", [(0, 1), (1, 0), (2, 3)])
def test_coordinate_values_off_alignment(nacho, oracle, total, shift):
    """Values whose place in memory sits differently on 16-byte boundaries than their coordinates': no bulk copy can bring them to the
    coordinates' words."""
    import torch
    dims = (1000, 800, 600)
    rng = np.random.default_rng(total)
    ka, kb = key_pair(total, dims[0] * dims[1] * dims[2], 0.3, rng)

    def moved(x, by):
        t = torch.empty(len(x) + by, dtype=torch.from_numpy(x).dtype, device="cuda")[by:]
        return t.copy_(torch.from_numpy(x))

    def tensors(key, by):
        t = COO3(dims, (key // 480000).astype(np.int32), (key // 600 % 800).astype(np.int32), (key % 600).astype(np.int32),
                 rng.uniform(-1, 1, len(key)).astype(np.float32))
        return t, nacho.COO3_gpu(*(moved(x, by[0]) for x in (t.i, t.j, t.k)), moved(t.val, by[1]), torch.tensor(dims, dtype=torch.int32))

    from test_tensor3_gpu import coo3_from_gpu
    (a, ga), (b, gb) = tensors(ka, shift), tensors(kb, shift[::-1])
    assert_same(coo3_from_gpu(nacho.gpu_coo3d_add_f32(ga, gb)), oracle.coo3_add(a, b, 8), "coo3 add")
    _, at_a, at_b = np.intersect1d(ka, kb, assume_unique=True, return_indices=True)
    terms = a.val[at_a].astype(np.float64) * b.val[at_b]
    assert abs(float(nacho.gpu_inner_prod_coo_f32(ga, gb).values.cpu()[0]) - terms.sum()) <= 1e-5 * np.abs(terms).sum() + 1e-30


# Where tiles change size, and where a second tile begins: 31 entries per thread for matrices from more small tiles on than are at work at once,
# 11 and 17 for sums of coordinates (7 and 17 for their reductions), 21 for the fibres of trees, 23 for the levels above.
SWITCH = RESIDENT * SMALL_STEP + 1
SUM_STEP, FIBRE_STEP, LEVEL_STEP = 256 * 11 - 1, 256 * 21 - 1, 256 * 23 - 1


@pytest.mark.parametrize("shape", ["one row", "rows of an entry", "rows of ten", "wide rows", "equal operands"])
@pytest.mark.parametrize("total", [SWITCH - 1, SWITCH, SWITCH + 1])
def test_csr_tiles_where_they_grow(nacho, oracle, total, shape):
    """The last small tiles and the first large ones, for every shape of a tile."""
    test_csr_tiles(nacho, oracle, total, shape)


@pytest.mark.parametrize("tiles", [31, 32, 33, 34, 64, 65, 66, 97])
def test_windows_of_counts(nacho, oracle, tiles):
    """A tile reads the counts in front of it 32 at a time: as many tiles as fill one window or two, one less and one more."""
    test_csr_tiles(nacho, oracle, tiles * SMALL_STEP, "rows of ten")
    test_coordinate_tiles(nacho, oracle, tiles * SUM_STEP, (1 << 9, 1 << 10, 1 << 11))


@pytest.mark.parametrize("dims", [(3, 4, 1 << 28), (1 << 26, 9, 5), (1 << 20, 1 << 21, 1 << 22)])
@pytest.mark.parametrize("total", [SUM_STEP - 1, SUM_STEP, SUM_STEP + 1, 2 * SUM_STEP, 2 * SUM_STEP + 1])
def test_coordinate_tiles_of_a_sum(nacho, oracle, total, dims):
    """One and two tiles of a sum, an entry more and less."""
    test_coordinate_tiles(nacho, oracle, total, dims)


@pytest.mark.parametrize("total", [SUM_STEP - 2, SUM_STEP + 1, 2 * SUM_STEP + 5, RESIDENT * SUM_STEP + 1])
@pytest.mark.parametrize("shift", [(0, 1), (3, 2)])
def test_coordinate_values_off_alignment_in_sums(nacho, oracle, total, shift):
    test_coordinate_values_off_alignment(nacho, oracle, total, shift)


@pytest.mark.parametrize("gap", [3000, 1_200_000])
def test_runs_of_empty_rows_between_large_tiles(nacho, oracle, gap):
    """More large tiles than are at work at once, so that the CTAs in front of them make the cuts, with runs of empty rows between."""
    rng = np.random.default_rng(gap)
    clusters, entries, cols = 16, 250_000, 5000
    rows = clusters * (gap + 1000)
    ka = np.concatenate([np.sort(rng.choice(1000 * cols, entries, replace=False)) + c * (gap + 1000) * cols for c in range(clusters)])
    kb = np.unique(np.concatenate([ka[::3], ka[1::4] + 1]))
    a, b = csr_of_keys(ka, rows, cols, rng), csr_of_keys(kb[kb < rows * cols], rows, cols, rng)
    assert len(a.col) + len(b.col) > max(700 * LARGE_STEP, 6_000_000)  # from where tiles are large whatever the rows
    ga, gb = csr_to_gpu(a), csr_to_gpu(b)
    assert_same(csr_from_gpu(nacho.gpu_csr_add_f32(ga, gb)), oracle.csr_add(a, b, 8), "add")
    assert_same(csr_from_gpu(nacho.gpu_csr_mul_f32(ga, gb)), oracle.csr_mul(a, b, 8), "mul")


AHEAD = 148  # tiles in front of a tile whose row offsets it asks for


@pytest.mark.parametrize("total", [9, 2 * SMALL_STEP + 5, SWITCH + 3, 5_200_000])
@pytest.mark.parametrize("dims", [(4000, 3000, 500), (2000, 130, 2000)])
@pytest.mark.parametrize("shift", [0, 1, 3])
def test_trees_of_many_tiles(nacho, oracle, total, dims, shift):
    """Trees of about an entry in a fibre, and of twenty, from one tile to more on both lower levels than are at work at once, so that some
    find their cuts and the offsets they ask for ahead made by the CTAs in front of them; with values that lie on 16-byte
    boundaries differently from their coordinates, too."""
    import torch
    from test_tensor3_gpu import csf3_from_gpu
    rng = np.random.default_rng(total + dims[1])

    def tree(key, by):
        ij, k = np.divmod(key, dims[2])
        new = np.flatnonzero(np.diff(ij, prepend=-1))
        i, j = np.divmod(ij[new], dims[1])
        first = np.flatnonzero(np.diff(i, prepend=-1))
        t = CSF3(dims, i[first].astype(np.int32), np.append(first, len(new)).astype(np.int32), j.astype(np.int32), np.append(new, len(key)).astype(np.int32),
                 k.astype(np.int32), rng.uniform(-1, 1, len(key)).astype(np.float32))
        to = lambda x: torch.from_numpy(x).cuda()
        val = torch.empty(len(key) + by, dtype=torch.float32, device="cuda")[by:].copy_(to(t.val))
        return t, nacho.CSF3_gpu(to(t.i_idx), to(t.j_ptr), to(t.j_idx), to(t.k_ptr), to(t.k_idx), val, torch.tensor(dims, dtype=torch.int32))

    ka, kb = key_pair(total, dims[0] * dims[1] * dims[2], 0.3, rng)
    (a, ga), (b, gb) = tree(ka, shift), tree(kb, (4 - shift) % 4)
    if total > 5_000_000:
        assert total > (RESIDENT + AHEAD) * FIBRE_STEP
        assert dims[1] != 3000 or len(a.j_idx) + len(b.j_idx) > (RESIDENT + AHEAD) * LEVEL_STEP
    assert_same(csf3_from_gpu(nacho.gpu_csf_add_f32(ga, gb)), oracle.csf3_add(a, b), "csf3")


@pytest.mark.parametrize("each", [1, 2, 5])
@pytest.mark.parametrize("total", [RESIDENT * SMALL_STEP + more for more in (0, 1)] + [RESIDENT * LARGE_STEP + more for more in (0, 1)] + [5_999_999, 6_000_000])
def test_row_lists_on_either_side_of_the_tiles_they_take(nacho, oracle, total, each):
    """Rows of one entry, of two and of five, in lists whose entries are merged in small tiles and in large ones."""
    from test_family_gpu import _dcsr_expected, csr_to_dcsr, dcsr_from_gpu, dcsr_to_gpu
    rows, cols = 4 * total if each == 1 else total // (2 * each), 4000
    rng = np.random.default_rng(total + each)
    ka, kb = key_pair(total, rows * cols, 0.3, rng)
    a, b = csr_of_keys(ka, rows, cols, rng), csr_of_keys(kb, rows, cols, rng)
    da, db = dcsr_to_gpu(nacho, csr_to_dcsr(a)), dcsr_to_gpu(nacho, csr_to_dcsr(b))
    assert_same(dcsr_from_gpu(nacho.gpu_dcsr_add_f32(da, db)), _dcsr_expected(oracle.csr_add(a, b, 8), a, b, False), "dcsr add")
    assert_same(dcsr_from_gpu(nacho.gpu_dcsr_mul_f32(da, db)), _dcsr_expected(oracle.csr_mul(a, b, 8), a, b, True), "dcsr mul")


@pytest.mark.parametrize("total", [RESIDENT * LARGE_STEP - 5, RESIDENT * LARGE_STEP + 5, 5_900_000])
@pytest.mark.parametrize("per_row,bits", [(3.3, 20), (10, 22), (100, 25), (35, 25), (60, 28)])
def test_tiles_on_either_side_of_wide_keys(nacho, oracle, total, per_row, bits):
    """Rows and columns with which a large tile's keys take 64 bits and a small one's 32, and with which both take 64."""
    rows, cols = int(total / per_row), 1 << bits
    rng = np.random.default_rng(total + bits)
    ka, kb = key_pair(total, rows * cols, 0.3, rng)
    a, b = csr_of_keys(ka, rows, cols, rng), csr_of_keys(kb, rows, cols, rng)
    ga, gb = csr_to_gpu(a), csr_to_gpu(b)
    assert_same(csr_from_gpu(nacho.gpu_csr_add_f32(ga, gb)), oracle.csr_add(a, b, 8), "add")
    assert_same(csr_from_gpu(nacho.gpu_csr_mul_f32(ga, gb)), oracle.csr_mul(a, b, 8), "mul")
    assert_same(csr_from_gpu(nacho.gpu_csr_add_3_f32(ga, gb, ga)), oracle.csr_add_3(a, b, a, 8), "add_3")


def test_stored_empty_rows_and_fibres(nacho, oracle):
    """Row lists that hold rows without entries, and trees that hold slices and fibres without any, come out without them."""
    from test_family_gpu import dcsr_from_gpu, dcsr_to_gpu
    from test_tensor3_gpu import _seeded, csf3_from_gpu
    import torch
    rng = np.random.default_rng(7)
    rows, cols = 5000, 800
    ops = []
    for _ in range(2):
        stored = np.sort(rng.choice(rows, 3000, replace=False))
        length = np.zeros(rows, np.int64)
        length[stored] = rng.integers(0, 9, len(stored))
        m = csr_of_keys(np.concatenate([r * cols + np.sort(rng.choice(cols, n, replace=False)) for r, n in enumerate(length)]).astype(np.int64), rows, cols, rng)
        ops.append((m, DCSR(rows, cols, stored.astype(np.int32), np.append(m.row_ptr[stored], m.row_ptr[-1]).astype(np.int32), m.col, m.val)))
    (a, da), (b, db) = ops
    z = oracle.csr_add(a, b)
    held = np.flatnonzero(np.diff(z.row_ptr)).astype(np.int32)
    want = DCSR(rows, cols, held, np.append(z.row_ptr[held], z.row_ptr[-1]).astype(np.int32), z.col, z.val)
    assert_same(dcsr_from_gpu(nacho.gpu_dcsr_add_f32(dcsr_to_gpu(nacho, da), dcsr_to_gpu(nacho, db))), want, "dcsr")

    dims = (40, 50, 60)
    (ca, va), (cb, vb) = _seeded(dims, 3000, 8)
    fa, fb = CSF3(dims, *csf3_levels(ca), va), CSF3(dims, *csf3_levels(cb), vb)
    j = np.setdiff1d(np.arange(dims[1]), fa.j_idx[:fa.j_ptr[1]])[:1]  # a fibre that slice 0 of A lacks, now stored without entries
    at = int(np.searchsorted(fa.j_idx[:fa.j_ptr[1]], j[0]))
    j_ptr = fa.j_ptr.copy()
    j_ptr[1:] += 1
    k_ptr = np.insert(fa.k_ptr, at, fa.k_ptr[at])
    to = lambda x: torch.from_numpy(np.ascontiguousarray(x)).cuda()
    plain = nacho.to_csf3(ca, va, dims, "cuda")
    hollow = type(plain)(to(fa.i_idx), to(j_ptr), to(np.insert(fa.j_idx, at, j[0]).astype(np.int32)), to(k_ptr.astype(np.int32)),
                         to(fa.k_idx), to(fa.val), torch.tensor(dims, dtype=torch.int32))
    gb = nacho.to_csf3(cb, vb, dims, "cuda")
    assert_same(csf3_from_gpu(nacho.gpu_csf_add_f32(hollow, gb)), oracle.csf3_add(fa, fb), "csf3")


@pytest.mark.parametrize("entries,length", [(1, 32), (4, 8), (6, 5), (8, 4), (9, 3), (4, 9), (1, 33), (3, 85), (2, 128), (1, 256), (64, 4), (300, 40)])
def test_product_rows(nacho, oracle, entries, length):
    """Rows of A of `entries` entries that select rows of B of `length`: up to 8 and 32 products in one pass, up to
    256 sorted, more ranked; at the tile of 128 rows and beyond 128 such tiles."""
    from test_spgemm_gpu import check
    rng = np.random.default_rng(entries * 1000 + length)
    inner, cols = 400, 5000
    rows = 128 * DIRECT_TILES + 1 if entries * length <= 33 else 129
    keys = lambda r, c, n: (np.arange(r)[:, None] * c + np.sort(np.argsort(rng.random((r, c)), axis=1)[:, :n], axis=1)).ravel()
    a = csr_of_keys(keys(rows, inner, entries), rows, inner, rng)
    b = csr_of_keys(keys(inner, cols, length), inner, cols, rng)
    check(nacho, oracle, a, b)


def test_many_ranked_rows(nacho, oracle):
    """8192 rows of 300 products and more: their CTAs hold sums in shared memory, and some rows more than those hold."""
    from test_spgemm_gpu import check
    rng = np.random.default_rng(3)
    rows, inner, cols = 8192 + 40, 600, 20000
    keys = lambda r, c, n: np.unique(np.repeat(np.arange(r), n) * c + rng.integers(0, c, r * n))
    length = np.full(inner, 110)
    length[:20] = 3000
    b_key = np.unique(np.concatenate([r * cols + rng.integers(0, cols, n) for r, n in enumerate(length)]))
    check(nacho, oracle, csr_of_keys(keys(rows, inner, 5), rows, inner, rng), csr_of_keys(b_key, inner, cols, rng))


def check_masked(nacho, oracle, a, b, c):
    """gpu_sssmm_f32 against the oracle's product on the mask's positions."""
    full, v64, abs64, _ = oracle.spgemm(a, b, 8, extras=True)
    key = lambda m: np.repeat(np.arange(m.rows, dtype=np.int64), np.diff(m.row_ptr)) * m.cols + m.col
    z = csr_from_gpu(nacho.gpu_sssmm_f32(csr_to_gpu(a), csr_to_gpu(b), csr_to_gpu(c)))
    common, i_f, i_c = np.intersect1d(key(full), key(c), return_indices=True)
    assert np.array_equal(key(z), common)
    bound = 1e-5 * abs64[i_f] * np.abs(c.val[i_c]) + 1e-30
    assert np.all(np.abs(z.val.astype(np.float64) - v64[i_f] * c.val[i_c].astype(np.float64)) <= bound)


@pytest.mark.parametrize("cols", [60000, 300000])
def test_masked_rows_by_words(nacho, oracle, cols):
    """A second operand of 2^18 entries and more: mask rows up to the bitmaps' largest, products that miss, meet one column of a
    bitmap's word or all 32."""
    rng = np.random.default_rng(cols)
    rows, inner = 60, 1200
    b_rows = [np.sort(rng.choice(cols, 240, replace=False)) if r % 3 else np.arange(q := int(rng.integers(0, cols - 400)), q + 250 + r % 60) for r in range(inner)]
    b = csr_of_keys(np.concatenate([r * cols + k for r, k in enumerate(b_rows)]).astype(np.int64), inner, cols, rng)
    assert len(b.col) >= 1 << 18
    per_row = np.array([0, 1, 8, 63, 64, 65, 200, 400, 1000, 1200] * 6)
    a = csr_of_keys(np.concatenate([r * inner + np.sort(rng.choice(inner, n, replace=False)) for r, n in enumerate(per_row)]).astype(np.int64), rows, inner, rng)
    masks = [0, 1, 40, 300, 2000, 2048, 2049, 8000, 8192, 20000]
    c = csr_of_keys(np.concatenate([r * cols + np.sort(rng.choice(cols, masks[(r + r // 10) % 10], replace=False)) for r in range(rows)]).astype(np.int64), rows, cols, rng)
    check_masked(nacho, oracle, a, b, c)


@pytest.mark.parametrize("cols", [40000, 65536, 70000])
def test_rows_by_result_length(nacho, oracle, cols):
    """Enough rows and products for the rows of B to be walked as bitmap words and the result's rows to be sorted by length:
    results from 300 entries to all columns, in rows of B that are scattered, solid runs, and runs that meet in one word; ranks in 16
    and (70000 columns) 32 bits."""
    from test_spgemm_gpu import check
    rng = np.random.default_rng(cols)
    inner, rows = 320, 8192 + 64
    b_rows = [np.sort(rng.choice(cols, 2400, replace=False)) for _ in range(200)]
    b_rows += [np.arange(q, q + n) for q, n in zip(rng.integers(0, cols - 4200, 118), rng.integers(300, 4200, 118))]
    b_rows += [np.arange(0, 17), np.arange(19, 2100)]  # neighbouring rows that end and begin in one word
    b_key = np.concatenate([r * cols + k for r, k in enumerate(b_rows)]).astype(np.int64)
    per_row = np.full(rows, 2)
    per_row[rng.integers(0, rows, 300)] = rng.integers(3, 60, 300)
    per_row[5:9] = 120, 200, 320, 319
    a_key = np.concatenate([r * inner + np.sort(rng.choice(inner, n, replace=False)) for r, n in enumerate(per_row)]).astype(np.int64)
    _, products = check(nacho, oracle, csr_of_keys(a_key, rows, inner, rng), csr_of_keys(b_key, inner, cols, rng))
    assert products >= 32 << 20


@pytest.mark.parametrize("cols", [65535, 65536, 65537])
def test_full_heavy_row(nacho, oracle, cols):
    """A row of more than 65535 products that reaches every column, at the width up to which positions fit 16 bits."""
    from test_spgemm_gpu import check
    rng = np.random.default_rng(cols)
    every = np.arange(cols)
    b_key = np.unique(np.concatenate([(every % 40) * cols + every, rng.integers(0, 40 * cols, 30000)]))  # 40 rows that cover all columns
    a_key = np.concatenate([np.arange(40), [40 + 3, 40 + 7], 80 + np.arange(40)])
    check(nacho, oracle, csr_of_keys(a_key, 3, 40, rng), csr_of_keys(b_key, 40, cols, rng))


@pytest.mark.parametrize("mask", [1, 31, 32, 33, 64, 65, 128, 129, 500])
def test_masked_rows_looked_up(nacho, oracle, mask):
    """Mask rows at the lengths where their look-up changes, under rows of A around its units of 8 entries."""
    rng = np.random.default_rng(mask)
    rows, inner, cols = 40, 3000, 100000
    per_row = np.array([1, 7, 8, 9, 64, 65, 300, 0] * 5)
    a = csr_of_keys(np.concatenate([r * inner + np.sort(rng.choice(inner, n, replace=False)) for r, n in enumerate(per_row)]).astype(np.int64), rows, inner, rng)
    b = csr_of_keys(np.unique(rng.integers(0, inner * cols, inner * 400)), inner, cols, rng)
    full, v64, abs64, _ = oracle.spgemm(a, b, 8, extras=True)
    key = lambda m: np.repeat(np.arange(m.rows, dtype=np.int64), np.diff(m.row_ptr)) * m.cols + m.col
    reached = [np.flatnonzero(key(full) // cols == r) for r in range(rows)]
    picks = [key(full)[rng.permutation(q)[:mask - mask // 3]] for q in reached]
    c = csr_of_keys(np.unique(np.concatenate(picks + [r * cols + rng.choice(cols, mask // 3, replace=False) for r in range(rows)])).astype(np.int64), rows, cols, rng)
    z = csr_from_gpu(nacho.gpu_sssmm_f32(csr_to_gpu(a), csr_to_gpu(b), csr_to_gpu(c)))
    common, i_f, i_c = np.intersect1d(key(full), key(c), return_indices=True)
    assert np.array_equal(key(z), common)
    bound = 1e-5 * abs64[i_f] * np.abs(c.val[i_c]) + 1e-30
    assert np.all(np.abs(z.val.astype(np.float64) - v64[i_f] * c.val[i_c].astype(np.float64)) <= bound)


def test_threads_share_a_stream(nacho, oracle):
    """Calls of several host threads on one stream, and on streams of their own with operands of another, as if alone."""
    import torch
    rng = np.random.default_rng(11)
    jobs = []
    for total in (200, 4000, 50_000, 700_000):
        ka, kb = key_pair(total, 3000 * 5000, 0.3, rng)
        a, b = csr_of_keys(ka, 3000, 5000, rng), csr_of_keys(kb, 3000, 5000, rng)
        jobs.append((csr_to_gpu(a), csr_to_gpu(b), oracle.csr_add(a, b, 8), oracle.csr_mul(a, b, 8)))
    torch.cuda.synchronize()
    wrong = []

    def work(job, stream):
        ga, gb, add, mul = job
        try:
            with torch.cuda.stream(stream):
                for _ in range(20):
                    z, p = nacho.gpu_csr_add_f32(ga, gb), nacho.gpu_csr_mul_f32(ga, gb)
                    assert_same(csr_from_gpu(z), add, "add")
                    assert_same(csr_from_gpu(p), mul, "mul")
        except BaseException as e:  # reported by the main thread
            wrong.append(e)

    for streams in ([torch.cuda.current_stream()] * 4, [torch.cuda.Stream() for _ in range(4)]):
        threads = [threading.Thread(target=work, args=(j, s)) for j, s in zip(jobs, streams)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        assert not wrong, wrong[0]
