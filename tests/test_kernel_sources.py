"""CPU suite: rules that a compiled kernel cannot show and its source can."""
import os
import re
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "nacho_b200", "csrc")


def source(name):
    text = open(os.path.join(CSRC, name)).read()
    return re.sub(r"//[^\n]*", "", text)


def parameters(text, kernel):
    """The parameter list of a kernel's definition."""
    return re.search(re.escape(kernel) + r"\(([^{;]*)\)\s*\{", text).group(1)


def test_steps_of_an_unrolled_merge_hold_no_loops():
    """What a step of a tile's merge holds is in its kernel once for every entry of a thread, for both operands. With a search there the
    kernels of 64-bit keys wait for their instructions: the search is a call."""
    text = source("csr_merge.cu")
    assert re.search(r"__noinline__\s+int\s+far_row\(", text)
    body = text[text.index("auto marked_row = "):]
    body = body[:body.index("};")]
    assert "far_row(" in body and not re.search(r"\b(for|while|do)\b", body)


def test_the_choice_of_tiles_knows_the_rows_of_row_lists():
    """Only the device knows how many rows two row lists have together, the call knows the most there can be: large tiles lose to small ones
    where rows hold an entry, so it has to say."""
    merges = re.findall(r"csr2_enqueue\((.*?)\)\)\)?\s", source("formats2d.cu"), re.S)
    of_entries = [m for m in merges if "&rows_ctl->total}" in m]
    assert of_entries and all("RowCount{(int32_t)std::min<int64_t>(stored, a->rows), &rows_ctl->total}" in m for m in of_entries)
    assert re.search(r"tile_v\(total, rows\.value, cols\b", source("csr_merge.cu"))


@pytest.mark.skipif(not shutil.which("g++"), reason="no host compiler")
def test_keys_of_a_large_tile_are_no_wider_than_need_be(tmp_path):
    """The choice of tiles by itself: a large one whose keys take 64 bits gives way to a small one that gets by with 32."""
    text = source("csr_merge.cu")
    rule = text[text.index("inline int tile_v("):]
    rule = rule[:rule.index("\n}\n") + 3]
    cases = [(2_500_000, 30_000, 20, 31), (2_500_000, 750_000, 20, 15), (2_500_000, 750_000, 14, 31), (2_500_000, 250_000, 22, 15), (2_500_000, 25_000, 25, 15),
             (4_000_000, 1_200_000, 20, 15), (5_900_000, 60_000, 25, 15), (5_900_000, 590_000, 22, 15), (5_900_000, 590_000, 16, 31), (6_000_000, 750_000, 20, 31),
             (2_272_688, 10, 10, 15), (2_272_689, 10, 10, 31), (4_000_000, 10, 31, 31), (4_900_000, 10, 31, 15)]
    (tmp_path / "rule.cpp").write_text("""
#include <cstdint>
#include <cstdio>
constexpr int RESIDENT = 592, V_SMALL = 15, V_LARGE = 31;
constexpr int tile_step(int v) { return 256 * v - 1; }
constexpr int64_t LARGE_FROM = (int64_t)RESIDENT * tile_step(V_SMALL) + 1, LARGE_ALWAYS_FROM = 6000000;
template <int V, bool L> struct TilePlan { static constexpr int ROWS = 1856; };
static int col_bits(int32_t cols) { int b = 1; while (b < 32 && (int64_t(1) << b) < cols) ++b; return b; }
""" + rule + "int main() {" + "".join('printf("%%d ", tile_v(%d, %d, (int32_t)%dll));' % (total, rows, min(1 << bits, 2**31 - 1)) for total, rows, bits, _ in cases) + "}")
    subprocess.run(["g++", "-std=c++17", "-o", str(tmp_path / "rule"), str(tmp_path / "rule.cpp")], check=True)
    got = subprocess.run([str(tmp_path / "rule")], check=True, capture_output=True, text=True).stdout.split()
    assert [int(v) for v in got] == [want for *_, want in cases]


def test_the_merge_does_not_wait_for_values_of_another_alignment():
    """What brings a tile's values into shared memory stands in front of its merge: an array that no bulk copy can bring is not loaded by the
    threads, which would wait for it there, but copied word by word, and landed before the values are used."""
    text = source("coo3_merge.cu")
    body = text[text.index("bool coo3_stage_values("):text.index("void coo3_tile(")]
    loop = body[body.index("for (int e = tid"):]
    assert "copy_word(" in loop[:loop.index(";", loop.index(")"))] and "__ldg" not in loop[:loop.index("else if")]
    tile = text[text.index("void coo3_tile("):]
    waits = [m.start() for m in re.finditer(r"mbar_wait_bounded\(&sh\.mbar, 1, MBAR_POLL_LIMIT\);\n\s*if \(!__syncthreads_and", tile)]
    assert len(waits) == 2 and all("if (word_by_word) copies_landed();" in tile[at - 150:at] for at in waits)
    assert re.search(r"return nv\[0\] == 0 \|\| nv\[1\] == 0;", body) and "word_by_word = STAGED && coo3_stage_values(" in tile


def test_no_read_only_loads_of_what_an_overlapped_kernel_waits_for():
    """A kernel that starts beside the one in front of it must not use read-only loads (ld.global.nc, or a const
    __restrict__ parameter that the compiler turns into one) for what that kernel writes: they may be issued before the
    wait. All kernels of the CSR merge start like that, and their operands may be an earlier call's result."""
    for name in ("csr_merge.cu", "csr_common.cuh"):
        text = source(name)
        assert not re.search(r"\bld_nc\b|\b__ldg\b|\b__ldcs\b|__restrict__", text), name
    late = {("spgemm_esc.cu", "k_esc_rowwork"): ["P"], ("spgemm_masked.cu", "k_sssmm_bitmap"): ["units", "ctl"],
            ("spgemm_masked.cu", "k_sssmm_scan"): ["pos", "acc"], ("spgemm_masked.cu", "k_sssmm_row_offsets"): ["pos"]}
    for (name, kernel), arrays in late.items():
        text = source(name)
        given = parameters(text, kernel)
        for a in arrays:
            assert re.search(r"\*" + a + r"\b", given), (kernel, a)
            assert not re.search(r"__restrict__\s+" + a + r"\b", given), (kernel, a)
        body = text[text.index(given):]
        body = body[:re.search(r"\n\}", body).start()]
        for a in arrays:
            assert not re.search(r"(ld_nc|__ldg|__ldcs)\(" + a + r"\b", body), (kernel, a)
