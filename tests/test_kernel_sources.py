"""CPU suite: rules that a compiled kernel cannot show and its source can."""
import os
import re

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
    assert "tile_v(total, rows.value, cols)" in source("csr_merge.cu")


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
