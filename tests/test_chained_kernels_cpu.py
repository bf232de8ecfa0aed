"""Kernels started by launch_chained run while their predecessor writes their operands, so nothing
that a kernel may have written goes through the read-only path (__ldg, or a const __restrict__
pointer parameter): only plan tables, which uploads write, do. Checked on the source text."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "mps_gb300", "csrc")
# element types of plan tables (uploaded by the host, never written by a kernel)
TABLES = {"Problem", "Tile", "int2", "int4", "AxisEntry", "MapBlock", "SmallProblem", "ThinUnit",
          "ThinOffset", "int64_t", "BulkRow"}
LDG_TABLES = re.compile(r"__ldg\((&?probs\b|ax \+|ke \+|vals \+|prefix \+|reinterpret_cast<const int4\*>|"
                        r"p\), y = __ldg\(p \+ 1\)|p \+ 1\)|b\), y = __ldg\(b \+ 1\)|b \+ 1\))")


def source(name):
    with open(os.path.join(CSRC, name)) as f:
        return re.sub(r"//[^\n]*", "", f.read())


def chained():
    """{kernel: file} of every kernel that a launch_chained call names (`kern` picks among the
    instances of the thin kernel)."""
    out = {}
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu"))):
        name = os.path.basename(path)
        for k in re.findall(r"launch_chained\(\s*(\w+)", source(name)):
            out["contract_thin_kernel" if k == "kern" else k] = name
    return out


def test_finds_the_kernels():
    assert len(chained()) >= 9


@pytest.mark.parametrize("kernel,name", sorted(chained().items()) + [
    ("split_gemm_fast_kernel", "kernels_split.cu")])
def test_operands_are_not_read_only(kernel, name):
    m = re.search(r"__global__[^;{]*?\b" + kernel + r"\((.*?)\)\s*\{", source(name), re.S)
    assert m, kernel
    for p in m.group(1).split(","):
        q = re.match(r"\s*const (\w+)\s*\*\s*__restrict__", p)
        assert q is None or q.group(1) in TABLES, f"{kernel}: {p.strip()}"


@pytest.mark.parametrize("name", sorted(set(chained().values())))
def test_ldg_reads_tables_only(name):
    text = source(name)
    if name == "kernels_copy.cu":  # the warp-unit kernel there is launched without overlap
        text = text[text.index("copy_rows_bulk_kernel("):text.index("copy_tasks_kernel<<<")
                    if "copy_tasks_kernel<<<" in text else None]
    for m in re.finditer(r"__ldg\(", text):
        rest = text[m.start():m.start() + 80].split("\n")[0]
        assert LDG_TABLES.match(rest), f"{name}: {rest}"
