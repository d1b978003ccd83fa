"""A kernel launched ahead of its turn reads what the grid before it writes by
ordinary loads behind its wait (csrc/wk_loads.cuh), never as memory that is
read-only for the kernel's lifetime.  Read from the source: each array that the
grid before may still be writing, in the kernels that are launched ahead."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "wukonggpu_gb300" / "csrc"

# file -> function whose body is checked, the arrays (as the source names them)
READS = [
    ("wk_kernels.cu", "k2u_count_kernel", ["hist"]),
    ("wk_kernels.cu", "plan_group", ["a.group_sums", "a.blk_sum", "a.err"]),
    ("wk_kernels.cu", "publish_kernel", ["pub.src"]),
    ("wk_kernels.cu", "k2u_expand_kernel", ["head", "slices"]),
    ("wk_kernels.cu", "filter_probe_kernel", ["hist"]),
    ("wk_kernels.cu", "filter_write_kernel", ["mask", "blk_nz", "group_sums"]),
    ("wk_fused.cu", "count_blocks", ["a.hist"]),
    ("wk_fused.cu", "copy_row_regs", ["src"]),
    ("wk_fused.cu", "write_k2u", ["a.nbr", "a.blk_nz"]),
    ("wk_fused.cu", "write_filter", ["hb", "a.mask", "a.blk_nz"]),
    ("wk_part.cu", "part_move_kernel", ["start"]),
    ("wk_batch.cu", "find_query", ["off"]),
    ("wk_batch.cu", "find_query_warp", ["off"]),
    ("wk_batch.cu", "find_queries", ["off"]),
    ("wk_batch.cu", "count_phase", ["row", "io.in_row_off"]),
    ("wk_tc_gemm.cuh", "sum_rows", ["part"]),
]


def _body(text, name):
    """The text of function `name` from its name to the brace that closes it."""
    at = re.search(rf"\b{name}\(", text).start()
    i, depth = text.index("{", at), 0
    for j in range(i, len(text)):
        depth += {"{": 1, "}": -1}.get(text[j], 0)
        if depth == 0:
            return text[at:j + 1]
    raise AssertionError(name)


@pytest.mark.parametrize("file,name,arrays", READS, ids=lambda x: x if isinstance(x, str) else "")
def test_no_read_only_loads(file, name, arrays):
    body = re.sub(r"//[^\n]*", "", _body((CSRC / file).read_text(), name))
    inside = body[body.index("{"):]
    for a in arrays:
        n = re.escape(a)
        # __ldg / __ldcg of an address formed from the array, or the array dereferenced
        assert not re.search(rf"__ldc?g\((?:reinterpret_cast<[^>]*>\()?{n}\b", inside), (name, a)
        assert not re.search(rf"(?<![\w.)]){n}\[", inside), (name, a)
        assert not re.search(rf"(?:[=(,!<>&|]|return)\s*\*{n}\b", inside), (name, a)
        assert re.search(rf"ld_(?:prior|l2)\((?:reinterpret_cast<[^>]*>\()?{n}\b", inside) or a == "slices", (name, a)
