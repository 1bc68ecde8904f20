"""Dynamic shared memory that 16-byte asynchronous copies write is declared with that
alignment (a declaration promises no more than its type's otherwise, and where the
array starts then depends on the static shared memory beside it)."""
from __future__ import annotations

import re
from pathlib import Path

CSRC = Path(__file__).resolve().parents[1] / "physim_gb300" / "csrc"


def test_asynchronous_copies_write_aligned_arrays():
    text = (CSRC / "bh.cu").read_text()
    copies = re.findall(r"cp\.async\.\w+\.shared\.global \[%0\], \[%1\], (\d+);", text)
    assert copies == ["16"]  # in rank_sort_body alone
    body = text.index("rank_sort_body(const TreeSortArgs")
    assert body < text.index("cp.async") < text.index("rank_sort_kernel", body)
    kernel = text[text.index("rank_sort_kernel(TreeSortArgs"):]
    kernel = kernel[:kernel.index("\n}")]
    found = re.search(r"extern __shared__ __align__\((\d+)\) \w+ (\w+)\[\];", kernel)
    assert found and int(found.group(1)) >= 16
    assert f"rank_sort_body(a, {found.group(2)})" in kernel
