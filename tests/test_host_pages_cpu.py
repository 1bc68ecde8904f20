"""Whether a caller's array can be written in place (physim_gb300/csrc/host_pages.h),
compiled here: yes for memory that may be written, its pages touched or not, from any
byte of a page on, with its contents kept; no for a mapping that may only be read, and
for one that ends before the array does, on which a kernel's write would fault."""
from __future__ import annotations

import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "physim_gb300" / "csrc"

MAIN = r"""
#include <stdio.h>
#include <string.h>
#include "host_pages.h"
int main()
{
    const size_t page = (size_t)sysconf(_SC_PAGESIZE), bytes = 8 * page;
    char *rw = (char *)mmap(0, bytes, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0);
    char *ro = (char *)mmap(0, bytes, PROT_READ, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0);
    char *cut = (char *)mmap(0, bytes, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0);
    if (!pg::populate_pages(rw, bytes, true)) return 77;  // a kernel without the advice
    munmap(cut + 4 * page, 4 * page);
    rw[3] = 5;
    printf("%d %d %d %d %d %d\n", pg::populate_pages(rw + 3, bytes - 9, true), (int)rw[3],
           pg::populate_pages(ro, bytes, false), pg::populate_pages(ro + 8, 80, true),
           pg::populate_pages(cut, 4 * page, true), pg::populate_pages(cut, 4 * page + 8, true));
    return 0;
}
"""


def test_pages(tmp_path):
    src, exe = tmp_path / "pages.cpp", tmp_path / "pages"
    src.write_text(MAIN)
    subprocess.run(["g++", "-O2", "-std=c++17", f"-I{CSRC}", str(src), "-o", str(exe)], check=True)
    run = subprocess.run([str(exe)], capture_output=True, text=True)
    if run.returncode == 77:
        pytest.skip("the kernel maps no pages on request")
    assert run.returncode == 0
    assert run.stdout.split() == ["1", "5", "1", "0", "1", "0"]


def test_downloads_ask():
    """The answer decides between the kernel and the copy."""
    text = (CSRC / "integrate.cu").read_text()
    body = text[text.index("int download_direct("):]
    assert "populate_pages(p, bytes, true)" in body[:body.index("\n}")]
