"""Kernels of a chain of dependent launches read what the launch before wrote (or may still be writing) through
ordinary loads only: ld.global.nc, from __ldg or from a const restrict parameter, may be moved above the wait."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "enblend-enfuse_gb300" / "csrc"
TABLE = re.compile(r"&(a\.tab|tab|g_div_table)\.")


def _code(path):
    text = re.sub(r"//[^\n]*", "", path.read_text())
    return re.sub(r"/\*.*?\*/", "", text, flags=re.S)


def _balanced(text, start):
    """The parenthesised or braced text that opens at or after start."""
    i = start
    while text[i] not in "({":
        i += 1
    depth, j = 0, i
    while True:
        depth += (text[j] in "({") - (text[j] in ")}")
        j += 1
        if depth == 0:
            return text[i:j], j


SOURCES = [p for p in sorted(CSRC.glob("*.cu*")) if p.suffix == ".cuh" or "griddep_wait()" in _code(p)]


@pytest.mark.parametrize("path", SOURCES, ids=lambda p: p.name)
def test_read_only_loads_are_of_tables(path):
    code = _code(path)
    bad = [code[m.end():m.end() + 60] for m in re.finditer(r"__ldg\(", code) if not TABLE.match(code[m.end():])]
    assert not bad, bad


@pytest.mark.parametrize("path", SOURCES, ids=lambda p: p.name)
def test_waiting_kernels_have_no_restrict_parameters(path):
    code = _code(path)
    for m in re.finditer(r"__global__ void( __launch_bounds__\([^)]*\))? (\w+)\(", code):
        params, end = _balanced(code, m.end() - 1)
        body, _ = _balanced(code, end)
        if "griddep_wait()" in body:
            assert "__restrict__" not in params, m.group(2)
