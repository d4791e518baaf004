"""CPU: kernels that wait for their predecessor inside the kernel (programmatic dependent launch) read what it writes by ordinary
loads: the read-only path (__ldg, const __restrict__ parameters) is for memory that stays unchanged while the kernel runs.
Checked on the source text: __ldg only on the job's vectors and the plan's tables, and no restrict-qualified input pointer."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "mpfs250t-sar-ifp_b200" / "csrc"
FILES = sorted(p for p in CSRC.glob("*.cu") if "pdl_wait()" in p.read_text())
# job vectors and plan tables: uploaded by copies before the frame's first kernel
CONSTANT = re.compile(r"a\.(tan_s|kr_grid|kc_grid|krp|kcp|tabq)\b|^(t4 \+ c|src \+ tid)|reinterpret_cast<const uint4 \*>\((a\.tabq|src)\)")


def _args(text, name):
    for m in re.finditer(name + r"\(", text):
        depth, i = 1, m.end()
        while depth:
            depth += {"(": 1, ")": -1}.get(text[i], 0)
            i += 1
        yield text[m.end():i - 1]


@pytest.mark.parametrize("path", FILES, ids=lambda p: p.name)
def test_written_memory_is_read_by_ordinary_loads(path):
    text = path.read_text()
    bad = [a for a in _args(text, "__ldg") if not CONSTANT.search(a)]
    assert not bad, bad
    for sig in re.findall(r"__global__[^{;]*\{", text):
        assert not re.search(r"const \w+ \*__restrict__", sig), sig


def test_the_check_sees_the_kernels():
    assert {p.name for p in FILES} >= {"pfa_display.cu", "pfa_fixed.cu", "pfa_fixed_runs.cu", "pfa_resample2.cu", "pfa_autofocus.cu"}
    assert not CONSTANT.search("a.y1 + (size_t)jr * N + k") and not CONSTANT.search("p1row + nat(l)")
