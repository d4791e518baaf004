"""CPU: the host-side decisions of csrc/host_rules.h, compiled with g++ behind a small C shim: how a plan's buffers share device
allocations, checked for overlap, alignment and the limit of each allocation."""
import ctypes as C
import random
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "mpfs250t-sar-ifp_b200" / "csrc"
MIB = 1 << 20
SHIM = r"""
#include "host_rules.h"
extern "C" int pack(const size_t *bytes, int n, size_t head, size_t *block, int *in, size_t *offset) {
    const pfa::Packing p = pfa::pack_buffers(std::vector<size_t>(bytes, bytes + n), head);
    std::copy(p.block.begin(), p.block.end(), block);
    std::copy(p.in.begin(), p.in.end(), in);
    std::copy(p.offset.begin(), p.offset.end(), offset);
    return (int)p.block.size();
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("host_rules")
    (d / "shim.cpp").write_text(SHIM)
    subprocess.run(["g++", "-std=c++17", "-O2", "-shared", "-fPIC", f"-I{CSRC}", "-o", str(d / "shim.so"), str(d / "shim.cpp")],
                   check=True)
    return C.CDLL(str(d / "shim.so"))


def _pack(lib, sizes, head):
    n = len(sizes)
    arr = (C.c_size_t * n)(*sizes)
    block, inn, off = (C.c_size_t * n)(), (C.c_int * n)(), (C.c_size_t * n)()
    k = lib.pack(arr, n, C.c_size_t(head), block, inn, off)
    return list(block[:k]), list(inn), list(off)


def _check(sizes, head, block, inn, off):
    used = [0] * len(block)
    for s, b, o in zip(sizes, inn, off):                     # in order, gapless, so disjoint and as aligned as the sizes
        assert o == used[b]
        used[b] += s
    assert used == block and len(block) <= 12
    at = 0
    for s, b, o in zip(sizes[:head], inn[:head], off[:head]):    # the head in a row at the start of the first allocation
        assert (b, o) == (0, at)
        at += s
    for k, total in enumerate(block):                        # a small allocation, or one buffer by itself
        assert len(block) == 1 or total <= MIB or (total <= 5 * MIB // 4 and (inn.count(k) == 1 or inn[:head].count(k) == inn.count(k)))


def test_packing(lib):
    rng = random.Random(1)
    for _ in range(3000):
        head = rng.randint(0, 6)
        sizes = [256 * rng.randint(1, rng.choice([8, 400, 4096, 9000])) for _ in range(head + rng.randint(1, 9))]
        block, inn, off = _pack(lib, sizes, head)
        _check(sizes, head, block, inn, off)
        if max(sizes[head:]) > 5 * MIB // 4 or sum(sizes[:head]) > 5 * MIB // 4:
            assert block == [sum(sizes)]
        elif sum(sizes) <= MIB:
            assert block == [sum(sizes)]


def test_small_plans_stay_within_the_mapped_sizes(lib):
    # buffers of a 256 x 256 float plan: three allocations of at most 1 MiB instead of one of 1.1; a large plan takes one
    k = 1024
    block, *_ = _pack(lib, [2 * k] * 10 + [30 * k, 512 * k, 514 * k], 10)
    assert len(block) == 2 and max(block) <= MIB
    block, *_ = _pack(lib, [8 * k] * 10 + [30 * k, 8 * MIB, 8 * MIB], 10)
    assert len(block) == 1
