"""CPU: the host-side decisions of csrc/host_rules.h, compiled with g++ behind a small C shim: how a plan's buffers share device
allocations, checked for overlap, alignment and the limit of each allocation; and which jobs the passes in runs take, for the
scenes on which the GPU tests rely to reach one kernel or the other and for vectors that no pass in runs may get."""
import ctypes as C
import random
import subprocess
from pathlib import Path

import numpy as np
import pytest

from pfa_b200 import geometry, synth

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
extern "C" int float_p1(int m, int n, const double *f0, const double *df, const double *fl, const double *pr, const double *kr) {
    return pfa::float_pass1_rule(m, n, f0, df, fl, pr, kr).runs;
}
extern "C" int fixed_p1(int m, int n, const float *f0, const float *df, const float *fac, const float *kr) {
    return pfa::fixed_pass1_rule(m, n, f0, df, fac, kr).runs;
}
extern "C" int float_p2(int m, int n, const double *tn, const double *kc, const double *kr) {
    return pfa::pass2_rule(m, n, tn, kc, kr, 1).runs;
}
extern "C" int fixed_p2(int m, int n, const float *tn, const float *kc, const float *kr) {
    return pfa::pass2_rule(m, n, tn, kc, kr, 8).runs;
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


# ------------------------------------------------------------------------------------------ routes
def _p(a):
    return C.c_void_p(a.ctypes.data)


def _float(lib, job):
    j = {k: np.ascontiguousarray(job[k], np.float64) for k in ("f0", "df", "f_last", "pr", "KR", "KC", "tan_s")}
    m, n = job["m"], job["n"]
    return (bool(lib.float_p1(m, n, *(_p(j[k]) for k in ("f0", "df", "f_last", "pr", "KR")))),
            bool(lib.float_p2(m, n, *(_p(j[k]) for k in ("tan_s", "KC", "KR")))))


def _fixed(lib, job):
    fac = (np.float32(2.0) * job["pr"]) / np.float32(299792458.0)
    m, n = job["m"], job["n"]
    return (bool(lib.fixed_p1(m, n, _p(job["f0"]), _p(job["df"]), _p(fac), _p(job["krp"]))),
            bool(lib.fixed_p2(m, n, _p(job["tan_s"]), _p(job["kcp"]), _p(job["krp"]))))


def _tables(m, n, jitter=0.0, bw=600e6, aperture_deg=3.0, seed=1, descending=False):
    t = dict(geometry.prepare_tables_from_scene(synth.make_scene(m, n, n_targets=2, seed=seed, jitter=jitter, bw=bw,
                                                                 aperture_deg=aperture_deg)))
    if descending:
        t["freq"] = -t["freq"]
        t["KR"] = -t["KR"][::-1]
    return t


@pytest.mark.parametrize("m,n,kw,runs,split", [
    (300, 260, dict(jitter=0.0), True, True), (290, 150, dict(jitter=0.1), True, True), (2050, 70, dict(jitter=0.3), True, True),
    (900, 1000, dict(jitter=0.1), True, True), (257, 1000, dict(jitter=0.2, bw=113.6e6), True, True),
    (256, 240, dict(jitter=0.3), True, False),               # few pulses: the fused pass 2
    (300, 260, dict(jitter=2.0), True, False), (4099, 300, dict(jitter=2.0, seed=4099), True, False),
    (1030, 200, dict(jitter=2.0, seed=1230), True, False), (2100, 333, dict(jitter=2.0, seed=2433), True, False),
    (1030, 200, dict(jitter=0.3, descending=True), False, False), (290, 150, dict(jitter=0.4, descending=True), False, False),
    (257, 1000, dict(bw=113.6e6, aperture_deg=10.0), False, True)])
def test_routes_of_scenes(lib, m, n, kw, runs, split):
    t = _tables(m, n, **kw)
    assert _float(lib, geometry.float_job(t)) == (runs, split)
    assert _fixed(lib, geometry.fixed_job(t, geometry.pow2(max(m, n))))[1] == split


def test_vectors_that_no_pass_in_runs_may_get(lib):
    t = _tables(300, 260, jitter=0.1)
    fl, fx = geometry.float_job(t), geometry.fixed_job(t, 512)
    assert _float(lib, fl) == (True, True) and _fixed(lib, fx) == (True, True)
    for bad in (np.nan, np.inf, -np.inf):
        for at in (0, 100, -1):
            for key, which in (("KR", (0, 1)), ("KC", (1,)), ("tan_s", (1,)), ("pr", (0,)), ("df", (0,)), ("f0", (0,)), ("f_last", (0,))):
                j = dict(fl, **{key: fl[key].copy()})
                j[key][at] = bad
                assert not any(_float(lib, j)[w] for w in which), (key, bad, at)
        for at in (0, 100):
            for key, which in (("krp", (0, 1)), ("kcp", (1,)), ("tan_s", (1,)), ("pr", (0,)), ("df", (0,)), ("f0", (0,))):
                j = dict(fx, **{key: fx[key].copy()})
                j[key][at] = bad
                assert not any(_fixed(lib, j)[w] for w in which), (key, bad, at)
    # an end sample that is not where the affine axis has it
    j = dict(fl, f_last=fl["f_last"].copy())
    j["f_last"][7] -= 20 * fl["df"][7]
    assert _float(lib, j) == (False, True)
    # queries that turn back, and sources that do
    for key in ("KC", "tan_s", "KR"):
        j = dict(fl, **{key: fl[key].copy()})
        j[key][50], j[key][51] = j[key][51], j[key][50]
        assert not _float(lib, j)[0 if key == "KR" else 1]
