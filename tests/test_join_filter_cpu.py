"""The tensor-core join's filter (kgraph_b200/csrc/kg_join_filter.h), compiled for the host.

The join skips a pair when its lower bound, formed from per-row terms and the
Gram entry of the rounded rows, lies above both endpoints' radii.  Here the
same lines are fed Gram entries of BF16 and of scaled E4M3 rows (with as much
accumulation error as the margin allows for) and compared with the oracle's
canonical FP32 distance and with FP64: the bound lies below both, no pair that
a pool would take is skipped, and pairs well outside are.  The audit that the
join runs on a sample of nodes must flag each kind of mistake.
"""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT
from oracle import kgoracle as ko
from test_filter_bound_cpu import bf16, e4m3

HARNESS = r"""
#include "kg_join_filter.h"
using namespace kgb;
extern "C" {
void row(int m, float h, float c, float nrm, float qn, float gam, float rad, float *out) {
  const FilterRow r = filter_row((FilterMetric)m, h, c, nrm, qn, gam, rad);
  out[0] = r.A; out[1] = r.s; out[2] = r.rad; out[3] = r.C; out[4] = r.nrm;
}
void pair(int m, float g, float t2, float gam, const float *u, const float *j, float *out) {
  const FilterTest t = filter_pair((FilterMetric)m, g, t2, gam, u[0], j[0], u[2], j[2], u[3], j[3], u[4], j[4]);
  out[0] = t.lhs; out[1] = t.rhs;
}
float et8(float fu, float fj, float g8) { return filter_et8(fu, fj, g8); }
int wrong(int m, float lhs, int skip, float rad, float nu, float nj, double d64, float dc) {
  return filter_wrong((FilterMetric)m, lhs, skip != 0, rad, nu, nj, d64, dc);
}
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("filter")
    (d / "h.cpp").write_text(HARNESS)
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-shared", "-fPIC", "-I",
                           os.path.join(ROOT, "kgraph_b200", "csrc"), str(d / "h.cpp"), "-o", str(d / "h.so")])
    L = C.CDLL(str(d / "h.so"))
    f, i, fp = C.c_float, C.c_int, C.POINTER(C.c_float)
    L.row.argtypes = [i, f, f, f, f, f, f, fp]
    L.pair.argtypes = [i, f, f, f, fp, fp, fp]
    L.et8.argtypes, L.et8.restype = [f, f, f], f
    L.wrong.argtypes = [i, f, i, f, f, f, C.c_double, f]
    return L


def rows(kind, n, d, rng):
    if kind == "near":       # a node's neighbourhood
        return (rng.standard_normal(d) * 3 + rng.standard_normal((n, d))).astype(np.float32)
    if kind == "offset":     # far from the origin: the canonical distance cancels
        return (rng.standard_normal((n, d)) + 300).astype(np.float32)
    if kind == "integers":
        return rng.integers(0, 200, (n, d)).astype(np.float32)
    if kind == "tiny":       # products of differences underflow
        return (rng.standard_normal((n, d)) * 1e-22).astype(np.float32)
    x = (rng.standard_normal(d) + 0.3 * rng.standard_normal((n, d))).astype(np.float32)
    return (x / np.linalg.norm(x, axis=1, keepdims=True)).astype(np.float32)


def exact(X, metric):
    x = X.astype(np.float64)
    if metric == "angular":
        n = np.sqrt((x * x).sum(1))
        return -(x @ x.T) / (n[:, None] * n[None] + np.finfo(np.float32).eps)
    d2 = ((x[:, None] - x[None]) ** 2).sum(-1)
    return d2 if metric == "l2sqr" else 0.5 * d2


@pytest.mark.parametrize("prec", ["bf16", "fp8"])
@pytest.mark.parametrize("metric", ["euclidean", "angular", "l2sqr"])
@pytest.mark.parametrize("kind,d", [("near", 20), ("near", 64), ("near", 128), ("near", 300), ("offset", 96),
                                    ("integers", 128), ("sphere", 96), ("tiny", 64)])
def test_bound_and_skip(lib, prec, metric, kind, d):
    rng = np.random.default_rng(d + 7 * len(kind))
    n = 40
    X = rows(kind, n, d, rng)
    X[5] = X[6]              # equal rows
    X[7] = X[0]              # the node itself
    o, m, d64 = ko.Oracle(X, metric), ko.METRICS[metric], exact(X, metric)
    f = np.float32
    gam = f(d + 4) * f(5.9605e-8)
    et = f(0.00390625) + f(7.63e-6) + f(d + 4) * f(1.1921e-7)
    g8 = f(d + 4) * f(9.5367e-7) + f(8) * f(5.9605e-8)
    v = X - X[0]
    hs, c, qn = (v * v).sum(1, dtype=f), (v * X[0]).sum(1, dtype=f), f((X[0] * X[0]).sum(dtype=f))
    if prec == "bf16":
        q, scale, rel = bf16(v).astype(np.float64), np.ones(n, f), np.zeros(n, f)
    else:
        mx = np.abs(v).max(1)
        scale = np.where(mx > 0, mx / f(448), f(1)).astype(f)
        scale[scale == 0] = np.finfo(f).smallest_subnormal
        q = np.stack([e4m3(v[k].astype(np.float64) / scale[k]) for k in range(n)])
        err = np.sqrt((((v.astype(np.float64) - q * scale[:, None].astype(np.float64))) ** 2).sum(1))
        rel = np.where(hs > 0, err / np.sqrt(np.maximum(hs.astype(np.float64), 1e-300)) * (1 + 1e-5), 0).astype(f)
    buf = lambda: (C.c_float * 5)()

    def term(u, rad):
        r = buf()
        lib.row(m, f(0.5) * hs[u], c[u], o.norms[u], qn, gam, rad, r)
        return r

    big, outside = np.finfo(f).max, 0
    for u in range(n):
        for j in range(u + 1, n):
            dc = f(o.pair(u, j))
            gram = f((q[u] * q[j]).sum())
            gram += f(rng.choice([-1, 1]) * np.abs(q[u] * q[j]).sum() * d * 2.0 ** -24)
            if prec == "fp8":
                gram = f(f(gram * scale[u]) * scale[j])
            t0 = term(u, 0.0)
            e = et if prec == "bf16" else f(lib.et8(f(1) + rel[u], f(1) + rel[j], g8))
            for radu, radj in [(dc, -big), (-big, dc), (dc, dc), (big, big), (-big, -big)]:
                ru, rj = term(u, radu), term(j, radj)
                t2 = f(f(f(2) * e) * f(ru[1])) * f(rj[1])
                out = (C.c_float * 2)()
                lib.pair(m, gram, t2, gam, ru, rj, out)
                skip = out[0] > out[1]
                if max(radu, radj) >= dc:
                    assert not skip, (u, j, radu, radj, dc, out[0], out[1])
                assert not lib.wrong(m, out[0], skip, max(ru[2], rj[2]), ru[4], rj[4], d64[u, j], dc), (u, j)
            # well outside: skipped
            ss = float(t0[1]) * float(rj[1])
            unit = float(o.norms[u]) * float(o.norms[j]) if metric == "angular" else 1.0
            slack = (0.05 if prec == "bf16" else 0.4) * (2 if metric == "l2sqr" else 1) * ss / unit if unit else 0
            if kind not in ("offset", "tiny") and ss > 0:
                rad = f(float(dc) - slack)
                ru, rj = term(u, rad), term(j, rad)
                lib.pair(m, gram, t2, gam, ru, rj, out)
                assert out[0] > out[1], (u, j, dc, rad, out[0], out[1])
                outside += 1
    assert outside > 600 or kind in ("offset", "tiny")


@pytest.mark.parametrize("metric", ["euclidean", "angular", "l2sqr"])
def test_audit_flags_a_wrong_bound_and_a_wrong_skip(lib, metric):
    m = ko.METRICS[metric]
    rng = np.random.default_rng(m)
    for _ in range(200):
        nu, nj = rng.uniform(0.5, 3, 2).astype(np.float32)
        dist = float(rng.uniform(0.1, 2)) * (-1 if metric == "angular" else 1)
        dc = np.float32(dist)
        unit = {"euclidean": 1.0, "l2sqr": 0.5, "angular": float(nu) * float(nj)}[metric]
        half = 0.5 if metric == "l2sqr" else 1.0   # the test holds l2sqr radii halved
        below, above = np.float32(dist - 0.01), np.float32(dist + 0.01)
        good, bad = np.float32((dist - 0.02) * unit), np.float32((dist + 0.02) * unit)
        assert not lib.wrong(m, good, 0, above * half, nu, nj, dist, dc)
        assert not lib.wrong(m, good, 1, below * half, nu, nj, dist, dc)
        assert lib.wrong(m, bad, 0, above * half, nu, nj, dist, dc)       # a bound above the distance
        assert lib.wrong(m, good, 1, above * half, nu, nj, dist, dc)      # skipped inside the radius
        assert lib.wrong(m, good, 1, dc * np.float32(half), nu, nj, dist, dc)   # at the radius a pool still takes it
        assert not lib.wrong(m, np.float32(np.nan), 0, below * half, nu, nj, dist, dc)
