"""Reverse completion of lists with NaN distances: no edge lost, none doubled,
the serial introsort's order (kg_sort.h, compiled for the host)."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

HARNESS = r"""
#include "kg_sort.h"
#include <vector>
#include <utility>
struct Rec { float d; unsigned id; };
struct Acc {
  Rec *v; int n; int *out;
  bool in(int i) const { if (i < 0 || i >= n) { ++*out; return false; } return true; }
  float key(int i) const { return in(i) ? v[i].d : -__builtin_inff(); }   // outside: stops the scan
  void swap(int i, int j) { if (in(i) && in(j)) std::swap(v[i], v[j]); }
  Rec get(int i) const { return in(i) ? v[i] : Rec{0, 0xFFFFFFFFu}; }
  void put(int i, Rec r) { if (in(i)) v[i] = r; }
  float rkey(Rec r) const { return r.d; }
};
extern "C" int sort_ids(const float *d, int n, unsigned *ids) {
  std::vector<Rec> a(n);
  for (int i = 0; i < n; ++i) a[i] = Rec{d[i], (unsigned)i};
  int out = 0;
  Acc acc{a.data(), n, &out};
  kgb::gnu_sort(acc, 0, n);
  for (int i = 0; i < n; ++i) ids[i] = a[i].id;
  return out;
}
"""


def host_sort(path):
    (path / "h.cpp").write_text(HARNESS)
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-I",
                           os.path.join(ROOT, "kgraph_b200", "csrc"), str(path / "h.cpp"), "-o", str(path / "h.so")])
    lib = C.CDLL(str(path / "h.so"))
    lib.sort_ids.argtypes = [np.ctypeslib.ndpointer(np.float32, flags="C_CONTIGUOUS"), C.c_int,
                             np.ctypeslib.ndpointer(np.uint32, flags="C_CONTIGUOUS")]

    def order(d):
        d = np.ascontiguousarray(d, np.float32)
        ids = np.zeros(max(1, len(d)), np.uint32)
        return lib.sort_ids(d, len(d), ids), ids[:len(d)]
    return order


@pytest.mark.parametrize("seed,share", [(1, 0.002), (2, 0.1), (3, 0.6)])
def test_reverse_keeps_every_edge(gpu_ctx, tmp_path, seed, share):
    order = host_sort(tmp_path)
    rng = np.random.default_rng(seed)
    n, M = 900, 12
    ids = np.where(rng.random((n, M)) < 0.3, rng.integers(0, 12, (n, M)), rng.integers(0, n, (n, M))).astype(np.uint32)
    d = rng.integers(0, 50, (n, M)).astype(np.float32)
    d[rng.random((n, M)) < share] = np.nan
    gpu_ctx.set_data(rng.random((n, 4), dtype=np.float32), "l2sqr")
    gpu_ctx.set_graph(np.arange(0, n * M + 1, M), ids, d, np.full(n, M))
    gpu_ctx.reverse(-1)
    off, gi, gd, _ = gpu_ctx.graph()
    lists = [[] for _ in range(n)]   # the reference's push order (kgraph.cpp:667-702)
    for i in range(n):
        for t, x in zip(ids[i], d[i]):
            lists[i].append((int(t), x))
            lists[t].append((i, x))
    for i in range(n):
        out, at = order(np.array([x for _, x in lists[i]], np.float32))
        assert out == 0
        want = [lists[i][k] for k in at]
        want = [w for k, w in enumerate(want) if k == 0 or w[0] != want[k - 1][0]]
        a, b = int(off[i]), int(off[i + 1])
        assert [w[0] for w in want] == gi[a:b].tolist(), i
        assert np.array_equal(np.array([w[1] for w in want], np.float32).view(np.uint32), gd[a:b].view(np.uint32)), i
