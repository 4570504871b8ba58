"""Elimination plans on the CPU: the builder's plans, run pass by pass in Python,
solve their systems, with no slot written twice in a pass or read beside its write
(what the kernel's threads rely on); plans appended to one set are the plans of
their systems alone, and a pattern without a plan leaves the set as it was."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "cfdrs_b200", "csrc")
SHIM = """
#include <algorithm>
#include "ls_plan.h"
using namespace cfd;
static LsPlanSet S; static LsPlanWork W;
extern "C" int build(int n, const int* rp, const int* col, unsigned short* init, LsPlanHead* h) {
  return ls_plan_build(n, rp, col, W, S, init, *h);
}
extern "C" void clear() { S = LsPlanSet{}; }
extern "C" long words(unsigned short* out) {
  if (out) std::copy(S.words.begin(), S.words.end(), out);
  return (long)S.words.size();
}
extern "C" long rounds(int* out) {
  if (out) std::copy(&S.rounds[0].at_l, &S.rounds[0].at_l + 8 * S.rounds.size(), out);
  return (long)S.rounds.size();
}
"""


class Head(C.Structure):
    _fields_ = [(f, C.c_int32) for f in ("ok", "slots", "b0", "round0", "rounds", "core", "at_core", "entries",
                                         "at_entries", "pad")] + [("words", C.c_int64)]


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("ls_plan")
    (d / "shim.cpp").write_text(SHIM)
    so = str(d / "shim.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-I", CSRC, "-o", so, str(d / "shim.cpp"),
                    os.path.join(CSRC, "ls_plan.cpp")], check=True)
    L = C.CDLL(so)
    L.words.restype = L.rounds.restype = C.c_long
    return L


def build(lib, n, rp, col):
    h, init = Head(), np.zeros(len(col), np.uint16)
    ok = lib.build(n, rp.ctypes.data_as(C.c_void_p), col.ctypes.data_as(C.c_void_p),
                   init.ctypes.data_as(C.c_void_p), C.byref(h))
    assert bool(ok) == bool(h.ok)
    return h, init


def the_set(lib):
    w = np.zeros(max(1, lib.words(None)), np.uint16)
    lib.words(w.ctypes.data_as(C.c_void_p))
    r = np.zeros((max(1, lib.rounds(None)), 8), np.int32)
    if lib.rounds(None):
        lib.rounds(r.ctypes.data_as(C.c_void_p))
    return w, r


def solve(h, init, words, rounds, rp, val, b):
    """k_ls_sparse's passes, one thread after another."""
    n, w = len(b), words[h.words:].astype(np.int64)
    v = np.zeros(h.slots)
    np.add.at(v, init, val)
    v[h.b0:h.b0 + n] = b
    for at_l, nl, at_t, nt, pairs, at_x, nx, xpairs in rounds[h.round0:h.round0 + h.rounds]:
        div = w[at_l:at_l + 2 * nl].reshape(-1, 2)
        assert len(set(div[:, 0])) == nl and not set(div[:, 0]) & set(div[:, 1])
        v[div[:, 0]] /= v[div[:, 1]]
        written, read = set(), set()
        for t, first, count in w[at_t:at_t + 3 * nt].reshape(-1, 3):
            p = w[pairs + 2 * first:pairs + 2 * (first + count)].reshape(-1, 2)
            assert t not in written and count > 0
            written.add(t)
            read.update(p.ravel().tolist())
            for i, j in p:
                v[t] -= v[i] * v[j]
        assert not written & read
    core = w[h.at_core:h.at_core + h.core]
    M = np.zeros((h.core, h.core))
    for s, i, j in w[h.at_entries:h.at_entries + 3 * h.entries].reshape(-1, 3):
        M[i, j] += v[s]
    if h.core:
        v[h.b0 + core] = np.linalg.solve(M, v[h.b0 + core])
    for at_l, nl, at_t, nt, pairs, at_x, nx, xpairs in rounds[h.round0:h.round0 + h.rounds][::-1]:
        x = w[at_x:at_x + 4 * nx].reshape(-1, 4)
        own = set(x[:, 0])
        for s, d, first, count in x:
            p = w[xpairs + 2 * first:xpairs + 2 * (first + count)].reshape(-1, 2)
            assert not own & set(p[:, 1].tolist())
            v[s] = (v[s] - (v[p[:, 0]] * v[p[:, 1]]).sum()) / v[d]
    return v[h.b0:h.b0 + n]


def pattern(kind, n, rng):
    ent = {(i, i) for i in range(n)}

    def edge(i, j):
        if i != j:
            ent.update({(i, j), (j, i)})
    if kind in ("tree", "loops"):
        for i in range(1, n):
            edge(i, int(rng.integers(i)))
    if kind == "loops":
        for _ in range(n // 5):
            edge(*rng.integers(n, size=2).tolist())
    if kind == "chain":
        for i in range(1, n):
            edge(i, i - 1)
    if kind == "star":
        for i in range(1, n):
            edge(i, 0)
    if kind == "one_sided":
        for i in range(1, n):
            ent.add((i, int(rng.integers(i))))
    if kind == "pieces":
        for i in range(n):
            if i % 3:
                edge(i, i - 1)
    if kind == "dense":
        ent = {(i, j) for i in range(n) for j in range(n)}
    rows = [[] for _ in range(n)]
    for i, j in sorted(ent):
        rows[i].append(j)
    if kind == "loops":  # columns in any order, an entry stored twice
        rows = [rng.permutation(r + r[:1]).tolist() for r in rows]
    rp = np.concatenate([[0], np.cumsum([len(r) for r in rows])]).astype(np.int32)
    col = np.concatenate([np.array(r) for r in rows]).astype(np.int32)
    return rp, col


KINDS = [("tree", 1), ("tree", 2), ("tree", 37), ("tree", 400), ("loops", 20), ("loops", 300), ("loops", 900),
         ("chain", 257), ("star", 64), ("one_sided", 150), ("pieces", 100), ("diagonal", 50)]


@pytest.mark.parametrize("kind,n", KINDS)
def test_plans_solve(lib, kind, n):
    rng = np.random.default_rng(n)
    rp, col = pattern(kind, n, rng)
    row = np.repeat(np.arange(n), np.diff(rp))
    val = rng.uniform(-1.0, -0.1, len(col))
    D = np.zeros((n, n))
    np.add.at(D, (row, col), np.where(row == col, 0.0, val))
    dom = np.abs(D).sum(1) + np.abs(D).sum(0) + 1.0  # dominant in rows and columns
    copies = np.bincount(row[row == col], minlength=n)
    val = np.where(row == col, dom[row] / copies[row], val)
    D = np.zeros((n, n))
    np.add.at(D, (row, col), val)
    b = rng.uniform(-1, 1, n)
    lib.clear()
    h, init = build(lib, n, rp, col)
    assert h.ok
    x = solve(h, init, *the_set(lib), rp, val, b)
    # diagonally dominant: growth at most 2, kappa at most the ratio of the row sums
    kappa = np.abs(D).sum(1).max() / 1.0
    assert np.abs(x - np.linalg.solve(D, b)).max() <= 64 * n * np.finfo(float).eps * kappa * np.abs(x).max()


def test_one_set(lib):
    rng = np.random.default_rng(1)
    pats = [pattern(k, n, rng) for k, n in KINDS]
    alone = []
    for rp, col in pats:
        lib.clear()
        h, init = build(lib, len(rp) - 1, rp, col)
        alone.append((h, init, *the_set(lib)))
    lib.clear()
    heads = []
    for k, (rp, col) in enumerate(pats):
        heads.append(build(lib, len(rp) - 1, rp, col))
        if k == 4:
            before = lib.words(None), lib.rounds(None)
            assert not build(lib, 60, *pattern("dense", 60, rng))[0].ok
            assert (lib.words(None), lib.rounds(None)) == before
    words, rounds = the_set(lib)
    for (h, init), (a, ainit, aw, ar) in zip(heads, alone):
        np.testing.assert_array_equal(init, ainit)
        np.testing.assert_array_equal(words[h.words:h.words + len(aw)], aw)
        np.testing.assert_array_equal(rounds[h.round0:h.round0 + h.rounds], ar)
        assert [getattr(h, f) for f in ("slots", "b0", "core", "at_core", "entries", "at_entries")] == \
            [getattr(a, f) for f in ("slots", "b0", "core", "at_core", "entries", "at_entries")]


def test_a_hub_costs_no_more_than_a_tree(lib):
    """A node with all others for neighbours: the builder must not search its list for
    every one of them (a manifold of 2000 pipes took 12 times a random tree's time)."""
    import time
    rng = np.random.default_rng(3)
    best = {}
    for kind in ("star", "tree"):
        rp, col = pattern(kind, 2000, rng)
        times = []
        for _ in range(7):
            lib.clear()
            t = time.perf_counter()
            build(lib, 2000, rp, col)
            times.append(time.perf_counter() - t)
        best[kind] = min(times)
    assert best["star"] <= 4 * best["tree"]
