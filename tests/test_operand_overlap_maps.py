"""The aliasing test of the sliced products for operands that pick buffers by
class maps of their own, as the batched tau2d sweeps do (pairs of buffers,
several principal layers as classes), and for operands of fewer rows than
their leading dimension (depth halves), against a brute-force intersection
(CPU)."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def overlap(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("ovm") / "libovm.so")
    subprocess.run(["g++", "-O2", "-shared", "-fPIC", "-I/usr/local/cuda/include", "-o", so,
                    os.path.join(ROOT, "tests", "harness", "overlap_maps_host.cpp")], check=True)
    L = ctypes.CDLL(so)
    ll, i, p = ctypes.c_longlong, ctypes.c_int, ctypes.c_void_p
    L.overlap_maps_eval.argtypes = [ll, p, ll, p, ll, ll, i, i, i, i]

    L.overlap_rows_eval.argtypes = [ll, i, ll, i, ll, ll, i, i, i, i]

    def go(offa, mapa, offb, mapb, sk, sc, ld, nk, n):
        a, b = (np.ascontiguousarray(m, np.int32) for m in (mapa, mapb))
        return L.overlap_maps_eval(offa, a.ctypes.data, offb, b.ctypes.data, sk, sc, ld, nk, len(a), n)
    go.rows = L.overlap_rows_eval
    return go


def _elems(off, mp, sk, sc, ld, nk, n):
    return {off + k * sk + c * sc + j * ld + r for k in range(nk) for c in mp for j in range(n) for r in range(n)}


@pytest.mark.parametrize("nprc,nc", [(1, 1), (2, 1), (3, 2), (4, 3), (5, 2), (7, 1)])
def test_pairs_of_buffers(overlap, nprc, nc):
    """Every pair of buffer pairs of the tau2d work layout: apart exactly when they share no buffer."""
    n, nbuf, nk = 3, 5 * nprc + 4, 2
    MB = n * n
    pairs = [(f, b) for f in range(0, nbuf, 2) for b in range(1, nbuf, 3)]
    rng = np.random.default_rng(nprc)
    for q in rng.integers(0, len(pairs), size=(300, 2)):
        (f1, b1), (f2, b2) = (pairs[i] for i in q)
        m1, m2 = ([s * nbuf + x for x in p for s in range(nc)] for p in ((f1, b1), (f2, b2)))
        assert overlap(0, m1, 0, m2, nc * nbuf * MB, MB, n, nk, n) == bool({f1, b1} & {f2, b2})


@pytest.mark.parametrize("nprc,nc", [(3, 1), (4, 2), (8, 2)])
def test_groups_of_layers(overlap, nprc, nc):
    """Several layers of one kind of buffer against those of another."""
    n, nbuf, nk = 3, 5 * nprc + 4, 3
    MB = n * n
    for p0 in range(0, nprc, 2):
        np_ = min(2, nprc - p0)
        many = lambda b0: [s * nbuf + b0 + q for q in range(np_) for s in range(nc)]  # noqa: E731
        for k1 in range(5):
            for k2 in range(5):
                got = overlap(0, many(k1 * nprc + p0), 0, many(k2 * nprc + p0), nc * nbuf * MB, MB, n, nk, n)
                assert got == (k1 == k2)


def test_never_apart_when_sharing(overlap):
    rng = np.random.default_rng(5)
    for _ in range(600):
        n = int(rng.integers(1, 4))
        ld = n + int(rng.integers(0, 3))
        nk, nc = int(rng.integers(1, 4)), int(rng.integers(1, 5))
        sc = n * ld * int(rng.integers(0, 3))
        sk = n * ld * int(rng.integers(0, 8))
        m1, m2 = (rng.integers(0, 6, size=nc).tolist() for _ in range(2))
        o1, o2 = (int(rng.integers(0, 30)) for _ in range(2))
        true = bool(_elems(o1, m1, sk, sc, ld, nk, n) & _elems(o2, m2, sk, sc, ld, nk, n))
        if true:
            assert overlap(o1, m1, o2, m2, sk, sc, ld, nk, n) == 1, (o1, m1, o2, m2, sk, sc, ld, nk, n)


def test_depth_halves_end_with_their_matrix(overlap):
    """The two halves of every buffer of an item against every whole buffer: apart from all but their own, the
    last buffer's second half from the next item's first buffer too."""
    n, nbuf, nc, nk = 4, 3, 2, 3
    MB = n * n
    for b1 in range(nbuf):
        for half in (0, n // 2):
            for b2 in range(nbuf):
                got = overlap.rows(b1 * MB + half, n // 2, b2 * MB, n, nc * nbuf * MB, nbuf * MB, n, nk, nc, n)
                assert got == (b1 == b2)


def test_row_ranges_are_never_apart_when_sharing(overlap):
    rng = np.random.default_rng(6)
    for _ in range(600):
        n = int(rng.integers(1, 5))
        ra, rb = (int(rng.integers(1, n + 1)) for _ in range(2))
        ld = n + int(rng.integers(0, 3))
        nk, nc = int(rng.integers(1, 4)), int(rng.integers(1, 4))
        sc, sk = int(rng.integers(0, 2 * n * ld)), int(rng.integers(0, 6 * n * ld))
        o1, o2 = (int(rng.integers(0, 40)) for _ in range(2))
        el = [{o + k * sk + c * sc + j * ld + q for k in range(nk) for c in range(nc) for j in range(n) for q in range(r)}
              for o, r in ((o1, ra), (o2, rb))]
        if el[0] & el[1]:
            assert overlap.rows(o1, ra, o2, rb, sk, sc, ld, nk, nc, n) == 1, (o1, ra, o2, rb, sk, sc, ld, nk, nc, n)
