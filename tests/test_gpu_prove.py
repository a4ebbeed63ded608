"""The publication proofs of device builds accept what the host's accept and reject
what they reject: trees as built, a table of single-word corruptions (one for each
check), and flips of random bits.  The proofs read words; nothing is traced."""
import numpy as np
import pytest

from vitrum_b200 import _native as N
from vitrum_b200 import bvh as vb
from vitrum_b200 import scenes

pytestmark = pytest.mark.gpu

BUILD = 6
LEAF = 0xFFFF0000


def _ptr(a):
    return None if a is None else a.ctypes.data


def _accepts(on_device, binary=None, wide=None, recs=None, triangles=0, stack=64):
    try:
        N.call("vt_debug_prove_bvh", on_device, _ptr(binary), 0 if binary is None else len(binary), _ptr(wide),
               0 if wide is None else len(wide), _ptr(recs), 0 if recs is None else len(recs), triangles, stack)
        return True
    except N.VtError as e:
        assert e.status == BUILD, e
        return False


def _both(**kw):
    host, device = _accepts(0, **kw), _accepts(1, **kw)
    assert host == device, (host, device)
    return host


@pytest.fixture(scope="module")
def tree():
    m = scenes.random_triangles(700, seed=11)
    with vb.build_compressed_wide_bvh(m.positions, m.indices) as g:
        binary, _ = g.export_binary()
        words, recs = g.export_wide()
    return binary, words.reshape(-1, 20), recs.reshape(-1, 16)


def _interior(b, k):
    return int(np.flatnonzero(b[:, 7] < 3)[k])


def _leaf(b, k, least=1):
    return int(np.flatnonzero((b[:, 7] >= LEAF) & ((b[:, 7] & 0xFFFF) >= least))[k])


def _f(b, i, j):
    return b.view(np.float32)[i, j]


BINARY = {
    "lower bound not finite": lambda b: b.view(np.float32).__setitem__((_leaf(b, 3), 0), np.nan),
    "upper bound not finite": lambda b: b.view(np.float32).__setitem__((0, 5), np.inf),
    "bounds inverted": lambda b: b.view(np.float32).__setitem__((_leaf(b, 0), 1), _f(b, _leaf(b, 0), 4) + 1),
    "child outside its parent": lambda b: b.view(np.float32).__setitem__(
        (_interior(b, 4), 3), np.nextafter(_f(b, _interior(b, 4), 3), np.float32(-np.inf))),
    "split axis": lambda b: b.__setitem__((_interior(b, 2), 7), 3),
    "right child offset 0": lambda b: b.__setitem__((_interior(b, 2), 6), 0),
    "right child is the left one": lambda b: b.__setitem__((_interior(b, 2), 6), 1),
    "right child outside": lambda b: b.__setitem__((_interior(b, 2), 6), len(b)),
    "right child far outside": lambda b: b.__setitem__((_interior(b, 2), 6), 0xFFFFFFFF),
    "shared child": lambda b: b.__setitem__((_interior(b, 1), 6), b[_interior(b, 1), 6] - 1),
    "unreachable nodes": lambda b: b.__setitem__((_interior(b, 5), 7), LEAF),
    "leaf range overlaps": lambda b: b.__setitem__((_leaf(b, 2), 7), b[_leaf(b, 2), 7] + 1),
    "leaf range leaves a gap": lambda b: b.__setitem__((_leaf(b, 2, 2), 7), b[_leaf(b, 2, 2), 7] - 1),
    "leaf starts elsewhere": lambda b: b.__setitem__((_leaf(b, 5), 6), b[_leaf(b, 5), 6] + 1),
    "leaf range outside": lambda b: b.__setitem__((_leaf(b, 5), 6), 0xFFFFFFF0),
}


@pytest.mark.parametrize("what", BINARY)
def test_corrupt_binary_trees_are_rejected(cuda, tree, what):
    binary = tree[0].copy()
    assert _both(binary=binary, triangles=700)
    BINARY[what](binary)
    assert not _both(binary=binary, triangles=700)


def test_binary_triangle_count_and_stack(cuda, tree):
    binary = tree[0]
    assert not _both(binary=binary, triangles=699)
    assert not _both(binary=binary, triangles=701)
    verdicts = [_both(binary=binary, triangles=700, stack=s) for s in range(1, 40)]
    assert not verdicts[0] and verdicts[-1] and verdicts == sorted(verdicts)


def _bytes(w):
    return w.view(np.uint8).reshape(len(w), 80)


def _slot(w, kind, k=0):
    """(node, slot) of the k-th internal, leaf or empty slot below the root."""
    b = _bytes(w)
    inner = (b[:, 15, None] >> np.arange(8)) & 1
    nib = (w[:, 6, None] >> (4 * np.arange(8))) & 15
    pick = {"internal": inner == 1, "leaf": (inner == 0) & (nib > 0), "empty": (inner == 0) & (nib == 0)}[kind]
    n, s = np.nonzero(pick)
    keep = n > 0
    return int(n[keep][k]), int(s[keep][k])


def _box(kind, low, step, k=0):
    def f(w, r):
        n, s = _slot(w, kind, k)
        at = n, (32 if low else 56) + s
        _bytes(w)[at] = (int(_bytes(w)[at]) + step) & 255
    return f


def _nibble(value):
    def f(w, r):
        n, s = _slot(w, "leaf")
        w[n, 6] = (int(w[n, 6]) & ~(0xF << 4 * s)) | value << 4 * s
    return f


def _node(kind, word, change):
    def f(w, r):
        n, _ = _slot(w, kind)
        w[n, word] = change(int(w[n, word])) & 0xFFFFFFFF
    return f


def _record(word, value):
    def f(w, r):
        n, s = _slot(w, "leaf")
        r.view(np.uint32)[int(w[n, 5]) + 4 * s, word] = value(r.view(np.uint32))
    return f



WIDE = {
    "child base shifted": _node("internal", 4, lambda x: x + 1),
    "child base outside": _node("internal", 4, lambda x: 0xFFFFFFF0),
    "child base at the root (a cycle)": _node("internal", 4, lambda x: 0),
    "internal slot owns records": lambda w, r: w.__setitem__(
        (_slot(w, "internal")[0], 6), int(w[_slot(w, "internal")[0], 6]) | 1 << 4 * _slot(w, "internal")[1]),
    "internal slot gone": _node("internal", 3, lambda x: x & 0x00FFFFFF),
    "record mask not contiguous": _nibble(0b101),
    "records dropped": _nibble(0),
    "a record too many": _nibble(0b1111),
    "record base shifted": _node("leaf", 5, lambda x: x + 1),
    "record base outside": _node("leaf", 5, lambda x: 0x3FFFFFFF),
    "record names no triangle": _record(3, lambda u: 700),
    "record names a triangle twice": lambda w, r: r.view(np.uint32).__setitem__(
        (int(w[_slot(w, "leaf", 1)[0], 5]) + 4 * _slot(w, "leaf", 1)[1], 3),
        r.view(np.uint32)[int(w[_slot(w, "leaf")[0], 5]) + 4 * _slot(w, "leaf")[1], 3]),
    "vertex outside its box": _record(0, lambda u: np.float32(1e6).view(np.uint32)),
    "vertex NaN": _record(4, lambda u: np.float32(np.nan).view(np.uint32)),
    "leaf box a step too small below": _box("leaf", True, 1),
    "leaf box a step too small above": _box("leaf", False, -1),
    "ancestor box a step too small below": _box("internal", True, 1),
    "ancestor box a step too small above": _box("internal", False, -1),
    "empty slot with a box": _box("empty", True, -1),
    "grid origin NaN": _node("leaf", 0, lambda x: 0x7FC00000),
    "grid origin infinite": _node("leaf", 1, lambda x: 0xFF800000),
    "grid exponent a step too small": _node("leaf", 3, lambda x: x - 1),
}


@pytest.mark.parametrize("what", WIDE)
def test_corrupt_wide_trees_are_rejected(cuda, tree, what):
    wide, recs = tree[1].copy(), tree[2].copy()
    assert _both(wide=wide, recs=recs, triangles=700)
    WIDE[what](wide, recs)
    assert (wide != tree[1]).any() or (recs.view(np.uint32) != tree[2].view(np.uint32)).any()
    assert not _both(wide=wide, recs=recs, triangles=700)


def test_wide_triangle_count_and_stack(cuda, tree):
    _, wide, recs = tree
    assert not _both(wide=wide, recs=recs, triangles=699)
    assert not _both(wide=wide, recs=recs, triangles=701)
    last = int(np.flatnonzero(recs[:, 15] != 0).max())     # the last valid record (padding may follow it)
    assert _both(wide=wide, recs=recs[:last + 1], triangles=700)
    assert not _both(wide=wide, recs=recs[:last], triangles=700)
    verdicts = [_both(wide=wide, recs=recs, triangles=700, stack=s) for s in range(1, 40)]
    assert not verdicts[0] and verdicts[-1] and verdicts == sorted(verdicts)


@pytest.mark.parametrize("which", ["binary", "wide", "records"])
def test_random_bit_flips_get_the_same_verdict(cuda, tree, which):
    rng = np.random.default_rng(5)
    accepted = 0
    for _ in range(400):
        b, w, r = (a.copy() for a in tree)
        a = {"binary": b, "wide": w, "records": r.view(np.uint32)}[which].reshape(-1)
        a[rng.integers(len(a))] ^= np.uint32(1 << int(rng.integers(32)))
        if which == "binary":
            accepted += _both(binary=b, triangles=700)
        else:
            accepted += _both(wide=w, recs=r, triangles=700)
    assert 0 < accepted < 400
