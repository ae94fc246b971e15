"""Nested-dissection fronts of the bordered Newton Jacobian: the symbolic phase
of the tree elimination in ``frontal.py``.

The elements are bisected recursively by their centroids, at every level where
a cut along x, y or a diagonal leaves the fewest nodes on it, into a complete
binary tree of element sets (heap numbering: root 1, children 2t and 2t + 1).  A node is
eliminated with the smallest set that holds all of its elements; the *front* of
a set is made of the unknowns eliminated with it (its pivots) and those of its
elements' nodes that are eliminated further up.  Fronts of one depth are
independent of each other, so a whole depth is factorised at once, and the
serial chain is the pivots along one path to the root instead of every unknown.
"""
from __future__ import annotations

import math

import numpy as np

# elements per leaf on average: 2, 4, 8 cost 62.0, 63.0, 66.9 G multiply-adds at
# 20,000 quads (median cuts); a leaf of 4 halves the fronts of 2 and stores 5% less
LEAF = 4


# A cut may lie this far from the middle (of the elements), and larger sets than
# MEDIAN also try the diagonals.  Multiply-adds of the elimination, 20,000 quads:
# medians along x or y 63.0 G, and +-20% 54.1 G, and diagonals 49.2 G (2,000
# quads: 2.3, 2.1, 1.8 G); +-30% 49.5 G.  Sets of up to MEDIAN elements take the
# median along x or y: they are most of the sets and hardly any of the work.
SLACK = 0.2
MEDIAN = 24


def _split(c: np.ndarray, sel: np.ndarray, en: np.ndarray, first: np.ndarray, last: np.ndarray):
    """(score, lower, upper) of the best cut of the elements ``sel`` in the order
    of ``c``: nodes on the cut, times 1 + its distance from the middle."""
    n = len(sel)
    order = sel[np.argsort(c[sel], kind="stable")]
    v = en[order].reshape(-1)
    pos = np.repeat(np.arange(n), en.shape[1])
    first[v[::-1]] = pos[::-1]
    last[v] = pos
    own = first[v] == pos                               # every node once
    cut = np.cumsum(np.bincount(pos[own] + 1, minlength=n + 2) - np.bincount(last[v[own]] + 1, minlength=n + 2))
    slack = SLACK if n > MEDIAN else 0.0
    k = np.arange(max(1, int(n * (0.5 - slack))), max(int(n * (0.5 + slack)), n // 2) + 1)
    score = cut[k] * (1.0 + np.abs(k / n - 0.5))
    j = int(np.argmin(score)) if slack else 0
    k = int(k[j]) if slack else n // 2
    return cut[k] * (1.0 + abs(k / n - 0.5)), order[:k], order[k:]


def bisect(en: np.ndarray, cen: np.ndarray, leaf: int):
    """Heap id of every element's leaf set, and the depth of the tree."""
    nel = en.shape[0]
    depth = max(0, math.ceil(math.log2(max(1.0, nel / leaf))))
    ids = np.ones(nel, dtype=np.int64)
    first = np.empty(int(en.max()) + 1, dtype=np.int64)
    last = np.empty_like(first)
    axes = [cen[0], cen[1], cen[0] + cen[1], cen[0] - cen[1]]
    stack = [(np.arange(nel), 1, 0)]
    while stack:
        sel, node, d = stack.pop()
        if d == depth or len(sel) < 2:
            # a set too small to cut goes down the lower side
            ids[sel] = node << (depth - d)
            continue
        best = min((_split(c, sel, en, first, last) for c in axes[:2 if len(sel) <= MEDIAN else 4]),
                   key=lambda s: s[0])
        stack.append((best[1], 2 * node, d + 1))
        stack.append((best[2], 2 * node + 1, d + 1))
    return ids, depth


def _common(lo: np.ndarray, hi: np.ndarray) -> np.ndarray:
    """Lowest common ancestor of the leaves lo..hi (heap ids of one depth)."""
    x, up = lo ^ hi, np.zeros_like(lo)
    while (x > 0).any():
        up += x > 0
        x = x >> 1
    return lo >> up


class Tree:
    """Fronts of a mesh, deepest level first; per front t of ``nfront``:
    ``heap[t]``, ``p[t]`` pivots and ``n[t]`` unknowns in all, which are
    ``ids[idx_off[t]:idx_off[t + 1]]``, the pivots first and both parts by
    unknown id; ``levels``: (first, end) fronts of each depth, deepest first.
    ``owner``: heap id of the front every unknown is eliminated with."""

    def __init__(self, en, xy, nn, neq, nborder, leaf=LEAF, delay_field=None):
        nel, nbf = en.shape
        N = nn * neq + nborder
        leafid, depth = bisect(en, xy, leaf)
        ev, el = en.reshape(-1), np.repeat(leafid, nbf)
        lo, hi = np.full(nn, np.iinfo(np.int64).max), np.full(nn, -1, dtype=np.int64)
        np.minimum.at(lo, ev, el)
        np.maximum.at(hi, ev, el)
        if (hi < 0).any():
            raise ValueError("a node belongs to no element")
        own_node = _common(lo, hi)
        owner = np.repeat(own_node, neq).reshape(nn, neq)
        if delay_field is not None:
            # this field goes with the set that holds every element touching
            # any node of its node's elements
            elo, ehi = lo[en].min(axis=1), hi[en].max(axis=1)
            lo2, hi2 = lo.copy(), hi.copy()
            np.minimum.at(lo2, ev, np.repeat(elo, nbf))
            np.maximum.at(hi2, ev, np.repeat(ehi, nbf))
            owner[:, delay_field] = _common(lo2, hi2)
        owner = np.concatenate([owner.reshape(-1), np.ones(nborder, dtype=np.int64)])
        # (set, unknown) pairs of one depth from those of the depth below; a
        # node's unknowns travel together unless one field is delayed
        per = 1 if delay_field is not None else neq
        nent = nn * (neq // per)
        ent_owner = owner[:nn * neq:per]
        if per == 1:
            pairs = (el[:, None] * nent + ev[:, None] * neq + np.arange(neq)).reshape(-1)
        else:
            pairs = el * nent + ev
        border = np.arange(nn * neq, N, dtype=np.int64)
        heap, p_sz, n_sz, ids, self.levels = [], [], [], [], []
        for d in range(depth, -1, -1):
            pairs = np.unique(pairs)
            s, u = pairs // nent, pairs % nent
            up = ent_owner[u] != s                       # eliminated further up
            o = np.lexsort((u, up, s))
            s, u, up = s[o], u[o], up[o]
            first, count = 1 << d, 1 << d
            n_ent = np.bincount(s - first, minlength=count)
            p = np.bincount((s - first)[~up], minlength=count) * per
            n = n_ent * per + nborder
            if d == 0:
                p = p + nborder
            full = np.empty(int(n.sum()), dtype=np.int64)
            end = np.cumsum(n)
            bpos = (end[:, None] - nborder + np.arange(nborder)).reshape(-1)
            body = np.ones(len(full), dtype=bool)
            body[bpos] = False
            full[bpos] = np.tile(border, count)
            full[body] = (u[:, None] * per + np.arange(per)).reshape(-1)
            t0 = sum(len(h) for h in heap)
            self.levels.append((t0, t0 + count))
            heap.append(np.arange(first, first + count, dtype=np.int64))
            p_sz.append(p)
            n_sz.append(n)
            ids.append(full)
            pairs = (s[up] >> 1) * nent + u[up]
        self.depth, self.N, self.owner = depth, N, owner
        self.heap = np.concatenate(heap)
        self.p, self.n = np.concatenate(p_sz).astype(np.int64), np.concatenate(n_sz).astype(np.int64)
        self.ids = np.concatenate(ids)
        self.idx_off = np.concatenate([[0], np.cumsum(self.n)])
        self.nfront = len(self.heap)
        # front index of a heap id
        self.front_of = np.empty(2 << depth, dtype=np.int64)
        self.front_of[self.heap] = np.arange(self.nfront)
