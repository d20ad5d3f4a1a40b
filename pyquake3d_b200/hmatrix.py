"""H-matrix structure (host) and the packed device operator.

Host part (FP64, numpy), a restatement of src/Hmatrix.py:
  * build_cluster_tree  <- build_block_tree   (:143-182)  bisection of the
    longest bounding-box axis at its midpoint, leaves of <= min_size elements;
  * is_admissible       <- is_admissible      (:88-103)   min(diam) <= eta*dist;
  * build_blocks        <- create_recursive_blocks + collect_blocks (:1611-1672,
    :1291-1297) quad-split, a leaf when admissible or when either cluster has
    <= mini_leaf elements; leaves listed depth-first (the reference's order);
  * ACA vs dense        <- BlockTree.ACA_worker (:1014-1066): ACA when both
    dimensions exceed mini_leaf, dense otherwise.
Every cluster is also given its range in tree order (depth-first, left child
first), the layout of all device vectors.

Device part: DeviceHMatrix assembles the operator on the GPU (dense near field
with the FP64 Green's function, admissible blocks with batched ACA), packs it
for one or more storage precisions and applies it with pq3d_hmatvec.
"""
import math
import os

import numpy as np

from . import _lib
from ._lib import ptr, check

# ----------------------------------------------------------------------------- host tree


class ClusterNode:
    __slots__ = ("indices", "left", "right", "start", "level", "bbox_min", "bbox_max", "leaf_id", "_box")

    def __init__(self, indices, level):
        self.indices = indices
        self.left = None
        self.right = None
        self.start = 0
        self.level = level
        self.bbox_min = None
        self.bbox_max = None
        self._box = None
        self.leaf_id = -1


def build_cluster_tree(points, min_size=16):
    """Cluster tree of build_block_tree (src/Hmatrix.py:143-182).

    Returns (root, perm, leaves): perm[p] = element at tree position p."""
    root = ClusterNode(np.arange(len(points)), 0)
    stack = [(root, points)]
    while stack:
        node, pts = stack.pop()
        cl = node.indices
        node.bbox_min = np.min(pts, axis=0)
        node.bbox_max = np.max(pts, axis=0)
        if len(cl) <= min_size:
            continue
        alpha, beta = node.bbox_min, node.bbox_max
        j = int(np.argmax(beta - alpha))
        gamma = (alpha[j] + beta[j]) / 2
        i1 = pts[:, j] <= gamma
        i2 = pts[:, j] > gamma
        t1, t2 = cl[i1], cl[i2]
        if len(t1) == 0 or len(t2) == 0:
            continue
        node.left = ClusterNode(t1, node.level + 1)
        node.right = ClusterNode(t2, node.level + 1)
        stack.append((node.right, pts[i2]))
        stack.append((node.left, pts[i1]))
    # tree-order ranges (left first) and leaves
    perm = np.empty(len(points), dtype=np.int64)
    leaves = []
    pos = 0
    st = [root]
    while st:
        nd = st.pop()
        nd.start = pos if nd.left is None else nd.start
        if nd.left is None:
            nd.start = pos
            nd.leaf_id = len(leaves)
            leaves.append(nd)
            perm[pos:pos + len(nd.indices)] = nd.indices
            pos += len(nd.indices)
        else:
            st.append(nd.right)
            st.append(nd.left)
    _fix_starts(root)
    return root, perm, leaves


def _fix_starts(root):
    st = [root]
    order = []
    while st:
        nd = st.pop()
        order.append(nd)
        if nd.left is not None:
            st.append(nd.right)
            st.append(nd.left)
    for nd in reversed(order):
        if nd.left is not None:
            nd.start = nd.left.start


def _box(nd):
    """(bbox_min, bbox_max as floats, diameter) of a cluster, computed once."""
    if nd._box is None:
        lo, hi = [float(v) for v in nd.bbox_min], [float(v) for v in nd.bbox_max]
        e = [h - l for l, h in zip(lo, hi)]
        nd._box = (lo, hi, math.sqrt((e[0] * e[0] + e[1] * e[1]) + e[2] * e[2]))
    return nd._box


def is_admissible(a, b, eta):
    """min(diam_a, diam_b) <= eta * dist(bbox_a, bbox_b).  The sums run in numpy's
    order for three terms ((t0 + t1) + t2) and every operation is correctly rounded,
    so the decisions are those of the reference's numpy expression."""
    alo, ahi, da = _box(a)
    blo, bhi, db = _box(b)
    t = []
    for k in range(3):
        u = max(0.0, blo[k] - ahi[k])
        v = max(0.0, alo[k] - bhi[k])
        t.append(u * u + v * v)
    dq = math.sqrt((t[0] + t[1]) + t[2])
    return min(da, db) <= eta * dq


class LeafBlock:
    """A leaf of the block tree: rows = row cluster, cols = col cluster."""
    __slots__ = ("row", "col", "aca", "admissible", "level")

    def __init__(self, row, col, aca, admissible, level):
        self.row = row
        self.col = col
        self.aca = aca
        self.admissible = admissible
        self.level = level

    @property
    def row_cluster(self):
        return self.row.indices

    @property
    def col_cluster(self):
        return self.col.indices

    @property
    def judaca(self):
        return self.aca


def build_blocks(row_root, col_root, eta=2.0, mini_leaf=32):
    """Leaves of create_recursive_blocks in collect_blocks (depth-first) order."""
    out = []
    st = [(row_root, col_root, 0)]
    while st:
        r, c, lev = st.pop()
        adm = is_admissible(r, c, eta)
        if adm or len(r.indices) <= mini_leaf or len(c.indices) <= mini_leaf or \
                r.left is None or r.right is None or c.left is None or c.right is None:
            aca = len(r.indices) > mini_leaf and len(c.indices) > mini_leaf
            out.append(LeafBlock(r, c, aca, bool(adm), lev))
            continue
        st.append((r.right, c.right, lev + 1))
        st.append((r.right, c.left, lev + 1))
        st.append((r.left, c.right, lev + 1))
        st.append((r.left, c.left, lev + 1))
    return out


class HStructure:
    """Cluster trees and leaf blocks of the operator (the part QDsim.__init__ builds)."""

    def __init__(self, xg, mini_leaf=32, eta=2.0, min_size=16):
        self.n = len(xg)
        self.mini_leaf = mini_leaf
        self.eta = eta
        self.min_size = min_size
        self.row_root, self.perm, self.leaves = build_cluster_tree(xg, min_size)
        # the reference builds the column tree with the same call: identical tree
        self.col_root = self.row_root
        self.iperm = np.empty_like(self.perm)
        self.iperm[self.perm] = np.arange(self.n)
        self.blocks = build_blocks(self.row_root, self.col_root, eta, mini_leaf)

    def stats(self):
        nd = sum(1 for b in self.blocks if not b.aca)
        na = len(self.blocks) - nd
        dense_entries = sum(len(b.row.indices) * len(b.col.indices) for b in self.blocks if not b.aca)
        aca_mn = sum(len(b.row.indices) + len(b.col.indices) for b in self.blocks if b.aca)
        return dict(n=self.n, blocks=len(self.blocks), dense_blocks=nd, aca_blocks=na,
                    dense_entries=dense_entries, aca_m_plus_n=aca_mn, leaves=len(self.leaves))


def aca_start_indices(blocks, seed):
    """Starting reference row/col of every ACA pass, drawn as the reference does
    (np.random.randint(n_rows) - 3, np.random.randint(n_cols) - 3 for the strike
    pass, then again for the dip pass, src/Hmatrix.py:660-661 and :888-889), with
    a seeded legacy RandomState and blocks taken in list order."""
    sizes = [(len(b.row.indices), len(b.col.indices)) * 2 for b in blocks if b.aca]
    if not sizes:
        return []
    # one draw over the array of bounds gives the numbers of a draw per bound
    r = np.random.RandomState(seed).randint(np.array(sizes, dtype=np.int64).reshape(-1)) - 3
    return [((a, b), (c, d)) for a, b, c, d in r.reshape(-1, 4).tolist()]


# ----------------------------------------------------------------------------- packed layout (host)


def x_stride(n):
    """Plane stride of the device deficit vector (hm_layout.cuh x_stride)."""
    return ((n + 16 + 7) // 8) * 8


def pack_x(x1, x2, n):
    """Deficit vector in the device layout: interleaved pairs, then strike and dip
    planes (x1, x2 already in tree order)."""
    P = x_stride(n)
    x = np.zeros(4 * P)
    x[0:2 * n:2] = x1
    x[1:2 * n:2] = x2
    x[2 * P:2 * P + n] = x1
    x[3 * P:3 * P + n] = x2
    return x


def _expand(counts):
    """For counts[i] consecutive items of each owner i: (owner, index within the owner)."""
    counts = np.asarray(counts, dtype=np.int64)
    owner = np.repeat(np.arange(len(counts)), counts)
    return owner, np.arange(len(owner)) - (np.cumsum(counts) - counts)[owner]


def _offsets(sizes):
    """Exclusive running sum of sizes, and the total."""
    t = np.cumsum(sizes, dtype=np.int64)
    return t - sizes, int(t[-1]) if len(t) else 0


def _fields(dtype, n, **cols):
    """n records of `dtype` from columns (at least one zero record, for the uploads)."""
    rec = np.zeros(max(n, 1), dtype=dtype)
    for k, v in cols.items():
        rec[k][:n] = v
    return rec


def _check32(**sizes):
    """The records hold these in 32 bits, and an assignment to a column wraps silently: refuse a
    plan beyond that before its items are made."""
    for k, v in sizes.items():
        if v > 0x7fffffff:
            raise OverflowError("%s of the plan: %d does not fit the work items' 32 bits" % (k, v))


def workspace_table(ntasks):
    """Where every ACA task's factors are: workspace, offset in it and room for terms (none:
    ntasks 0, as an operator read from a checkpoint has it)."""
    return {k: np.zeros(ntasks, np.int64) for k in ("ws", "off", "kmax")}


def _block_geometry(blocks):
    """(m, n, first row, first column, lo, hi) of blocks in tree order; [lo, hi) are the
    block-local rows the plan computes (all, unless a row partition clipped them)."""
    g = np.array([(len(b.row.indices), len(b.col.indices), b.row.start, b.col.start) + getattr(b, "rows", (0, -1))
                  for b in blocks], dtype=np.int64).reshape(-1, 6).T
    return g[0], g[1], g[2], g[3], g[4], np.where(g[5] < 0, g[0], g[5])


def dense_layout(dense_blocks):
    """DenseBlock records with FP64 / FP32 offsets, and the two array sizes.  Stored
    columns start at the column-group-aligned c0 - (c0 % CW)."""
    m, n, r0, c0, _, _ = _block_geometry(dense_blocks)
    off64, n64 = _offsets(_cdiv(n + c0 % 2, 2) * m * 12)
    off32, n32 = _offsets(_cdiv(n + c0 % 4, 4) * m * 24)
    recs = np.zeros(len(dense_blocks), dtype=_lib.DENSE_BLOCK)
    for k, v in dict(off64=off64, off32=off32, m=m, n=n, r0=r0, c0=c0).items():
        recs[k] = v
    return recs, n64, n32


_PACK = np.dtype([("bi", "i8"), ("pass_", "i8"), ("u_off", "i8"), ("v_off", "i8"), ("K", "i8"), ("Q", "i8"), ("kS", "i8"),
                  ("kD", "i8")])
_PACK_M = np.dtype([("bi", "i8"), ("pass_", "i8")] + [(k, "i8", 3) for k in ("u_off", "v_off", "kS", "kD", "Q", "K", "sb")])


def build_plan_arrays(struct, dense_recs, kS, kD, code, dense_chunk=64, v_chunk=256, u_rows=512):
    """Matvec work items, slot layout and per-leaf slot lists for storage code
    (0 FP64, 1 FP32, 2 FP32 dense + BF16 low rank).  Pure numpy.

    Slots: every dense (block, column chunk) and every low-rank block owns m
    consecutive slots (one per block row); row i of a block with slot base s
    and first row r0 writes slot s + (i - r0).  leaf_off lists, per leaf
    cluster, the offsets s - r0 of all slot owners covering that leaf."""
    cwd, cwl = _CW_DENSE[code], _CW_LR[code]
    n = struct.n
    dense_off = dense_recs["off64"] if code == 0 else dense_recs["off32"]
    ditems, slot_rows, slot0 = _dense_items(dense_recs, cwd, dense_off, dense_chunk)
    m, nn, row0, c0, lo, hi = _block_geometry([b for b in struct.blocks if b.aca])
    ks, kd = np.asarray(kS, np.int64)[:len(m)], np.asarray(kD, np.int64)[:len(m)]
    lr_entries = int((3 * (ks + kd) * ((hi - lo) + nn)).sum())
    on = np.nonzero(ks + kd > 0)[0]                     # blocks with terms
    m, nn, row0, c0, lo, hi, ks, kd = (a[on] for a in (m, nn, row0, c0, lo, hi, ks, kd))
    lr = dict(vitems=_fields(_lib.V_ITEM, 0), utasks=_fields(_lib.U_TASK, 0), n_vitems=0, n_utasks=0, n_slots=slot0,
              n_tpart=0, kmax=0, u_size=0, v_size=0, pack=np.zeros(0, dtype=_PACK))
    if len(on):
        lr, rows = _lowrank_items(m, nn, row0, c0, lo, hi, ks, kd, on, cwl, v_chunk, u_rows, slot0)
        slot_rows = np.concatenate([slot_rows, rows])
    L = _leaf_lists(struct, slot_rows)
    esz_d = 8 if code == 0 else 4
    esz_l = {0: 8, 1: 4, 2: 2}[code]
    dense_entries = int(np.sum(dense_recs["m"].astype(np.int64) * dense_recs["n"])) if len(dense_recs) else 0
    nd = len(ditems)
    return dict(ditems=_fields(_lib.DENSE_ITEM, 0) if nd == 0 else ditems, n_ditems=nd,
                alg_bytes=dense_entries * 6 * esz_d + lr_entries * esz_l + 2 * n * esz_d + 3 * n * 8, **lr, **L)


def _lowrank_items(m, nn, row0, c0, lo, hi, ks, kd, on, cwl, v_chunk, u_rows, slot0):
    """The low-rank part of build_plan_arrays for the blocks with terms (their geometry, terms per
    pass and numbers `on`), slots from slot0: (plan entries, slot owners)."""
    K, Q, lead = _cdiv(ks + kd, cwl) * cwl, 3 * (ks + kd), c0 % cwl
    ngv = _cdiv(nn + lead, cwl)
    nch = _cdiv(ngv, v_chunk)
    u_off, u_size = _offsets((K // cwl) * m * 3 * cwl)
    v_off, v_size = _offsets(Q * ngv * cwl)
    tp, n_tpart = _offsets(nch * Q)
    slot, n_slots = _offsets(hi - lo)
    slot, n_slots = slot + slot0, n_slots + slot0
    _check32(slots=n_slots, t_positions=n_tpart)
    # V items: per column chunk, the strike rows then the dip rows, 32 to an item
    nS, nD = _cdiv(3 * ks, 32), _cdiv(3 * kd, 32)
    b, i = _expand(nch * (nS + nD))
    ch, i = i // (nS + nD)[b], i % (nS + nD)[b]
    dip = i >= nS[b]
    q = np.where(dip, 3 * ks[b] + 32 * (i - nS[b]), 32 * i)
    nv = len(b)
    vitems = _fields(_lib.V_ITEM, nv, off=v_off[b], Q=Q[b], q=q, nr=np.minimum(32, np.where(dip, Q[b], 3 * ks[b]) - q),
                     g0=ch * v_chunk, g1=np.minimum(ngv[b], (ch + 1) * v_chunk), c0=(c0 - lead)[b], s=dip,
                     tp=tp[b] + ch * Q[b])
    # U tasks; row r of the block writes slot (slot - lo) + r, for r in [lo, hi)
    b, i = _expand(_cdiv(hi - lo, u_rows))
    r0 = lo[b] + i * u_rows
    nu = len(b)
    utasks = _fields(_lib.U_TASK, nu, off=u_off[b], m=m[b], r0=r0, r1=np.minimum(hi[b], r0 + u_rows), K=K[b], kS=ks[b],
                     kD=kd[b], Q=Q[b], tp=tp[b], nch=nch[b], slot=(slot - lo)[b])
    pack = np.zeros(2 * len(on), dtype=_PACK)
    for k, v in dict(bi=on, u_off=u_off, v_off=v_off, K=K, Q=Q, kS=ks, kD=kd).items():
        pack[k] = np.repeat(v, 2)
    pack["pass_"] = np.tile([0, 1], len(on))
    return dict(vitems=vitems, utasks=utasks, n_vitems=nv, n_utasks=nu, n_slots=n_slots, n_tpart=n_tpart,
                kmax=int(K.max()), u_size=u_size, v_size=v_size, pack=pack), np.stack([slot, row0 + lo, hi - lo], axis=1)


def _dense_items(dense_recs, cwd, dense_off, dense_chunk):
    """Dense work items (one warp: 32 rows x a chunk of column groups) and their slots:
    every (block, column chunk) owns m consecutive slots."""
    m, nn, r0, c0 = (dense_recs[k].astype(np.int64) for k in ("m", "n", "r0", "c0"))
    lead = c0 % cwd
    ng = _cdiv(nn + lead, cwd)
    nch, nr = _cdiv(ng, dense_chunk), _cdiv(m, 32)
    ob, ch = _expand(nch)                              # slot owners: (block, column chunk)
    slot, n_slots = _offsets(m[ob])
    _check32(slots=n_slots)
    o, i = _expand(nr[ob])
    b = ob[o]
    ditems = np.zeros(len(o), dtype=_lib.DENSE_ITEM)
    for k, v in dict(off=np.asarray(dense_off)[b], m=m[b], r=32 * i, g0=ch[o] * dense_chunk,
                     g1=np.minimum(ng[b], (ch[o] + 1) * dense_chunk), c0=(c0 - lead)[b], slot=slot[o]).items():
        ditems[k] = v
    return ditems, np.stack([slot, r0[ob], m[ob]], axis=1).reshape(-1, 3), n_slots


def _leaf_lists(struct, slot_rows):
    """Per leaf cluster, the offsets (slot - first row) of every slot owner covering it."""
    n = struct.n
    nleaf = len(struct.leaves)
    start = np.array([lf.start for lf in struct.leaves], dtype=np.int64)
    leaf_id = np.array([lf.leaf_id for lf in struct.leaves], dtype=np.int32)
    leaf_of_row = np.repeat(leaf_id, [len(lf.indices) for lf in struct.leaves])
    if len(start) and (np.diff(start) < 0).any():      # leaves listed out of row order
        order = np.argsort(start, kind="stable")
        leaf_of_row = np.repeat(leaf_id[order], [len(struct.leaves[i].indices) for i in order])
    sr = np.array(slot_rows, dtype=np.int64).reshape(-1, 3)
    first = leaf_of_row[sr[:, 1]].astype(np.int64)
    last = leaf_of_row[sr[:, 1] + sr[:, 2] - 1].astype(np.int64)
    cnt = last - first + 1
    rep_leaf = np.repeat(first, cnt) + (np.arange(cnt.sum()) - np.repeat(np.cumsum(cnt) - cnt, cnt))
    rep_off = np.repeat(sr[:, 0] - sr[:, 1], cnt)
    order = np.argsort(rep_leaf, kind="stable")
    leaf_off = rep_off[order].astype(np.int32)
    leaf_ptr = np.concatenate([[0], np.cumsum(np.bincount(rep_leaf, minlength=nleaf))]).astype(np.int32)
    return dict(leaf_of_row=leaf_of_row, leaf_ptr=leaf_ptr,
                leaf_off=leaf_off if len(leaf_off) else np.zeros(1, np.int32), slot_rows=sr)


# ----------------------------------------------------------------------------- mixed storage (host)

MIXED_CW = (4, 8, 16)               # column groups of the FP32 / FP16 / INT8 term classes
MIXED_BYTES = (4, 2, 1)
# relative rounding of a stored entry against its vector's largest magnitude
MIXED_EPS = (2.0 ** -24, 2.0 ** -11, 0.5 / 127.0)


def classify_terms(wS, wD, tol):
    """The rule of classify_blocks, stated for one block (the plans use the former; tests
    compare the two): classes (0 FP32, 1 FP16, 2 INT8) of the block's ACA terms from their weights
    w = max_i(|u_i| / R_i) ||v||_1 (strike terms wS, dip terms wD, in ACA order).

    A term needs FP32 when 2 eps_FP16 w > tol (quantising u and v to FP16 would move a
    row by more than tol times its near-field absolute row sum), FP16 when 2 eps_INT8 w
    > tol, else INT8 suffices.  Each class's column count is padded to its column
    group (4, 8, 16); the padding is filled by promoting the next most important terms
    instead of storing zeros, and an INT8 remnant of at most 8 terms (or an FP16
    remnant of at most 4 after FP32 and with no INT8 terms) moves up a class at no
    extra storage.  Returns (cls_S, cls_D) arrays of class codes."""
    w = np.concatenate([np.asarray(wS, dtype=np.float64), np.asarray(wD, dtype=np.float64)])
    K = len(w)
    if K == 0:
        return np.zeros(0, np.int32), np.zeros(0, np.int32)
    req = np.where(2 * MIXED_EPS[1] * w > tol, 0, np.where(2 * MIXED_EPS[2] * w > tol, 1, 2))
    n0, n1 = int((req == 0).sum()), int((req == 1).sum())
    n0p = min(K, _cdiv(n0, 4) * 4) if n0 else 0
    rem1 = max(0, n0 + n1 - n0p)
    left = K - n0p
    n1p = min(left, _cdiv(rem1, 8) * 8) if rem1 else 0
    n2p = left - n1p
    if 0 < n2p <= 8:
        n1p, n2p = n1p + n2p, 0
    if n2p == 0 and 0 < n1p <= 4 and n0p % 4 == 0:
        n0p, n1p = n0p + n1p, 0
    order = np.argsort(-w, kind="stable")
    cls = np.empty(K, np.int32)
    cls[order[:n0p]] = 0
    cls[order[n0p:n0p + n1p]] = 1
    cls[order[n0p + n1p:]] = 2
    return cls[:len(wS)], cls[len(wS):]


def classify_blocks(w, offs, tol):
    """classify_terms over all blocks at once: w holds every term's weight in task order
    (block by block, strike terms then dip), offs the tasks' offsets (two per block and
    the total).  Returns the class of every term."""
    K = offs[2::2] - offs[:-1:2]
    blk = np.repeat(np.arange(len(K)), K)
    first = (np.cumsum(K) - K)[blk]
    w = w[:len(blk)]
    req = np.where(2 * MIXED_EPS[1] * w > tol, 0, np.where(2 * MIXED_EPS[2] * w > tol, 1, 2))
    n0 = np.bincount(blk[req == 0], minlength=len(K))
    n1 = np.bincount(blk[req == 1], minlength=len(K))
    n0p = np.where(n0 > 0, np.minimum(K, _cdiv(n0, 4) * 4), 0)
    rem1 = np.maximum(0, n0 + n1 - n0p)
    left = K - n0p
    n1p = np.where(rem1 > 0, np.minimum(left, _cdiv(rem1, 8) * 8), 0)
    n2p = left - n1p
    up = (n2p > 0) & (n2p <= 8)
    n1p, n2p = np.where(up, n1p + n2p, n1p), np.where(up, 0, n2p)
    up = (n2p == 0) & (n1p > 0) & (n1p <= 4) & (n0p % 4 == 0)
    n0p, n1p = np.where(up, n0p + n1p, n0p), np.where(up, 0, n1p)
    order = np.lexsort((-w, blk))                      # stable: block by block, largest weight first
    rank = np.empty(len(blk), np.int64)
    rank[order] = np.arange(len(blk)) - first
    return np.where(rank < n0p[blk], 0, np.where(rank < (n0p + n1p)[blk], 1, 2)).astype(np.int32)


def class_counts(cls, offs):
    """Terms per (block, pass, class) of classes in task order."""
    task = np.repeat(np.arange(len(offs) - 1), np.diff(offs))
    return np.bincount(3 * task + cls[:len(task)], minlength=3 * (len(offs) - 1)).reshape(-1, 2, 3)


def build_plan_arrays_mixed(struct, dense_recs, cls_lists, dense_chunk=16, v_chunk=32, u_rows=512, stream=False,
                            ncta=148, nwarps=None, counts=None):
    """Work items, slot layout and packing records of the mixed storage (code 3):
    FP32 dense items as in the FP32 plan; per low-rank block and term class c
    (FP32, FP16, INT8) the class's own U / V arrays with column groups MIXED_CW[c].
    counts[bi, pass, class]: terms of each class (class_counts of classify_blocks), or
    cls_lists[bi] = (cls_S, cls_D), the classes of one block's terms.  Pure numpy.

    stream=True lays the work out for the persistent bulk-copy kernel k_stream:
    StreamTask lists of phase A (dense tasks of at most STREAM_DENSE_ROWS rows and
    1,024 columns; V tasks over all rows of one class of one block and at most
    1,024 columns) and phase B (U tasks of at most STREAM_ROWS rows), each list
    split over `ncta` persistent CTAs balanced by the bytes they stream, plus
    one TGather record per low-rank block (the t it gathers into tfull)."""
    if stream:
        return _build_stream_mixed(struct, dense_recs, cls_lists, ncta)
    ditems, slot_rows, slot0 = _dense_items(dense_recs, 4, dense_recs["off32"], dense_chunk)
    if counts is None:
        counts = np.array([[np.bincount(c, minlength=3) for c in cl] for cl in cls_lists], np.int64).reshape(-1, 2, 3)
    lr = dict(vitems=_fields(_lib.V_ITEM_M, 0), vwarp=np.zeros(9, np.int32), vrows=_fields(_lib.V_ROW, 0),
              utasks=_fields(_lib.U_TASK_M, 0), n_utasks=0, n_slots=slot0, n_tpart=0, n_scales=0, kmax=0,
              u_sizes=[0, 0, 0], v_sizes=[0, 0, 0], pack=np.zeros(0, dtype=_PACK_M),
              class_terms=np.zeros((3, 2), np.int64))
    lr_bytes = 0
    if counts.any():
        lr, rows, lr_bytes = _lowrank_items_mixed(struct, counts, v_chunk, u_rows, slot0, nwarps or VMIX_WARPS)
        slot_rows = np.concatenate([slot_rows, rows])
    A = _leaf_lists(struct, slot_rows)
    dense_entries = int(np.sum(dense_recs["m"].astype(np.int64) * dense_recs["n"])) if len(dense_recs) else 0
    n = struct.n
    nd = len(ditems)
    A.update(ditems=_fields(_lib.DENSE_ITEM, 0) if nd == 0 else ditems, n_ditems=nd, n_vitems=int(lr["vwarp"][-1]),
             stream=False, alg_bytes=dense_entries * 6 * 4 + lr_bytes + 2 * n * 4 + 3 * n * 8, **lr)
    return A


def _lowrank_items_mixed(struct, counts, v_chunk, u_rows, slot0, nwarps):
    """The low-rank part of build_plan_arrays_mixed, slots from slot0: (plan entries, slot owners,
    bytes of the factors)."""
    CW = np.array(MIXED_CW)
    m, nn, row0, c0, lo, hi = _block_geometry([b for b in struct.blocks if b.aca])
    on = np.nonzero(counts.sum(axis=(1, 2)) > 0)[0]              # blocks with terms
    m, nn, row0, c0, lo, hi = (a[on] for a in (m, nn, row0, c0, lo, hi))
    ks, kd = counts[on, 0], counts[on, 1]                        # (block, class)
    K = _cdiv(ks + kd, CW) * CW
    Q = 3 * (ks + kd)
    lead = c0[:, None] % CW
    ngv = _cdiv(nn[:, None] + lead, CW)
    nch = np.where(K > 0, _cdiv(ngv, v_chunk), 0)
    # class arrays one after the other within a class; partials and scales over (block, class)
    u_off, v_off, u_size, v_size = np.zeros_like(K), np.zeros_like(K), [], []
    for c in range(3):
        u_off[:, c], t = _offsets(K[:, c] * m * 3)
        u_size.append(t)
        v_off[:, c], t = _offsets(Q[:, c] * ngv[:, c] * MIXED_CW[c])
        v_size.append(t)
    if max(v_size) >= 1 << 32:
        raise _lib.Pq3dError("a V class array of the mixed storage holds 2^32 elements or more")
    tp, n_tpart = _offsets((nch * Q).ravel())
    scaled = np.where(np.arange(3) > 0, Q, 0).ravel()
    sb, n_scales = _offsets(scaled)
    tp, sb = np.where(K > 0, tp.reshape(-1, 3), 0), np.where((K > 0) & (np.arange(3) > 0), sb.reshape(-1, 3), 0)
    slot, n_slots = _offsets(hi - lo)
    slot, n_slots = slot + slot0, n_slots + slot0
    _check32(slots=n_slots, t_positions=n_tpart, scales=n_scales, row_stride=int((Q * CW).max(initial=0)))
    # one entry per (block, class) with rows, for the merged V items
    b, c = np.nonzero(K > 0)
    vitems, vwarp, vrows = _merged_v_items(c0[b], nn[b], c, v_off[b, c], Q[b, c], 3 * ks[b, c], tp[b, c], v_chunk,
                                           nwarps)
    o, i = _expand(_cdiv(hi - lo, u_rows))
    r0 = lo[o] + i * u_rows
    nu = len(o)
    utasks = _fields(_lib.U_TASK_M, nu, off=u_off[o], m=m[o], r0=r0, r1=np.minimum(hi[o], r0 + u_rows),
                     slot=(slot - lo)[o], K=K[o], kS=ks[o], kD=kd[o], Q=Q[o], tp=tp[o], nch=nch[o], sb=sb[o])
    pack = np.zeros(2 * len(on), dtype=_PACK_M)
    for k, v in dict(bi=on, u_off=u_off, v_off=v_off, kS=ks, kD=kd, Q=Q, K=K, sb=sb).items():
        pack[k] = np.repeat(v, 2, axis=0)
    pack["pass_"] = np.tile([0, 1], len(on))
    lr_bytes = int((Q * ((hi - lo) + nn)[:, None] * np.array(MIXED_BYTES)).sum() + 4 * scaled.sum())
    return dict(vitems=vitems, vrows=vrows, vwarp=vwarp, utasks=utasks, n_utasks=nu, n_slots=n_slots, n_tpart=n_tpart,
                n_scales=n_scales, kmax=int(K.sum(axis=1).max()), u_sizes=u_size, v_sizes=v_size, pack=pack,
                class_terms=np.stack([ks.sum(axis=0), kd.sum(axis=0)], axis=1)), \
        np.stack([slot, row0 + lo, hi - lo], axis=1), lr_bytes


VMIX_WARPS = 8 * 148 * 4      # k_v_mixed warps when no device says otherwise (B200, 4 CTAs per SM)
VMIX_ROWS = 32                # rows per merged V item (k_v_mixed handles up to 32)


def _merged_v_items(col0, nn, cls, off, Q, ks3, tp, v_chunk, nwarps=VMIX_WARPS):
    """V items of the mixed storage's plain kernels (k_v_mixed): for each column
    cluster, class and slip, the V rows of all low-rank blocks with those columns
    (in block order), per column chunk, 32 rows to an item, so the x slice is loaded
    once for all of them.  One entry per (block, class): column start, columns, class,
    V offset in the class array, Q, strike rows, t base.  Returns the items
    ordered by warp, the per-warp offsets (nwarps + 1) and the row records.  Items go
    largest first to the least loaded of the nwarps warps (cost: row slots of 8 x
    column groups, plus a fixed start), so the persistent warps end together."""
    # entries grouped by (columns, class), groups in order of first appearance
    _, first, grp = np.unique(np.stack([col0, nn, cls], axis=1), axis=0, return_index=True, return_inverse=True)
    grp = np.argsort(np.argsort(first))[grp.ravel()]
    e = np.argsort(grp, kind="stable")
    grp, off, Q, ks3, tp = grp[e], off[e], Q[e], ks3[e], tp[e]
    g0 = np.sort(first)                                          # a group's first entry
    col0, nn, cls = col0[g0], nn[g0], cls[g0]
    cw = np.array(MIXED_CW)[cls]
    lead = col0 % cw
    ngv = _cdiv(nn + lead, cw)
    nch = _cdiv(ngv, v_chunk)
    ng = len(g0)
    # rows of group g, slip s: q in [0, ks3) or [ks3, Q) of its entries, in order
    cnt = np.stack([ks3, Q - ks3], axis=1)
    eo = np.lexsort((np.tile(np.arange(len(grp)), 2), np.concatenate([2 * grp, 2 * grp + 1])))
    ent, slip = eo % max(len(grp), 1), eo // max(len(grp), 1)
    o, q = _expand(cnt[ent, slip])
    ent, slip = ent[o], slip[o]
    q = q + np.where(slip == 1, ks3[ent], 0)
    gs = 2 * grp[ent] + slip                                     # sorted: rows of (group, slip) are consecutive
    nrows = np.bincount(gs, minlength=2 * ng)
    row0, _ = _offsets(nrows)
    # per (group, slip, chunk): the rows' records, then its items of 32 rows
    a, ch = _expand(np.where(nrows > 0, np.repeat(nch, 2), 0))
    rec0, nrec = _offsets(nrows[a])
    o, i = _expand(nrows[a])
    r = row0[a[o]] + i
    rec = _fields(_lib.V_ROW, nrec, base=off[ent[r]] + q[r] * cw[grp[ent[r]]], stride=Q[ent[r]] * cw[grp[ent[r]]],
                  out=tp[ent[r]] + ch[o] * Q[ent[r]] + q[r])
    o, i = _expand(_cdiv(nrows[a], VMIX_ROWS))
    g = a[o] // 2
    nitems = len(o)
    items = _fields(_lib.V_ITEM_M, nitems, rows=rec0[o] + VMIX_ROWS * i, nr=np.minimum(VMIX_ROWS, nrows[a[o]] - VMIX_ROWS * i),
                    g0=ch[o] * v_chunk, g1=np.minimum(ngv[g], (ch[o] + 1) * v_chunk), c0=(col0 - lead)[g],
                    s=a[o] % 2 | (cls[g] << 8))
    import heapq
    it = items[:nitems]
    cost = _cdiv(it["nr"], 8) * (it["g1"] - it["g0"]) + 16
    order = np.argsort(-cost, kind="stable")
    nwarps = max(8, min(int(nwarps), max(nitems, 1)) // 8 * 8)
    heap = [(0, w) for w in range(nwarps)]
    warp = np.empty(nitems, np.int32)
    for k, c in enumerate(cost[order].tolist()):
        load, w = heap[0]
        warp[k] = w
        heapq.heapreplace(heap, (load + c, w))
    vwarp = np.concatenate([[0], np.cumsum(np.bincount(warp, minlength=nwarps))]).astype(np.int32)
    items[:nitems] = it[order[np.argsort(warp, kind="stable")]]
    return items, vwarp, rec


def _balance(tasks, nbytes, ncta):
    """Tasks grouped by CTA (largest first to the least loaded CTA): (records sorted by
    CTA, per-CTA ranges of ncta' + 1 entries, ncta' = CTAs with work)."""
    import heapq
    if not tasks:
        return np.zeros(1, dtype=_lib.STREAM_TASK), np.zeros(1, np.int32), 0
    ncta = max(1, min(int(ncta), len(tasks)))
    heap = [(0, c) for c in range(ncta)]
    owner = np.empty(len(tasks), np.int64)
    for i in np.argsort(-np.asarray(nbytes, np.int64), kind="stable"):
        load, c = heapq.heappop(heap)
        owner[i] = c
        heapq.heappush(heap, (load + int(nbytes[i]), c))
    order = np.argsort(owner, kind="stable")
    rec = np.array([tasks[i] for i in order], dtype=_lib.STREAM_TASK)
    ptr = np.zeros(ncta + 1, np.int32)
    np.add.at(ptr, owner + 1, 1)
    return rec, np.cumsum(ptr).astype(np.int32), ncta


def _task(kind, **kw):
    t = dict(off=0, off1=0, off2=0, kind=kind, cls=0, m=0, r0=0, r1=0, g0=0, g1=0, c0=0, out=0, kS3=0, K0=0, K1=0,
             K2=0, tb=0)
    t.update(kw)
    return tuple(t[k] for k in _lib.STREAM_TASK.names)


def _build_stream_mixed(struct, dense_recs, cls_lists, ncta):
    """Task lists of the streamed mixed storage (build_plan_arrays_mixed, stream=True)."""
    DCOLS, VCOLS = 1024, 1024                  # columns of a dense / V task (x slice in shared memory)
    n = struct.n
    ta, ba, tb_, bb, gather = [], [], [], [], []
    slot_rows, slot = [], 0
    # dense tasks: (block, column chunk) owns m slots; row ranges share them
    for i in range(len(dense_recs)):
        m, nn, r0b, c0 = (int(dense_recs[k][i]) for k in ("m", "n", "r0", "c0"))
        lead = c0 % 4
        ng = _cdiv(nn + lead, 4)
        gch = DCOLS // 4
        for g0 in range(0, ng, gch):
            g1 = min(ng, g0 + gch)
            for r0 in range(0, m, _lib.STREAM_DENSE_ROWS):
                r1 = min(m, r0 + _lib.STREAM_DENSE_ROWS)
                ta.append(_task(0, off=int(dense_recs["off32"][i]), m=m, r0=r0, r1=r1, g0=g0, g1=g1, c0=c0 - lead,
                                out=slot))
                ba.append((g1 - g0) * (6 * (r1 - r0) * 16 + 32))
            slot_rows.append((slot, r0b, m))
            slot += m
    aca_blocks = [b for b in struct.blocks if b.aca]
    u_off, v_off = [0, 0, 0], [0, 0, 0]
    tp = sb = tb = 0
    pack = []
    lr_bytes = 0
    counts = np.zeros((3, 2), np.int64)
    for bi, b in enumerate(aca_blocks):
        m, nn = len(b.row.indices), len(b.col.indices)
        lo, hi = getattr(b, "rows", (0, m))
        cS, cD = cls_lists[bi]
        ks = np.bincount(cS, minlength=3).tolist()
        kd = np.bincount(cD, minlength=3).tolist()
        if sum(ks) + sum(kd) == 0:
            continue
        Ks = [_cdiv(ks[c] + kd[c], MIXED_CW[c]) * MIXED_CW[c] for c in range(3)]
        Qs = [3 * (ks[c] + kd[c]) for c in range(3)]
        if 3 * sum(Ks) > _lib.STREAM_BUF:
            raise _lib.Pq3dError("a block's t (%d values) exceeds the stream buffer" % (3 * sum(Ks)))
        rec_off, rec_voff, rec_tp, rec_nch, rec_sb = [0] * 3, [0] * 3, [0] * 3, [0] * 3, [0] * 3
        for c in range(3):
            counts[c] += (ks[c], kd[c])
            cw = MIXED_CW[c]
            lr_bytes += Qs[c] * ((hi - lo) + nn) * MIXED_BYTES[c] + (Qs[c] * 4 if c else 0)
            rec_off[c], rec_voff[c] = u_off[c], v_off[c]
            if Ks[c] == 0:
                continue
            if Qs[c] * 16 > _lib.STREAM_STAGE_BYTES:
                raise _lib.Pq3dError("a block's term class has %d V rows, more than one stream stage holds" % Qs[c])
            lead = b.col.start % cw
            ngv = _cdiv(nn + lead, cw)
            gch = VCOLS // cw
            nch = _cdiv(ngv, gch)
            for ch in range(nch):
                g0, g1 = ch * gch, min(ngv, (ch + 1) * gch)
                ta.append(_task(1, off=v_off[c], cls=c, m=Qs[c], g0=g0, g1=g1, c0=b.col.start - lead,
                                out=tp + ch * Qs[c], kS3=3 * ks[c]))
                ba.append((g1 - g0) * (Qs[c] * 16 + 8 * cw))
            rec_tp[c], rec_nch[c] = tp, nch
            tp += nch * Qs[c]
            if c:
                rec_sb[c] = sb
                sb += Qs[c]
            u_off[c] += Ks[c] * m * 3
            v_off[c] += Qs[c] * ngv * cw
        gather.append((Ks, ks, kd, Qs, rec_tp, rec_nch, rec_sb, tb, 0))
        for r0 in range(lo, hi, _lib.STREAM_ROWS):
            r1 = min(hi, r0 + _lib.STREAM_ROWS)
            tb_.append(_task(2, off=rec_off[0], off1=rec_off[1], off2=rec_off[2], m=m, r0=r0, r1=r1, out=slot - lo,
                             K0=Ks[0], K1=Ks[1], K2=Ks[2], tb=tb))
            bb.append(3 * (r1 - r0) * 16 * (Ks[0] // 4 + Ks[1] // 8 + Ks[2] // 16) + 12 * sum(Ks))
        tb += 3 * sum(Ks)
        slot_rows.append((slot, b.row.start + lo, hi - lo))
        for p in (0, 1):
            pack.append((bi, p, rec_off, rec_voff, ks, kd, Qs, Ks, rec_sb))
        slot += hi - lo
    A = _leaf_lists(struct, slot_rows)
    tasks_a, cta_a, ncta_a = _balance(ta, ba, ncta)
    tasks_b, cta_b, ncta_b = _balance(tb_, bb, ncta)
    dense_entries = int(np.sum(dense_recs["m"].astype(np.int64) * dense_recs["n"])) if len(dense_recs) else 0
    A.update(ditems=_rec([], _lib.DENSE_ITEM), vitems=_rec([], _lib.V_ITEM), utasks=_rec([], _lib.U_TASK_M),
             n_ditems=0, n_vitems=0, n_utasks=0, n_slots=slot, n_tpart=tp, n_scales=sb, kmax=0, u_sizes=u_off,
             v_sizes=v_off, pack=pack, stream=True, class_terms=counts,
             tasks_a=tasks_a, cta_a=cta_a, ncta_a=ncta_a, tasks_b=tasks_b, cta_b=cta_b, ncta_b=ncta_b,
             gather=_rec(gather, _lib.T_GATHER), n_gather=len(gather), n_tfull=tb,
             alg_bytes=dense_entries * 6 * 4 + lr_bytes + 2 * n * 4 + 3 * n * 8)
    return A


def _rec(rows, dt):
    return np.array(rows, dtype=dt) if rows else np.zeros(1, dtype=dt)


# ----------------------------------------------------------------------------- plan cache

PLAN_CACHE = os.path.join(os.path.dirname(os.path.abspath(__file__)), "plan_cache.json")
_plan_cache = None


def _entry_n(e):
    """Element count of the workload a cache entry was tuned on."""
    if "n" in e:
        return int(e["n"])
    import re
    m = re.search(r"\((\d+) triangles\)", e.get("workload", ""))
    return int(m.group(1)) if m else None


def plan_cache_entry(gpu_name, dtype, n=None):
    """Work-item shapes measured by pyquake3d_b200.autotune for this GPU model and
    storage, or None.  The cache may hold entries tuned on workloads of several
    sizes (a list); the one tuned on the size closest to n (log scale) is used."""
    global _plan_cache
    if _plan_cache is None:
        _plan_cache = {}
        if os.path.exists(PLAN_CACHE):
            import json
            with open(PLAN_CACHE) as f:
                _plan_cache = json.load(f)
    ent = _plan_cache.get(gpu_name, {}).get(dtype)
    if ent is None or isinstance(ent, dict):
        return ent
    sized = [e for e in ent if _entry_n(e)]
    if n is None or not sized:
        return ent[0] if ent else None
    return min(sized, key=lambda e: abs(np.log(_entry_n(e) / float(n))))


# ----------------------------------------------------------------------------- device operator

DTYPES = {"fp64": 0, "fp32": 1, "bf16": 2, "mixed": 3}
# default term-class tolerance of the mixed storage: a quantised term may move a row
# by at most 2^-22 of its near-field absolute row sum (4 ulps of FP32 storage)
MIXED_TOL = 2.0 ** -22
_CW_DENSE = {0: 2, 1: 4, 2: 4, 3: 4}
_CW_LR = {0: 2, 1: 4, 2: 8}


def _cdiv(a, b):
    return (a + b - 1) // b


class DeviceHMatrix:
    """The packed operator on one GPU.

    assemble() computes dense blocks and ACA factors in FP64 on the device;
    plan(dtype) packs them into the matvec layout of one storage precision
    ("fp64": FP64 everywhere; "fp32": FP32 everywhere; "bf16": FP32 dense,
    BF16 low rank).  matvec(x_dev, dtype) returns y (n x 3, FP64, tree order)."""

    # work-item shapes per storage code (0 FP64, 1 FP32, 2 BF16 low rank, 3 mixed): these
    # defaults unless the plan cache written by pyquake3d_b200.autotune has an entry for
    # this GPU and storage (shapes()).
    DENSE_CHUNK_GROUPS = {0: 64, 1: 16, 2: 16, 3: 16}   # column groups per dense work item
    V_CHUNK_GROUPS = {0: 128, 1: 32, 2: 32, 3: 32}      # column groups per V work item
    U_ROWS = 512                                        # rows per U task (one CTA)

    def __init__(self, struct, xg, ev, nodes, tri, mu, lam, device="cuda", aca_tol=0.01, aca_rel=False,
                 aca_seed=0, kcap=96, ws_budget_bytes=8 << 30, keep_factors=False, halfspace=0,
                 mixed_tol=MIXED_TOL):
        """halfspace: 0 full space; 1 half space, a triangle side along z adds no
        free-surface term; 2 half space with the side handling of the reference's
        compiled library (the values its H-matrix assembly uses).  mixed_tol: the
        term-class tolerance of the "mixed" storage (classify_blocks)."""
        self.mixed_tol = float(mixed_tol)
        self.mixed_stream = False      # mixed storage: True selects the bulk-copy (streamed) kernels
        self.use_plan_cache = True
        import torch
        self.torch = torch
        self.L = _lib.load()
        self.s = struct
        self.n = struct.n
        self.mu, self.lam = float(mu), float(lam)
        self.dev = torch.device(device)
        self.aca_tol, self.aca_rel, self.aca_seed = float(aca_tol), bool(aca_rel), int(aca_seed)
        self.kcap = int(kcap)
        self.keep_factors = bool(keep_factors)
        self.ws_budget = int(ws_budget_bytes)
        f64 = dict(dtype=torch.float64, device=self.dev)
        self.xg = torch.tensor(np.ascontiguousarray(xg), **f64)
        self.ev = torch.tensor(np.ascontiguousarray(ev), **f64)
        self.nodes = torch.tensor(np.ascontiguousarray(nodes), **f64)
        self.tri = torch.tensor(np.ascontiguousarray(tri, dtype=np.int64), dtype=torch.int64, device=self.dev)
        self.perm = torch.tensor(struct.perm.astype(np.int32), dtype=torch.int32, device=self.dev)
        self.iperm = torch.tensor(struct.iperm.astype(np.int32), dtype=torch.int32, device=self.dev)
        rb = self.L.pq3d_src_record_bytes()
        self.rec = torch.empty((self.n * rb + 7) // 8, **f64)
        self._stream = _lib.stream_ptr()
        check(self.L.pq3d_src_records(ptr(self.nodes), ptr(self.tri), self.n, ptr(self.rec), self._stream),
              "pq3d_src_records")
        self.halfspace = int(halfspace)
        self.hs = None
        if self.halfspace:
            hb = self.L.pq3d_hs_record_bytes()
            self.hs = torch.empty((self.n * hb + 7) // 8, **f64)
            check(self.L.pq3d_hs_records(ptr(self.nodes), ptr(self.tri), self.n, ptr(self.hs), self._stream),
                  "pq3d_hs_records")
        self.dense_blocks = [b for b in struct.blocks if not b.aca]
        self.aca_blocks = [b for b in struct.blocks if b.aca]
        self.plans = {}
        self.assembled = False
        self.timings = {}

    # ------------------------------------------------------------------ assembly
    def assemble(self, want=("fp64", "bf16")):
        """Dense near field + ACA factors (FP64 on device), then pack for each dtype."""
        import time
        torch = self.torch
        want = tuple(want)
        torch.cuda.synchronize()
        t0 = time.perf_counter()
        self._assemble_dense(want)
        torch.cuda.synchronize()
        t1 = time.perf_counter()
        self._run_aca()
        torch.cuda.synchronize()
        t2 = time.perf_counter()
        self.timings.update(dense_s=t1 - t0, aca_s=t2 - t1)
        for d in want:
            self.plan(d)
        torch.cuda.synchronize()
        self.timings["pack_s"] = time.perf_counter() - t2
        self.assembled = True
        if not self.keep_factors:
            # packed copies are all that the matvec needs: release the FP64 ACA workspaces
            self.aca_ws = [None] * len(self.aca_ws)
            torch.cuda.empty_cache()
        return self

    def _assemble_dense(self, want):
        torch = self.torch
        need64 = "fp64" in want
        need32 = any(d in want for d in ("fp32", "bf16", "mixed"))
        recs, off64, off32 = dense_layout(self.dense_blocks)
        order = np.argsort(-(recs["m"].astype(np.int64) * recs["n"]), kind="stable")
        self.dense_recs = recs
        self.dense64 = torch.zeros(max(off64, 1), dtype=torch.float64, device=self.dev) if need64 else None
        self.dense32 = torch.zeros(max(off32, 1), dtype=torch.float32, device=self.dev) if need32 else None
        if len(recs):
            d_recs = torch.from_numpy(recs[order].view(np.uint8)).to(self.dev)
            check(self.L.pq3d_dense_assemble(ptr(self.xg), ptr(self.ev), ptr(self.rec), ptr(self.perm), ptr(d_recs),
                                             len(recs), self.mu, self.lam, ptr(self.dense64), ptr(self.dense32),
                                             ptr(self.hs), self.halfspace, self._stream), "pq3d_dense_assemble")
            torch.cuda.synchronize()

    def _run_aca(self):
        """Batched ACA over all admissible blocks; ranks and FP64 factors kept per task."""
        torch = self.torch
        if not self.aca_blocks:
            self.aca_ranks, self.aca_flags = np.zeros(0, np.int32), np.zeros(0, np.int32)
            self.aca_ws, self.task_ws = [], workspace_table(0)
            return
        starts = getattr(self.s, "aca_starts", None)
        if starts is None:
            starts = aca_start_indices(self.s.blocks, self.aca_seed)
        blocks = self.aca_blocks
        nt = 2 * len(blocks)                     # tasks: strike and dip pass of every block
        m, n = (np.repeat(v, 2) for v in _block_geometry(blocks)[:2])
        start = np.array(starts, dtype=np.int64).reshape(-1, 2)
        # row and column lists stored separately
        self.rowlist = torch.from_numpy(np.concatenate([b.row.indices for b in blocks]).astype(np.int32)).to(self.dev)
        self.collist = torch.from_numpy(np.concatenate([b.col.indices for b in blocks]).astype(np.int32)).to(self.dev)
        ro, co = self._row_offsets()
        self.aca_ranks = np.zeros(nt, dtype=np.int32)
        self.aca_flags = np.zeros(nt, dtype=np.int32)
        self.aca_ws = []                         # workspaces; a task's is task_ws["ws"][task]
        self.task_ws = workspace_table(nt)
        kcap = np.minimum(np.minimum(m, n), self.kcap)
        pending = np.arange(nt)
        while len(pending):
            # batches bounded by the workspace budget, largest tasks first
            pending = pending[np.argsort(-(m + n)[pending], kind="stable")]
            retry = []
            i0 = 0
            while i0 < len(pending):
                t = pending[i0:]
                end = np.cumsum(3 * kcap[t] * (m[t] + n[t]) + 6 * (m[t] + n[t]))        # pq3d_aca_ws_doubles
                t = t[:max(1, int(np.searchsorted(end * 8, self.ws_budget, side="right")))]
                end = end[:len(t)]
                i0 += len(t)
                rec = np.zeros(len(t), dtype=_lib.ACA_TASK)
                for k, v in dict(rows_off=ro[t // 2], cols_off=co[t // 2], ws_off=np.concatenate([[0], end[:-1]]), m=m[t],
                                 n=n[t], kmax=kcap[t], pass_=t % 2, iref0=start[t, 0], jref0=start[t, 1]).items():
                    rec[k] = v
                if int(end[0]) != self.L.pq3d_aca_ws_doubles(int(m[t[0]]), int(n[t[0]]), int(kcap[t[0]])):
                    raise _lib.Pq3dError("ACA workspace layout mismatch")
                max_mn = int(max(m[t].max(), n[t].max()))
                ws = torch.empty(int(end[-1]), dtype=torch.float64, device=self.dev)
                d_rec = torch.from_numpy(rec.view(np.uint8)).to(self.dev)
                d_out = torch.zeros((2, len(t)), dtype=torch.int32, device=self.dev)      # ranks, flags
                check(self.L.pq3d_aca_batched(ptr(self.xg), ptr(self.ev), ptr(self.rec), ptr(self.rowlist),
                                              ptr(self.collist), ptr(d_rec), len(t), ptr(ws), self.mu, self.lam,
                                              self.aca_tol, 1 if self.aca_rel else 0, max_mn, ptr(d_out[0]),
                                              ptr(d_out[1]), ptr(self.hs), self.halfspace, self._stream),
                      "pq3d_aca_batched")
                ranks, flags = d_out.cpu().numpy()
                if (flags & 8).any():
                    raise _lib.Pq3dError("pq3d_aca_batched: a task has more rows or columns than the batch's "
                                         "max_mn (not run)")
                # flag 4 (every remaining pivot candidate excluded) ends a task normally: the
                # factors found so far are the block's approximation, as in the reference loop
                full = np.minimum(m[t], n[t])
                again = (flags & 1 != 0) & (kcap[t] < full)
                done = t[~again]
                self.aca_ranks[done] = ranks[~again]
                self.aca_flags[done] = flags[~again]
                self.task_ws["ws"][done] = len(self.aca_ws)
                self.task_ws["off"][done] = rec["ws_off"][~again]
                self.task_ws["kmax"][done] = kcap[done]
                self.aca_ws.append(ws)
                kcap[t[again]] = np.minimum(2 * kcap[t], full)[again]
                retry.append(t[again])
            pending = np.concatenate(retry)

    def ranks(self):
        """(kS, kD) per ACA block."""
        r = self.aca_ranks.reshape(-1, 2)
        return r[:, 0], r[:, 1]

    # ------------------------------------------------------------------ packing / plans
    def plan(self, dtype):
        if dtype in self.plans:
            return self.plans[dtype]
        if self.assembled and not self.keep_factors and self.aca_blocks:
            raise _lib.Pq3dError("ACA factors were released after assembly; request every precision in "
                                 "assemble(want=...) or construct with keep_factors=True")
        torch = self.torch
        code = DTYPES[dtype]
        if code == 3:
            return self._plan_mixed()
        A = self.plan_arrays(dtype)
        lr_dtype = torch.float64 if code == 0 else (torch.float32 if code == 1 else torch.bfloat16)
        Ubuf = torch.zeros(max(A["u_size"], 8), dtype=lr_dtype, device=self.dev)
        Vbuf = torch.zeros(max(A["v_size"], 8), dtype=lr_dtype, device=self.dev)
        # pack every ACA task into the layout, one launch per workspace batch
        K = A["pack"]
        if len(K) == 0:
            return self._finish_plan(dtype, A, Ubuf, Vbuf)
        ti = 2 * K["bi"] + K["pass_"]
        rec = self._task_records(_lib.PACK_TASK, ti)
        for k in ("u_off", "v_off", "kS", "kD", "K", "Q"):
            rec[k] = K[k]
        for wi, d_rec, k in self._by_workspace(rec, ti):
            check(self.L.pq3d_aca_pack(ptr(d_rec), k, ptr(self.aca_ws[wi]), ptr(self.rowlist), ptr(self.collist),
                                       ptr(self.iperm), code, ptr(Ubuf), ptr(Vbuf), self._stream), "pq3d_aca_pack")
        return self._finish_plan(dtype, A, Ubuf, Vbuf)

    def shapes(self, dtype):
        """(dense_chunk, v_chunk, u_rows) of a storage: an explicit override
        (set_shapes), else the plan cache's entry for this GPU, else the defaults."""
        code = DTYPES[dtype]
        ov = getattr(self, "_shape_override", {}).get(dtype)
        if ov is not None:
            return ov
        if self.use_plan_cache:
            ent = plan_cache_entry(self.torch.cuda.get_device_name(self.dev), dtype, self.n)
            if ent is not None:
                return int(ent["dense_chunk"]), int(ent["v_chunk"]), int(ent["u_rows"])
        return self.DENSE_CHUNK_GROUPS[code], self.V_CHUNK_GROUPS[code], self.U_ROWS

    def set_shapes(self, dtype, dense_chunk, v_chunk, u_rows):
        """Rebuild one storage's work items with other shapes; the packed operator data
        does not depend on them and is kept (the autotuner's move)."""
        if not hasattr(self, "_shape_override"):
            self._shape_override = {}
        self._shape_override[dtype] = (int(dense_chunk), int(v_chunk), int(u_rows))
        P = self.plans.get(dtype)
        if P is None:
            return None
        if DTYPES[dtype] == 3:
            offs = np.concatenate([[0], np.cumsum(np.asarray(self.aca_ranks, np.int64))])
            A = self._mixed_arrays(self.mixed_tmap & 3, offs)
            A["mixed"] = P["mixed"]
        else:
            A = self.plan_arrays(dtype)
        del self.plans[dtype]
        return self._finish_plan(dtype, A, P["U"], P["V"])

    def plan_arrays(self, dtype):
        """Host work-item arrays of one storage precision (deterministic from the
        structure and the ACA ranks)."""
        code = DTYPES[dtype]
        kS, kD = self.ranks()
        dc, vc, ur = self.shapes(dtype)
        return build_plan_arrays(self.s, self.dense_recs, kS, kD, code, dc, vc, ur)

    def _task_records(self, dtype, ti):
        """Pack records (PACK_TASK or PACK_TASK_M) of tasks ti: workspace, lists, sizes, rank."""
        m, n, r0, c0, _, _ = (v[ti // 2] for v in _block_geometry(self.aca_blocks))
        ro, co = (v[ti // 2] for v in self._row_offsets())
        rec = np.zeros(len(ti), dtype=dtype)
        for k, v in dict(ws_off=self.task_ws["off"][ti], rows_off=ro, cols_off=co, m=m, n=n, kmax=self.task_ws["kmax"][ti],
                         k=self.aca_ranks[ti], pass_=ti % 2, r0=r0, c0=c0, zeroB=self.aca_flags[ti] & 2 != 0).items():
            rec[k] = v
        return rec

    def _by_workspace(self, rec, ti):
        """(workspace, records on the device, their number) per workspace batch."""
        ws = self.task_ws["ws"][ti]
        for wi in np.unique(ws):
            r = rec[ws == wi]
            yield int(wi), self.torch.from_numpy(r.view(np.uint8)).to(self.dev), len(r)

    def _plan_mixed(self):
        """Mixed storage (code 3): FP32 dense near field; ACA terms in FP32 / FP16 / INT8
        classes chosen from their weights against the near-field row sums."""
        torch = self.torch
        if self.dense32 is None:
            raise _lib.Pq3dError("the mixed plan needs the FP32 dense blocks: request it in assemble(want=...)")
        L = self.L
        st = self._stream
        offs, tmap = np.zeros(1, np.int64), np.zeros(1, np.int32)
        if self.aca_blocks:
            rec, offs, tmap = self._term_classes()
        self.mixed_tmap = tmap[:int(offs[-1])]
        A = self._mixed_arrays(self.mixed_tmap & 3, offs)
        # INT8-class entries are stored as b + 128: the fill 128 decodes to zero, so padding
        # columns (a block's lead and tail columns, its K padding) contribute nothing
        tdt, fill = (torch.float32, torch.float16, torch.uint8), (0, 0, 128)
        Ub = [torch.full((max(int(A["u_sizes"][c]), 16),), fill[c], dtype=tdt[c], device=self.dev) for c in range(3)]
        Vb = [torch.full((max(int(A["v_sizes"][c]), 16),), fill[c], dtype=tdt[c], device=self.dev) for c in range(3)]
        scales = torch.zeros(max(A["n_scales"], 4), dtype=torch.float32, device=self.dev)
        d_tmap = torch.from_numpy(tmap).to(self.dev)
        K = A["pack"]                              # blocks with terms
        if len(K):
            if A.get("stream"):
                K = np.array([tuple(k) for k in K], dtype=_PACK_M)
            ti = 2 * K["bi"] + K["pass_"]
            rec = rec[ti]
            for k in ("u_off", "v_off", "kS", "kD", "Q", "K", "sb"):
                rec[k] = K[k]
            for wi, d_rec, k in self._by_workspace(rec, ti):
                check(L.pq3d_aca_pack_mixed(ptr(d_rec), k, ptr(self.aca_ws[wi]), ptr(self.rowlist), ptr(self.collist),
                                            ptr(self.iperm), ptr(d_tmap), ptr(Ub[0]), ptr(Ub[1]), ptr(Ub[2]), ptr(Vb[0]),
                                            ptr(Vb[1]), ptr(Vb[2]), ptr(scales), st), "pq3d_aca_pack_mixed")
        A["mixed"] = dict(U=Ub, V=Vb, scales=scales, tol=self.mixed_tol, class_terms=A["class_terms"].tolist())
        return self._finish_plan("mixed", A, Ub[0], Vb[0])

    def _term_classes(self):
        """Packing records of all tasks, the tasks' term offsets, and every term's class and
        position among its task's terms of that class (class | position << 2), from the terms'
        weights."""
        torch = self.torch
        n = self.n
        L = self.L
        st = self._stream
        # near-field absolute row sums (tree order), largest component
        R3 = torch.zeros(3 * n, dtype=torch.float64, device=self.dev)
        recs = self.dense_recs
        if len(recs):
            d_recs = torch.from_numpy(np.ascontiguousarray(recs).view(np.uint8)).to(self.dev)
            check(L.pq3d_nearfield_rowabs(ptr(self.dense32), ptr(d_recs), len(recs), n, ptr(R3), st),
                  "pq3d_nearfield_rowabs")
        R = R3.view(3, n).max(dim=0).values.contiguous()
        # every task's weights, and the offset of its terms (tasks in block order, strike first)
        tasks = np.arange(2 * len(self.aca_blocks))
        offs = np.concatenate([[0], np.cumsum(self.aca_ranks, dtype=np.int64)])
        rec = self._task_records(_lib.PACK_TASK_M, tasks)
        rec["tmap_off"] = offs[:-1]
        w = torch.zeros(max(int(offs[-1]), 1), dtype=torch.float64, device=self.dev)
        for wi, d_rec, k in self._by_workspace(rec, tasks):
            check(L.pq3d_aca_term_weights(ptr(d_rec), k, ptr(self.aca_ws[wi]), ptr(self.rowlist), ptr(self.iperm),
                                          ptr(R), ptr(w), st), "pq3d_aca_term_weights")
        # every term's class, and its position within its task's terms of that class
        cls = classify_blocks(w.cpu().numpy()[:int(offs[-1])], offs, self.mixed_tol)
        key = 3 * np.repeat(tasks, self.aca_ranks) + cls
        order = np.argsort(key, kind="stable")
        pos = np.empty(len(cls), np.int64)
        pos[order] = _expand(np.bincount(key, minlength=3 * len(tasks)))[1]
        tmap = np.zeros(max(len(cls), 1), np.int32)
        tmap[:len(cls)] = cls | (pos << 2)
        return rec, offs, tmap

    def _mixed_arrays(self, cls, offs):
        """Plan arrays from every term's class (task order) and the tasks' term offsets."""
        dc, vc, ur = self.shapes("mixed")
        if self.mixed_stream:
            ncta = self.L.pq3d_stream_ctas()
            if ncta > 0:
                try:
                    cls_lists = [(cls[offs[i]:offs[i + 1]], cls[offs[i + 1]:offs[i + 2]])
                                 for i in range(0, len(offs) - 1, 2)]
                    return build_plan_arrays_mixed(self.s, self.dense_recs, cls_lists, dc, vc, ur, stream=True,
                                                   ncta=ncta)
                except _lib.Pq3dError:
                    pass               # a term class too large for a stream stage: the plain kernels
        nw = self.L.pq3d_vmix_ctas()
        return build_plan_arrays_mixed(self.s, self.dense_recs, None, dc, vc, ur,
                                       nwarps=8 * nw if nw > 0 else VMIX_WARPS, counts=class_counts(cls, offs))

    def install_mixed(self, tmap, U, V, scales):
        """Register a mixed plan whose class arrays come from elsewhere (an operator
        checkpoint): tmap holds every term's class code (bits 0-1) in task order."""
        offs = np.concatenate([[0], np.cumsum(np.asarray(self.aca_ranks, np.int64))])
        self.mixed_tmap = np.asarray(tmap, np.int32)
        A = self._mixed_arrays(self.mixed_tmap & 3, offs)
        A["mixed"] = dict(U=list(U), V=list(V), scales=scales, tol=self.mixed_tol,
                          class_terms=A["class_terms"].tolist())
        return self._finish_plan("mixed", A, U[0], V[0])

    def install_plan(self, dtype, Ubuf, Vbuf):
        """Register a plan whose packed low-rank buffers were produced elsewhere (an
        operator checkpoint); dense blocks must already be in dense64/dense32."""
        return self._finish_plan(dtype, self.plan_arrays(dtype), Ubuf, Vbuf)

    def _finish_plan(self, dtype, A, Ubuf, Vbuf):
        torch = self.torch
        code = DTYPES[dtype]

        def dev_rec(a):
            return torch.from_numpy(np.ascontiguousarray(a).view(np.uint8)).to(self.dev)

        acc = torch.float64 if code == 0 else torch.float32
        dense = self.dense64 if code == 0 else self.dense32
        if A["n_ditems"] > 0 and dense is None:
            raise _lib.Pq3dError(f"dense blocks of the {dtype} plan were not assembled")
        P = dict(code=code, dtype=dtype, acc=acc,
                 dense=self.dense64 if code == 0 else self.dense32, U=Ubuf, V=Vbuf,
                 ditems=dev_rec(A["ditems"]), vitems=dev_rec(A["vitems"]), utasks=dev_rec(A["utasks"]),
                 leaf_of_row=torch.tensor(A["leaf_of_row"], device=self.dev),
                 leaf_ptr=torch.tensor(A["leaf_ptr"], device=self.dev),
                 leaf_off=torch.tensor(A["leaf_off"], device=self.dev),
                 n_ditems=A["n_ditems"], n_vitems=A["n_vitems"], n_utasks=A["n_utasks"],
                 n_slots=A["n_slots"], n_tpart=A["n_tpart"], kmax=A["kmax"])
        P["slots"] = torch.empty(3 * max(P["n_slots"], 1), dtype=acc, device=self.dev)
        P["tpart"] = torch.empty(max(P["n_tpart"], 1), dtype=acc, device=self.dev)
        hp = np.zeros(1, dtype=_lib.HM_PLAN)
        hp["n"] = self.n
        hp["dtype"] = code
        for k in ("dense", "U", "V", "ditems", "vitems", "utasks", "leaf_of_row", "leaf_ptr", "leaf_off"):
            hp[k] = P[k].data_ptr() if P[k] is not None else 0
        for k in ("n_ditems", "n_vitems", "n_utasks", "n_slots", "n_tpart", "kmax"):
            hp[k] = P[k]
        if code == 3:
            M = A["mixed"]
            P["mixed"] = M
            hp["U16"], hp["U8"] = M["U"][1].data_ptr(), M["U"][2].data_ptr()
            hp["V16"], hp["V8"] = M["V"][1].data_ptr(), M["V"][2].data_ptr()
            hp["scales"] = M["scales"].data_ptr()
            P["status"] = torch.zeros(1, dtype=torch.int32, device=self.dev)
            hp["status"] = P["status"].data_ptr()
            hp["stream"] = 1 if A.get("stream") else 0
            P["stream"] = bool(A.get("stream"))
            if not P["stream"]:
                P["vrows"] = dev_rec(A["vrows"])
                hp["vrows"] = P["vrows"].data_ptr()
                P["vwarp"] = torch.tensor(A["vwarp"], dtype=torch.int32, device=self.dev)
                hp["vwarp"], hp["n_vwarp"] = P["vwarp"].data_ptr(), len(A["vwarp"]) - 1
            if P["stream"]:
                for k in ("tasks_a", "tasks_b", "gather"):
                    P[k] = dev_rec(A[k])
                    hp[k] = P[k].data_ptr()
                for k in ("cta_a", "cta_b"):
                    P[k] = torch.tensor(A[k], dtype=torch.int32, device=self.dev)
                    hp[k] = P[k].data_ptr()
                P["tfull"] = torch.zeros(max(A["n_tfull"], 4), dtype=torch.float32, device=self.dev)
                hp["tfull"] = P["tfull"].data_ptr()
                hp["n_gather"], hp["ncta_a"], hp["ncta_b"] = A["n_gather"], A["ncta_a"], A["ncta_b"]
        P["host_plan"] = hp
        P["alg_bytes"] = A["alg_bytes"]
        P["stored_bytes"] = (P["dense"].numel() * P["dense"].element_size() if P["dense"] is not None else 0) + \
            Ubuf.numel() * Ubuf.element_size() + Vbuf.numel() * Vbuf.element_size()
        if code == 3:
            P["stored_bytes"] += sum(t.numel() * t.element_size() for t in P["mixed"]["U"][1:] + P["mixed"]["V"][1:])
        self.plans[dtype] = P
        return P

    def _row_offsets(self):
        """Offsets of every ACA block's rows and columns in rowlist and collist."""
        m, n = _block_geometry(self.aca_blocks)[:2]
        return _offsets(m)[0], _offsets(n)[0]

    def kernel_status(self, dtype):
        """Status word of a plan's streamed kernels: 0, 1 after a timed-out wait, 2 after a
        task of a size they do not take (nothing of the kind is expected)."""
        P = self.plans.get(dtype)
        return int(P["status"].item()) if P is not None and "status" in P else 0

    def new_x(self, dtype):
        """Zero deficit buffer (tree order, device layout of pack_x) for the given plan."""
        P = self.plan(dtype)
        return self.torch.zeros(4 * x_stride(self.n), dtype=P["acc"], device=self.dev)

    def matvec(self, x, dtype, y=None, add=(None, None, None), stream=None, slots_only=False):
        """y[i, c] = sum_j K_c(i, j) x  (tree order, FP64 output).  slots_only: write the
        per-row partial sums only (the step kernel reduces them)."""
        P = self.plan(dtype)
        if y is None and not slots_only:
            y = self.torch.empty((self.n, 3), dtype=self.torch.float64, device=self.dev)
        P["slots_owner"] = None     # the slots now hold this call's products
        st = _lib.stream_ptr(stream)
        check(self.L.pq3d_hmatvec(P["host_plan"].ctypes.data, ptr(x), ptr(P["slots"]), ptr(P["tpart"]),
                                  ptr(add[0]), ptr(add[1]), ptr(add[2]), None if slots_only else ptr(y), st),
              "pq3d_hmatvec")
        return y

    def apply(self, x1, x2, dtype="fp64"):
        """Host convenience: (y1, y2, yB) in element order for deficits x1, x2 (element order)."""
        torch = self.torch
        P = self.plan(dtype)
        xt = pack_x(np.asarray(x1)[self.s.perm], np.asarray(x2)[self.s.perm], self.n)
        x = torch.tensor(xt, dtype=P["acc"], device=self.dev)
        y = self.matvec(x, dtype).cpu().numpy()
        out = np.empty_like(y)
        out[self.s.perm] = y
        return out[:, 0], out[:, 1], out[:, 2]


def export_blocks(op):
    """Host copy of the FP64 operator per block, in the reference's block format:
    list of ("dense", rows, cols, M[6][m][n]) or ("aca", rows, cols, S, D) with
    S/D dicts of U1 V1 U2 V2 UB VB (rows/cols are element ids in tree order).
    Used to run the reference's CPU step on the same operator."""
    P = op.plan("fp64")
    perm = op.s.perm
    dense = op.dense64.cpu().numpy() if op.dense64 is not None else None
    U = P["U"].cpu().numpy()
    V = P["V"].cpu().numpy()
    out = []
    recs = op.dense_recs
    for i in range(len(recs)):
        m, n, r0, c0 = (int(recs[k][i]) for k in ("m", "n", "r0", "c0"))
        lead = c0 % 2
        ng = _cdiv(n + lead, 2)
        a = dense[int(recs["off64"][i]):int(recs["off64"][i]) + ng * m * 12].reshape(ng, 3, 2, m, 2)
        # (group, comp, slip, row, t) -> (slip, comp, row, col)
        M = a.transpose(2, 1, 3, 0, 4).reshape(2, 3, m, ng * 2)[:, :, :, lead:lead + n].reshape(6, m, n)
        out.append(("dense", perm[r0:r0 + m], perm[c0:c0 + n], np.ascontiguousarray(M)))
    kS, kD = op.ranks()
    u_off = v_off = 0
    for bi, b in enumerate(op.aca_blocks):
        m, n = len(b.row.indices), len(b.col.indices)
        ks, kd = int(kS[bi]), int(kD[bi])
        rows = perm[b.row.start:b.row.start + m]
        cols = perm[b.col.start:b.col.start + n]
        if ks + kd == 0:
            z = dict(U1=np.zeros((m, 0)), V1=np.zeros((0, n)), U2=np.zeros((m, 0)), V2=np.zeros((0, n)), UB=[], VB=[])
            out.append(("aca", rows, cols, z, dict(z)))
            continue
        K = _cdiv(ks + kd, 2) * 2
        Q = 3 * (ks + kd)
        lead = b.col.start % 2
        ngv = _cdiv(n + lead, 2)
        Ub = U[u_off:u_off + K // 2 * m * 6].reshape(K // 2, 3, m, 2).transpose(1, 2, 0, 3).reshape(3, m, K)
        Vb = V[v_off:v_off + ngv * Q * 2].reshape(ngv, Q, 2).transpose(1, 0, 2).reshape(Q, ngv * 2)[:, lead:lead + n]
        S, D = {}, {}
        for c, (un, vn) in enumerate((("U1", "V1"), ("U2", "V2"), ("UB", "VB"))):
            S[un] = np.ascontiguousarray(Ub[c, :, :ks])
            S[vn] = np.ascontiguousarray(Vb[c * ks:(c + 1) * ks])
            D[un] = np.ascontiguousarray(Ub[c, :, ks:ks + kd])
            D[vn] = np.ascontiguousarray(Vb[3 * ks + c * kd:3 * ks + (c + 1) * kd])
        out.append(("aca", rows, cols, S, D))
        u_off += K // 2 * m * 6
        v_off += ngv * Q * 2
    return out
