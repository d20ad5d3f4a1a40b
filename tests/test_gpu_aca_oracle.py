"""Blocks of every ACA kernel (one CTA, clusters of two and of eight, at and beside 256 and 1,024 rows
or columns), full and half space, against the oracle's ACA run on the device's own entries of
the same block, and against the stop rule evaluated from the device's own factors.

 * ranks are the oracle's, and the first terms' A1 factors to 1e-9 of their largest entry;
 * the products U V of all three operators agree within 2 tol of the A1 product's largest entry:
   a term is about tol times the first one when it is added, and where two pivot candidates
   are nearly equal the entries' last bits pick one or the other (test_gpu_aca_rel.py);
 * while the factors are the oracle's, a term's row and column vanish in the residual at the
   oracle's pivots: to 1e-9 of the block's largest entry;
 * ||u_k|| ||v_k|| <= tol ||S_k||_F holds at no term before the last, and at the last one unless the
   block ended as the oracle's did, at a pivot below 1e-4 or with all rows used; the norm summed
   here in FP64 from the same factors: at most 2,400 terms and 300 cross terms, 1e-6 of slack.

Blocks of more than 128 terms, the cross terms reduced at a time, keep the stop rule too."""
import numpy as np
import pytest

import qd_oracle

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

SIZES = [(33, 33), (256, 255), (257, 256), (64, 1024), (1025, 300), (700, 1100)]


@pytest.fixture(scope="module")
def fault(tmp_path_factory):
    from pyquake3d_b200 import QDsim, meshgen, read_mshV2
    msh, para = meshgen.make_case("thrust20k", str(tmp_path_factory.mktemp("acaor")), n_target=5000)
    nodes, tris = read_mshV2(msh)
    sim = QDsim(tris, nodes, para)
    return sim, np.argsort(sim.xg[:, 0], kind="stable")


def _operator(sim, half):
    from pyquake3d_b200.hmatrix import DeviceHMatrix
    return DeviceHMatrix(sim.tree_block.struct, sim.xg, sim.eleVec, sim.nodelst, sim.elelst, sim.mu, sim.lambda_,
                         halfspace=half)


def _aca(op, blocks, tol, kmax):
    """(U, V, rank, flag) of (rows, cols, pass, iref0, jref0) tasks, relative stop, one batch."""
    from pyquake3d_b200 import _lib
    from pyquake3d_b200._lib import ptr
    L = op.L
    rec = np.zeros(len(blocks), dtype=_lib.ACA_TASK)
    ro = co = ws = 0
    for k, (r, c, p, i0, j0) in enumerate(blocks):
        km = min(len(r), len(c), kmax)
        rec[k] = (ro, co, ws, len(r), len(c), km, p, i0, j0)
        ro, co, ws = ro + len(r), co + len(c), ws + L.pq3d_aca_ws_doubles(len(r), len(c), km)
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to("cuda")
    rl, cl = (dev(np.concatenate([b[q] for b in blocks]).astype(np.int32)) for q in (0, 1))
    w = torch.full((ws,), float("nan"), dtype=torch.float64, device="cuda")
    out = torch.full((2, len(blocks)), -1, dtype=torch.int32, device="cuda")
    d = dev(rec.view(np.uint8))
    _lib.check(L.pq3d_aca_batched(ptr(op.xg), ptr(op.ev), ptr(op.rec), ptr(rl), ptr(cl), ptr(d), len(blocks), ptr(w),
                                  op.mu, op.lam, tol, 1, int(max(rec["m"].max(), rec["n"].max())), ptr(out[0]),
                                  ptr(out[1]), ptr(op.hs), op.halfspace, op._stream), "pq3d_aca_batched")
    w, (rank, flag), res = w.cpu().numpy(), out.cpu().numpy(), []
    for t, r, f in zip(rec, rank, flag):
        m, n, km = int(t["m"]), int(t["n"]), int(t["kmax"])
        a = t["ws_off"]
        res.append((w[a:a + 3 * km * m].reshape(km, 3, m)[:r], w[a + 3 * km * m:a + 3 * km * (m + n)].reshape(km, 3, n)[:r],
                    int(r), int(f)))
    return res


class _Entries:
    """The device's entries of one block, as the oracle's geometry hands them out."""

    def __init__(self, op, rows, cols):
        from pyquake3d_b200 import _lib
        from pyquake3d_b200._lib import ptr
        r = torch.from_numpy(np.repeat(rows, len(cols)).astype(np.int64)).to("cuda")
        c = torch.from_numpy(np.tile(cols, len(rows)).astype(np.int64)).to("cuda")
        o = torch.empty((len(r), 6), dtype=torch.float64, device="cuda")
        _lib.check(op.L.pq3d_traction_pairs(ptr(op.xg), ptr(op.ev), ptr(op.rec), ptr(r), ptr(c), len(r), op.mu, op.lam,
                                            ptr(o), ptr(op.hs), op.halfspace, op._stream), "pq3d_traction_pairs")
        self.K = np.ascontiguousarray(np.moveaxis(o.cpu().numpy().reshape(len(rows), len(cols), 2, 3), (2, 3), (0, 1)))
        self.ri, self.ci = ({int(e): k for k, e in enumerate(v)} for v in (rows, cols))

    def gf_block(self, rows, cols, which):
        i, j = [self.ri[int(e)] for e in rows], [self.ci[int(e)] for e in cols]
        return self.K[which - 1][:, i][:, :, j].copy()


def _stopped(u, v, tol):
    """Whether the last term meets the stop rule; none before it may."""
    uu, vv = u @ u.T, v @ v.T
    frob2 = np.cumsum([2.0 * (uu[k, :k] * vv[k, :k]).sum() + uu[k, k] * vv[k, k] for k in range(len(u))])
    step, lim = np.sqrt(np.diag(uu) * np.diag(vv)), tol * np.sqrt(np.abs(frob2))
    assert (step[:-1] > lim[:-1] * (1 - 1e-6)).all()
    return bool(step[-1] <= lim[-1] * (1 + 1e-6))


@pytest.mark.parametrize("half", [0, 2])
@pytest.mark.parametrize("tol", [1e-4, 1e-5])
def test_blocks_against_oracle(fault, half, tol):
    sim, order = fault
    op = _operator(sim, half)
    blocks = [(np.sort(order[:m]), np.sort(order[-n:]), p, m // 3, n // 4) for m, n in SIZES for p in (0, 1)]
    got = _aca(op, blocks, tol, 96)
    for (rows, cols, p, i0, j0), (U, V, r, flag) in zip(blocks, got):
        size = (len(rows), len(cols), p)
        E = _Entries(op, rows, cols)
        o = qd_oracle.aca_plus(E, rows, cols, p + 1, tol, i0, j0, rel=True)
        u1, v1 = np.asarray(o["U1"]), np.asarray(o["V1"])
        assert flag in (0, 2) and r == u1.shape[1], size
        assert np.abs(U[0, 0] - u1[:, 0]).max() <= 1e-9 * np.abs(u1[:, 0]).max(), size
        assert np.abs(V[0, 0] - v1[0]).max() <= 1e-9 * np.abs(v1[0]).max(), size
        scale = np.abs(u1 @ v1).max()
        for c, (un, vn) in enumerate((("U1", "V1"), ("U2", "V2"), ("UB", "VB"))):
            po = np.asarray(o[un]) @ np.asarray(o[vn]) if len(o[un]) else 0.0
            assert np.abs(U[:, c].T @ V[:, c] - po).max() <= 2 * tol * scale, size + (c,)
        A = E.K[p, 0]
        R, same = A.copy(), 0
        for k in range(r):
            R -= np.outer(U[k, 0], V[k, 0])
            if np.abs(U[k, 0] - u1[:, k]).max() > 1e-9 * np.abs(A).max():
                break
            same += 1
            I, J = int(o["prevI"][k]), int(o["prevJ"][k])
            assert max(np.abs(R[I]).max(), np.abs(R[:, J]).max()) <= 1e-9 * np.abs(A).max(), size + (k,)
        assert same >= 1
        assert _stopped(U[:, 0], V[:, 0], tol) == _stopped(u1.T, v1, tol), size


@pytest.mark.parametrize("half", [0, 2])
@pytest.mark.parametrize("m,n", [(256, 256), (600, 500), (1200, 1200)])
def test_many_terms(fault, half, m, n):
    """Neighbouring element sets at a tight stop: more terms than are reduced at a time.  (The stop
    is a heuristic: the oracle's blocks of these sets end 7e-7 to 3e-9 from the exact ones.)"""
    sim, order = fault
    op = _operator(sim, half)
    tol = 1e-9
    b = (np.sort(order[:m]), np.sort(order[m:m + n]), 0, 5, 7)
    U, V, r, flag = _aca(op, [b], tol, 400)[0]
    assert flag in (0, 2) and 128 < r < min(m, n, 400)
    A = _Entries(op, b[0], b[1]).K[0, 0]
    assert np.linalg.norm(A - U[:, 0].T @ V[:, 0]) <= 1e-4 * np.linalg.norm(A)
    assert _stopped(U[:, 0], V[:, 0], tol)
