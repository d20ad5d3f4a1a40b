"""The array forms of the plan builders against their per-block statements: term classes of
all blocks at once, the ACA starting indices in one draw, and an operator without low-rank
blocks or with blocks that keep no term."""
import numpy as np
import pytest

from pyquake3d_b200 import meshgen
from pyquake3d_b200.hmatrix import (HStructure, aca_start_indices, build_plan_arrays, build_plan_arrays_mixed,
                                    class_counts, classify_blocks, classify_terms, dense_layout)


@pytest.mark.parametrize("tol", [0.0, 2.0 ** -22, 2.0 ** -16])
def test_classify_blocks_is_classify_terms_per_block(tol):
    rng = np.random.default_rng(7)
    ranks = rng.integers(0, 30, 400)
    ranks[rng.random(400) < 0.1] = 0
    offs = np.concatenate([[0], np.cumsum(ranks)])
    w = 10.0 ** rng.uniform(-8, 1, offs[-1])
    w[rng.random(len(w)) < 0.2] = 1e-4                 # ties keep the terms' order
    w[rng.random(len(w)) < 0.02] = 0.0
    ref = [classify_terms(w[offs[i]:offs[i + 1]], w[offs[i + 1]:offs[i + 2]], tol) for i in range(0, 400, 2)]
    got = classify_blocks(w, offs, tol)
    assert np.array_equal(got, np.concatenate([np.concatenate(r) for r in ref]))
    cnt = class_counts(got, offs)
    assert np.array_equal(cnt, np.array([[np.bincount(c, minlength=3) for c in r] for r in ref]))


def _structure(n, leaf):
    P, T = meshgen.planar(20.0, 8.0, 60.0, n // 16, 8, jitter=0.1, seed=1)
    return HStructure(meshgen.centroids_km(P, T) * 1e3, mini_leaf=leaf)


def test_starting_indices_are_the_draws_in_block_order():
    s = _structure(2000, 32)
    for seed in (0, 3):
        rs, ref = np.random.RandomState(seed), []
        for b in s.blocks:
            if b.aca:
                m, n = len(b.row.indices), len(b.col.indices)
                ref.append(((rs.randint(m) - 3, rs.randint(n) - 3), (rs.randint(m) - 3, rs.randint(n) - 3)))
        assert aca_start_indices(s.blocks, seed) == ref and len(ref) > 100


def test_plans_without_terms():
    for leaf in (32, 100000):                           # every rank zero; no low-rank blocks at all
        s = _structure(600, leaf)
        recs, _, _ = dense_layout([b for b in s.blocks if not b.aca])
        nb = sum(b.aca for b in s.blocks)
        z = np.zeros(nb, np.int64)
        A = build_plan_arrays(s, recs, z, z, 1, 16, 32, 512)
        assert A["n_vitems"] == A["n_utasks"] == A["u_size"] == A["n_tpart"] == 0 and len(A["pack"]) == 0
        assert A["n_ditems"] == len(A["ditems"]) > 0
        M = build_plan_arrays_mixed(s, recs, None, 16, 32, 512, counts=np.zeros((nb, 2, 3), np.int64))
        assert M["n_vitems"] == M["n_utasks"] == M["n_scales"] == 0 and M["vwarp"][-1] == 0
        assert np.array_equal(M["ditems"], A["ditems"]) and M["n_slots"] == A["n_slots"]
