"""Rows per task of the ensemble step: every task has a CTA of its own whenever tasks of the
largest size would, however uneven the faults; multiples of 16; short for small ensembles."""
import numpy as np
import pytest

from pyquake3d_b200.ensemble import ensemble_task_rows, ensemble_tasks

CTAS, MOST = 296, 256


def _tasks(sizes, rows):
    row0 = np.concatenate([[0], np.cumsum(sizes)])
    return len(ensemble_tasks(row0, rows)[1])


@pytest.mark.parametrize("sizes", [
    [200] * 100 + [50] * 100, [200] * 148 + [20] * 148, [257] * 148, [256] * 296, [17] * 296, [1] * 296,
    [20000] + [40] * 200, [500, 900, 1300, 2000, 3000, 4900], [75000], [1], [33, 4000]])
def test_a_cta_per_task_where_there_is_one(sizes):
    row0 = np.concatenate([[0], np.cumsum(sizes)])
    rows = ensemble_task_rows(row0, CTAS, MOST)
    assert rows % 16 == 0 and 16 <= rows <= MOST
    assert _tasks(sizes, MOST) <= CTAS and _tasks(sizes, rows) <= CTAS
    # not longer than needed: shorter tasks would not fit, or would take more than half the CTAs
    assert rows == 16 or _tasks(sizes, rows - 16) > CTAS or sum(sizes) > (rows - 16) * (CTAS // 2)


@pytest.mark.parametrize("sizes", [[60] * 320, [80000], [257] * 149, [20000] * 4])
def test_longest_tasks_in_lock_step(sizes):
    assert _tasks(sizes, MOST) > CTAS
    assert ensemble_task_rows(np.concatenate([[0], np.cumsum(sizes)]), CTAS, MOST) == MOST


def test_seeded_random_ensembles():
    rng = np.random.default_rng(3)
    for _ in range(300):
        sizes = rng.integers(1, int(rng.choice([40, 300, 2000])), int(rng.integers(1, 330)))
        rows = ensemble_task_rows(np.concatenate([[0], np.cumsum(sizes)]), CTAS, MOST)
        assert (_tasks(sizes, rows) <= CTAS) == (_tasks(sizes, MOST) <= CTAS)


def test_no_device_grid():
    assert ensemble_task_rows([0, 5000], -1, MOST) == MOST
