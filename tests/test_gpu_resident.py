"""Small problems: the steps between two evaluations as one cooperative launch with the
plan, its average and the cost in shared memory (the automatic choice), against the CUDA
graph of the primal pass and the dual step (persistent=False). Every CTA range, dual
block and order of addition is the kernels' own, so iterates, duals and every record
are the same bit for bit."""
import numpy as np
import pytest

import pdot
from pdot import instances

pytestmark = pytest.mark.gpu


def _records(o):
    return [(s.iteration_number, s.step_size, s.primal_weight, int(s.restart_used), s.cumulative_kkt_matrix_passes,
             *vars(s.convergence_information[0]).values()) for s in o.iteration_stats]


def _same(a, b):
    assert a.iteration_count == b.iteration_count
    assert a.termination_reason == b.termination_reason
    for f in ("primal_solution", "dual_source_solution", "dual_target_solution"):
        assert np.array_equal(getattr(a, f), getattr(b, f)), f
    assert _records(a) == _records(b)


# fewer units than CTA ranges, one row or column, a ragged last panel, CTA ranges of two
# panels, a warp and a thread per dual row, the largest that fit and the first that do not
SHAPES = [(1, 1, 300), (1, 300, 300), (300, 1, 300), (68, 40, 900), (127, 93, 400), (256, 256, 300), (257, 130, 300),
          (1000, 1000, 700), (2050, 300, 300), (100, 8000, 200), (5000, 60, 300), (1216, 900, 200), (1217, 960, 200),
          (2400, 450, 200)]


@pytest.mark.parametrize("m,n,limit", SHAPES)
def test_resident_steps_match_the_graph(cuda, m, n, limit):
    prob = instances.uniform_sqeuclid(m, n, seed=m + n)
    params = pdot.default_parameters(1e-9, iteration_limit=limit)
    _same(pdot.optimize(params, prob, persistent=False), pdot.optimize(params, prob))


@pytest.mark.parametrize("primal_pass", ["staged", "direct"])
@pytest.mark.parametrize("cost,dim", [("f32", 2), ("bf16", 2), ("sqeuclid", 1), ("sqeuclid", 2), ("sqeuclid", 3),
                                      ("sqeuclid", 4), ("l1", 1), ("l1", 2), ("l1", 3), ("l1", 4)])
def test_resident_steps_match_the_graph_in_mixed_precision(cuda, cost, dim, primal_pass):
    rng = np.random.default_rng(5)
    for m, n in ((1208, 900), (311, 205)):  # 16-byte loads, and single rows
        xs, ys = (rng.uniform(0, 1, (k, dim)).astype(np.float32) for k in (m, n))
        prob = instances.uniform_sqeuclid(m, n, seed=5)
        kw = {"precision": "f32", "cost": cost, "primal_pass": primal_pass}
        if cost in ("sqeuclid", "l1"):
            kw["points"] = (xs, ys)
        params = pdot.default_parameters(1e-7, iteration_limit=400)
        _same(pdot.optimize(params, prob, persistent=False, **kw), pdot.optimize(params, prob, **kw))


def test_resident_steps_end_where_the_graph_ends(cuda):
    """To a tolerance; with a constant step; evaluated every 5 and every 3 iterations (the latter too few
    steps for a launch); from a warm start; and with a pass limit."""
    prob = instances.uniform_sqeuclid(600, 500, seed=8)
    params = pdot.default_parameters(1e-4, iteration_limit=20_000)
    cold = pdot.optimize(params, prob, persistent=False)
    assert cold.termination_reason == pdot.TerminationReason.TERMINATION_REASON_OPTIMAL
    _same(cold, pdot.optimize(params, prob))
    warm = (0.9 * cold.dual_source_solution, 0.9 * cold.dual_target_solution)
    _same(pdot.optimize(params, prob, warm_start=warm, persistent=False), pdot.optimize(params, prob, warm_start=warm))
    for change in ({"step_size_policy_params": pdot.ConstantStepsizeParams()}, {"termination_evaluation_frequency": 5},
                   {"termination_evaluation_frequency": 3}, {"step_size_policy_params": pdot.AdaptiveStepsizeParams(0.7, 0.6)}):
        p = pdot.default_parameters(1e-6, iteration_limit=301)
        for k, v in change.items():
            setattr(p, k, v)
        _same(pdot.optimize(p, prob, persistent=False), pdot.optimize(p, prob))
    p = pdot.default_parameters(1e-9, iteration_limit=5000)
    p.termination_criteria.kkt_matrix_pass_limit = 700.0
    _same(pdot.optimize(p, prob, persistent=False), pdot.optimize(p, prob))


def test_resident_solver_in_pieces(cuda):
    prob = instances.uniform_sqeuclid(700, 650, seed=4)
    params = pdot.default_parameters(1e-4, iteration_limit=5000)
    ref = pdot.optimize(params, prob, persistent=False)
    s = pdot.Solver(params, prob)
    try:
        for k in (3, 70, 129, 1, 2, 256, 5000):
            s.iterate(k)
        _same(ref, s.finish())
        s.reset()
        _same(ref, s.finish())
    finally:
        s.close()


def test_resident_solves_on_several_threads(cuda):
    """Solves of several host threads at once, each on its own stream: their CTAs share SMs, so that some
    run far behind others, and their blocks and status slots are their own."""
    from concurrent.futures import ThreadPoolExecutor

    probs = [instances.uniform_sqeuclid(200 + 37 * k, 150 + 11 * k, seed=k) for k in range(8)]
    params = pdot.default_parameters(1e-5, iteration_limit=2000)
    want = [pdot.optimize(params, p, persistent=False) for p in probs]
    with ThreadPoolExecutor(8) as pool:
        for _ in range(12):
            for a, b in zip(want, pool.map(lambda p: pdot.optimize(params, p), probs)):
                _same(a, b)
