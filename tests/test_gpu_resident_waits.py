"""The grid barriers of a small problem's resident steps, when a wait runs out: no fault
and no hang, every CTA leaves, and the context serves the next solve."""
import numpy as np
import pytest

import pdot
from pdot import _abi, instances

pytestmark = pytest.mark.gpu


def _same(a, b):
    assert a.iteration_count == b.iteration_count
    assert a.termination_reason == b.termination_reason
    for f in ("primal_solution", "dual_source_solution", "dual_target_solution"):
        assert np.array_equal(getattr(a, f), getattr(b, f)), f


# one CTA, a few, and one on every SM; FP64, and an FP32 plan with a computed cost
@pytest.mark.parametrize("m,n,cost", [(20, 1, "f64"), (127, 93, "f64"), (600, 500, "f64"), (700, 600, "sqeuclid")])
def test_a_run_out_barrier_ends_the_call(cuda, m, n, cost):
    """One CTA's wait reports a run-out at the second barrier of the launch; the others, which wait for it,
    leave on its error. Then the same solve, unhooked, is the graph's bit for bit."""
    rng = np.random.default_rng(2)
    prob = instances.uniform_sqeuclid(m, n, seed=2)
    kw = {"primal_pass": "direct"}
    if cost != "f64":
        kw.update(precision="f32", cost=cost, points=tuple(rng.uniform(0, 1, (k, 2)).astype(np.float32) for k in (m, n)))
    params = pdot.default_parameters(1e-9, iteration_limit=150)
    for _ in range(3):
        with pytest.raises(_abi.PdotError) as ei:
            pdot.optimize(params, prob, fail_bounded_waits=True, **kw)
        assert ei.value.code == _abi.PDOT_ERR_CUDA
        assert "resident steps" in str(ei.value)
    _same(pdot.optimize(params, prob, persistent=False, **kw), pdot.optimize(params, prob, **kw))


@pytest.mark.parametrize("m,n,cost", [(600, 500, "f64"), (1216, 900, "f64"), (700, 601, "sqeuclid")])
def test_a_busy_sm_does_not_hold_a_solve_up(cuda, m, n, cost):
    """Beside a kernel of another stream that keeps one SM for a second and more, the resident steps find no
    room for all their CTAs: the solve takes the launches of the graph, ends long before that kernel, and is
    bit-identical; so it is when the kernel has gone and the resident steps come back."""
    import torch

    rng = np.random.default_rng(2)
    prob = instances.uniform_sqeuclid(m, n, seed=2)
    kw = {}
    if cost != "f64":
        kw.update(precision="f32", cost=cost, points=tuple(rng.uniform(0, 1, (k, 2)).astype(np.float32) for k in (m, n)))
    params = pdot.default_parameters(1e-9, iteration_limit=6000)
    ref = pdot.optimize(params, prob, persistent=False, **kw)
    side = torch.cuda.Stream()
    pdot.optimize(params, prob, **kw)
    s = pdot.Solver(params, prob, **kw)
    try:
        for pieces in ((300, 77, 500), (5, 1000)):
            s.reset()
            s.iterate(200)
            with torch.cuda.stream(side):
                torch.cuda._sleep(2_500_000_000)  # cycles of one thread
                over = torch.cuda.Event()
                over.record()
            for k in pieces:
                s.iterate(k)
            assert not over.query()
            over.synchronize()
            _same(ref, s.finish())
    finally:
        s.close()


@pytest.mark.parametrize("freq,limit", [(3000, 7000), (1027, 2600), (50_000, 2060)])
def test_evaluations_far_apart_take_several_launches(cuda, freq, limit):
    """More steps between two evaluations than one launch may take: the next launch goes on, without an
    evaluation in between; the last steps of an interval may be too few for a launch of their own."""
    prob = instances.uniform_sqeuclid(300, 200, seed=9)
    params = pdot.default_parameters(1e-9, iteration_limit=limit)
    params.termination_evaluation_frequency = freq
    want, got = (pdot.optimize(params, prob, persistent=p) for p in (False, None))
    _same(want, got)
    assert [s.iteration_number for s in want.iteration_stats] == [s.iteration_number for s in got.iteration_stats]
    s = pdot.Solver(params, prob)
    try:
        s.iterate(1500)
        s.iterate(3)
        _same(want, s.finish())
    finally:
        s.close()
