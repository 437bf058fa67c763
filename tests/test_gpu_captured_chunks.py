"""Solves whose regular chunks are CUDA graphs beside a thread that synchronises the device:
the driver refuses that call while a stream is captured and drops the capture. The solve
then launches the chunk kernel by kernel, with the same results."""
import threading

import numpy as np
import pytest

import pdot
from pdot import instances

pytestmark = pytest.mark.gpu


def test_a_spoiled_capture_does_not_fail_the_solve(cuda):
    import torch

    params = pdot.default_parameters(1e-9, iteration_limit=400)
    prob = instances.uniform_sqeuclid(200, 150, seed=1)
    batch = [instances.uniform_sqeuclid(60 + k, 50, seed=k) for k in range(4)]
    want = pdot.optimize(params, prob, persistent=False)
    want_batch = pdot.optimize_batched(params, batch)[0]
    stop = threading.Event()
    refused = [0]

    def synchronise():
        while not stop.is_set():
            try:
                torch.cuda.synchronize()
            except RuntimeError:  # while a chunk is captured
                refused[0] += 1

    thread = threading.Thread(target=synchronise)
    thread.start()
    try:
        for _ in range(150):
            got = pdot.optimize(params, prob, persistent=False)
            assert got.iteration_count == want.iteration_count
            assert np.array_equal(got.primal_solution, want.primal_solution)
        for _ in range(30):
            for a, b in zip(want_batch, pdot.optimize_batched(params, batch)[0]):
                assert np.array_equal(a.primal_solution, b.primal_solution)
    finally:
        stop.set()
        thread.join()
    print(f"{refused[0]} synchronisations refused")
