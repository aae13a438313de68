"""Threads with a context each (marked gpu): launches of one kernel with different shared-memory sizes do not get into
each other's way, and every trajectory is the one it has alone."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def work(slsf, dims, call, rounds):
    with slsf.Context() as ctx:
        if call == "stream":
            ctx.tune_set(dims, "stream", 1, 256)
        if call == "cluster":
            ctx.tune_set(dims, "cluster", 1, 512)
        t = slsf.Task(ctx, dims, np.full(dims[2], 1.2), np.full(dims[2], 1.0), 1.2, wolff_steps=1, seed=8)
        t.init_random()
        for _ in range(rounds):
            if call == "sweep":
                t.sweep(1)
            elif call == "correlations":
                t.correlations(min(dims[0], dims[1]) // 2, dims[2] // 2)
            else:
                ctx.batch_run([t], 1)
        theta = t.theta
        t.close()
        return theta


@pytest.mark.parametrize("call,small,large", [("sweep", (4, 4, 4), (20, 20, 20)), ("batch", (6, 4, 4), (32, 32, 32)),
                                              ("stream", (12, 6, 20), (64, 64, 64)), ("cluster", (8, 8, 8), (32, 32, 32)),
                                              ("correlations", (400, 4, 4), (700, 2, 2))])
def test_two_threads_with_launches_of_different_size(slsf, call, small, large):
    slsf.build()
    rounds = 1500
    want = [work(slsf, d, call, rounds) for d in (small, large)]
    got, errors = [None, None], []

    def run(k, dims):
        try:
            got[k] = work(slsf, dims, call, rounds)
        except slsf.SlsfError as e:
            errors.append((dims, str(e)))

    threads = [threading.Thread(target=run, args=(k, d)) for k, d in enumerate((small, large))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors
    for a, b in zip(got, want):
        assert np.array_equal(a.view(np.uint32), b.view(np.uint32))
