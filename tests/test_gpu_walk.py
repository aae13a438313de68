"""Edges of the batched one-CTA kernel's walks (marked gpu): lattices whose sides are the smallest, odd multiples of
four, not multiples of the thread patch or of the warp, with one and with many planes per walk.  The batched
trajectory equals the one-task trajectory bit for bit, and the binned sums equal the one-task measurements to FP64
summation order, also for zero couplings and for couplings too large for the biased sums."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx(slsf):
    slsf.build()
    c = slsf.Context()
    yield c
    c.close()


@pytest.mark.parametrize("threads", [0, 64, 512, 1024])
@pytest.mark.parametrize("dims,j", [((4, 2, 2), 1.2), ((4, 4, 6), 1.2), ((6, 2, 10), 1.2), ((8, 2, 34), 1.2),
                                    ((12, 6, 10), 1.2), ((20, 70, 4), 1.2), ((28, 14, 6), 1.2), ((30, 34, 2), 1.2),
                                    ((32, 32, 32), 1.2), ((16, 8, 8), 0.0), ((16, 8, 8), 1e31)])
def test_batched_walk_equals_one_task(slsf, ctx, dims, j, threads):
    jz = np.linspace(0.5, 1.5, dims[2]) * (j / 1.2)
    sweeps, make = 4, lambda: slsf.Task(ctx, dims, np.full(dims[2], j), jz, 1.2, seed=11, thermalization=0, binsize=1,
                                        n_bins=4)
    a, b = make(), make()
    a.init_random()
    b.init_random()
    if threads:
        ctx.tune_set(dims, "resident", 1, threads)
    stats = ctx.batch_run([a], sweeps)[0]
    rows, accepted, sites = [], 0, 0
    for _ in range(sweeps):
        st = b.sweep(1)
        accepted += st["accepted"]
        sites += st["wolff_cluster_sites"]
        o = b.measure()
        rows.append([o["energy"], o["magnetization_squared"], o["cos_x"], o["cos_y"], o["cos_z"], o["sin_x"], o["sin_y"],
                     o["sin_z"]])
    assert np.array_equal(a.theta.view(np.uint32), b.theta.view(np.uint32))
    assert (stats["accepted"], stats["wolff_cluster_sites"]) == (accepted, sites)
    got = a.bins()[0][:, [0, 2, 3, 4, 5, 6, 7, 8]]
    # the sums differ by their FP64 (or value-and-remainder) rounding: at most 2^-36 of the terms' total magnitude
    v = float(np.prod(dims))
    scale = np.array([3 * j, 1, v * j, v * j, v * j, v * j, v * j, v * j]) * 1.3 + 1e-30
    assert np.all(np.abs(got - np.array(rows)) <= 2.0 ** -36 * scale), (got, rows)


@pytest.mark.parametrize("dims", [(12, 6, 20), (12, 34, 6), (32, 32, 34), (36, 40, 44), (40, 6, 10), (48, 48, 48), (64, 64, 64),
                                  (64, 2, 8), (60, 128, 32)])
def test_stream_kernels_equal_one_task(slsf, ctx, dims):
    """The stream kernels (one launch per phase for many replicas, in one and in two parts) give every replica the
    one-task trajectory and measurements, also through a session whose replays continue the counters."""
    jz = np.linspace(0.5, 1.5, dims[2])
    make = lambda i: slsf.Task(ctx, dims, np.full(dims[2], 1.2), jz, 1.1 + 0.1 * i, wolff_steps=1 + i % 2, seed=21 + i,
                               thermalization=1, binsize=1, n_bins=6)
    batch, alone = [make(i) for i in range(3)], [make(i) for i in range(3)]
    for t in batch + alone:
        t.init_random()
    ctx.tune_set(dims, "stream", 1, 256)
    stats = [ctx.batch_run(batch[:1], 2)[0]] + ctx.batch_run(batch[1:], 2)
    with ctx.session(batch, 2) as s:
        for _ in range(2):
            for total, more in zip(stats, s.step()):
                for k in total:
                    total[k] += more[k]
    for t, st, u in zip(batch, stats, alone):
        rows, want = [], {k: 0 for k in st}
        for n in range(6):
            for k, v in u.sweep(1).items():
                want[k] += v
            o = u.measure()
            if n > 0:
                rows.append([o[k] for k in ("energy", "magnetization_squared", "cos_x", "cos_y", "cos_z", "sin_x", "sin_y",
                                            "sin_z")])
        assert np.array_equal(t.theta.view(np.uint32), u.theta.view(np.uint32))
        assert st == want
        got = t.bins()[0][:5, [0, 2, 3, 4, 5, 6, 7, 8]]
        v = float(np.prod(dims))
        assert np.all(np.abs(got - np.array(rows)) <= 2.0 ** -36 * np.array([3, 1, v, v, v, v, v, v]) * 1.6)
