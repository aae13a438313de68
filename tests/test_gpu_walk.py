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
