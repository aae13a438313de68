"""Correlations inside the batched sweeps of a shape that no cluster holds (marked gpu): the tuner may give the shape to the
stream kernel, and such a task still runs through the grid-wide kernels, as without a tuned entry."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LONG = (40, 4, 1018)  # 509 planes of 160 sites, the smallest equal slabs but one, are 326 KB


@pytest.fixture(scope="module")
def ctx(slsf):
    slsf.build()
    c = slsf.Context()
    yield c
    c.close()


def task(slsf, ctx, dims):
    jz = np.linspace(0.5, 1.5, dims[2])
    t = slsf.Task(ctx, dims, np.full(dims[2], 1.2), jz, 1.2, wolff_steps=1, seed=9, thermalization=1, binsize=2, n_bins=2)
    t.init_random()
    t.corr_setup(2, 0, 1, 3)
    return t


def fused_run(slsf, ctx, dims):
    t = task(slsf, ctx, dims)
    t.corr_fuse(1)
    ctx.batch_run([t], 4)
    out = t.theta.view(np.uint32).copy(), t.corr_bins(), t.bins()
    t.close()
    return out


def test_fused_correlations_after_autotune(slsf, ctx):
    assert ctx.tune_get(LONG)["kind"] == "grid"
    theta, (corr, n), (bins, m) = fused_run(slsf, ctx, LONG)
    assert ctx.autotune(LONG, 1)["kind"] in ("grid", "stream")
    for tuned in (None, ("stream", 1, 256)):
        if tuned:
            ctx.tune_set(LONG, *tuned)
        theta2, (corr2, n2), (bins2, m2) = fused_run(slsf, ctx, LONG)
        assert n == n2 == 3 and m == m2 == 3
        assert np.array_equal(theta, theta2)
        assert np.array_equal(corr, corr2)
        assert np.array_equal(bins, bins2)


def test_stream_shapes_that_a_cluster_holds_stay_refused(slsf, ctx):
    t = task(slsf, ctx, (48, 48, 48))
    assert ctx.tune_get((48, 48, 48))["kind"] == "stream"
    with pytest.raises(slsf.SlsfError, match="correlations inside the sweeps"):
        t.corr_fuse(1)
    t.close()
