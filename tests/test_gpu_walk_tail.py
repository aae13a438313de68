"""Walks whose runs of planes are odd, or a single plane (marked gpu): their last terms reach the FP64 sums, with the
tolerance of test_gpu_sums.py."""
import numpy as np
import pytest

from test_gpu_sums import BIN_COLS, FIELDS, TOLERANCE, bounds, fp64_sums

pytestmark = pytest.mark.gpu


def couplings(dims):
    return np.full(dims[2], 1.2), np.linspace(0.5, 1.5, dims[2])


def make(slsf, ctx, dims, bins=0):
    jx, jzz = couplings(dims)
    t = slsf.Task(ctx, dims, jx, jzz, 1.2, wolff_steps=1, seed=31, thermalization=0, binsize=1, n_bins=bins)
    t.init_random()
    return t


@pytest.mark.parametrize("dims", [(4, 2, 3), (36, 6, 7), (72, 6, 9), (100, 90, 71), (256, 256, 5)])
def test_single_measurement_of_odd_heights(slsf, dims):
    with slsf.Context() as ctx:
        t = make(slsf, ctx, dims)
        got = t.measure()
        want = fp64_sums(slsf, t.theta, dims, *couplings(dims))
        assert np.all(np.abs(np.array([got[f] for f in FIELDS]) - want) <= TOLERANCE * bounds(dims, *couplings(dims)))
        t.close()


# one CTA: four segments of 3, 3, 3 and 1 planes, three of 2, two of 3; the stream kernel: 4 and 2; the grid: of any length
@pytest.mark.parametrize("dims,choice", [((16, 16, 10), ("resident", 1, 128)), ((16, 16, 6), ("resident", 1, 128)),
                                         ((32, 32, 6), ("resident", 1, 256)), ((40, 4, 6), ("stream", 1, 256)),
                                         ((256, 256, 10), ("grid", 1, 256)), ((100, 90, 26), ("grid", 1, 256))])
def test_measured_sweeps_of_odd_runs(slsf, dims, choice):
    with slsf.Context() as ctx:
        ctx.tune_set(dims, *choice)
        batch, alone = make(slsf, ctx, dims, 3), make(slsf, ctx, dims)
        ctx.batch_run([batch], 3)
        bins = batch.bins()[0][:, BIN_COLS]
        for s in range(3):
            alone.sweep(1)
            want = fp64_sums(slsf, alone.theta, dims, *couplings(dims))
            assert np.all(np.abs(bins[s] - want) <= TOLERANCE * bounds(dims, *couplings(dims))), s
        batch.close()
        alone.close()
