"""The stream kernel (many replicas with their state in global memory, one persistent launch) in the regimes that its
launch rules make (marked gpu): trajectories, statistics and binned measurements equal the one-task path's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
COLS = ("energy", "magnetization_squared", "cos_x", "cos_y", "cos_z", "sin_x", "sin_y", "sin_z")


@pytest.fixture
def ctx(slsf):
    slsf.build()
    c = slsf.Context()
    yield c
    c.close()


def make(slsf, ctx, dims, i, bins=0, wolff_steps=1, temperature=None, j=1.2, cold=False):
    t = slsf.Task(ctx, dims, np.full(dims[2], j), np.linspace(0.5, 1.5, dims[2]) * (j / 1.2),
                  temperature or 0.9 + 0.05 * (i % 12), wolff_steps=wolff_steps, seed=1000 + i, thermalization=1, binsize=1,
                  n_bins=bins)
    t.init_cold() if cold else t.init_random()
    return t


def same_angles(a, b):
    return np.array_equal(a.theta.view(np.uint32), b.theta.view(np.uint32))


@pytest.mark.parametrize("dims", [(36, 8, 512), (36, 256, 12), (16, 64, 64), (64, 64, 40), (40, 2, 1000)])
@pytest.mark.parametrize("n", [1, 3])
def test_few_replicas_of_long_lattices(slsf, ctx, dims, n):
    """Grown by several CTAs together."""
    assert ctx.tune_get(dims)["kind"] == "stream"
    batch, alone = ([make(slsf, ctx, dims, i) for i in range(n)] for _ in range(2))
    for t, st, u in zip(batch, ctx.batch_run(batch, 3), alone):
        assert st == u.sweep(3)
        assert same_angles(t, u)
        t.close()
        u.close()
