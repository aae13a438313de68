"""Wolff updates of lattices of extreme form (marked gpu): the joins between tiles keep their trees shallow, so that no device
loop takes a number of steps that grows with the lattice's length, and the cluster is the seed's component."""
import numpy as np
import pytest
from scipy.sparse import coo_matrix
from scipy.sparse.csgraph import connected_components

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx(slsf):
    slsf.build()
    c = slsf.Context()
    yield c
    c.close()


@pytest.mark.parametrize("temperature", [0.4, 1.3])
@pytest.mark.parametrize("dims", [(32, 8, 4096), (4, 4, 20000), (20000, 4, 4), (4, 20000, 2)])
def test_rows_of_tiles_join_in_few_steps(slsf, dims, temperature):
    # 1,024 to 5,000 tiles in a row: 128 steps are far above the logarithm of either
    with slsf.Context() as ctx:
        t = slsf.Task(ctx, dims, np.full(dims[2], 1.2), np.full(dims[2], 1.0), temperature, wolff_steps=1, seed=7)
        t.init_cold()
        ctx.set_loop_limit(128)
        for _ in range(4):
            t.metropolis_sweep()
            t.wolff_step()
        t.close()


# rows of tiles; then both sides of the choice between tiles and growth on bits, from 2^21 sites on: whole and cut words,
# rows of less than a word, an odd number of planes
@pytest.mark.parametrize("dims", [(32, 8, 1024), (4, 4, 3001), (5001, 4, 4), (4, 3000, 2), (160, 160, 160), (100, 160, 160),
                                  (100, 160, 161), (6, 600, 600), (6, 590, 601), (64, 64, 512), (2048, 32, 32), (31, 10, 7000)])
def test_cluster_is_the_seeds_component(slsf, ctx, dims):
    t = slsf.Task(ctx, dims, np.full(dims[2], 1.2), np.linspace(0.5, 1.5, dims[2]), 0.8, wolff_steps=1, seed=9)
    t.init_cold()
    lx, ly, lz = dims
    site = np.arange(t.volume).reshape(lz, ly, lx)
    for _ in range(3 if t.volume < 2 ** 20 else 1):
        dbg = t.wolff_step_debug()
        bonds = dbg["bonds"].reshape(lz, ly, lx)
        ends = [(site[bonds & (1 << bit) != 0], np.roll(site, -1, axis)[bonds & (1 << bit) != 0])
                for bit, axis in ((0, 2), (1, 1), (2, 0))]
        a, b = (np.concatenate([e[k] for e in ends]) for k in (0, 1))
        label = connected_components(coo_matrix((np.ones(a.size, np.int8), (a, b)), shape=(t.volume,) * 2), directed=False)[1]
        x, y, z = dbg["seed_site"]
        assert np.array_equal(dbg["cluster"].astype(bool), label == label[site[z, y, x]])
    t.close()


@pytest.mark.parametrize("dims", [(4, 4, 130), (4, 8, 256), (8, 8, 128), (8, 8, 300), (4, 64, 64), (6, 10, 60)])
def test_batched_thin_replicas(slsf, dims):
    """The one-CTA kernel's default block keeps the rows of thin lattices in registers (four a thread up to 512
    threads), and their trajectories are the one-task trajectories."""
    with slsf.Context() as ctx:
        choice = ctx.tune_get(dims)
        assert choice["kind"] == "resident" and 4 * choice["threads"] >= min(dims[1] * dims[2], 2048)
        make = lambda: slsf.Task(ctx, dims, np.full(dims[2], 1.2), np.linspace(0.5, 1.5, dims[2]), 0.9, wolff_steps=1, seed=4)
        a, b = make(), make()
        a.init_random()
        b.init_random()
        stats, alone = ctx.batch_run([a], 4)[0], b.sweep(4)
        assert stats == alone
        assert np.array_equal(a.theta.view(np.uint32), b.theta.view(np.uint32))
        a.close()
        b.close()
