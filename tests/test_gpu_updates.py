"""The single-task updates (marked gpu) at the sizes where their kernels change: the one-launch sweep and updates of
small lattices against the grid-wide kernels, a site per lane against the patch walk, union-find tiles against the
growth on bits.  Whole trajectories are equal bit for bit; a cluster is the seed's connected component over the
recorded bonds."""
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


def task(slsf, ctx, dims, temperature=1.2):
    t = slsf.Task(ctx, dims, np.full(dims[2], 1.2), np.linspace(0.5, 1.5, dims[2]), temperature, seed=31, wolff_steps=1)
    t.init_random()
    return t


@pytest.mark.parametrize("dims", [(4, 4, 4), (6, 8, 16), (8, 8, 14), (8, 8, 16), (4, 2, 128), (10, 10, 6), (16, 16, 20),
                                  (18, 18, 16), (20, 20, 20), (18, 22, 22), (24, 26, 28), (34, 10, 24)])
def test_sweep_and_single_updates_equal_grid_wide(slsf, ctx, dims):
    sweep, calls, grid = (task(slsf, ctx, dims) for _ in range(3))
    for _ in range(3):
        st = sweep.sweep(1)
        accepted = calls.metropolis_sweep() * calls.volume
        size = calls.wolff_step()
        # colour by colour and with the cluster written out, the updates run on the grid-wide kernels
        n = sum(grid.metropolis_color(c)[0] for c in (0, 1))
        grid.counters = (grid.counters[0] + 1, grid.counters[1])
        dbg = grid.wolff_step_debug()
        assert (st["accepted"], st["wolff_cluster_sites"]) == (n, dbg["size"])
        assert (round(accepted), size) == (n, dbg["size"])
        assert sweep.counters == calls.counters == grid.counters
        assert np.array_equal(sweep.theta.view(np.uint32), grid.theta.view(np.uint32))
        assert np.array_equal(calls.theta.view(np.uint32), grid.theta.view(np.uint32))


@pytest.mark.parametrize("temperature", [0.9, 2.2])
@pytest.mark.parametrize("dims", [(2, 2, 2), (5, 3, 7), (33, 9, 5), (32, 32, 32), (34, 66, 30), (100, 90, 70), (128, 128, 126),
                                  (132, 126, 128), (128, 128, 129), (1030, 34, 62)])
def test_cluster_is_the_seeds_component(slsf, ctx, dims, temperature):
    t, u = task(slsf, ctx, dims, temperature), task(slsf, ctx, dims, temperature)
    lx, ly, lz = dims
    site = np.arange(t.volume).reshape(lz, ly, lx)
    for _ in range(2):
        before = t.theta
        dbg = t.wolff_step_debug()
        bonds = dbg["bonds"].reshape(lz, ly, lx)
        ends = [(site[bonds & (1 << bit) != 0], np.roll(site, -1, axis)[bonds & (1 << bit) != 0])
                for bit, axis in ((0, 2), (1, 1), (2, 0))]
        a, b = (np.concatenate([e[k] for e in ends]) for k in (0, 1))
        label = connected_components(coo_matrix((np.ones(a.size, np.int8), (a, b)), shape=(t.volume,) * 2), directed=False)[1]
        x, y, z = dbg["seed_site"]
        member = label == label[site[z, y, x]]
        assert np.array_equal(dbg["cluster"].astype(bool), member)
        assert dbg["size"] == member.sum() == u.wolff_step()
        assert np.array_equal(t.theta[~member].view(np.uint32), before[~member].view(np.uint32))
        assert np.array_equal(t.theta.view(np.uint32), u.theta.view(np.uint32))
