"""The measured sums of the patch walks (marked gpu) against the same FP32 terms summed in FP64: slsf_measure_noalloc,
which does not know the couplings' size, sums term by term in FP64 on the same device arithmetic.  Tolerances scale with
each direction's own coupling: FP64 sums in two orders differ by at most 2^-53 of the terms' total for each of the some
fifty additions that a term goes through."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
FIELDS = ("energy", "magnetization_squared", "cos_x", "cos_y", "cos_z", "sin_x", "sin_y", "sin_z")
BIN_COLS = [0, 2, 3, 4, 5, 6, 7, 8]
TOLERANCE = 2.0 ** -47


def fp64_sums(slsf, theta, dims, jxy, jz):
    import torch

    dev = torch.device("cuda", 0)
    arrays = [torch.from_numpy(np.ascontiguousarray(a, dtype=np.float32)).to(dev) for a in (theta, jxy, jz)]
    torch.cuda.synchronize(dev)
    out = slsf.Observables()
    rc = slsf.load().slsf_measure_noalloc(*(C.c_void_p(a.data_ptr()) for a in arrays), *dims,
                                          C.c_void_p(torch.cuda.current_stream(dev).cuda_stream), C.byref(out))
    assert rc == slsf.OK, slsf.last_error()
    d = out.as_dict()
    return np.array([d[f] for f in FIELDS])


def bounds(dims, jxy, jz):
    """Sums of the terms' largest magnitudes, per field."""
    v, plane = float(np.prod(dims)), float(dims[0] * dims[1])
    x, z = plane * np.sum(jxy), plane * np.sum(jz)
    return np.array([(2 * x + z) / v, 1.0, x, x, z, x, x, z])


@pytest.mark.parametrize("jxy,jz", [(1.2, 1.0), (1.2, 1e-5), (1e-6, 1.0), (3e4, 2e-4)])
@pytest.mark.parametrize("dims,kind", [((32, 32, 32), "resident"), ((16, 8, 200), "resident"), ((40, 40, 40), "stream"),
                                       ((64, 64, 64), "stream"), ((100, 90, 70), "grid"), ((64, 64, 256), "grid")])
def test_walk_sums_equal_fp64_sums(slsf, dims, kind, jxy, jz):
    jx, jzz = np.full(dims[2], jxy), np.linspace(0.5, 1.5, dims[2]) * jz
    scale = bounds(dims, jx, jzz)
    with slsf.Context() as ctx:
        assert ctx.tune_get(dims)["kind"] == kind
        make = lambda: slsf.Task(ctx, dims, jx, jzz, 1.2 * max(jxy, jz), wolff_steps=1, seed=17, thermalization=0, binsize=1,
                                 n_bins=4)
        batch, alone = make(), make()
        batch.init_random()
        alone.init_random()
        ctx.batch_run([batch], 4)
        bins = batch.bins()[0][:, BIN_COLS]
        for s in range(4):
            alone.sweep(1)
            want = fp64_sums(slsf, alone.theta, dims, jx, jzz)
            got = alone.measure()
            for have in (np.array([got[f] for f in FIELDS]), bins[s]):
                assert np.all(np.abs(have - want) <= TOLERANCE * scale), (s, (have - want) / scale)
        batch.close()
        alone.close()


@pytest.mark.parametrize("dims,threads", [((32, 32, 32), 64), ((16, 16, 64), 64), ((8, 8, 512), 64), ((32, 32, 32), 512)])
def test_long_walks_over_layers_of_any_strength(slsf, dims, threads):
    """Couplings spread over six decades from layer to layer, many planes a thread: weak layers' terms are summed to the
    same precision as strong ones'."""
    rng = np.random.default_rng(5)
    jx, jzz = (10.0 ** rng.uniform(-6, 0, dims[2]) for _ in range(2))
    scale = bounds(dims, jx, jzz)
    with slsf.Context() as ctx:
        ctx.tune_set(dims, "resident", 1, threads)
        make = lambda: slsf.Task(ctx, dims, jx, jzz, 0.5, wolff_steps=1, seed=23, thermalization=0, binsize=1, n_bins=8)
        batch, alone = make(), make()
        batch.init_random()
        alone.init_random()
        ctx.batch_run([batch], 8)
        bins = batch.bins()[0][:, BIN_COLS]
        for s in range(8):
            alone.sweep(1)
            want = fp64_sums(slsf, alone.theta, dims, jx, jzz)
            assert np.all(np.abs(bins[s] - want) <= TOLERANCE * scale), (s, (bins[s] - want) / scale)
        batch.close()
        alone.close()
