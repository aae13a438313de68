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


def rows_of(u, sweeps):
    """Sweeps and measurements of one task alone: [sweeps, 8], and its summed statistics."""
    rows, stats = [], None
    for _ in range(sweeps):
        st = u.sweep(1)
        stats = st if stats is None else {k: v + st[k] for k, v in stats.items()}
        o = u.measure()
        rows.append([o[k] for k in COLS])
    return np.array(rows), stats


def bins_match(bins, rows, volume):
    # FP64 sums of the same FP32 terms in two orders: some fifty additions of 2^-53 of the terms' total each
    scale = np.array([3, 1, volume, volume, volume, volume, volume, volume]) * 1.6
    return np.all(np.abs(bins[:, [0, 2, 3, 4, 5, 6, 7, 8]] - rows) <= 2.0 ** -47 * scale)


@pytest.mark.parametrize("dims,n", [((64, 64, 64), 40), ((64, 64, 64), 300), ((60, 62, 64), 130), ((36, 40, 44), 200),
                                    ((32, 64, 64), 200)])
def test_many_replicas(slsf, ctx, dims, n):
    """One CTA grows a cluster (up to the full 4,096 rows), and chunks take several blocks with a ragged last chunk."""
    assert ctx.tune_get(dims)["kind"] == "stream"
    batch = [make(slsf, ctx, dims, i, bins=3) for i in range(n)]
    stats = ctx.batch_run(batch, 4)
    for i in {0, 1, 7, n // 2, n - 1}:
        u = make(slsf, ctx, dims, i)
        rows, want = rows_of(u, 4)
        assert stats[i] == want
        assert same_angles(batch[i], u)
        assert bins_match(batch[i].bins()[0], rows[1:], u.volume)  # the first sweep is thermalization
        u.close()
    for t in batch:
        t.close()


@pytest.mark.parametrize("session", [False, True])
def test_launch_cut_into_spans_of_sweeps(slsf, ctx, session):
    """The work queue holds the chunks of some 450 sweeps of these replicas: a longer call is several launches, over whose
    seams sweeps, measurements and counters carry on."""
    dims, n, sweeps = (64, 64, 64), 40, 500
    batch = [make(slsf, ctx, dims, i, bins=2 * sweeps) for i in range(n)]
    before = ctx.launches
    if session:
        with ctx.session(batch, sweeps) as s:
            stats = s.step()
            stats = [{k: a[k] + b[k] for k in a} for a, b in zip(stats, s.step())]
        total = 2 * sweeps
    else:
        stats = ctx.batch_run(batch, sweeps)
        assert ctx.launches - before >= 4  # two of each span
        total = sweeps
    for i in (0, n - 1):
        u = make(slsf, ctx, dims, i)
        rows, want = rows_of(u, total)
        assert stats[i] == want
        assert batch[i].counters == u.counters
        assert same_angles(batch[i], u)
        assert bins_match(batch[i].bins()[0][:total - 1], rows[1:], u.volume)
        u.close()
    for t in batch:
        t.close()


def test_mixed_shapes_and_sweep_counts(slsf, ctx):
    import ctypes as C

    shapes = [(36, 40, 44), (48, 48, 48), (64, 16, 30), (36, 8, 200)]
    batch = [make(slsf, ctx, shapes[i % 4], i, bins=8, wolff_steps=i % 3) for i in range(64)]
    sweeps = np.array([(5 * i) % 8 for i in range(64)], dtype=np.uint32)  # some of them 0
    stats = (slsf.SweepStats * 64)()
    slsf.check(slsf.load().slsf_batch_run_v(ctx.h, ctx.handle_array(batch), 64, sweeps.ctypes.data_as(C.POINTER(C.c_uint32)),
                                            stats))
    for i in range(0, 64, 5):
        u = make(slsf, ctx, shapes[i % 4], i, wolff_steps=i % 3)
        assert stats[i].sweeps == sweeps[i]
        if sweeps[i]:
            rows, want = rows_of(u, int(sweeps[i]))
            assert stats[i].as_dict() == want
            assert bins_match(batch[i].bins()[0][:max(0, sweeps[i] - 1)], rows[1:], u.volume)
        assert same_angles(batch[i], u)
        u.close()
    for t in batch:
        t.close()


@pytest.mark.parametrize("wolff_steps,j", [(1025, 1.2), (1024, 1.2), (1, 1e31)])
def test_tasks_that_the_stream_kernel_does_not_take(slsf, ctx, wolff_steps, j):
    """Beyond 1,024 Wolff steps and for couplings from 1e30 the shape's tasks run on the cluster kernel."""
    dims = (40, 6, 10)
    ctx.tune_set(dims, "stream", 1, 256)
    t, u = (make(slsf, ctx, dims, 3, wolff_steps=wolff_steps, j=j) for _ in range(2))
    assert ctx.batch_run([t], 2)[0] == u.sweep(2)
    assert same_angles(t, u)
    t.close()
    u.close()


@pytest.mark.parametrize("choice", [("stream", 1, 256), ("resident", 1, 64)])
@pytest.mark.parametrize("dims", [(8, 8, 8), (16, 16, 16), (32, 32, 32), (48, 48, 48), (64, 64, 64), (24, 16, 32), (8, 80, 8),
                                  (8, 8, 64), (40, 34, 8)])
def test_choices_give_the_one_task_trajectory(slsf, ctx, dims, choice):
    if choice[0] == "resident" and dims[0] > 32:
        with pytest.raises(slsf.SlsfError):
            ctx.tune_set(dims, *choice)
        return
    ctx.tune_set(dims, *choice)
    t, u = make(slsf, ctx, dims, 5, bins=3), make(slsf, ctx, dims, 5)
    stats = [ctx.batch_run([t], 2)[0], ctx.batch_run([t], 2)[0]]
    rows, want = rows_of(u, 4)
    assert {k: stats[0][k] + stats[1][k] for k in want} == want
    assert same_angles(t, u)
    assert bins_match(t.bins()[0], rows[1:], u.volume)
    t.close()
    u.close()


@pytest.mark.parametrize("dims", [(66, 50, 40), (66, 66, 66), (72, 60, 40)])
def test_grid_path_measures_every_sweep(slsf, ctx, dims):
    """Lattices too large for a cluster, rows of 2 mod 4 sites and of a multiple of four."""
    ctx.tune_set(dims, "grid", 1, 256)
    t, u = make(slsf, ctx, dims, 2, bins=4), make(slsf, ctx, dims, 2)
    stats = ctx.batch_run([t], 5)[0]
    rows, want = rows_of(u, 5)
    assert stats == want
    assert same_angles(t, u)
    assert bins_match(t.bins()[0], rows[1:], u.volume)
    t.close()
    u.close()


@pytest.mark.parametrize("dims,path", [((8, 8, 8), "single"), ((16, 16, 20), "wolff"), ((64, 64, 64), "batched"),
                                       ((36, 8, 512), "batched")])
def test_bounded_loops_give_up(slsf, ctx, dims, path):
    """The one-launch single-task calls and the growth by several CTAs, with device loops bounded at one step."""
    ctx.set_loop_limit(1)
    t = make(slsf, ctx, dims, 1, temperature=0.5, cold=True)
    with pytest.raises(slsf.SlsfError) as e:
        if path == "single":
            t.sweep(3)
        elif path == "wolff":
            t.wolff_step()
        else:
            ctx.batch_run([t], 3)
    assert e.value.code == slsf.ERR_TIMEOUT
    t.close()
    ctx.set_loop_limit(0)
    t, u = make(slsf, ctx, dims, 9), make(slsf, ctx, dims, 9)
    assert ctx.batch_run([t], 2)[0] == u.sweep(2)
    assert same_angles(t, u)
    t.close()
    u.close()


@pytest.mark.parametrize("L,T,states", [(32, 1.3, 8), (64, 1.3, 8)])
def test_default_kernels_measure_to_the_parity_bars(slsf, ctx, orc, L, T, states):
    """The measurements of the default batched kernels against FP64 evaluation of the same states."""
    dims, v = (L, L, L), float(L ** 3)
    jxy, jz = np.full(L, 1.2), slsf.uniform_layer_disorder(L, 0.5, 1.5, 20260710)
    new = lambda bins: slsf.Task(ctx, dims, jxy, jz, T, wolff_steps=1, seed=77, thermalization=0, binsize=1, n_bins=bins)
    t, u = new(states), new(0)
    t.init_random()
    u.init_random()
    ctx.batch_run([t], states)
    bins = t.bins()[0][:, [0, 2, 3, 4, 5, 6, 7, 8]]
    for s in range(states):
        u.sweep(1)
        ref = orc.measure_f32(dims, u.theta, jxy.astype(np.float32), jz.astype(np.float32))
        err = np.abs(bins[s] - np.array([ref[k] for k in COLS]))
        assert np.all(err < np.array([2e-5, 1e-5] + [2e-5 * v] * 6)), err
    t.close()
    u.close()
