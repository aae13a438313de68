"""A task's couplings on the device (marked gpu), around the number of layers that one launch carries and the number
that travels by launches at all, and for a long lattice in a bounded number of launches."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
HEADER = 24 + 8 + 16 + 16 + 16 + 32 + 32 + 8  # the state blob's header, before the couplings as the device holds them


@pytest.mark.parametrize("lz", [1, 2, 255, 256, 257, 1023, 1024, 1025, 1026, 5000])
def test_couplings_arrive(slsf, lz):
    rng = np.random.default_rng(lz)
    jxy, jz = rng.uniform(0.1, 2.0, lz), rng.uniform(0.1, 2.0, lz)
    with slsf.Context() as ctx:
        t = slsf.Task(ctx, (4, 2, lz), jxy, jz, 1.2, seed=3)
        blob = np.frombuffer(t.save_state(), dtype=np.uint8)
        got = blob[HEADER:HEADER + 8 * lz].view(np.float32)
        assert np.array_equal(got, np.concatenate([jxy, jz]).astype(np.float32))
        t.close()


def test_long_lattice_takes_few_launches(slsf):
    lz = 1 << 16
    with slsf.Context() as ctx:
        before = ctx.launches
        t = slsf.Task(ctx, (4, 2, lz), np.full(lz, 1.2), np.full(lz, 1.0), 1.2, seed=3)
        assert ctx.launches - before <= 4
        t.close()
