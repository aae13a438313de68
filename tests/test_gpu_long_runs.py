"""Statistics of one long call (marked gpu): a call's acceptances and cluster sites are counted in 64 bits, also where
all of its sweeps run in one launch."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("batched", [False, True])
def test_counts_past_32_bits(slsf, batched):
    # proposals of width 0 are all accepted, and at T -> 0 every bond of an ordered lattice is active, so each sweep
    # counts the volume twice; the call passes 2^32 of each by one sweep
    dims = (16, 16, 32)
    v = int(np.prod(dims))
    sweeps = 2 ** 32 // v + 1
    with slsf.Context() as ctx:
        t = slsf.Task(ctx, dims, np.full(dims[2], 1.2), np.full(dims[2], 1.0), 1e-30, proposal_width=0.0, wolff_steps=1,
                      seed=5)
        t.init_cold()
        st = ctx.batch_run([t], sweeps)[0] if batched else t.sweep(sweeps)
        assert (st["sweeps"], st["wolff_clusters"]) == (sweeps, sweeps)
        assert (st["accepted"], st["wolff_cluster_sites"]) == (v * sweeps, v * sweeps)
        t.close()
