"""The context's launch count over correlation measurements (marked gpu): the kernels that each combination of radii
launches -- the lines of x, y and of z off the spectral route, the spectral z lines, many layers' sums, the finalize."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims,radii,kernels", [((16, 16, 64), (0, 32), ("zfft", "finalize")),
                                                ((16, 16, 24), (0, 12), ("lines", "finalize")),
                                                ((16, 16, 24), (8, 12), ("lines", "finalize")),
                                                ((16, 16, 8), (8, 0), ("lines", "finalize")),
                                                ((16, 16, 64), (2, 32), ("lines", "zfft", "finalize")),
                                                ((16, 16, 512), (7, 0), ("lines", "finalize")),
                                                ((16, 16, 512), (8, 0), ("lines", "layers", "finalize")),
                                                ((128, 64, 128), (32, 64), ("lines", "zfft", "layers", "finalize"))])
def test_correlation_launches(slsf, dims, radii, kernels):
    with slsf.Context() as ctx:
        t = slsf.Task(ctx, dims, np.full(dims[2], 1.2), np.full(dims[2], 1.0), 1.2, seed=3)
        t.init_random()
        before = ctx.launches
        t.correlations(*radii)
        assert ctx.launches - before == len(kernels)
        t.close()
