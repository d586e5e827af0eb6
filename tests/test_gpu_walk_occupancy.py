"""walk_blocks_per_sm in contexts of few groups: 0 walks each group with two
warps, any other value with one, and the accelerations are the same bits - at
theta 0 too, where every node is opened (the pair of kernels compared, which a
larger context would compare only at its own size)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [33, 1408, 4831, 20000])
@pytest.mark.parametrize("theta,leaf,batch,pot,frontier", [(0.0, 16, 64, 0, 1), (0.0, 16, 64, 1, 0), (0.5, 8, 64, 1, 1),
                                                           (0.5, 1, 32, 0, 1), (1.0, 32, 32, 0, 0), (0.7, 4, 17, 1, 1)])
def test_occupancies_same_bits(gcs_mod, n, theta, leaf, batch, pot, frontier):
    gcs = gcs_mod
    if theta == 0.0 and n > 5000:
        n = 5000  # every pair of particles
    st = gcs.collision_pair(max(n, 64), 0.6, 6.0, 0.5, 40.0, 3)[:n]
    p = gcs.reference_params(bounds_mode=gcs.BOUNDS_DEVICE, theta=theta, epsilon_sq=4e-4, leaf_size=leaf,
                             walk_batch=batch, com_fp64=1, with_potential=pot)
    with gcs.Context(n) as ctx:
        ctx.set_walk_frontier(frontier)
        ctx.upload(st)
        ctx.run_stages(p, gcs.STAGE_BOUNDS, gcs.STAGE_WALK)
        two = ctx.read(gcs.BUF_ACCEL)
        assert np.abs(two).max() > 0
        for bps in (1, 4):
            p.walk_blocks_per_sm = bps
            ctx.run_stages(p, gcs.STAGE_WALK, gcs.STAGE_WALK)
            np.testing.assert_array_equal(ctx.read(gcs.BUF_ACCEL), two)
        assert ctx.device_status() == 0
