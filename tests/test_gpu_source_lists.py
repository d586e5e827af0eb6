"""The walk's source lists stand in the array of the aggregation's FP64 sums: an
aggregation after a walk, with and without a build before it, gives the nodes
it gave, and so the walk its accelerations; segments of every small size beside
a large one have the accelerations they have alone (their lists are packed)."""
import numpy as np
import pytest

from conftest import small_collision

pytestmark = pytest.mark.gpu


def _params(gcs, **kw):
    return gcs.reference_params(bounds_mode=gcs.BOUNDS_DEVICE, theta=0.5, epsilon_sq=4e-4, leaf_size=16, walk_batch=64,
                                com_fp64=1, **kw)


@pytest.mark.parametrize("n", [1500, 2048, 2049, 40000])
def test_aggregation_after_a_walk(gcs_mod, n):
    gcs = gcs_mod
    p = _params(gcs)
    with gcs.Context(n) as ctx:
        ctx.upload(gcs.collision_pair(n, 0.6, 6.0, 0.5, 40.0, 4))
        ctx.run_stages(p, gcs.STAGE_BOUNDS, gcs.STAGE_WALK)
        nodes, acc = ctx.read(gcs.BUF_NODES), ctx.read(gcs.BUF_ACCEL)
        for first in ([gcs.STAGE_AGGREGATE], [gcs.STAGE_BUILD], [gcs.STAGE_BUILD, gcs.STAGE_WALK]):
            for s in first:
                ctx.run_stages(p, s, s)
            ctx.device_status(clear=True)  # (a walk over nodes without mass may complain)
            ctx.run_stages(p, gcs.STAGE_AGGREGATE, gcs.STAGE_WALK)
            assert ctx.device_status() == 0
            assert ctx.read(gcs.BUF_NODES).tobytes() == nodes.tobytes()
            assert ctx.read(gcs.BUF_ACCEL).tobytes() == acc.tobytes()


@pytest.mark.parametrize("width", [32, 64, 52])
def test_packed_lists(gcs_mod, width):
    gcs = gcs_mod
    counts = list(range(1, 30)) + [193, 208, 209, 257, 1023, 1024, 1025, 3000, 20000] + [1] * 40
    parts = [np.resize(small_collision(2048, 512, 256, seed=k), c) for k, c in enumerate(counts)]
    rng = np.random.default_rng(3)
    for s in parts:
        s["x"] += rng.normal(0, 1e-2, len(s)).astype(np.float32)
    p = _params(gcs)
    with gcs.Context(sum(counts), len(counts)) as ctx:
        ctx.set_segments(counts)
        ctx.set_group_width(width)
        ctx.upload(np.concatenate(parts))
        ctx.run_stages(p, gcs.STAGE_BOUNDS, gcs.STAGE_WALK)
        acc = ctx.read(gcs.BUF_ACCEL)
        assert ctx.device_status() == 0
    at = 0
    for s in parts:
        if len(s) > 1 and len(s) not in (2, 7):
            with gcs.Context(len(s)) as ctx:
                ctx.set_group_width(width)
                ctx.upload(s)
                ctx.run_stages(p, gcs.STAGE_BOUNDS, gcs.STAGE_WALK)
                np.testing.assert_array_equal(ctx.read(gcs.BUF_ACCEL), acc[at:at + len(s)])
        at += len(s)
