"""A walk stage on its own after a graph-captured step uses records of its own G
and leaf size, also where stages ran with those between two launches of the
graph: accelerations the same bits as the same calls without graphs."""
import numpy as np
import pytest

from conftest import small_collision

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1408, 60000])
@pytest.mark.parametrize("change", [{"G": 2.0}, {"leaf_size": 8}, {}])
def test_stages_between_captured_steps(gcs_mod, n, change):
    import torch
    gcs = gcs_mod
    st = np.resize(small_collision(), n)
    st["x"] += np.random.default_rng(1).normal(0, 1e-2, n).astype(np.float32)
    p = gcs.reference_params(bounds_mode=gcs.BOUNDS_DEVICE, theta=0.5, epsilon_sq=4e-4, dt=1e-3, leaf_size=2)
    q = gcs.reference_params(bounds_mode=gcs.BOUNDS_DEVICE, theta=0.5, epsilon_sq=4e-4, dt=1e-3, leaf_size=2)
    for k, v in change.items():
        setattr(q, k, v)
    acc = []
    stream = torch.cuda.Stream()
    for graphs in (False, True):
        with gcs.Context(n) as ctx:
            ctx.set_stream(stream.cuda_stream)
            ctx.upload(st)
            ctx.set_graphs(graphs)
            ctx.step(p)
            ctx.run_stages(q, gcs.STAGE_AGGREGATE, gcs.STAGE_WALK)
            first = ctx.read(gcs.BUF_ACCEL)
            ctx.step(p)
            ctx.run_stages(q, gcs.STAGE_WALK, gcs.STAGE_WALK)
            second = ctx.read(gcs.BUF_ACCEL)
            ctx.run_stages(p, gcs.STAGE_WALK, gcs.STAGE_WALK)
            acc.append((first, second, ctx.read(gcs.BUF_ACCEL)))
            assert ctx.device_status() == 0
    for eager, captured in zip(*acc):
        assert np.abs(eager).max() > 0
        np.testing.assert_array_equal(eager, captured)
