"""The sort stage run again on its own, after a call that sorted and after the
stages behind it: the sorted keys and positions stay those of the first sort
(the pairs are sorted already), also where the first sort was the small
scenarios' one launch and after a graph-captured step."""
import numpy as np
import pytest

from conftest import small_collision

pytestmark = pytest.mark.gpu


def _stars(n, seed):
    st = np.resize(small_collision(2048, 512, 256, seed=seed), n)
    rng = np.random.default_rng(seed)
    for f in ("x", "y", "z"):
        st[f] += np.where(rng.random(n) < 0.8, rng.normal(0, 1e-2, n), 0.0).astype(np.float32)
    return st


def _same_again(gcs, ctx, p):
    keys, index = ctx.read(gcs.BUF_KEYS), ctx.read(gcs.BUF_INDEX)
    for _ in range(2):
        ctx.run_stages(p, gcs.STAGE_SORT, gcs.STAGE_SORT)
        np.testing.assert_array_equal(ctx.read(gcs.BUF_KEYS), keys)
        np.testing.assert_array_equal(ctx.read(gcs.BUF_INDEX), index)
    assert ctx.device_status() == 0


@pytest.mark.parametrize("last", ["SORT", "GATHER", "WALK", "INTEGRATE"])
@pytest.mark.parametrize("n", [1, 1408, 49152, 49153])
def test_one_segment(gcs_mod, n, last):
    gcs = gcs_mod
    p = gcs.reference_params(bounds_mode=gcs.BOUNDS_DEVICE)
    with gcs.Context(n) as ctx:
        ctx.upload(_stars(n, 5))
        ctx.run_stages(p, gcs.STAGE_BOUNDS, getattr(gcs, "STAGE_" + last))
        _same_again(gcs, ctx, p)


@pytest.mark.parametrize("last", ["SORT", "BUILD", "AGGREGATE", "INTEGRATE"])
@pytest.mark.parametrize("counts", [[1, 700, 5000], [1000] * 3 + [1] * 300, [30000, 40000]])
def test_segments(gcs_mod, counts, last):
    gcs = gcs_mod
    p = gcs.reference_params(bounds_mode=gcs.BOUNDS_DEVICE)
    with gcs.Context(sum(counts), len(counts)) as ctx:
        ctx.set_segments(counts)
        ctx.upload(_stars(sum(counts), 7))
        ctx.run_stages(p, gcs.STAGE_BOUNDS, getattr(gcs, "STAGE_" + last))
        _same_again(gcs, ctx, p)


def test_after_a_captured_step(gcs_mod):
    import torch
    gcs = gcs_mod
    p = gcs.reference_params(bounds_mode=gcs.BOUNDS_DEVICE)
    stream = torch.cuda.Stream()
    with gcs.Context(5000) as ctx:
        ctx.set_stream(stream.cuda_stream)
        ctx.upload(_stars(5000, 6))
        ctx.set_graphs(True)
        for _ in range(2):
            ctx.step(p)
            _same_again(gcs, ctx, p)
