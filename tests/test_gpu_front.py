"""Bounds, encode and sort of a small scenario in one launch against the
separate stages and numpy's stable sort: every cluster shape at its edges,
duplicate keys, caller and device bounds, bounds given by an earlier stage
(the chunked host step), and the non-finite status bit."""
import numpy as np
import pytest

from conftest import small_collision

pytestmark = pytest.mark.gpu

K = 512  # pairs a block holds per item and thread


def _stars(n, seed):
    rng = np.random.default_rng(seed)
    st = np.resize(small_collision(2048, 512, 256, seed=seed), n)
    jitter = rng.random(n) < 0.8  # the rest keeps duplicate positions
    for f in ("x", "y", "z"):
        st[f] += np.where(jitter, rng.normal(0, 1e-2, n), 0.0).astype(np.float32)
    return st


@pytest.mark.parametrize("n", [1, 2, 33, K, 8 * K, 8 * K + 1, 16 * K, 16 * K + 1, 32 * K + 1, 48 * K + 1, 64 * K,
                               64 * K + 1, 96 * K - 1, 96 * K, 96 * K + 1])
@pytest.mark.parametrize("caller", [0, 1])
def test_front_equals_stages(gcs_mod, n, caller):
    gcs = gcs_mod
    st = _stars(n, n % 89)
    p = gcs.reference_params(bounds_mode=gcs.BOUNDS_CALLER if caller else gcs.BOUNDS_DEVICE, global_min=-20.0,
                             global_max=25.0)
    with gcs.Context(n) as ctx:
        ctx.upload(st)
        ctx.run_stages(p, gcs.STAGE_BOUNDS, gcs.STAGE_SORT)
        keys, index = ctx.read(gcs.BUF_KEYS), ctx.read(gcs.BUF_INDEX)
        if not caller:
            lo, hi = ctx.read(gcs.BUF_BOUNDS)[0]
            xyz = np.stack([st[f] for f in ("x", "y", "z")])
            assert (lo, hi) == (xyz.min(), xyz.max())
        ctx.run_stages(p, gcs.STAGE_BOUNDS, gcs.STAGE_BOUNDS)
        ctx.run_stages(p, gcs.STAGE_ENCODE, gcs.STAGE_ENCODE)
        unsorted = ctx.read(gcs.BUF_KEYS_UNSORTED)
        order = np.argsort(unsorted, kind="stable")
        np.testing.assert_array_equal(keys, unsorted[order])
        np.testing.assert_array_equal(index, order)
        # encode and sort with the bounds of the stage above
        ctx.run_stages(p, gcs.STAGE_ENCODE, gcs.STAGE_SORT)
        np.testing.assert_array_equal(ctx.read(gcs.BUF_KEYS), keys)
        np.testing.assert_array_equal(ctx.read(gcs.BUF_INDEX), index)
        assert ctx.device_status() == 0


def test_front_reports_nonfinite(gcs_mod):
    gcs = gcs_mod
    st = _stars(5000, 4)
    st["y"][4321] = np.nan
    with gcs.Context(len(st)) as ctx:
        ctx.upload(st)
        ctx.run_stages(gcs.reference_params(bounds_mode=gcs.BOUNDS_DEVICE), gcs.STAGE_BOUNDS, gcs.STAGE_SORT)
        assert ctx.device_status(clear=True) == gcs.DEV_NONFINITE_POSITION
