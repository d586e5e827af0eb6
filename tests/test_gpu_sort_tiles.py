"""The radix sort at the edges of its tile rule: the last size of the
1,024-key tiles and the first of the wider ones, partial tiles and look-back
groups, one full wave of tiles and more than one, with duplicate keys and
(for segments) the segment-id passes, against numpy's stable sort."""
import numpy as np
import pytest

from conftest import small_collision

pytestmark = pytest.mark.gpu

WAVE = 296 * 512  # kSortWave * kSortThreads


@pytest.mark.parametrize("n", [1023, 1025, 16 * 1024, 16 * 1024 + 1, 148 * 1024, 148 * 1024 + 1, 2 * WAVE, 2 * WAVE + 1,
                               7 * WAVE, 8 * WAVE + 1])
def test_sort_at_tile_rule_edges(gcs_mod, n):
    gcs = gcs_mod
    rng = np.random.default_rng(n)
    stars = np.resize(small_collision(4096, 1024, 512, seed=n % 97), n)  # every key many times over
    jitter = rng.random(n) < 0.7
    for f in ("x", "y", "z"):
        stars[f] += np.where(jitter, rng.normal(0, 1e-2, n), 0.0).astype(np.float32)
    p = gcs.reference_params(bounds_mode=gcs.BOUNDS_DEVICE)
    for counts in ([n], [n // 3, 1, n - n // 3 - 1]):
        with gcs.Context(n, len(counts)) as ctx:
            ctx.set_segments(counts)
            ctx.upload(stars)
            ctx.run_stages(p, gcs.STAGE_BOUNDS, gcs.STAGE_ENCODE)
            keys = ctx.read(gcs.BUF_KEYS_UNSORTED)
            ctx.run_stages(p, gcs.STAGE_SORT, gcs.STAGE_SORT)
            order, at = [], 0
            for c in counts:
                order.append(at + np.argsort(keys[at:at + c], kind="stable"))
                at += c
            order = np.concatenate(order)
            np.testing.assert_array_equal(ctx.read(gcs.BUF_INDEX), order)
            np.testing.assert_array_equal(ctx.read(gcs.BUF_KEYS), keys[order])
            assert ctx.device_status() == 0
