"""The aggregation above its blocks: sizes around the blocks' run of
particles and the largest context one block takes whole (2,048), segments
that end inside and at the edge of a run, duplicate
positions (deep chains of equal keys), and an aggregation run again without a
build.  Node masses, widths, boxes and centres of mass bit-exact against the
oracle, segment by segment."""
import numpy as np
import pytest

from conftest import small_collision

pytestmark = pytest.mark.gpu

RUN = 256  # particles an aggregation block owns


def _stars(n, seed, dup):
    rng = np.random.default_rng(seed)
    st = np.resize(small_collision(2048, 512, 256, seed=seed), n)
    for f in ("x", "y", "z"):
        st[f] += rng.normal(0, 1e-2, n).astype(np.float32)
    if dup:  # long runs of equal keys
        k = rng.integers(0, max(1, n // 700), n)
        for f in ("x", "y", "z"):
            st[f] = st[f][k]
    return st


@pytest.mark.parametrize("dup", [0, 1])
@pytest.mark.parametrize("com_fp64", [0, 1])
@pytest.mark.parametrize("counts", [[2], [RUN - 1], [RUN], [RUN + 1], [2 * RUN], [1023], [1025], [2048], [2049], [20000], [1200, 1, 847],
                                    [RUN, 1, RUN - 1, 2 * RUN, 3, 5000, 1]])
def test_nodes_above_blocks(gcs_mod, oracle_mod, counts, com_fp64, dup):
    gcs = gcs_mod
    n = sum(counts)
    parts = [_stars(c, 7 + k, dup) for k, c in enumerate(counts)]
    p = gcs.reference_params(bounds_mode=gcs.BOUNDS_DEVICE, theta=0.5, epsilon_sq=4e-4, com_fp64=com_fp64)
    with gcs.Context(n, len(counts)) as ctx:
        ctx.set_segments(counts)
        ctx.upload(np.concatenate(parts))
        ctx.run_stages(p, gcs.STAGE_BOUNDS, gcs.STAGE_AGGREGATE)
        for again in range(2):  # the second without a build in front
            pos, nodes, bd = ctx.read(gcs.BUF_POS), ctx.read(gcs.BUF_NODES), ctx.read(gcs.BUF_BUILD)
            assert ctx.device_status() == 0
            off = 0
            for k, c in enumerate(counts):
                seg = nodes[off - k: off - k + c - 1].copy()
                for f in ("child_left", "child_right"):
                    v = seg[f].astype(np.int64)
                    leaf = v >= n - len(counts)
                    seg[f] = np.where(leaf, v - (n - len(counts)) - off + (c - 1), v - (off - k))
                ref, box = oracle_mod.aggregate(pos[off:off + c], seg["child_left"], seg["child_right"],
                                                seg["range_end"] - off, com_fp64=bool(com_fp64))
                b = bd[off - k: off - k + c - 1]
                for f in ("mass", "width", "com_x", "com_y", "com_z"):
                    np.testing.assert_array_equal(seg[f], ref[f], err_msg=f)
                np.testing.assert_array_equal(np.stack([b["min_x"], b["min_y"], b["min_z"]], 1), box[:, :3])
                np.testing.assert_array_equal(np.stack([b["max_x"], b["max_y"], b["max_z"]], 1), box[:, 3:])
                off += c
            ctx.run_stages(p, gcs.STAGE_AGGREGATE, gcs.STAGE_AGGREGATE)
