"""Deep one-sided trees: corner chains and steep density profiles, where a
256-particle run of the sorted order holds more than 32 finished subtrees for
the aggregation's second kernel (one a lane and turn of its warp).

On the CPU: that the inputs have such runs, and that taking a run's subtrees in
the order of position always finishes while the order in which they were
finished does not.  On the GPU: nodes bit for bit the oracle's, alone and as
segments, again without a build; accelerations against the oracle's walk; and
whole steps without a device status bit."""
import numpy as np
import pytest

import steep_inputs as S
from conftest import small_collision

INPUTS = {
    "chain": lambda gcs: S.corner_chain(gcs),
    "mirror": lambda gcs: S.corner_chain(gcs, mirror=True),
    "steep": lambda gcs: S.steep_profile(gcs),
    "steep_small": lambda gcs: S.steep_profile(gcs, n_outer=600, seed=2),
}


@pytest.mark.parametrize("name", INPUTS)
def test_subtrees_by_position_always_finish(oracle_mod, name):
    import gcs
    st = INPUTS[name](gcs)
    tree = S.sorted_tree(oracle_mod, st)
    runs = S.subtrees(tree, len(st))
    assert max(len(r) for r in runs) > S.LANES
    assert S.replay(tree, len(st), S.by_position) == 0
    # a right child waits, a left child never does: the mirror image has none to wait
    assert (S.replay(tree, len(st), S.by_completion) > 0) == (name != "mirror")


def _check_nodes(gcs, oracle, ctx, counts, com_fp64):
    n, leaf0 = sum(counts), sum(counts) - len(counts)
    pos, nodes, bd = ctx.read(gcs.BUF_POS), ctx.read(gcs.BUF_NODES), ctx.read(gcs.BUF_BUILD)
    off = 0
    for k, c in enumerate(counts):
        seg, b = nodes[off - k:off - k + c - 1].copy(), bd[off - k:off - k + c - 1]
        for f in ("child_left", "child_right"):
            v = seg[f].astype(np.int64)
            seg[f] = np.where(v >= leaf0, v - leaf0 - off + c - 1, v - (off - k))
        ref, box = oracle.aggregate(pos[off:off + c], seg["child_left"], seg["child_right"], seg["range_end"] - off,
                                    com_fp64=bool(com_fp64))
        for f in ("mass", "width", "com_x", "com_y", "com_z"):
            np.testing.assert_array_equal(seg[f], ref[f], err_msg=f)
        np.testing.assert_array_equal(np.stack([b[f] for f in ("min_x", "min_y", "min_z")], 1), box[:, :3])
        np.testing.assert_array_equal(np.stack([b[f] for f in ("max_x", "max_y", "max_z")], 1), box[:, 3:])
        off += c
    assert off == n


@pytest.mark.gpu
@pytest.mark.parametrize("com_fp64", [0, 1])
@pytest.mark.parametrize("names", [[k] for k in INPUTS] + [["steep_small", "chain", "", "mirror", "steep"]])
def test_nodes(gcs_mod, oracle_mod, names, com_fp64):
    gcs = gcs_mod
    parts = [INPUTS[k](gcs) if k else small_collision(300, 50, 27, seed=3) for k in names]
    counts = [len(s) for s in parts]
    p = gcs.reference_params(bounds_mode=gcs.BOUNDS_DEVICE, theta=0.5, epsilon_sq=4e-4, com_fp64=com_fp64)
    with gcs.Context(sum(counts), len(counts)) as ctx:
        ctx.set_segments(counts)
        ctx.upload(np.concatenate(parts))
        ctx.run_stages(p, gcs.STAGE_BOUNDS, gcs.STAGE_AGGREGATE)
        for _ in range(2):
            assert ctx.device_status() == 0
            _check_nodes(gcs, oracle_mod, ctx, counts, com_fp64)
            ctx.run_stages(p, gcs.STAGE_AGGREGATE, gcs.STAGE_AGGREGATE)


@pytest.mark.gpu
@pytest.mark.parametrize("graphs", [0, 1])
def test_steps(gcs_mod, oracle_mod, graphs):
    """Accelerations of every particle of the first step within 2e-5 of the sum
    of its terms' sizes (up to 6,200 terms of FP32 rounding 2^-24 each, summed
    in two orders: below 1e-5 were all at one standard deviation)."""
    import torch
    gcs = gcs_mod
    st = INPUTS["steep"](gcs)
    p = gcs.reference_params(bounds_mode=gcs.BOUNDS_DEVICE, theta=0.5, epsilon_sq=4e-4, com_fp64=1, leaf_size=8,
                             walk_batch=64, dt=1e-5)
    stream = torch.cuda.Stream()
    with gcs.Context(len(st)) as ctx:
        ctx.set_stream(stream.cuda_stream)
        ctx.upload(st)
        ctx.run_stages(p, gcs.STAGE_BOUNDS, gcs.STAGE_WALK)
        pos, acc, nodes = ctx.read(gcs.BUF_POS), ctx.read(gcs.BUF_ACCEL), ctx.read(gcs.BUF_NODES)
        ref = oracle_mod.walk(pos, nodes, p.G, p.epsilon_sq, p.theta, p.leaf_size)
        x = pos.astype(np.float64)
        size = np.empty(len(x))
        for i0 in range(0, len(x), 512):
            d = x[None, :, :3] - x[i0:i0 + 512, None, :3]
            r2 = (d * d).sum(-1)
            size[i0:i0 + 512] = (x[:, 3] * np.sqrt(r2) / (r2 + p.epsilon_sq) ** 1.5).sum(1)
        err = np.linalg.norm(acc[:, :3].astype(np.float64) - ref[:, :3], axis=1)
        assert (err <= 2e-5 * p.G * size).all(), (err / (p.G * size)).max()
        ctx.set_graphs(bool(graphs))
        for _ in range(4):
            ctx.step(p)
        assert ctx.device_status() == 0
        assert np.isfinite(ctx.read(gcs.BUF_POS)).all()
