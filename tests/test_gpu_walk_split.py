"""Walk groups split into parts: segments at both sides of every size where
the number of parts changes.  Accelerations of sampled targets against the
oracle's walk of the same tree (the walk tolerance of the parity tests:
1e-5 relative at the 99.9th percentile, 1e-4 at most), each segment's bits
the same alone and beside others, and the host step (whose chunks of groups
must not cut a split group) the same bits as the device step."""
import numpy as np
import pytest

from conftest import rel_err

pytestmark = pytest.mark.gpu

EDGES = [24 * 1024, 24 * 1024 + 1, 64 * 1024, 64 * 1024 + 1, 160 * 1024, 160 * 1024 + 1]


def _stars(gcs, n, seed):
    return gcs.collision_pair(n, 0.6, 6.0, 0.5, 40.0, seed)


def _params(gcs, **kw):
    return gcs.reference_params(bounds_mode=gcs.BOUNDS_DEVICE, theta=0.5, epsilon_sq=0.02 ** 2, dt=0.0025, leaf_size=8,
                                walk_batch=64, com_fp64=1, **kw)


@pytest.mark.parametrize("n", [33, 700] + EDGES)
@pytest.mark.parametrize("frontier", [1, 0])
def test_split_groups_match_oracle(gcs_mod, oracle_mod, n, frontier):
    gcs = gcs_mod
    p = _params(gcs, with_potential=1)
    with gcs.Context(n) as ctx:
        ctx.upload(_stars(gcs, n, n))
        ctx.set_walk_frontier(frontier)
        ctx.run_stages(p, gcs.STAGE_BOUNDS, gcs.STAGE_WALK)
        pos, acc, nodes = ctx.read(gcs.BUF_POS), ctx.read(gcs.BUF_ACCEL), ctx.read(gcs.BUF_NODES)
        assert ctx.device_status() == 0
    t = np.unique(np.random.default_rng(n).integers(0, n, 1024))
    t[-1] = n - 1  # the last, partial group
    ref, _ = oracle_mod.walk_targets(pos, nodes, p.G, p.epsilon_sq, p.theta, p.leaf_size, t)
    scale = np.median(np.linalg.norm(ref[:, :3], axis=1))
    e = rel_err(acc[t][:, :3], ref[:, :3], floor=1e-3 * scale)
    assert np.percentile(e, 99.9) <= 1e-5 and e.max() <= 1e-4, (np.percentile(e, 99.9), e.max())
    np.testing.assert_allclose(acc[t][:, 3], ref[:, 3], rtol=1e-5)


def test_split_groups_alone_and_mixed_same_bits(gcs_mod):
    gcs = gcs_mod
    counts = [EDGES[0], 100, EDGES[3], EDGES[1], EDGES[5]]
    parts = [_stars(gcs, n, k) for k, n in enumerate(counts)]
    p = _params(gcs)
    with gcs.Context(sum(counts), len(counts)) as ctx:
        ctx.set_segments(counts)
        ctx.upload(np.concatenate(parts))
        for _ in range(2):
            ctx.step(p)
        mixed, acc = ctx.download(), ctx.read(gcs.BUF_ACCEL)
        assert ctx.device_status() == 0
    at = 0
    for st in parts:
        with gcs.Context(len(st)) as ctx:
            ctx.upload(st)
            for _ in range(2):
                ctx.step(p)
            assert ctx.download().tobytes() == mixed[at:at + len(st)].tobytes()
            assert ctx.read(gcs.BUF_ACCEL).tobytes() == acc[at:at + len(st)].tobytes()
        at += len(st)


@pytest.mark.parametrize("frontier", [1, 0])
@pytest.mark.parametrize("n", [5000, EDGES[0], EDGES[4]])
def test_split_groups_host_step_same_bits(gcs_mod, n, frontier):
    gcs = gcs_mod
    st = _stars(gcs, n, 3)
    p = _params(gcs)
    with gcs.Context(n) as ctx:
        ctx.set_walk_frontier(frontier)
        ctx.upload(st)
        ctx.step(p)
        ref = ctx.download()
        out = np.zeros(n, gcs.STAR_DTYPE)
        for _ in range(2):
            ctx.upload(st)
            ctx.step_host(p, out)
            assert out.tobytes() == ref.tobytes()
        ctx.step_host_io(p, st, out)
        assert out.tobytes() == ref.tobytes()
        assert ctx.device_status() == 0
