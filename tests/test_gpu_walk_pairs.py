"""The walk of a group by two warps (contexts of few groups) and by one:
accelerations of sampled targets against the oracle's walk of the same tree
(the walk tolerance of the parity tests: 1e-5 relative at the 99.9th
percentile, 1e-4 at most); a scenario's bits the same alone, where its
groups get two warps, and beside others, where they get one; and the host
step the same bits as the device step."""
import numpy as np
import pytest

from conftest import rel_err

pytestmark = pytest.mark.gpu

LAST = 20 * 148 * 32  # the last size of two warps a group on 148 SMs
EDGES = [4097, 45056, LAST, LAST + 1]


def _stars(gcs, n, seed):
    return gcs.collision_pair(max(n, 64), 0.6, 6.0, 0.5, 40.0, seed)[:n]


def _params(gcs, **kw):
    return gcs.reference_params(bounds_mode=gcs.BOUNDS_DEVICE, theta=0.5, epsilon_sq=0.02 ** 2, dt=0.0025, leaf_size=8,
                                walk_batch=64, com_fp64=1, **kw)


@pytest.mark.parametrize("n", [2, 33, 700] + EDGES)
@pytest.mark.parametrize("frontier", [1, 0])
def test_small_walk_matches_oracle(gcs_mod, oracle_mod, n, frontier):
    gcs = gcs_mod
    p = _params(gcs, with_potential=1)
    with gcs.Context(n) as ctx:
        ctx.upload(_stars(gcs, n, n))
        ctx.set_walk_frontier(frontier)
        ctx.run_stages(p, gcs.STAGE_BOUNDS, gcs.STAGE_WALK)
        pos, acc, nodes = ctx.read(gcs.BUF_POS), ctx.read(gcs.BUF_ACCEL), ctx.read(gcs.BUF_NODES)
        assert ctx.device_status() == 0
    t = np.unique(np.random.default_rng(n).integers(0, n, 1024))
    if n < 64:
        t = np.arange(n)
    t[-1] = n - 1  # the last, partial group
    ref, _ = oracle_mod.walk_targets(pos, nodes, p.G, p.epsilon_sq, p.theta, p.leaf_size, t)
    scale = np.median(np.linalg.norm(ref[:, :3], axis=1))
    e = rel_err(acc[t][:, :3], ref[:, :3], floor=1e-3 * scale)
    assert np.percentile(e, 99.9) <= 1e-5 and e.max() <= 1e-4, (np.percentile(e, 99.9), e.max())
    np.testing.assert_allclose(acc[t][:, 3], ref[:, 3], rtol=1e-5)


@pytest.mark.parametrize("leaf,batch,theta,pot,frontier", [(8, 64, 0.5, 0, 1), (1, 32, 0.7, 1, 1), (32, 64, 0.7, 1, 1),
                                                           (4, 17, 0.5, 0, 0), (16, 64, 0.0, 0, 1)])
def test_alone_and_mixed_same_bits(gcs_mod, leaf, batch, theta, pot, frontier):
    gcs = gcs_mod
    counts = [1, 2, 31, 700, 4097] + ([30000, 90000] if theta > 0 else [])
    parts = [_stars(gcs, max(n, 64), k)[:n] for k, n in enumerate(counts)]
    p = _params(gcs, with_potential=pot)
    p.leaf_size, p.walk_batch, p.theta = leaf, batch, theta
    fill = _stars(gcs, 100000, 99) if theta > 0 else _stars(gcs, 2000, 99)
    with gcs.Context(sum(counts) + len(fill), len(counts) + 1) as ctx:
        ctx.set_walk_frontier(frontier)
        ctx.set_segments(counts + [len(fill)])
        ctx.upload(np.concatenate(parts + [fill]))
        for _ in range(2):
            ctx.step(p)
        mixed, acc = ctx.download(), ctx.read(gcs.BUF_ACCEL)
        assert ctx.device_status() == 0
    at = 0
    for st in parts:
        with gcs.Context(len(st)) as ctx:
            ctx.set_walk_frontier(frontier)
            ctx.upload(st)
            for _ in range(2):
                ctx.step(p)
            assert ctx.download().tobytes() == mixed[at:at + len(st)].tobytes()
            assert ctx.read(gcs.BUF_ACCEL).tobytes() == acc[at:at + len(st)].tobytes()
        at += len(st)


@pytest.mark.parametrize("frontier", [1, 0])
@pytest.mark.parametrize("n", [5000, 45056, LAST])
def test_host_step_same_bits(gcs_mod, n, frontier):
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
