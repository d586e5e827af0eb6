"""The helper threads of pageable copies sleep while a host step's walk has no
finished chunk to copy: over host steps whose walk takes far longer than the
copies, the process uses not much more than the calling thread's own time (the
helpers' share is the copying: 32 MB a step, some 3 ms of their time, and about
as much of waking and waiting for pieces on their way)."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_helpers_sleep_through_the_walk(gcs_mod):
    gcs = gcs_mod
    n = 1000000
    p = gcs.reference_params(bounds_mode=gcs.BOUNDS_DEVICE, theta=0.3, epsilon_sq=4e-4, leaf_size=8, walk_batch=64)
    out = np.zeros(n, gcs.STAR_DTYPE)
    with gcs.Context(n) as ctx:
        ctx.upload(gcs.collision_pair(n, 0.6, 6.0, 0.5, 40.0, 2))
        for _ in range(4):  # 64 MiB: the helpers exist
            ctx.step_host(p, out)
        shares = []
        for _ in range(5):
            cpu, wall = time.process_time(), time.perf_counter()
            ctx.step_host(p, out)
            shares.append((time.process_time() - cpu) / (time.perf_counter() - wall))
        assert ctx.device_status() == 0
    assert np.median(shares) < 2.5, shares  # all four threads awake: near 4


def test_helpers_sleep_behind_queued_steps(gcs_mod):
    """A download queued behind steps: its helpers sleep until the first piece
    has landed."""
    gcs = gcs_mod
    n = 1000000
    p = gcs.reference_params(bounds_mode=gcs.BOUNDS_DEVICE, theta=0.5, epsilon_sq=4e-4, leaf_size=8, walk_batch=64)
    out = np.zeros(n, gcs.STAR_DTYPE)
    with gcs.Context(n) as ctx:
        ctx.upload(gcs.collision_pair(n, 0.6, 6.0, 0.5, 40.0, 2))
        for _ in range(4):
            ctx.download(out=out)
        shares = []
        for _ in range(3):
            cpu, wall = time.process_time(), time.perf_counter()
            for _ in range(20):
                ctx.step(p)
            ctx.download(out=out)
            shares.append((time.process_time() - cpu) / (time.perf_counter() - wall))
        assert ctx.device_status() == 0
    assert np.median(shares) < 2.0, shares
