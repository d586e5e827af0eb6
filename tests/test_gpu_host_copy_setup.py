"""When the pinned pieces and helper threads of pageable copies are made: not
for the first copies (a program with few would wait longer for them than for
its copies), once 64 MiB have been copied plainly, and given back with the last
context that copied.  Copies on both sides of that, and across it, are right."""
import gc
import os

import numpy as np
import pytest

from conftest import small_collision

pytestmark = pytest.mark.gpu

PIECE = (512 << 10) // 32  # Stars


def _threads():
    return set(os.listdir("/proc/self/task"))


def _stars(gcs, n, seed):
    st = np.resize(small_collision(1024, 256, 128, seed=seed), n)
    st["x"] = np.arange(n, dtype=np.float32)
    return st


@pytest.mark.parametrize("n", [2 * PIECE, 2 * PIECE + 1, 8 * PIECE + 3, 21 * PIECE + 17])
def test_set_up_once_earned(gcs_mod, n):
    gcs = gcs_mod
    assert os.cpu_count() >= 2
    gc.collect()  # no context of another test is still to go
    st = _stars(gcs, n, 1)
    for _ in range(2):
        with gcs.Context(n) as ctx:
            ctx.upload(st)
            before = _threads()
            plain = -(-(64 << 20) // (32 * n))  # downloads that make 64 MiB
            for k in range(plain):
                assert ctx.download().tobytes() == st.tobytes()
                assert not _threads() - before, k
            for _ in range(3):
                assert ctx.download().tobytes() == st.tobytes()
            assert 1 <= len(_threads() - before) <= 3
            odd = np.zeros(n * 32 + 1, np.uint8)[1:].view(gcs.STAR_DTYPE)
            assert ctx.download(out=odd).tobytes() == st.tobytes()
            assert ctx.download(5, n - 9).tobytes() == st[5:n - 4].tobytes()
            np.testing.assert_array_equal(ctx.download_playback()["x"], st["x"])
        assert _threads() <= before


def _blocked(task):
    with open(f"/proc/self/task/{task}/status") as f:
        return int(next(line.split()[1] for line in f if line.startswith("SigBlk")), 16)


def test_helpers_take_no_signals(gcs_mod):
    """The caller's handlers run on the caller's threads only."""
    import signal
    gcs = gcs_mod
    n = 21 * PIECE
    gc.collect()
    with gcs.Context(n) as ctx:
        ctx.upload(_stars(gcs, n, 1))
        before, mask = _threads(), signal.pthread_sigmask(signal.SIG_BLOCK, [])
        for _ in range(8):
            ctx.download()
        helpers = _threads() - before
        assert helpers
        for s in (signal.SIGINT, signal.SIGTERM, signal.SIGALRM, signal.SIGUSR1, signal.SIGCHLD):
            assert all(_blocked(t) >> (s - 1) & 1 for t in helpers)
        assert signal.pthread_sigmask(signal.SIG_BLOCK, []) == mask


def test_host_steps_across_it(gcs_mod):
    """Host steps into pageable memory before, at and after the set-up: the same
    Stars as device steps."""
    gcs = gcs_mod
    n = 300000
    st = gcs.collision_pair(n, 0.6, 6.0, 0.5, 40.0, 2)
    p = gcs.reference_params()
    out = np.zeros(n, gcs.STAR_DTYPE)
    with gcs.Context(n) as a, gcs.Context(n) as b:
        a.upload(st)
        b.upload(st)
        for _ in range(10):  # 9.6 MB each
            a.step_host(p, out)
            b.step(p)
            assert out.tobytes() == b.download().tobytes()
        assert a.device_status() == 0
