"""Copies into pageable host memory through the pinned pieces: sizes around
the threshold (1 MiB), the piece (512 KiB) and a full ring (8 pieces), from
two threads at once (one of them copies plainly), again after every context
that held the threads is gone, and into memory at an odd address."""
import threading

import numpy as np
import pytest

from conftest import small_collision

pytestmark = pytest.mark.gpu

PIECE = (512 << 10) // 32  # Stars


def _stars(gcs, n, seed):
    st = np.resize(small_collision(1024, 256, 128, seed=seed), n)
    st["x"] = np.arange(n, dtype=np.float32)
    return st


@pytest.mark.parametrize("n", [2 * PIECE - 1, 2 * PIECE, 2 * PIECE + 1, 8 * PIECE, 8 * PIECE + 3, 21 * PIECE + 17])
def test_download_pageable(gcs_mod, n):
    gcs = gcs_mod
    st = _stars(gcs, n, 1)
    for _ in range(2):  # the second makes the threads again
        with gcs.Context(n) as ctx:
            ctx.upload(st)
            odd = np.zeros(n * 32 + 1, np.uint8)[1:].view(gcs.STAR_DTYPE)
            assert ctx.download(out=odd).tobytes() == st.tobytes()
            assert ctx.download(5, n - 9).tobytes() == st[5:n - 4].tobytes()
            pb = ctx.download_playback()
            np.testing.assert_array_equal(pb["x"], st["x"])
            np.testing.assert_array_equal(pb["r"], st["r"])


def test_download_two_threads(gcs_mod):
    gcs = gcs_mod
    n, errors = 9 * PIECE, []

    def one(seed):
        try:
            st = _stars(gcs, n, seed)
            with gcs.Context(n) as ctx:
                ctx.upload(st)
                for _ in range(8):
                    assert ctx.download().tobytes() == st.tobytes()
        except Exception as e:  # reported by the test's thread
            errors.append(e)

    threads = [threading.Thread(target=one, args=(k,)) for k in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
