"""A context takes no more device memory than the same context took before the
sort's smaller tiles and the longer source lists of super-groups, so a server
under a fixed budget admits what it did.  Bytes of that version, 148 SMs."""
import pytest

pytestmark = pytest.mark.gpu

BEFORE = {(1, 1): 562568, (1, 1024): 77191224, (64, 4): 1134292, (100, 1): 1115956, (1000, 1): 8766836,
          (1000, 32): 11153188, (5000, 1): 43175412, (5000, 1024): 119806116, (20000, 1): 171014836,
          (20000, 4): 171572132, (37888, 1): 323975716, (100000, 32): 422731220, (300000, 1): 491256836,
          (1000000, 4): 732460116, (10000000, 1): 3829749476, (10000000, 1024): 3844268436,
          (300000000, 1): 103640353316}


@pytest.mark.parametrize("n,segments", BEFORE)
def test_no_more_than_before(gcs_mod, n, segments):
    assert gcs_mod.context_bytes(n, segments) <= BEFORE[n, segments]


@pytest.mark.parametrize("n,segments", [(5000, 1), (20000, 4), (100000, 32)])
def test_server_admits_what_it_did(gcs_mod, n, segments):
    gcs = gcs_mod
    p = gcs.reference_params(bounds_mode=gcs.BOUNDS_DEVICE)
    with gcs.Server(p, n, segments, float(BEFORE[n, segments])) as srv:
        assert srv.capacity == n
