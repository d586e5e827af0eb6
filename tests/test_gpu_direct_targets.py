"""The FP64 direct sum around the number of targets (eight an SM) up to which a
block takes two of them, in any order, against the oracle.  Bound: 700 terms of
random signs, some ten roundings of 2^-53 each, on the size of the largest sum."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_targets", [1, 2, 3, 1183, 1184, 1185, 1186, 1187, 1188])
@pytest.mark.parametrize("n", [700, 2500])
def test_direct_targets(gcs_mod, oracle_mod, n, n_targets):
    gcs = gcs_mod
    rng = np.random.default_rng(n_targets)
    st = np.zeros(n, gcs.STAR_DTYPE)
    for f in ("x", "y", "z"):
        st[f] = rng.normal(0, 3, n).astype(np.float32)
    st["mass"] = rng.random(n).astype(np.float32)
    targets = rng.integers(0, n, n_targets)
    p = gcs.reference_params(epsilon_sq=1e-2, G=1.5)
    with gcs.Context(n) as ctx:
        ctx.upload(st)
        got = ctx.direct_fp64(p, targets)
    ref = oracle_mod.direct_fp64(np.stack([st[f] for f in ("x", "y", "z", "mass")], 1), targets, p.G,
                                 float(p.epsilon_sq))
    np.testing.assert_allclose(got, ref, rtol=0, atol=1e-12 * np.abs(ref).max())
