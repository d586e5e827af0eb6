"""The FP64 direct sum with infinite and NaN positions and masses, coincident
particles without softening and infinite softening: the same NaN, infinite and
finite components as the oracle's sum (relative 1e-12: some 700 terms of one
sign pattern, each a few 2^-53)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

INF, NAN = np.inf, np.nan


@pytest.mark.parametrize("targets", [[3], [0, 1, 2, 3, 4, 600], list(range(0, 700, 7))])
@pytest.mark.parametrize("special,eps2", [({"x": INF}, 1e-4), ({"y": -INF}, 0.0), ({"x": INF, "z": -INF}, 1e-4),
                                          ({"x": INF, "mass": 0.0}, 1e-4), ({"y": NAN}, 1e-4), ({"mass": INF}, 1e-4),
                                          ({"mass": -INF}, 0.0), ({"mass": NAN}, 1e-4), ({"copy": 3}, 0.0),
                                          ({"copy": 3, "mass": 0.0}, 0.0), ({}, INF), ({"x": INF}, INF), ({}, 1e-4)])
def test_components(gcs_mod, oracle_mod, special, eps2, targets):
    gcs = gcs_mod
    rng = np.random.default_rng(11)
    st = np.zeros(700, gcs.STAR_DTYPE)
    for f in ("x", "y", "z"):
        st[f] = rng.normal(0, 3, 700).astype(np.float32)
    st["mass"] = rng.random(700).astype(np.float32) + 0.1
    for f, v in special.items():
        if f == "copy":
            for g in ("x", "y", "z"):
                st[g][250] = st[g][v]
        else:
            st[f][250] = v
    p = gcs.reference_params(epsilon_sq=eps2, G=1.5)
    with gcs.Context(700) as ctx:
        ctx.upload(st)
        got = ctx.direct_fp64(p, np.array(targets))
    xyzm = np.stack([st[f] for f in ("x", "y", "z", "mass")], 1)
    ref = oracle_mod.direct_fp64(xyzm, targets, p.G, float(p.epsilon_sq))
    with np.errstate(all="ignore"):
        scale = np.abs(ref[np.isfinite(ref)]).max() if np.isfinite(ref).any() else 1.0
    np.testing.assert_array_equal(np.isnan(got), np.isnan(ref))
    np.testing.assert_array_equal(np.isinf(got), np.isinf(ref))
    np.testing.assert_allclose(got, ref, rtol=1e-12, atol=1e-12 * scale, equal_nan=True)
