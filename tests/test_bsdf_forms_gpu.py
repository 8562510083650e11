"""The warp-wide BSDF of the default Shade kernels against the out-of-line one:
re_bsdf_probe runs them on alternate warps of queries."""
import numpy as np
import pytest

import bsdf_cases as B
from renderingengine_b200 import _native as N

pytestmark = pytest.mark.gpu


def _hostile(q):
    """A fifth of the queries with what the checks refuse or barely pass."""
    q = q.copy()
    rng = np.random.default_rng(len(q))
    for field, values in (("perceptual_roughness", (0.0, 1e-4, 1.5, np.nan)), ("wo", ((0, 0, 0), (1, 0, 0), (0, 0, -1))),
                          ("wi", ((0, 0, 0), (np.inf, 0, 0))), ("random", ((0, 0, 0), (1, 0, 0), (0.999999, 0, 0.5))),
                          ("eta_incident", (0.0, -1.0)), ("allowed_lobes", (0, 1, 2, 4, 8))):
        at = rng.choice(len(q), len(q) // 25, replace=False)
        q[field][at] = np.array(values, q[field].dtype)[rng.integers(0, len(values), len(at))]
    return q


def _bits(results):
    return np.ascontiguousarray(results).view(np.uint32).reshape(results.size, -1)


@pytest.mark.parametrize("hostile", [False, True])
@pytest.mark.parametrize("model", list(B.MODELS) + ["mixed"])
def test_warp_form_equals_out_of_line_form(native, model, hostile):
    n = 64 * 400
    if model == "mixed":
        parts = [B.random_queries(m, n, seed=900 + m) for m in B.MODELS.values()]
        q = np.stack(parts)[np.random.default_rng(1).integers(0, len(parts), n), np.arange(n)]
    else:
        q = B.random_queries(B.MODELS[model], n, seed=800 + B.MODELS[model])
    if hostile:
        q = _hostile(q)
    # Each 32 queries twice in a row: an even and an odd warp.
    twice = np.repeat(q.reshape(-1, 1, 32), 2, axis=1).reshape(-1)
    got = B.device_probe(N, twice).reshape(-1, 2, 32)
    assert got["sample_valid"].mean() > 0.1
    even, odd = _bits(got[:, 0]), _bits(got[:, 1])
    differ = (even != odd).any(1)
    assert not differ.any(), f"{differ.sum()} of {n} queries, words {np.flatnonzero((even != odd).any(0))}"


@pytest.mark.parametrize("n", [1, 31, 33, 95, 129])
def test_ragged_counts(native, n):
    q = B.random_queries(5, 256, seed=3)
    want = B.device_probe(N, q)[:n]
    np.testing.assert_array_equal(_bits(B.device_probe(N, q[:n])), _bits(want))
