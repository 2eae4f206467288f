"""The branch-free window rule of the kernels (phi_window_flat in velo_kernels.cuh: two halving
searches, the "found" flag from the elements beside the first one, the reference's own search
where rounding at the lower edge leaves it open), restated in float32, against the reference's
searches probe for probe (VeloTools.cuh:6-42), on the modules and edge values of the window
oracle's test."""
import numpy as np
import pytest

from oracle import mlp_oracle
from test_window_oracle import MARGIN, edge_values, module, scalar_window


def flat_window(a, value, margin):
    lo, hi = np.float32(value - margin), np.float32(value + margin)
    il = ih = 0
    left = len(a)
    while left > 1:
        half = left >> 1
        il += half if lo > a[il + half - 1] else 0
        ih += half if hi > a[ih + half - 1] else 0
        left -= half
    inside = lambda i: abs(np.float32(value - a[i])) < margin  # noqa: E731
    found = inside(il)
    if not found and not lo > a[il] and (a[il] < value or (il > 0 and inside(il - 1))):
        found = mlp_oracle.window_first(a, value, margin) != -1
    return (il, il + max(ih - il + inside(ih), 1)) if found else (-1, -1)


@pytest.mark.parametrize("sizes", [(1, 5), (60, 70), (120, 260)])
def test_flat_rule_equals_reference_searches(sizes):
    rng = np.random.default_rng(17)
    for trial in range(60):
        n = int(rng.integers(*sizes))
        a = module(rng, n, trial % 3)
        v = np.concatenate([rng.uniform(-3.5, 3.5, 10).astype(np.float32), a[rng.integers(0, n, 5)],
                            edge_values(rng, a, 25)])
        for x in v:
            assert flat_window(a, x, MARGIN) == scalar_window(a, x), (trial, n, x)
