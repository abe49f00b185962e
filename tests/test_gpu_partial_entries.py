"""Partial traces of pure states with few traced configurations run one thread per entry, the others as
staged products: both sides of the rule, against numpy sums over the same amplitudes. An entry adds at most 2^6
products of total weight <= 1, so its rounding error stays below 2^6 * 2.3e-16 = 1.5e-14."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# (n, kept, batch, one thread per entry)
@pytest.mark.parametrize("n,keep,B,entries", [
    (2, [2], 1, True), (3, [1, 3], 1, True), (4, [2, 3], 5, True), (5, [4], 1, True), (6, [1, 2, 3, 4, 6], 1, True),
    (6, [5], 1, False), (8, [2, 3, 5, 8], 1, True), (8, [1, 4, 6], 1, False), (10, [1, 3, 5, 7, 9, 10], 3, True),
    (11, [1, 2, 4, 6, 8, 11], 1, True), (11, [1, 2, 4, 6, 8], 1, False), (9, [1, 2, 3, 4, 5, 6, 7, 9], 8, True),
    (9, [1, 2, 3, 4, 5, 6, 7, 9], 9, False), (10, list(range(2, 11)), 1, True), (12, list(range(3, 13)), 1, False)])
def test_both_sides(mq, n, keep, B, entries):
    from mossquantum_b200 import _native as N
    rng = np.random.default_rng(7 * n + B)
    v = rng.normal(size=(1 << n, B)) + 1j * rng.normal(size=(1 << n, B))
    v /= np.linalg.norm(v, axis=0)
    traced = [q for q in range(1, n + 1) if q not in keep]
    N.profile(True)
    got = [mq.partial_tr(mq.StateVector(v[:, 0]), traced)] if B == 1 else mq.partial_tr(mq.BatchStateVector(v), traced)
    seen = N.profile_report()
    N.profile(False)
    assert ("k_partial_entries" in seen, "k_partial_outer" in seen) == (entries, not entries)
    order = [n - q for q in reversed(traced)] + [n - q for q in reversed(keep)]
    for b in range(B):
        m = v[:, b].reshape([2] * n).transpose(order).reshape(-1, 1 << len(keep))
        assert np.max(np.abs(got[b].to_numpy() - m.T @ m.conj())) <= 1.5e-14
