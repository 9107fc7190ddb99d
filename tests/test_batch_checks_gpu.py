"""River subgames without a bet (no chips behind: check, check, showdown) have their own CFR kernel when
they fill a batch's class. Against the general kernel, which solves the same subgames in a batch that
also holds one with bets, every regret and average sum agrees bit for bit (the arithmetic is the same,
operand for operand; the general kernel is held against the oracle by the other batch tests). Batches of 1, of one and two subgames per resident CTA and a remainder, uniform and linear sums."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _checks(P, n, seed):
    specs, ranges = P.random_subgames(n, seed=seed)
    specs["stack"] = 0.0
    return specs, ranges


@pytest.mark.parametrize("n", [1, 5, 592, 700, 1185])
@pytest.mark.parametrize("average,linear", [(False, False), (True, False), (True, True)])
def test_checks_match_the_general_kernel(n, average, linear):
    import pokerrust_b200 as P
    specs, ranges = _checks(P, n, seed=31)
    one, one_range = P.random_subgames(1, seed=32)
    rng = np.random.default_rng(33)
    got = P.Batch(specs, ranges)
    want = P.Batch(np.concatenate([specs, one]), np.concatenate([ranges, one_range]))
    assert got.shape(0)[1:] == (2, 1) and want.shape(n)[2] > 1
    for b in (got, want):
        if average:
            b.enable_average()
        if linear:
            b.set_linear_average(True)
    for s in {0, n // 2, n - 1}:  # one-action nodes play their action at every regret
        reg = (rng.random((2, P.HANDS), dtype=np.float32) - 0.25).clip(0) * 0.1
        got.set_regrets(s, reg)
        want.set_regrets(s, reg)
    for _ in range(2):
        got.iterate(2)
        want.iterate(2)
        for which in range(1 + average):
            assert np.array_equal(got.all_rows(which), want.all_rows(which)[:2 * n])
    got.close()
    want.close()
