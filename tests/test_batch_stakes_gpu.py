"""A fold that costs nothing: at the smallest pot half of it rounds to zero, so a fold before any bet of
the folder moves no chips and every hand's value there is zero, whether or not the fold's scan is shared
with its sibling call. Values and best responses in double precision against the oracle, to 1e-9 of the
largest entry, and one CFR iteration to 1e-4, as in the other batch tests."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("K", [2, 3, 4])
def test_folds_of_no_stake(K):
    import pokerrust_b200 as P
    specs, ranges = P.random_subgames(3, seed=51)
    specs["pot"] = np.finfo(np.float32).smallest_subnormal
    specs["stack"], specs["sizes"], specs["max_raises"] = 1.0, 4, 2
    b = P.Batch(specs, ranges)
    for c in range(2):
        b.set_config(c, K, 1, 0)
    rng = np.random.default_rng(52)
    oracles = []
    for s, sp in enumerate(specs):
        o = O.Subgame(int(sp["board"]), float(sp["pot"]), float(sp["stack"]), int(sp["sizes"]),
                      int(sp["max_raises"]), ranges[s, 0], ranges[s, 1])
        o.regrets = rng.random((o.edges, 1326), dtype=np.float32)
        b.set_regrets(s, o.regrets)
        oracles.append(o)
    br0, br1, _ = b.exploitability(use_average=False, fp64=True)
    values = [b.root_values(p)[0] for p in range(2)]
    for s, o in enumerate(oracles):
        for p, got in ((0, br0[s]), (1, br1[s])):
            want = o.best_response(p)[0]
            assert abs(got - want) <= 1e-9 * abs(want), p
            row = o.value(p)[1]
            assert np.abs(values[p][s] - row).max() <= 1e-9 * np.abs(row).max(), p
    b.iterate(1)
    for s, o in enumerate(oracles):
        o.iterate(1)
        live = (P.card_order() & np.uint64(specs[s]["board"])) == 0
        want = o.regrets[:, live]
        assert np.abs(b.regrets(s)[:, live] - want).max() <= 1e-4 * np.abs(want).max()
    b.close()
