"""Leaf counts at the edges of the leaf phase, which takes leaves in groups (16 in single, 8 in double
precision) and their scans in batches of 4 or 8: trees of 1, 5, 9, 13 and more leaves, at every number of
hands per thread. Best responses and strategy values run in double precision on both sides, so their root
vectors agree to 1e-9 of the largest entry, as in the other batch tests; the single-precision CFR
passes of every configuration agree bit for bit."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

# (chips behind in pots, bet sizes, raises)
SHAPES = [(0.0, 7, 1), (4.0, 4, 1), (4.0, 3, 1), (4.0, 7, 1), (4.0, 4, 3), (4.0, 1, 3), (4.0, 3, 2), (4.0, 7, 3)]


@pytest.mark.parametrize("K", [2, 3, 4])
def test_leaf_counts_match_the_oracle(K):
    import pokerrust_b200 as P
    specs, ranges = P.random_subgames(len(SHAPES), seed=41)
    for sp, (behind, sizes, raises) in zip(specs, SHAPES):
        sp["stack"], sp["sizes"], sp["max_raises"] = behind * sp["pot"], sizes, raises
    b = P.Batch(specs, ranges)
    plain = P.Batch(specs, ranges)  # the configuration a batch starts with
    leaves = [b.shape(s)[2] for s in range(b.count)]
    assert min(leaves) == 1 and {5, 9, 13} <= set(leaves) and max(leaves) > 16, leaves
    rng = np.random.default_rng(42)
    oracles = []
    for s, sp in enumerate(specs):
        o = O.Subgame(int(sp["board"]), float(sp["pot"]), float(sp["stack"]), int(sp["sizes"]),
                      int(sp["max_raises"]), ranges[s, 0], ranges[s, 1])
        o.regrets = rng.random((o.edges, 1326), dtype=np.float32)
        b.set_regrets(s, o.regrets)
        plain.set_regrets(s, o.regrets)
        oracles.append(o)
    for c in range(2):
        b.set_config(c, K, 1, 0)
    br0, br1, _ = b.exploitability(use_average=False, fp64=True)
    values = [b.root_values(p)[0] for p in range(2)]
    for s, o in enumerate(oracles):
        for p, got in ((0, br0[s]), (1, br1[s])):
            want = o.best_response(p)[0]
            assert abs(got - want) <= 1e-9 * abs(want), (leaves[s], p)
            row = o.value(p)[1]
            assert np.abs(values[p][s] - row).max() <= 1e-9 * np.abs(row).max(), (leaves[s], p)
    for x in (b, plain):
        x.enable_average()
        x.iterate(2)
    for which in range(2):
        assert np.array_equal(b.all_rows(which), plain.all_rows(which))
    b.close()
    plain.close()
