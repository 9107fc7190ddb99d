"""All-in leaves of a flop game: their betting-free river subgames run the kernel of their own with the
updater's range weighting the average sums and with root values going to the game. For both players and
every subgame (more than the resident CTAs take at once): a subgame's sums are the weight of the iteration
times the updater's reach, exactly (its only action is played with certainty), and the values of leaves
from the first to the last are those of the oracle, to 1e-4 of the largest (single-precision leaf
arithmetic)."""
import numpy as np
import pytest

from oracle import full_game as F
from oracle import oracle as O

pytestmark = pytest.mark.gpu

FLOP = (1 << 3) | (1 << 20) | (1 << 45)
STREETS = [((0.75,), True, 1), ((0.5,), True, 1)]


def test_all_in_leaves_of_both_players():
    import pokerrust_b200 as P
    (ff, fa, fr), (tf, ta, tr) = STREETS
    spec = P.full_spec(FLOP, 10.0, 100.0, flop_fracs=ff, flop_allin=fa, flop_raises=fr, turn_fracs=tf,
                       turn_allin=ta, turn_raises=tr, river_sizes=0b011, river_raises=2)
    rng = np.random.default_rng(6)
    init = rng.random((2, F.HANDS)).astype(np.float32)
    init[:, F.blocked(FLOP)] = 0.0
    init /= init.sum(axis=1, keepdims=True)
    g = P.FullGame(spec, init)
    tree = F.Tree(FLOP, 10.0, 100.0, STREETS)
    g.set_regrets((rng.random((g.edges, F.HANDS)) * 0.05).astype(np.float32))
    bt, leaves = g.batch(1), g.batch_leaves(1)
    assert bt.count == 48 * len(leaves) > 4 * 148 and bt.shape(0)[1:] == (2, 1)
    order = P.card_order()
    for p in range(2):
        before = bt.all_rows(1).reshape(bt.count, 2, F.HANDS)
        g.half_iteration(p)
        R, LV = g.reach(), g.leaf_values()
        sums = bt.all_rows(1).reshape(bt.count, 2, F.HANDS)
        assert np.array_equal(sums[:, 1 - p], before[:, 1 - p])
        checked = {0, len(leaves) // 3, 2 * len(leaves) // 3, len(leaves) - 1}
        s = 0
        for j, node in enumerate(leaves):
            board = tree.board[node]
            want = np.zeros(F.HANDS)
            for c in range(52):
                if board >> c & 1:
                    continue
                live = (order & np.uint64(board | (1 << c))) == 0
                assert np.array_equal(sums[s, p][live], R[node, p][live]), (p, s)
                s += 1
                if j in checked:
                    o = O.Subgame(board | (1 << c), tree.stake[node], tree.stack[node], 0b011, 2,
                                  R[node, 0], R[node, 1])
                    want += o.value(p)[1] / 48
            if j in checked:
                got = LV[tree.leaf_index[node]]
                assert np.abs(got - want).max() <= 1e-4 * np.abs(want).max(), (p, node)
    g.close()
