"""The work that users of this framework have it do, as measurable cases over its public
entry points (pokerrust_b200.interface and the C ABI behind it).

  river       CFR passes of both players over the river roots of the fixed-flop limit game, ranges
              and results on the device (pr_evaluate_device): one root is a query about one spot,
              441 roots are one flop betting line of the game (49 turn cards x 9 turn lines),
              27,783 are the whole game, the benchmark's workload.
  river_host  the same two passes as the reference's host program makes them: upload, evaluate_cuda,
              download of every root.
  river_br    double-precision best responses of both players at river roots (the exploitability
              check).
  game        one CFR iteration of the whole fixed-flop limit game with average strategies.
  batch       general river subgames solved for a number of iterations, average sums read back: one
              subgame is an interactive solve, 4096 the benchmark's batch.
  adjoint     gradients of subgame values at their average strategies, on the device.
  train       training steps of the turn-leaf value network over a set of minibatches, then its
              parameters read back.
  full        CFR iterations of a flop game with general bets on every street, then the flop and
              turn average sums; with net=True its turn leaves are answered by the value network.
"""
import math

import numpy as np
import torch

import pokerrust_b200.interface as P

HANDS = 1326
STRIDE = 1328
DEV = "cuda"


def listed():
    return [
        # a query about one river root: latency of one CTA's chain of 48 river cards
        {"name": "river_one", "kind": "river", "roots": 1},
        # one flop betting line of the limit game: a few CTAs per SM
        {"name": "river_line", "kind": "river", "roots": 441},
        # the whole game's river roots, the benchmark's step
        {"name": "river_all", "kind": "river", "roots": 27783},
        # the drop-in boundary with host buffers, as the reference's program drives it
        {"name": "river_host_all", "kind": "river_host", "roots": 27783},
        # the exploitability check's river part, double precision
        {"name": "river_br_line", "kind": "river_br", "roots": 441},
        # one iteration of the whole limit game (upper tree, river passes, average sums)
        {"name": "limit_game", "kind": "game", "iterations": 1},
        # an interactive solve of one river spot
        {"name": "batch_one", "kind": "batch", "subgames": 1, "iterations": 200},
        # the benchmark's batch of general subgames
        {"name": "batch_4096", "kind": "batch", "subgames": 4096, "iterations": 100},
        # gradients of subgame values with respect to ranges and root strategies
        {"name": "adjoint_1024", "kind": "adjoint", "subgames": 1024},
        # an epoch of value-network training at the benchmark's batch
        {"name": "train_4096", "kind": "train", "samples": 4096, "steps": 64},
        # a flop game with bets on every street, river subgames solved in the same pass
        {"name": "flop_game", "kind": "full", "stack_pots": 3.0, "raises": 1, "iterations": 10, "net": False},
        # the same with value-network leaves: many small launches and a forward pass per player
        {"name": "flop_game_net", "kind": "full", "stack_pots": 3.0, "raises": 1, "iterations": 10, "net": True},
    ]


def log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["river", "river", "river", "river_host", "river_br", "batch", "batch", "adjoint", "train",
                       "full"])
    if kind in ("river", "river_host"):
        return {"kind": kind, "roots": log_int(rng, 1, 27000)}
    if kind == "river_br":
        return {"kind": kind, "roots": log_int(rng, 1, 900)}
    if kind == "batch":
        n = log_int(rng, 1, 4000)
        return {"kind": kind, "subgames": n, "iterations": rng.randint(20, 100)}
    if kind == "adjoint":
        return {"kind": kind, "subgames": log_int(rng, 1, 1000)}
    if kind == "train":
        return {"kind": kind, "samples": log_int(rng, 100, 4096), "steps": rng.randint(16, 64)}
    return {"kind": kind, "stack_pots": float(rng.choice([0.5, 1.0, 2.0, 4.0, 10.0])), "raises": 1,
            "iterations": rng.randint(2, 10), "net": rng.random() < 0.5}


# ---- inputs, from the seed alone ----

def torch_rng(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    return g


def hand_cards():
    """The two cards (low, high) of every hand in colex order, [1326] each."""
    hi = np.repeat(np.arange(52), np.arange(52))
    lo = np.concatenate([np.arange(c) for c in range(52)])
    return lo, hi


def touches(board_cards):
    """[1326] bool: the hand holds a card of the board."""
    lo, hi = hand_cards()
    on = np.zeros(52, bool)
    on[list(board_cards)] = True
    return on[lo] | on[hi]


def river_spots(n, seed):
    """A flop and n river roots in the game's order: 9 turn lines per turn card, 49 turn cards per
    flop line; equal bets of the limit structure."""
    rng = np.random.default_rng(seed)
    flop = sorted(int(c) for c in rng.choice(52, 3, replace=False))
    turns = [c for c in range(52) if c not in flop]
    turn = np.array([turns[(i // 9) % 49] for i in range(n)])
    bets = (1 + rng.integers(0, 4, n) + rng.integers(0, 5, n) + 2 * rng.integers(0, 5, n)).astype(np.float32)
    return flop, turn, bets


def river_inputs(n, seed):
    """Opponent ranges [2][n][1328] (U(0,1), a quarter of the hands zero, hands on the 4-card board
    zero) and bucket regrets [n][26][256] (clipped ones zero) on the device."""
    flop, turn, bets = river_spots(n, seed)
    g = torch_rng(seed)
    r = torch.rand((2, n, STRIDE), device=DEV, generator=g)
    r *= torch.rand((2, n, STRIDE), device=DEV, generator=g) >= 0.25
    lo, hi = (torch.tensor(x, device=DEV) for x in hand_cards())
    t = torch.tensor(turn, device=DEV)[:, None]
    hit = (lo[None] == t) | (hi[None] == t)
    for c in flop:
        hit |= ((lo == c) | (hi == c))[None]
    r[:, :, :HANDS] *= ~hit
    r[:, :, HANDS:] = 0
    reg = torch.rand((n, 26, 256), device=DEV, generator=g) * 100 - 30
    reg.clamp_(min=0)
    return flop, turn, bets, r, reg


def river_builder(n, seed):
    flop, turn, bets, r, reg = river_inputs(n, seed)
    mask = sum(1 << c for c in flop)
    b = P.Builder()
    for t, bet in zip(turn.tolist(), bets.tolist()):
        b.add(mask | (1 << t), bet)
    b.set_regrets(reg.cpu().numpy())
    return b, P.build_flop_tables(mask), r


class Tables:
    """A table handle that is released with its state."""

    def __init__(self, ptr):
        self.ptr = ptr

    def __del__(self):
        P.free_eval(self.ptr)


def full_inputs(case, seed):
    rng = np.random.default_rng(seed)
    flop = sum(1 << int(c) for c in rng.choice(52, 3, replace=False))
    pot = float(rng.integers(10, 100))
    ranges = rng.random((2, HANDS), dtype=np.float32)
    ranges[rng.random((2, HANDS)) < 0.3] = 0
    spec = P.full_spec(flop, pot, case["stack_pots"] * pot, flop_fracs=(0.75,), flop_raises=case["raises"],
                       turn_fracs=(0.75,), turn_raises=case["raises"], river_sizes=0b011, river_raises=1)
    return spec, ranges


def net_parameters(seed):
    rng = np.random.default_rng(seed)
    out = []
    for l in range(5):
        o, i = (2652 if l == 4 else 1024), (2706 if l == 0 else 1024)
        bound = math.sqrt(6.0 / i) * (0.5 if l == 4 else 1.0)
        W = (rng.random((o, i), dtype=np.float32) * 2 - 1) * np.float32(bound)
        out.append((W, (rng.random(o, dtype=np.float32) - 0.5) * np.float32(0.02)))
    return out


def make_net(rows, seed):
    net = P.ValueNet(rows, seed)
    for l, (W, b) in enumerate(net_parameters(seed)):
        net.set_layer(l, W, b)
    return net


MINIBATCHES = 4


def train_data(case, seed):
    """Minibatches (ranges, boards, scalars, targets) of turn states: normalised ranges, 4-card
    boards, pot / 200 and stack / (10 pot), values of the order of the pot."""
    n = case["samples"]
    g = torch_rng(seed)
    out = []
    for _ in range(MINIBATCHES):
        r = torch.rand((n, 2, HANDS), device=DEV, generator=g)
        r *= torch.rand((n, 2, HANDS), device=DEV, generator=g) >= 0.25
        cards = torch.rand((n, 52), device=DEV, generator=g).topk(4, dim=1).indices
        boards = (torch.ones_like(cards) << cards).sum(dim=1)
        lo, hi = (torch.tensor(x, device=DEV) for x in hand_cards())
        hit = ((boards[:, None] >> lo[None]) | (boards[:, None] >> hi[None])) & 1
        r *= (hit == 0)[:, None]
        r /= r.sum(dim=2, keepdim=True)
        s = torch.rand((n, 2), device=DEV, generator=g)
        y = torch.randn((n, 2 * HANDS), device=DEV, generator=g) * 0.25
        out.append((r, boards, s, y))
    return out


def batch_inputs(case, seed):
    """Specs and ranges of general river subgames: the bet trees are those of random_subgames for
    this count, boards and ranges come from the seed (U(0,1), a quarter of the hands zero, hands on
    the board zero, summing to 1)."""
    n = case["subgames"]
    specs, _ = P.random_subgames(n, seed=4321)
    rng = np.random.default_rng(seed)
    cards = rng.permuted(np.tile(np.arange(52), (n, 1)), axis=1)[:, :5].astype(np.uint64)
    specs["board"] = (np.uint64(1) << cards).sum(axis=1)
    ranges = rng.random((n, 2, HANDS), dtype=np.float32)
    ranges[rng.random((n, 2, HANDS), dtype=np.float32) < 0.25] = 0
    lo, hi = (x.astype(np.uint64) for x in hand_cards())
    hit = ((specs["board"][:, None] >> lo) | (specs["board"][:, None] >> hi)) & np.uint64(1)
    ranges *= (hit == 0)[:, None]
    ranges /= ranges.sum(axis=2, keepdims=True)
    return specs, ranges


def average_rows(case, seed, edges):
    """Average sums of each subgame's edges, [edges][1326] f32 in subgame order."""
    return np.random.default_rng(seed + 1).random((edges, HANDS), dtype=np.float32)


# ---- what a program has in hand before the call ----

def prepare(case, seed):
    kind = case["kind"]
    st = {"kind": kind}
    if kind in ("river", "river_host", "river_br"):
        n = case["roots"]
        b, tables, r = river_builder(n, seed)
        st.update(builder=b, tables=Tables(tables))
        if kind == "river":
            st.update(ranges=r, results=[torch.zeros((n, STRIDE), device=DEV) for _ in range(2)])
        else:
            host = r[:, :, :HANDS].cpu().numpy()
            st.update(ranges=[np.ascontiguousarray(h, dtype=np.float64 if kind == "river_br" else np.float32)
                              for h in host])
            if kind == "river_host":
                st.update(results=[np.zeros((n, HANDS), np.float32) for _ in range(2)])
    elif kind == "game":
        rng = np.random.default_rng(seed)
        st.update(game=P.Game(sum(1 << int(c) for c in rng.choice(52, 3, replace=False))),
                  iterations=case["iterations"])
        st["game"].enable_average()
    elif kind in ("batch", "adjoint"):
        b = P.Batch(*batch_inputs(case, seed))
        b.enable_average()
        if kind == "batch" and case["subgames"] >= 256:
            b.tune()
        shapes = [b.shape(s)[1] for s in range(b.count)]
        st.update(batch=b)
        if kind == "batch":
            st.update(iterations=case["iterations"], rows=np.zeros((sum(shapes), HANDS), np.float32))
        else:
            rows, at = average_rows(case, seed, sum(shapes)), 0
            for s, e in enumerate(shapes):
                b.set_average(s, rows[at:at + e])
                at += e
            new = lambda *shape: torch.zeros(shape, device=DEV, dtype=torch.float64)  # noqa: E731
            st.update(grads=(new(b.count, HANDS), new(b.count, HANDS), new(b.count, 8, HANDS)))
    elif kind == "train":
        rows = -(-case["samples"] // 256) * 256
        st.update(net=make_net(rows, seed), data=train_data(case, seed), steps=case["steps"])
    else:
        st.update(game=P.FullGame(*full_inputs(case, seed)), iterations=case["iterations"])
        st["game"].tune()
        if case["net"]:
            st.update(net=make_net(4096, seed))
            st["game"].set_net(st["net"])
    return st


# ---- one pass ----

def run(state):
    kind = state["kind"]
    if kind == "river":
        for p in range(2):
            state["builder"].evaluate_device(state["tables"].ptr, p, False, state["ranges"][p].data_ptr(),
                                             state["results"][p].data_ptr())
        return state["results"]
    if kind == "river_host":
        for p in range(2):
            state["builder"].upload_all(state["ranges"][p])
            state["builder"].evaluate(state["tables"].ptr, p)
            state["builder"].download_all(state["results"][p])
        return state["results"]
    if kind == "river_br":
        return [state["builder"].best_response_f64(state["tables"].ptr, p, state["ranges"][p]) for p in range(2)]
    if kind == "game":
        state["game"].iterate(state["iterations"])
        return state["game"].root_values()
    if kind == "batch":
        state["batch"].iterate(state["iterations"])
        return state["batch"].all_rows(1, state["rows"])
    if kind == "adjoint":
        state["batch"].value_grad_device(*state["grads"], use_average=True)
        return state["grads"]
    if kind == "train":
        losses = [state["net"].train_step(*state["data"][k % MINIBATCHES], 1e-4) for k in range(state["steps"])]
        return {"loss": np.array(losses, np.float32), "layers": [state["net"].layer(l) for l in range(5)]}
    state["game"].iterate(state["iterations"])
    return state["game"].average()


# ---- what a pass cannot do without ----

def work(case):
    kind = case["kind"]
    if kind in ("river", "river_host", "river_br"):
        n = case["roots"]
        boards = 48 * min(49, -(-n // 9)) * (0.5 if n >= 441 else 1)
        wide = 2 if kind == "river_br" else 1
        # ranges and values, 26 regret rows read and 13 written (none by a best response), the
        # rank order and buckets of each board; 13 channels scanned three times and 17 leaf values
        # formed and weighted per hand and river card
        rows = 26 * 1024 + (0 if kind == "river_br" else 13 * 1024)
        return {"bytes": 2 * (n * (2 * HANDS * 4 * wide + rows) + boards * 1081 * 6),
                "flops": 2 * n * 48 * 1081 * (13 * 4 + 17 * 6)}
    if kind == "game":
        one = work({"kind": "river", "roots": 27783})
        # average sums read and written beside the regrets, the upper tree's vectors
        return {"bytes": case["iterations"] * (one["bytes"] + 2 * 27783 * 26 * 1024 + 2 * 55777 * 3 * HANDS * 4),
                "flops": case["iterations"] * one["flops"] * 1.05}
    if kind in ("batch", "adjoint"):
        n = case["subgames"]
        edges = 20.0 * n  # mean of random_subgames' trees
        if kind == "batch":
            return {"bytes": case["iterations"] * (edges * 1081 * 20 + 2 * n * (2 * HANDS * 4 + 1081 * 2)) + edges * HANDS * 4,
                    "flops": case["iterations"] * edges * 1081 * 2 * 14}
        return {"bytes": 2 * n * 2 * HANDS * 4 + 2 * edges * 1081 * 4 + n * 10 * HANDS * 8,
                "flops": edges * 1081 * 2 * 14}
    if kind == "train":
        n, params = case["samples"], 2706 * 1024 + 3 * 1024 * 1024 + 1024 * 2652
        return {"bytes": case["steps"] * (n * (2 * 2 * HANDS * 4 + 16) + params * 24),
                "flops": case["steps"] * 6.0 * n * params}
    _, _, edges, leaves = P.full_tree(full_inputs(case, 0)[0])
    rivers = leaves * 48
    upper = edges * HANDS * 4 * 5 * 2
    if case["net"]:
        n = case["iterations"] * 2 * leaves
        return {"bytes": n * 2 * HANDS * 8 + case["iterations"] * upper,
                "flops": n * 2.0 * (2706 * 1024 + 3 * 1024 * 1024 + 1024 * 2652)}
    river_edges = rivers * 12  # a check-bet-bet tree has 14 edges, an all-in leaf's 2
    return {"bytes": case["iterations"] * (river_edges * 1081 * 20 + upper),
            "flops": case["iterations"] * river_edges * 1081 * 2 * 14}


# ---- the same results in 64 bits, by plain torch ----

def hand_values(board):
    """Strength of every hand with the 5 board cards, [1326] int64 on the device (-1: the hand
    touches the board). Category first, then its ranks in order of importance."""
    lo, hi = (torch.tensor(x, device=DEV) for x in hand_cards())
    cards = torch.cat([torch.tensor(board, device=DEV).expand(HANDS, 5), lo[:, None], hi[:, None]], 1)
    rank, suit = cards % 13, cards // 13
    count = torch.zeros((HANDS, 13), dtype=torch.int64, device=DEV).scatter_add_(1, rank, torch.ones_like(rank))
    by_suit = torch.zeros((HANDS, 4, 13), dtype=torch.bool, device=DEV)
    by_suit[torch.arange(HANDS, device=DEV)[:, None], suit, rank] = True

    def straight(has):  # highest straight of a [.., 13] rank set, -1 for none (the wheel is 3)
        ext = torch.cat([has[..., 12:], has], -1)
        best = torch.full(has.shape[:-1], -1, dtype=torch.int64, device=DEV)
        for top in range(3, 13):
            run = ext[..., top - 3:top + 2].all(-1)
            best = torch.where(run, top, best)
        return best

    def top(has, k):  # the k highest ranks of a rank set as one base-13 number
        order = torch.where(has, torch.arange(13, device=DEV), -1).sort(-1, descending=True).values[..., :k]
        v = torch.zeros(has.shape[:-1], dtype=torch.int64, device=DEV)
        for i in range(k):
            v = v * 14 + order[..., i] + 1
        return v

    def keep(category, v):
        return category * 14 ** 5 + v

    one, two, three, four = (count >= k for k in (1, 2, 3, 4))
    value = keep(0, top(one, 5))
    pair = top(two, 1) - 1
    not_pair = one & (torch.arange(13, device=DEV)[None] != pair[:, None])
    value = torch.where(two.any(1), keep(1, (pair + 1) * 14 ** 3 + top(not_pair, 3)), value)
    second = torch.where(two.sum(1) >= 2, top(two, 2), 0)
    rest = one & (torch.arange(13, device=DEV)[None] != pair[:, None]) & \
        (torch.arange(13, device=DEV)[None] != (second % 14 - 1)[:, None])
    value = torch.where(two.sum(1) >= 2, keep(2, second * 14 + top(rest, 1)), value)
    trips = top(three, 1) - 1
    no_trips = torch.arange(13, device=DEV)[None] != trips[:, None]
    value = torch.where(three.any(1), keep(3, (trips + 1) * 14 ** 2 + top(one & no_trips, 2)), value)
    s = straight(one)
    value = torch.where(s >= 0, keep(4, s), value)
    flush = by_suit.sum(2) >= 5
    fl = torch.where(flush, top(by_suit, 5), 0).max(1).values
    value = torch.where(flush.any(1), keep(5, fl), value)
    other = two & no_trips
    full = three.any(1) & other.any(1)
    value = torch.where(full, keep(6, (trips + 1) * 14 + top(other, 1)), value)
    quads = top(four, 1) - 1
    kick = one & (torch.arange(13, device=DEV)[None] != quads[:, None])
    value = torch.where(four.any(1), keep(7, (quads + 1) * 14 + top(kick, 1)), value)
    sf = straight(by_suit).max(1).values
    value = torch.where(sf >= 0, keep(8, sf), value)
    return torch.where(torch.tensor(touches(board), device=DEV), -1, value)


def board_matrices(board):
    """compat[h][o] (1 where hands h and o share no card, o off the board), showdown[h][o] (its
    sign by strength), and each hand's bucket of 256."""
    value = hand_values(board)
    lo, hi = (torch.tensor(x, device=DEV) for x in hand_cards())
    clash = (lo[:, None] == lo) | (lo[:, None] == hi) | (hi[:, None] == lo) | (hi[:, None] == hi)
    live = value >= 0
    compat = (~clash & live[None]).double()
    sign = torch.sign(value[:, None] - value[None]).double() * compat
    wins, ties = (sign > 0).sum(1), compat.sum(1).long() - (sign != 0).sum(1)
    points = torch.where(live, (2 * wins + 2 * ties - 1) % (1 << 32), 0)
    bucket = torch.where(live, ((points * 256) % (1 << 32)) // 1980, 0)
    return compat, sign, bucket, live


class RiverTree:
    """The limit river tree: bets of 2, at most four; edges numbered as their child is finished.
    Nodes are ("node", actor, [(edge, child)]) or (kind, who folds, chips)."""

    def __init__(self):
        self.edges = 0
        self.root = self.node(0, 0.0, 0.0, 0, False)

    def node(self, actor, own, opp, raises, answered):
        """own / opp: the actor's and the other's chips on the river."""
        kids = [lambda: ("fold", actor, own)] if opp > own else []
        if opp > own or answered:
            kids.append(lambda: ("show", None, opp))
        else:
            kids.append(lambda: self.node(1 - actor, opp, own, raises, True))
        if raises < 4:
            kids.append(lambda: self.node(1 - actor, opp, opp + 2, raises + 1, True))
        out = []
        for kid in kids:
            child = kid()
            out.append((self.edges, child))
            self.edges += 1
        return ("node", actor, out)


def river_pass(tree, flop, turn, bets, r, reg, player, best):
    """One pass of `player` at every root: values [n][1328] and, unless `best`, the new regrets."""
    n = len(turn)
    reg = reg.double() if reg.dtype != torch.float64 else reg
    out = torch.zeros((n, STRIDE), device=DEV, dtype=torch.float64)
    new = None if best else reg.clone()
    boards = {}
    for t in sorted(set(turn.tolist())):
        at = torch.tensor(np.nonzero(turn == t)[0], device=DEV)
        g, x0 = reg[at], r[at, :HANDS].double()
        bet = torch.tensor(bets[at.cpu().numpy()], device=DEV, dtype=torch.float64)
        sigma = {}

        def strategies(nd):
            rows = [g[:, e] for e, _ in nd[2]]
            tot = sum(rows)
            for (e, c), row in zip(nd[2], rows):
                sigma[e] = torch.where(tot <= 1e-4, 1.0 / len(rows), row / tot.clamp(min=1e-300))
                if c[0] == "node":
                    strategies(c)

        strategies(tree.root)
        sums = {}  # leaf -> [m][256] bucket sums of values over the river cards
        total = torch.zeros_like(x0)
        for rc in range(52):
            if rc == t or rc in flop:
                continue
            key = tuple(sorted((t, rc)))
            if key not in boards:
                boards[key] = board_matrices(flop + list(key))
            compat, sign, bucket, live = boards[key]
            hot = torch.nn.functional.one_hot(bucket, 256).double()

            def walk(nd, opp, own):
                """Per-hand value [m][1326] (strategy-weighted or best) of the node."""
                if nd[0] != "node":
                    x = x0 * live * opp[:, bucket]
                    stake = bet + nd[2]
                    if nd[0] == "show":
                        v = stake[:, None] * (x @ sign.T)
                    else:
                        v = (-stake if nd[1] == player else stake)[:, None] * (x @ compat.T)
                    if not best:
                        sums[id(nd)] = sums.get(id(nd), 0) + v @ hot
                    return v
                vals = []
                for e, c in nd[2]:
                    s = sigma[e]
                    if nd[1] == player:
                        v = walk(c, opp, own)
                        vals.append(v if best else v * s[:, bucket])
                    else:
                        vals.append(walk(c, opp * s, own))
                if best and nd[1] == player:
                    return torch.stack(vals).max(0).values
                return sum(vals)

            ones = torch.ones((len(at), 256), device=DEV, dtype=torch.float64)
            total += walk(tree.root, ones, ones) * live
        out[at, :HANDS] = total / 48
        if not best:
            def update(nd):
                if nd[0] != "node":
                    return sums[id(nd)]
                kids = [(e, update(c)) for e, c in nd[2]]
                if nd[1] != player:
                    return sum(v for _, v in kids)
                value = sum(sigma[e] * v for e, v in kids)
                for e, v in kids:
                    new[at, e] = (g[:, e] + v - value).clamp(min=0)
                return value

            update(tree.root)
    return out, new


def exact_river(case, seed):
    flop, turn, bets, r, reg = river_inputs(case["roots"], seed)
    best = case["kind"] == "river_br"
    tree, reg, got = RiverTree(), reg.double(), []
    for p in range(2):
        v, new = river_pass(tree, flop, turn, bets, r[p], reg, p, best)
        reg = reg if best else new
        got.append(v if case["kind"] == "river" else v[:, :HANDS])
    return got


def bet_tree(pot, stack, sizes, raises):
    """General river tree: nodes ("node", actor, first edge, children) or (kind, who, stake); edges
    numbered by parent in pre-order."""
    f4 = np.float32
    count = [0]

    def node(actor, chips, done):
        own, opp = chips[actor], chips[1 - actor]
        behind, call, in_pot = f4(stack - own), f4(opp - own), f4(pot + chips[0]) + chips[1]
        acts = [("check", f4(0))] if call <= 0 else [("fold", f4(0)), ("call", call)]
        if done < raises and behind > max(call, f4(0)):
            for k in range(3):
                if not (sizes >> k) & 1:
                    continue
                put = behind if k == 2 else f4(call + f4((0.5, 1.0)[k]) * f4(in_pot + call))
                put = min(put, behind)
                if put > call and ("raise", put) not in acts:
                    acts.append(("raise", put))
        first = count[0]
        count[0] += len(acts)
        kids = []
        for name, put in acts:
            after = list(chips)
            if name == "fold":
                kids.append(("fold", actor, float(f4(0.5) * f4(pot) + own)))
            elif name == "call":
                kids.append(("show", None, float(f4(0.5) * f4(pot) + opp)))
            elif name == "check" and actor == 1:
                kids.append(("show", None, float(f4(0.5) * f4(pot) + chips[0])))
            else:
                after[actor] = f4(after[actor] + put)
                kids.append(node(1 - actor, after, done + (name == "raise")))
        return ("node", actor, first, kids)

    root = node(0, [f4(0), f4(0)], 0)
    return root, count[0]


def five(board):
    return [c for c in range(52) if (int(board) >> c) & 1]


def sigma_rows(src, first, n, cut):
    v = src[first:first + n].clamp(min=0)
    tot = v.sum(0)
    return torch.where(tot <= cut, torch.full_like(v, 1.0 / n), v / tot.clamp(min=1e-300))


def subgame_pass(root, mats, ranges, src, cut, player, regrets=None, sums=None, children=None):
    """Values [1326] of `player` under the strategies of the rows src; with `regrets`, its regrets
    (and average sums) are updated."""
    compat, sign, _, live = mats

    def walk(nd, opp, own):
        if nd[0] != "node":
            if nd[0] == "show":
                return nd[2] * (sign @ opp)
            return (-nd[2] if nd[1] == player else nd[2]) * (compat @ opp)
        _, actor, first, kids = nd
        s = sigma_rows(src, first, len(kids), cut)
        if actor != player:
            vals = [walk(c, opp * s[k], own) for k, c in enumerate(kids)]
            return sum(vals)
        vals = [walk(c, opp, own * s[k]) for k, c in enumerate(kids)]
        value = sum(s[k] * v for k, v in enumerate(vals))
        if nd is root and children is not None:
            children.extend(vals)
        if regrets is not None:
            for k, v in enumerate(vals):
                sums[first + k] += own * s[k]
                regrets[first + k] = (regrets[first + k] + v - value).clamp(min=0)
        return value

    opp = ranges[1 - player].double() * live
    return walk(root, opp, torch.ones_like(opp)) * live


def exact_batch(case, seed):
    if case["subgames"] * case["iterations"] > 800:
        return None
    specs, ranges = batch_inputs(case, seed)
    got = []
    for s, rr in zip(specs, ranges):
        root, edges = bet_tree(float(s["pot"]), float(s["stack"]), int(s["sizes"]), int(s["max_raises"]))
        mats, rr = board_matrices(five(s["board"])), torch.tensor(rr, device=DEV)
        reg = torch.zeros((edges, HANDS), device=DEV, dtype=torch.float64)
        avg = torch.zeros_like(reg)
        for _ in range(case["iterations"]):
            for p in range(2):
                subgame_pass(root, mats, rr, reg.clone(), 1e-4, p, reg, avg)
        got.append(avg * mats[3])
    return torch.cat(got)


def exact_adjoint(case, seed):
    specs, ranges = batch_inputs(case, seed)
    trees = [bet_tree(float(s["pot"]), float(s["stack"]), int(s["sizes"]), int(s["max_raises"])) for s in specs]
    rows, at = average_rows(case, seed, sum(e for _, e in trees)), 0
    n = case["subgames"]
    g0, g1 = (torch.zeros((n, HANDS), device=DEV, dtype=torch.float64) for _ in range(2))
    gs = torch.zeros((n, 8, HANDS), device=DEV, dtype=torch.float64)
    for i, (s, (root, edges)) in enumerate(zip(specs, trees)):
        mats, rr = board_matrices(five(s["board"])), torch.tensor(ranges[i], device=DEV)
        src = torch.tensor(rows[at:at + edges], device=DEV).double()
        at += edges
        kids = []
        g0[i] = subgame_pass(root, mats, rr, src, 0.0, 0, children=kids)
        g1[i] = -subgame_pass(root, mats, rr, src, 0.0, 1)
        for k, v in enumerate(kids):
            gs[i, k] = rr[0].double() * v * mats[3]
    return g0, g1, gs


def exact_train(case, seed):
    layers = [tuple(torch.tensor(t, device=DEV, dtype=torch.float64).requires_grad_() for t in wb)
              for wb in net_parameters(seed)]
    params = [t for wb in layers for t in wb]
    opt = torch.optim.Adam(params, lr=1e-4, betas=(0.9, 0.999), eps=1e-8)
    losses = []
    data = train_data(case, seed)
    bits = torch.arange(52, device=DEV)
    for k in range(case["steps"]):
        r, boards, s, y = data[k % MINIBATCHES]
        h = torch.cat([r.flatten(1), ((boards[:, None] >> bits) & 1).float(), s], 1).double()
        for l, (W, b) in enumerate(layers):
            h = h @ W.T + b
            h = torch.nn.functional.gelu(h) if l < 4 else h
        loss = ((h - y.double()) ** 2).mean()
        opt.zero_grad()
        loss.backward()
        opt.step()
        losses.append(loss.detach())
    return {"loss": torch.stack(losses), "layers": [tuple(t.detach() for t in wb) for wb in layers]}


def exact(case, seed):
    kind = case["kind"]
    if kind in ("river", "river_host", "river_br"):
        # 64-bit products of every board of the whole game take longer than a check should
        return exact_river(case, seed) if case["roots"] <= 2000 else None
    return {"batch": exact_batch, "adjoint": exact_adjoint, "train": exact_train}.get(kind, lambda c, s: None)(case, seed)
