"""Performance cases of the postflop engine, through its public Python API.

A case is one block of work as a solving program runs it: a number of CFR
iterations, the exploitability check that decides whether to go on, and the
strategies read back; a batch of spots solved side by side; the turn-leaf
network trained, or used by a depth-limited solve.  listed() holds the cases,
draw() gives more of the same ranges, prepare() builds what the program has in
hand (spot, host solver, engine or network), run() is one block, work() what
one block cannot do without, exact() the same results in 64 bits where plain
numpy gives them in reasonable time.
"""
import numpy as np

import gtopen_b200 as g
from gtopen_b200 import leafdata as LD
from gtopen_b200 import workloads as W

# The preflop ranges of a button v big blind single-raised pot (about 250 and
# 320 combos on a flop), and short late-street ranges (a few dozen combos).
WIDE_OOP = ("55-22,A8s-A2s,K9s-K6s,Q9s-Q6s,J9s-J7s,T8s-T7s,97s,98s,86s,87s,75s,76s,64s,65s,53s,54s,43s,AJo-A8o,"
            "KTo-K9o,QTo,QJo,JTo,T9o,98o")
WIDE_IP = "22+,A2s+,K6s+,Q8s+,J8s+,T8s+,97s+,87s,76s,65s,A8o+,KTo+,QTo+,JTo"
MID_OOP = "TT,99,88,77,AKs,AQs,AJs,JTs,T9s,87s,AKo,KQo"
MID_IP = "QQ,JJ,TT,AKs,KQs,QJs,T9s,98s,AQo"
TIGHT_OOP = "QQ,JJ,TT,99,AKs,87s"
TIGHT_IP = "AA,KK,AQs,JTs,T9s"
CLASSES = {"wide": (WIDE_OOP, WIDE_IP), "mid": (MID_OOP, MID_IP), "tight": (TIGHT_OOP, TIGHT_IP)}

# Sizes per tree: (flop, turn, river) of "bets OOP / bets IP / raises", the
# number of raises and the stack behind a pot of 100.
TREES = {
    "river3": {"bet": "33,75,a", "raise": "2.5x", "max_raises": 1, "stack": 400.0},
    "turn3": {"bet": "33,75,a", "raise": "2.5x", "max_raises": 2, "stack": 300.0},
    "turn4": {"bet": "33,75,150,a", "raise": "2.5x", "max_raises": 1, "stack": 600.0},
    "street1": {"bet": "50", "raise": "2.5x", "max_raises": 1, "stack": 330.0},
    "street2": {"bet": "50,125", "raise": "2.5x", "max_raises": 1, "stack": 500.0},
    "jam": {"bet": "75,a", "raise": "a", "max_raises": 2, "stack": 1770.0},
    "half": {"bet": "50", "raise": "", "max_raises": 0, "stack": 330.0},
    "srp": {"bet": "33/33,75|75|75", "raise": "60", "max_raises": 10, "stack": 1617.0},
}
STORAGE = {"f32": ("f32", None), "i16": ("compressed", None), "i16sr": ("compressed", "i16sr")}


def listed():
    return [
        # the smallest solve: a river spot, every combo on both sides; launches and latency count
        {"name": "river_f32", "kind": "solve", "cards": 5, "suits": "any", "ranges": "top", "oop": 1.0, "ip": 1.0,
         "tree": "river3", "arenas": "f32", "algo": "dcfr", "iso": True, "iterations": 20},
        # the ordinary turn solve, half of all combos on each side, exact arenas
        {"name": "turn_f32", "kind": "solve", "cards": 4, "suits": "any", "ranges": "top", "oop": 0.5, "ip": 0.5,
         "tree": "turn3", "arenas": "f32", "algo": "dcfr", "iso": True, "iterations": 100},
        # the same street in the memory-saving arenas with stochastic rounding, ranges of unequal, odd sizes
        {"name": "turn_i16sr", "kind": "solve", "cards": 4, "suits": "any", "ranges": "top", "oop": 0.31, "ip": 0.83,
         "tree": "turn3", "arenas": "i16sr", "algo": "dcfr", "iso": True, "iterations": 100},
        # the predictive variant, round-to-nearest 16-bit arenas
        {"name": "turn_pcfr_i16", "kind": "solve", "cards": 4, "suits": "any", "ranges": "top", "oop": 0.4, "ip": 0.55,
         "tree": "turn3", "arenas": "i16", "algo": "pcfr+", "iso": True, "iterations": 100},
        # five actions at a node (check and four sizes)
        {"name": "turn_wide_i16sr", "kind": "solve", "cards": 4, "suits": "any", "ranges": "top", "oop": 0.45,
         "ip": 0.5, "tree": "turn4", "arenas": "i16sr", "algo": "dcfr", "iso": True, "iterations": 50},
        # a flop between two tight ranges: many nodes, a few dozen hands each
        {"name": "flop_tight_f32", "kind": "solve", "cards": 3, "suits": "rainbow", "ranges": "tight", "oop": 0.0,
         "ip": 0.0, "tree": "street1", "arenas": "f32", "algo": "dcfr", "iso": True, "iterations": 50},
        # a two-tone flop, suit isomorphism at work, medium ranges
        {"name": "flop_iso_i16", "kind": "solve", "cards": 3, "suits": "twotone", "ranges": "mid", "oop": 0.0,
         "ip": 0.0, "tree": "street2", "arenas": "i16", "algo": "dcfr", "iso": True, "iterations": 50},
        # a flop with the full single-raised-pot hand counts (470 v 647) on a narrow tree
        {"name": "flop_jam_i16sr", "kind": "solve", "cards": 3, "suits": "rainbow", "ranges": "top", "oop": 0.4,
         "ip": 0.55, "tree": "jam", "arenas": "i16sr", "algo": "dcfr", "iso": True, "iterations": 20},
        # the largest: a single-raised pot on a flop, 1.2 million nodes
        {"name": "flop_srp_f32", "kind": "solve", "cards": 3, "suits": "rainbow", "ranges": "wide", "oop": 0.0,
         "ip": 0.0, "tree": "srp", "arenas": "f32", "algo": "dcfr", "iso": True, "iterations": 20},
        # turn spots solved side by side to a target (the leaf network's training data, and reports)
        {"name": "batch_turn", "kind": "batch", "spots": 8, "top": 0.5, "iterations": 200, "check": 20,
         "arenas": "i16sr"},
        # the turn-leaf network trained on the spots it was given
        {"name": "leaf_train", "kind": "train", "rows": 896, "batch": 256, "epochs": 30},
        # a flop solve cut at the turn, its leaves valued by the network
        {"name": "leaf_solve", "kind": "leaf", "top": 0.5, "tree": "street1", "iterations": 50, "arenas": "f32"},
    ]


def draw(rng):
    kind = rng.choice(["river", "turn", "turn", "flop", "flop", "batch", "train", "leaf"])
    arenas = rng.choice(["f32", "i16", "i16sr"])
    top = lambda lo, hi: round(lo * (hi / lo) ** rng.random(), 3)  # noqa: E731
    base = {"kind": "solve", "suits": "any", "ranges": "top", "arenas": arenas, "algo": "dcfr", "iso": True}
    if kind == "river":
        return dict(base, cards=5, oop=top(0.04, 1.0), ip=top(0.04, 1.0), tree="river3",
                    iterations=rng.randint(10, 60))
    if kind == "turn":
        algo = rng.choice(["dcfr", "dcfr", "pcfr+", "cfr+"])
        return dict(base, cards=4, oop=top(0.05, 0.9), ip=top(0.05, 0.9), algo=algo if arenas != "i16sr" else "dcfr",
                    tree=rng.choice(["turn3", "turn3", "turn4", "street2"]), iterations=rng.randint(20, 100))
    if kind == "flop" and rng.random() < 0.5:
        return dict(base, cards=3, suits=rng.choice(["rainbow", "twotone", "mono"]), ranges=rng.choice(["tight", "mid", "wide"]),
                    oop=0.0, ip=0.0, tree=rng.choice(["half", "street1", "street2"]), iterations=rng.randint(10, 40))
    if kind == "flop":
        return dict(base, cards=3, suits=rng.choice(["rainbow", "twotone", "mono"]), oop=top(0.03, 0.5), ip=top(0.03, 0.5),
                    tree=rng.choice(["half", "street1"]), iterations=rng.randint(10, 20))
    if kind == "batch":
        return {"kind": "batch", "spots": rng.randint(2, 8), "top": top(0.1, 0.5), "iterations": 20 * rng.randint(2, 10),
                "check": 20, "arenas": arenas}
    if kind == "train":
        return {"kind": "train", "rows": rng.randint(200, 1500), "batch": 128 * rng.randint(1, 4),
                "epochs": rng.randint(1, 6)}
    return {"kind": "leaf", "top": top(0.1, 0.6), "tree": rng.choice(["half", "street1"]),
            "iterations": rng.randint(10, 50), "arenas": rng.choice(["f32", "i16"])}


# ------------------------------------------------------------------ inputs
def _board(rng, n, suits):
    """n cards of the wanted suit pattern (flops: rainbow, two-tone, monotone)."""
    while True:
        b = W.draw_board(rng, n)
        k = len({c & 3 for c in b})
        if suits == "any" or k == {"rainbow": 3, "twotone": 2, "mono": 1}[suits]:
            return b


def _tree(name):
    t = TREES[name]
    lists = lambda s: W.sizes(*[x for x in s.split(",") if x])  # noqa: E731
    streets = t["bet"].split("|") * (3 if "|" not in t["bet"] else 1)
    sides = []
    for p in (0, 1):
        side = []
        for s in streets:
            mine = s.split("/")[p if "/" in s else 0]
            side.append({"bet": lists(mine), "raise": lists(t["raise"]), "donk": []})
        sides.append(side)
    return {"starting_pot": 100.0, "effective_stack": t["stack"], "rake_pct": 0.0, "rake_cap": 0.0, "oop": sides[0],
            "ip": sides[1], "allin_threshold": 0.85, "add_allin": False, "max_raises": t["max_raises"]}


def _config(case, seed):
    """The spot of a solve.  "top": a board from the seed, the top share of all
    combos by a seeded strength score, random weights.  Otherwise preflop
    classes, each class at a seeded weight, on the pattern's one board (so that
    the board blocks the same combos at every seed)."""
    rng = W.XorShift(0x51D0 + 7919 * int(seed))
    for _ in range(8):
        rng.next()
    fixed = W.XorShift(0xB0A2D)
    board = _board(rng if case["ranges"] == "top" else fixed, case["cards"], case["suits"])
    text = "".join(W.card_str(c) for c in board)
    if case["ranges"] == "top":
        r = [W.weighted_range(rng, W.top_fraction(rng, board, case[k], g.evaluate7), 0.2) for k in ("oop", "ip")]
    else:
        r = [",".join("%s:%.3f" % (c, 0.5 + 0.5 * rng.uniform()) for c in t.split(",")) for t in CLASSES[case["ranges"]]]
    return {"board": text, "range_oop": r[0], "range_ip": r[1], "tree": _tree(case["tree"])}


def _turn_spot(rng, top):
    board = W.draw_board(rng, 4)
    r = [W.weighted_range(rng, W.top_fraction(rng, board, top, g.evaluate7), 0.2) for _ in range(2)]
    return g.Spot({"board": "".join(W.card_str(c) for c in board), "range_oop": r[0], "range_ip": r[1],
                   "tree": _tree("turn3")})


DIMS = (2705, 1024, 3, 2652)  # inputs, width, hidden layers, outputs of the turn-leaf network


def _net_params(seed):
    """Weights as a freshly initialised network of this shape has them."""
    rng = np.random.default_rng(seed)
    din, dh, nh, dout = DIMS
    out = []
    for layer in range(nh + 1):
        fi, fo = din if layer == 0 else dh, dout if layer == nh else dh
        a = np.float32(np.sqrt(3.0 / fi) * (0.1 if layer == nh else 1.0))
        out.append(((rng.random((fo, fi), np.float32) * 2 - 1) * a, (rng.random(fo, np.float32) - 0.5) * np.float32(0.02)))
    return out


def _net(seed):
    net = g.LeafNet(*DIMS, seed=1 + seed)
    for layer, (w, b) in enumerate(_net_params(seed)):
        net.set_params(layer, w, b)
    return net


def _train_rows(case, seed):
    """Rows as the generator of turn spots makes them: the cards one-hot, the
    pot-to-stack ratio, both players' reach normalised over the combos;
    targets for the combos that the board leaves, a mask for them."""
    rng = np.random.default_rng(1000003 + seed)
    n, din, dout = case["rows"], DIMS[0], DIMS[3]
    x, m = np.zeros((n, din), np.float32), np.ones((n, dout), np.float32)
    hi, lo = np.array([(h, w) for h in range(52) for w in range(h)]).T
    reach = rng.random((n, 2, 1326), np.float32)
    reach *= rng.random((n, 2, 1326), np.float32) < 0.5
    for i in range(n):
        board = rng.permutation(52)[:4]
        x[i, board] = 1.0
        dead = np.isin(hi, board) | np.isin(lo, board)
        reach[i][:, dead] = 0.0
        m[i] = np.tile(~dead, 2)
    reach /= reach.sum(2, keepdims=True)
    x[:, 52] = rng.random(n, np.float32)
    x[:, 53:] = reach.reshape(n, -1)
    t = (rng.standard_normal((n, dout), np.float32) * np.float32(0.3)) * m
    return x, t, m


# ------------------------------------------------------------------- cases
def prepare(case, seed):
    kind = case["kind"]
    if kind == "solve":
        storage, fmt = STORAGE[case["arenas"]]
        host = g.Solver(g.Spot(_config(case, seed)), storage=storage, algo=case["algo"], use_iso=case["iso"])
        return {"case": case, "host": host, "gpu": g.GpuSolver(host, device_format=fmt)}
    if kind == "batch":
        rng = W.XorShift(0xBA7C + 104729 * int(seed))
        return {"case": case, "spots": [_turn_spot(rng, case["top"]) for _ in range(case["spots"])]}
    if kind == "train":
        return {"case": case, "net": _net(seed), "rows": _train_rows(case, seed)}
    storage, fmt = STORAGE[case["arenas"]]
    spot = g.Spot(_config(_leaf_solve(case), seed))
    host = g.Solver(spot, storage=storage)
    return {"case": case, "host": host, "gpu": g.dl_gpu_solver(host, _net(seed), device_format=fmt)}


def _leaf_solve(case):
    return {"cards": 3, "suits": "rainbow", "ranges": "top", "oop": case["top"], "ip": case["top"], "tree": case["tree"]}


def run(state):
    case = state["case"]
    if case["kind"] == "batch":
        storage, fmt = STORAGE[case["arenas"]]
        b = g.Batch(state["spots"], storage=storage, device_format=fmt, keep_solvers=False)
        b.run(max_iterations=case["iterations"], target_pct=0.1, check_every=case["check"])
        rows = b.rows()
        return {"iterations": np.array([r["iterations"] for r in rows], np.int64),
                "exploit_pct": np.array([r["exploit_pct"] for r in rows]), "ev": np.array([r["ev"] for r in rows]),
                "cfv": np.concatenate([b.root_cfv(i, p) for i in range(len(rows)) for p in (0, 1)])}
    if case["kind"] == "train":
        net = state["net"]
        losses = net.train(*state["rows"], epochs=case["epochs"], batch=case["batch"], lr=3e-4, seed=3)
        return {"losses": losses, "params": [net.params(layer) for layer in range(DIMS[2] + 1)]}
    gpu = state["gpu"]
    gpu.iterate(case["iterations"])
    out = {"exploitability": gpu.exploitability()}
    out["strategy"] = [gpu.export_arena(1, p) for p in (0, 1)]
    if case["kind"] == "solve" and case["cards"] > 3:  # small enough to keep for a resumed solve
        out["regrets"] = [gpu.export_arena(0, p) for p in (0, 1)]
    return out


def work(case):
    kind = case["kind"]
    din, dh, nh, dout = DIMS
    weights = din * dh + (nh - 1) * dh * dh + dh * dout
    if kind == "train":
        n, steps = case["rows"], case["epochs"] * max(1, case["rows"] // case["batch"])
        # inputs, targets and masks once; the parameters in and out
        return {"bytes": 4.0 * n * (din + 2 * dout) + 8.0 * weights,
                "flops": steps * min(n, case["batch"]) * (6.0 * weights - 2.0 * din * dh)}
    if kind == "batch":
        rng = W.XorShift(0xBA7C)
        one = _solve_work(_turn_spot(rng, case["top"]), case["arenas"], "dcfr", True, case["iterations"])
        checks = case["iterations"] / case["check"]
        return {"bytes": case["spots"] * (one["arena"] + checks * one["check"]), "flops": case["spots"] * one["flops"]}
    if kind == "leaf":
        spot = g.Spot(_config(_leaf_solve(case), 0))
        leaves, _, _, visited = g.dl_plan(spot)
        rows = 49 * len(leaves)
        w = _solve_work(spot, case["arenas"], "dcfr", True, case["iterations"], visited)
        sweeps = 2 * (case["iterations"] + 1)
        return {"bytes": w["arena"] + w["check"] + w["out"] + 2.0 * weights,
                "flops": w["flops"] + 2.0 * weights * rows * sweeps}
    spot = g.Spot(_config(case, 0))
    w = _solve_work(spot, case["arenas"], case["algo"], case["iso"], case["iterations"])
    return {"bytes": w["arena"] + w["check"] + w["out"], "flops": w["flops"]}


def _solve_work(spot, arenas, algo, iso, iterations, visited=None):
    """Arena bytes of the iterations (the regrets read by the other player's
    sweep, regrets and sums -- and PCFR+ predictions -- read and written by
    the owner's), of one check, and of the strategies handed back; about ten
    operations per arena entry and hand of a terminal."""
    t = spot.tree()
    if visited is None:
        visited = g.shard_visited(spot, 0, 1, use_iso=iso)
    vis = visited.astype(bool)
    entries = sum(float(t["nchild"][vis & (t["kind"] == 0) & (t["player"] == p)].sum()) * spot.nh[p] for p in (0, 1))
    terms = float((vis & (t["kind"] >= 2)).sum())
    b = 4 if arenas == "f32" else 2
    per = 5 * b + (3 * b if algo == "pcfr+" else 0)
    size = sum(spot.data_size)
    once = min(entries * 4 * b, 126e6)  # what fits the L2 cache is read and written once
    return {"arena": max(iterations * (entries * per - once), entries * 4 * b), "check": entries * b, "out": (8.0 if len(spot.config["board"]) > 6 else 4.0) * size,
            "flops": 10.0 * (2 * iterations + 2) * (entries / 2 + terms * (spot.nh[0] + spot.nh[1]) / 2)}


# ------------------------------------------------------------------- exact
def exact(case, seed):
    """River solves in exact arenas and the network's training, in 64 bits.
    Turn and flop solves, batches and depth-limited solves take plain numpy
    minutes (thousands to a million nodes, dozens of sweeps): None; 16-bit
    arenas are defined by their rounding: None."""
    if case["kind"] == "train":
        return _exact_train(case, seed)
    if case["kind"] == "solve" and case["cards"] == 5 and case["arenas"] == "f32" and case["algo"] == "dcfr":
        return _exact_river(case, seed)
    return None


def _strength(cards):
    """(category, ranks...) of the best five of seven cards."""
    ranks = sorted((c >> 2 for c in cards), reverse=True)

    def straight(rs):
        s = set(rs) | ({-1} if 12 in rs else set())
        return next((h for h in range(12, 2, -1) if all(h - k in s for k in range(5))), None)
    for suit in range(4):
        fl = sorted((c >> 2 for c in cards if c & 3 == suit), reverse=True)
        if len(fl) >= 5:
            top = straight(fl)
            return (8, top) if top is not None else (5,) + tuple(fl[:5])  # a flush rules out quads and full houses
    by = sorted(((ranks.count(r), r) for r in set(ranks)), reverse=True)
    if by[0][0] == 4:
        return (7, by[0][1], max(r for r in ranks if r != by[0][1]))
    if by[0][0] == 3 and by[1][0] >= 2:
        return (6, by[0][1], max(r for n, r in by[1:] if n >= 2))
    top = straight(ranks)
    if top is not None:
        return (4, top)
    rest = lambda used, n: tuple([r for r in ranks if r not in used][:n])  # noqa: E731
    if by[0][0] == 3:
        return (3, by[0][1]) + rest({by[0][1]}, 2)
    if by[0][0] == 2 and by[1][0] == 2:
        return (2, by[0][1], by[1][1]) + rest({by[0][1], by[1][1]}, 1)
    if by[0][0] == 2:
        return (1, by[0][1]) + rest({by[0][1]}, 3)
    return (0,) + tuple(ranks[:5])


def _cards(text):
    return ["23456789TJQKA".index(text[i]) * 4 + "cdhs".index(text[i + 1]) for i in range(0, len(text), 2)]


def _exact_river(case, seed):
    cfg = _config(case, seed)
    board, tree = _cards(cfg["board"]), cfg["tree"]
    hands, w = [], []
    for text in (cfg["range_oop"], cfg["range_ip"]):
        rows = sorted((tuple(_cards(tok.split(":")[0])), np.float32(tok.split(":")[1])) for tok in text.split(","))
        hands.append([r[0] for r in rows])
        w.append(np.array([r[1] for r in rows], np.float64))
    val = [[_strength(board + list(h)) for h in hs] for hs in hands]
    order = {v: i for i, v in enumerate(sorted(set(val[0]) | set(val[1])))}
    val = [np.array([order[v] for v in vs]) for vs in val]
    c = [np.array(hs) for hs in hands]
    meet = np.ones((len(c[0]), len(c[1])))
    for a in (0, 1):
        for b in (0, 1):
            meet[c[0][:, a][:, None] == c[1][:, b][None, :]] = 0.0
    sign = np.sign(val[0][:, None] - val[1][None, :]) * meet
    meet, sign = (meet, meet.T.copy()), (sign, -sign.T.copy())
    bets = [75.0 if b == {"PotPct": 75.0} else 33.0 for b in tree["oop"][2]["bet"] if b != "AllIn"]
    assert case["tree"] == "river3" and bets == [33.0, 75.0]
    pot, stack = tree["starting_pot"], tree["effective_stack"]
    nodes = []  # (player, children, arena offset) in the order of the arenas
    size = [0, 0]

    def cap(x, top):
        return top if x >= 0.85 * top - 1e-9 else x

    def node(p, put, bet, raises, inc, checked):
        left, facing = stack - (put[p] - pot / 2), bet[1 - p] - bet[p]
        me = {"p": p, "kids": []}
        kids = []
        if facing > 0:
            kids += [("fold",), ("call",)]
            if left > facing + 1e-9 and raises < tree["max_raises"]:
                x = cap(max(2.5 * bet[1 - p], bet[1 - p] + inc), bet[p] + left)
                kids.append(("to", x, raises + 1))
        else:
            sizes = sorted({cap(x, left) for x in [0.33 * sum(put), 0.75 * sum(put), left]})
            kids += [("check",)] + [("to", x, raises) for x in sizes]
        me["off"], me["na"] = size[p], len(kids)
        size[p] += len(kids) * len(w[p])
        nodes.append(me)
        for k in kids:
            if k[0] == "fold":
                me["kids"].append({"fold": p, "amount": put[p]})
            elif k[0] == "call":
                me["kids"].append({"show": put[1 - p]})
            elif k[0] == "check":
                me["kids"].append({"show": put[p]} if checked else node(1 - p, put, bet, raises, inc, True))
            else:
                to, at = list(put), list(bet)
                to[p] += k[1] - bet[p]
                at[p] = k[1]
                me["kids"].append(node(1 - p, to, at, k[2], max(inc, k[1] - bet[1 - p]), checked))
        return me

    root = node(0, [pot / 2, pot / 2], [0.0, 0.0], 0, 0.0, False)
    for n in nodes:
        n["r"] = np.zeros((n["na"], len(w[n["p"]])))
        n["s"] = np.zeros_like(n["r"])

    def share(x, floor):
        x = np.maximum(x, 0.0)
        t = x.sum(0)
        return np.where(t > floor, x / np.where(t > floor, t, 1.0), 1.0 / len(x))

    def walk(n, p, reach, opp, mode, disc):
        if "fold" in n:
            return (meet[p] @ opp) * (-n["amount"] if n["fold"] == p else n["amount"])
        if "show" in n:
            return (sign[p] @ opp) * n["show"]
        sig = share(n["r"] if mode == "cfr" else n["s"], 1e-12)
        if n["p"] != p:
            return sum(walk(k, p, reach, opp * sig[i], mode, disc) for i, k in enumerate(n["kids"]))
        v = np.array([walk(k, p, reach * sig[i], opp, mode, disc) for i, k in enumerate(n["kids"])])
        if mode == "best":
            return v.max(0)
        own = (sig * v).sum(0)
        n["r"] = n["r"] * np.where(n["r"] > 0, disc[0], 0.5) + (v - own)
        n["s"] = n["s"] * disc[1] + reach * sig
        return own

    for t in range(1, case["iterations"] + 1):
        d = (t ** 1.5 / (t ** 1.5 + 1), (t / (t + 1)) ** 2)
        for p in (0, 1):
            walk(root, p, w[p], w[1 - p], "cfr", d)
    pairs = w[0] @ meet[0] @ w[1]
    best = [w[p] @ walk(root, p, w[p], w[1 - p], "best", None) / pairs for p in (0, 1)]
    strat = [np.concatenate([n["s"].reshape(-1) for n in nodes if n["p"] == p]) for p in (0, 1)]
    regrets = [np.concatenate([n["r"].reshape(-1) for n in nodes if n["p"] == p]) for p in (0, 1)]
    return {"exploitability": sum(best) / 2, "strategy": strat, "regrets": regrets}


def _exact_train(case, seed):
    import torch
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    x, t, m = (torch.from_numpy(a).to(dev).double() for a in _train_rows(case, seed))
    ps = [torch.from_numpy(a).to(dev).double().requires_grad_() for wb in _net_params(seed) for a in wb]
    n, batch, mask64 = case["rows"], case["batch"], (1 << 64) - 1
    opt = torch.optim.Adam(ps, lr=3e-4)
    # the row order: a Fisher-Yates shuffle per epoch, drawn from xorshift64
    s = (3 * 0x9E3779B97F4A7C15 + 1) & mask64
    order, losses = list(range(n)), []
    for _ in range(case["epochs"]):
        for i in range(n - 1, 0, -1):
            s ^= (s << 13) & mask64
            s ^= s >> 7
            s ^= (s << 17) & mask64
            j = s % (i + 1)
            order[i], order[j] = order[j], order[i]
        total, nb = 0.0, max(1, n // batch)
        for k in range(nb):
            rows = torch.tensor(order[k * batch:min(n, (k + 1) * batch)], device=dev)
            h = x[rows]
            for layer in range(DIMS[2] + 1):
                h = h @ ps[2 * layer].T + ps[2 * layer + 1]
                if layer < DIMS[2]:
                    h = torch.nn.functional.gelu(h)
            loss = ((h - t[rows]) * m[rows]).square().mean()
            opt.zero_grad()
            loss.backward()
            opt.step()
            total += loss.item()
        losses.append(total / nb)
    return {"losses": np.array(losses),
            "params": [(ps[2 * i].detach().cpu().numpy(), ps[2 * i + 1].detach().cpu().numpy()) for i in range(DIMS[2] + 1)]}
