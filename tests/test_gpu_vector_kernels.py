"""The default engine's node, showdown and chance kernels against the plain
engine (one CTA and one launch per node kind, hands strided over the threads)
on the same spots: the arithmetic is the same, so after a few iterations every
arena entry, the exploitability and the root values are equal bit for bit.
Sizes sit at the edges of the kernels' forms: the warp-per-node forms end at
32, 64 and 128 hands, the showdown CTAs at 85, 170, 341 and 682 hands on a
board, vectors come in groups of four."""
import numpy as np
import pytest

import gtopen_b200 as g
from gtopen_b200 import workloads as W

pytestmark = pytest.mark.gpu


def _config(cards, n0, n1, bet, raise_, raises, seed, scale="%.6f", stack=400):
    """n0 / n1 combos of a seeded board, weights in (0, 1]."""
    rng = W.XorShift(seed)
    board = W.draw_board(rng, cards)
    combos = W.live_combos(board)
    ranges = []
    for n in (n0, n1):
        order = sorted(range(len(combos)), key=lambda _: rng.next())[:n]
        ranges.append(",".join("%s:%s" % (W.combo_str(*combos[i]), scale % (0.05 + 0.95 * rng.uniform()))
                               for i in sorted(order)))
    return {"board": "".join(W.card_str(c) for c in board), "range_oop": ranges[0], "range_ip": ranges[1],
            "tree": W.tree_config(100, stack, bet, raise_, raises)}


def _solve(cfg, engine, storage, fmt, algo, iters, lock):
    spot = g.Spot(cfg)
    host = g.Solver(spot, storage=storage, algo=algo)
    if lock:
        t = spot.tree()
        for n in np.nonzero((t["kind"] == 0) & (t["nchild"] == 3))[0][:3]:
            na, nh = int(t["nchild"][n]), spot.nh[int(t["player"][n])]
            s = np.random.default_rng(int(n)).random((na, nh), np.float32)
            host.set_lock(int(n), (s / s.sum(0)).reshape(-1))
    gpu = g.GpuSolver(host, device_format=fmt, engine=engine)
    gpu.iterate(iters)
    out = [gpu.exploitability()]
    out += [gpu.root_cfv(p, mode) for p in (0, 1) for mode in (0, 1)]
    gpu.iterate(1)  # after the evaluation sweeps rewrote the reach slots
    which = (0, 1, 2) if algo == "pcfr+" else (0, 1)
    return out + [gpu.export_arena(w, p) for w in which for p in (0, 1)]


def _equal(cfg, storage="f32", fmt=None, algo="dcfr", iters=3, lock=False):
    a = _solve(cfg, "staged", storage, fmt, algo, iters, lock)
    b = _solve(cfg, "plain", storage, fmt, algo, iters, lock)
    assert a[0] == b[0]
    for x, y in zip(a[1:], b[1:]):
        np.testing.assert_array_equal(x, y)
    assert all(np.isfinite(x).all() for x in a[1:])


FORMATS = [("f32", None, "dcfr"), ("compressed", None, "dcfr"), ("compressed", "i16sr", "dcfr"),
           ("f32", None, "pcfr+"), ("compressed", None, "pcfr+"), ("compressed", None, "cfr+")]


@pytest.mark.parametrize("storage,fmt,algo", FORMATS)
@pytest.mark.parametrize("n0,n1", [(1, 2), (31, 33), (32, 64), (65, 63), (127, 129), (128, 341), (130, 1081)])
def test_river_sizes(n0, n1, storage, fmt, algo):
    _equal(_config(5, n0, n1, ("33", "75", "a"), ("2.5x",), 1, seed=100 + n0), storage, fmt, algo)


@pytest.mark.parametrize("storage,fmt,algo", FORMATS)
@pytest.mark.parametrize("n0,n1", [(3, 5), (30, 90), (200, 171), (600, 100)])
def test_turn_sizes(n0, n1, storage, fmt, algo):
    _equal(_config(4, n0, n1, ("75",), ("2.5x",), 1, seed=n0), storage, fmt, algo)


@pytest.mark.parametrize("bets", [4, 6, 7])
@pytest.mark.parametrize("storage,fmt,algo", FORMATS)
def test_wide_nodes(bets, storage, fmt, algo):
    """5 to 8 actions at a node (check and 4 to 7 sizes): the wide records."""
    sizes = ("10", "20", "30", "45", "60", "80", "100")[:bets]
    _equal(_config(5, 150, 37, sizes, ("2.5x",), 1, seed=bets, stack=1000), storage, fmt, algo)


@pytest.mark.parametrize("storage,fmt,algo", FORMATS)
def test_locked_nodes(storage, fmt, algo):
    _equal(_config(4, 61, 142, ("33", "75"), ("2.5x",), 1, seed=9), storage, fmt, algo, lock=True)


@pytest.mark.parametrize("scale", ["%.6fe-20", "%.6fe-32", "%.6fe-37"])
def test_tiny_weights(scale):
    """Weights whose fixed-point scales pass 2^100 and 2^126."""
    _equal(_config(5, 90, 70, ("75",), ("2.5x",), 1, seed=4, scale=scale))


def test_suit_symmetric_flop():
    cfg = W.iso_spot()
    _equal(cfg)
    _equal(cfg, "compressed", "i16sr")


def test_export_of_an_engine_that_holds_few_nodes():
    """A depth-limited solve's export: its nodes' average strategies, zeros
    elsewhere (only the held blocks are read back)."""
    cfg = W.flop_spot(g.evaluate7, seed=6, bet=("50",), raise_=("2.5x",), max_raises=1, pot=100, stack=330,
                      frac=(0.15, 0.2))
    spot = g.Spot(cfg)
    host = g.Solver(spot)
    gpu = g.dl_gpu_solver(host, g.LeafNet(2705, 128, 1, 2652, seed=2))
    gpu.iterate(3)
    t = spot.tree()
    _, _, _, visited = g.dl_plan(spot)
    for p in (0, 1):
        assert spot.data_size[p] * 4 >= 8 << 20
        sums = gpu.export_arena(1, p)
        held = np.zeros(spot.data_size[p], bool)
        for n in np.nonzero(visited.astype(bool) & (t["kind"] == 0) & (t["player"] == p))[0]:
            na, off = int(t["nchild"][n]), int(t["data_off"][n])
            held[off:off + na * spot.nh[p]] = True
            s = np.maximum(sums[off:off + na * spot.nh[p]].reshape(na, -1), 0).astype(np.float64)
            total = s.sum(0)
            want = np.where(total > 1e-12, s / np.where(total > 0, total, 1), 1.0 / na)
            got = g.node_strategy(gpu, int(n), na, p)
            assert np.abs(got - want).max() <= 2e-7  # one f32 rounding of the same quotient
        assert held.any() and not sums[~held].any()


@pytest.mark.parametrize("m,n,k", [(128, 128, 64), (128, 256, 192), (256, 2688, 128), (1024, 1024, 64), (1024, 2048, 64),
                                   (2048, 2048, 64)])
def test_product_tile_widths(m, n, k):
    """The tcgen05 product at shapes that take each tile width (32 to 256
    columns): f32 accumulation against f64, 1e-5 of sum |a||b|."""
    rng = np.random.default_rng(m + n)
    a, b = (rng.normal(0, 1, (r, k)).astype(np.float32) for r in (m, n))
    bits = [(x.view(np.uint32) >> 16).astype(np.uint16) for x in (a, b)]
    a, b = (((x.astype(np.uint32)) << 16).view(np.float32).astype(np.float64) for x in bits)
    c = g.gemm_bf16(*bits)
    assert np.all(np.abs(c - a @ b.T) <= 1e-5 * (np.abs(a) @ np.abs(b).T) + 1e-6)


def test_one_adam_step():
    """One training step on one batch against Adam's formula on the gradients
    the network reports (padded, odd dimensions; every layer, weights and
    biases).  The first step moves an entry by lr g / (|g| + eps'): insensitive
    to the batch order's rounding where |g| is well above eps."""
    dims, n, lr = (70, 130, 2, 40), 128, 1e-2
    rng = np.random.default_rng(5)
    x, t = rng.normal(0, 1, (n, 70)).astype(np.float32), rng.normal(0, 1, (n, 40)).astype(np.float32)
    m = (rng.random((n, 40)) < 0.8).astype(np.float32)
    a, b = g.LeafNet(*dims, seed=3), g.LeafNet(*dims, seed=3)
    loss = a.gradients(x, t, m)
    losses = b.train(x, t, m, epochs=1, batch=n, lr=lr, seed=1)
    assert abs(losses[0] - loss) <= 1e-5 * loss
    for layer in range(dims[2] + 1):
        for w, gr, got in zip(a.params(layer), a.grads(layer), b.params(layer)):
            gr = gr.astype(np.float64)
            want = w - lr * gr / (np.abs(gr) + 1e-8)
            big = np.abs(gr) > 1e-5
            assert big.any() and np.abs(got - want)[big].max() <= 1e-2 * lr
            assert np.abs(got - w).max() <= lr * 1.001


@pytest.mark.parametrize("rows,batch", [(200, 128), (300, 512)])
def test_short_training_repeats(rows, batch):
    """A call's tables are on the device before its first step reads them: the
    same short training gives the same parameters every time, bit for bit
    (buffers are zeroed and filled on a stream that the network's does not
    wait for)."""
    dims = (2705, 128, 1, 2652)
    rng = np.random.default_rng(rows)
    x, t = (rng.standard_normal((rows, w), np.float32) for w in (dims[0], dims[3]))
    m = np.ones((rows, dims[3]), np.float32)
    first = None
    for _ in range(6):
        net = g.LeafNet(*dims, seed=4)
        net.train(x, t, m, epochs=2, batch=batch, lr=1e-3, seed=2)
        got = [a for layer in range(dims[2] + 1) for a in net.params(layer)]
        first = first or got
        assert all(np.array_equal(a, b) for a, b in zip(first, got))
