"""The vector kernels' large-launch forms and the inputs their usual sizes never
meet, bit for bit against the plain engine (or, for FP8 arenas, the persistent
batch kernel, which stages nodes in shared memory).  The form a launch takes
depends on its level's node count as well as on the hands, so each test first
checks from the plan's own levels that its form is taken."""
import numpy as np
import pytest

from test_gpu_vector_kernels import FORMATS, _config, _equal

import gtopen_b200 as g
from gtopen_b200 import workloads as W

pytestmark = pytest.mark.gpu
MINE = 6  # the batch queue's kind of a level's traverser nodes
FILL = 148 * 16  # warps that fill the device; half of it in warps of 128 hands is a large launch


def _large(cfg, p):
    """(some level's update of player p is a large launch: four hands a thread; its hands; the tree)"""
    spot = g.Spot(cfg)
    seg = g.batch_queue([spot])[0]
    counts = seg["count"][(seg["kind"] == MINE) & (seg["p"] == p)].astype(np.int64)
    return counts.max() * ((spot.nh[p] + 127) // 128) > FILL // 2, spot.nh[p], spot.tree()


@pytest.mark.parametrize("storage,fmt,algo", FORMATS)
def test_one_warp_of_four_hands_a_lane(storage, fmt, algo):
    """65 to 128 hands, thousands of nodes on a level: a warp per node."""
    cfg = W.flop_spot(g.evaluate7, seed=6, bet=("50",), raise_=(), max_raises=0, pot=100, stack=330, frac=(0.08, 0.095))
    for p in (0, 1):
        large, nh, _ = _large(cfg, p)
        assert large and 64 < nh <= 128
    _equal(cfg, storage, fmt, algo, iters=2)


@pytest.mark.parametrize("sizes,widest", [(("20", "40", "75", "a"), 5), (("10", "20", "30", "45", "60", "80", "100"), 8)])
@pytest.mark.parametrize("storage,fmt,algo", FORMATS)
def test_wide_records_on_large_levels(sizes, widest, storage, fmt, algo):
    """Nodes of 5 and 8 actions and several hundred hands: a CTA per node for
    the quantised update, warps of 128 hands for the rest."""
    cfg = _config(4, 500, 303, sizes, (), 0, seed=3, stack=1000)
    for p in (0, 1):
        large, nh, t = _large(cfg, p)
        assert large and nh > 128 and t["nchild"][t["kind"] == 0].max() == widest
    _equal(cfg, storage, fmt, algo, iters=2)


@pytest.mark.parametrize("storage", ["f32", "compressed"])
def test_predictions_on_large_levels(storage):
    cfg = W.turn_spot(g.evaluate7, seed=2)
    for p in (0, 1):
        large, nh, _ = _large(cfg, p)
        assert large and nh > 128
    _equal(cfg, storage, None, "pcfr+", iters=2)


def _fp8_config(name):
    if name == "flop":
        return W.flop_spot(g.evaluate7, seed=6, bet=("50",), raise_=(), max_raises=0, pot=100, stack=330, frac=(0.08, 0.095))
    cards, n0, n1 = name
    return _config(cards, n0, n1, ("33", "75", "a") if cards == 5 else ("75",), ("2.5x",), 1, seed=100 + n0)


@pytest.mark.parametrize("algo", ["dcfr", "pcfr+"])
@pytest.mark.parametrize("name", [(5, 1, 2), (5, 31, 33), (5, 65, 63), (5, 127, 129), (5, 130, 1081), (4, 200, 171), "flop"])
def test_fp8_sizes(tmp_path, monkeypatch, name, algo):
    monkeypatch.setenv("GTOB_TUNE_CACHE", str(tmp_path / "shapes.txt"))
    cfg, n = _fp8_config(name), 3
    spot = g.Spot(cfg)
    host = g.Solver(spot, storage="f32", algo=algo)
    gpu = g.GpuSolver(host, device_format="fp8")
    gpu.iterate(n)
    gpu.sync_to_cpu(host)
    batch = g.Batch([g.Spot(cfg)], storage="f32", algo=algo, device_format="fp8")
    batch.run(max_iterations=n, target_pct=0.0, check_every=n, persistent=True, window=1)
    row = batch.rows()[0]
    assert row["status"] == 0 and row["iterations"] == n, row
    for which in (0, 1):
        for p in (0, 1):
            a = host.arena(which, p)
            assert np.isfinite(a).all()
            np.testing.assert_array_equal(a, batch.solver(0).arena(which, p))


@pytest.mark.parametrize("storage,fmt,algo", FORMATS)
def test_locks_on_wide_nodes(storage, fmt, algo):
    """Nodes of 5 to 7 actions locked, one of each player."""
    cfg = _config(5, 150, 37, ("10", "20", "30", "45", "60", "80"), ("2.5x",), 1, seed=6, stack=1000)
    out = []
    for engine in ("staged", "plain"):
        spot = g.Spot(cfg)
        host = g.Solver(spot, storage=storage, algo=algo)
        t = spot.tree()
        for p in (0, 1):
            n = int(np.nonzero((t["kind"] == 0) & (t["player"] == p) & (t["nchild"] >= 5))[0][0])
            s = np.random.default_rng(n).random((int(t["nchild"][n]), spot.nh[p]), np.float32)
            host.set_lock(n, (s / s.sum(0)).reshape(-1))
        gpu = g.GpuSolver(host, device_format=fmt, engine=engine)
        gpu.iterate(3)
        out.append([gpu.exploitability()] + [gpu.root_cfv(p, m) for p in (0, 1) for m in (0, 1)])
        gpu.iterate(1)
        out[-1] += [gpu.export_arena(w, p) for w in (0, 1) for p in (0, 1)]
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("storage,fmt,algo", FORMATS)
@pytest.mark.parametrize("n0,n1", [(20, 40), (70, 130)])
def test_infinite_and_nan_values(n0, n1, storage, fmt, algo):
    """A pot whose payoffs times reach pass the largest float: values, regrets
    and the quantised blocks' maxima become infinite or NaN, on both engines
    alike."""
    cfg = _config(5, n0, n1, ("75",), ("2.5x",), 1, seed=11)
    cfg["tree"]["starting_pot"] = 3e38
    cfg["tree"]["effective_stack"] = 3e38
    out = []
    for engine in ("staged", "plain"):
        host = g.Solver(g.Spot(cfg), storage=storage, algo=algo)
        gpu = g.GpuSolver(host, device_format=fmt, engine=engine)
        gpu.iterate(3)
        out.append([gpu.root_cfv(p, m) for p in (0, 1) for m in (0, 1)])
        out[-1] += [gpu.export_arena(w, p) for w in (0, 1) for p in (0, 1)]
    assert not all(np.isfinite(a).all() for a in out[0])
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)
