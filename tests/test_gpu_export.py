"""Read-back of arenas: the packed export of an engine that holds a fraction of
its spot against the whole arena of one engine."""
import numpy as np
import pytest

import gtopen_b200 as g
from gtopen_b200 import workloads as W

pytestmark = pytest.mark.gpu


def _flop(frac=(0.15, 0.2)):
    return W.flop_spot(g.evaluate7, seed=6, bet=("50",), raise_=(), max_raises=0, pot=100, stack=330, frac=frac)


@pytest.mark.parametrize("fmt,algo", [("f32", "dcfr"), ("i16", "pcfr+"), ("i16sr", "dcfr"), ("fp8", "dcfr")])
def test_first_packed_export_of_a_shard(fmt, algo):
    """The first packed export uploads its table of blocks and uses it at once.
    Sixteen shards hold thousands of blocks each; their exports, put together,
    are one engine's arenas bit for bit."""
    host = g.Solver(g.Spot(_flop()), storage="f32", algo=algo, use_iso=False)
    assert min(host.spot.data_size) * 4 >= 8 << 20
    one = g.GpuSolver(host, device_format=fmt)
    sh = g.Shards(host, 16, device_format=fmt)
    one.iterate(2)
    sh.iterate(2)
    for which in (0, 1, 2) if algo == "pcfr+" else (0, 1):
        for p in (0, 1):
            np.testing.assert_array_equal(sh.export_arena(which, p), one.export_arena(which, p))


def test_engines_read_back_side_by_side():
    """Seven engines, each read back twice from a thread of its own: every arena
    as when read back alone."""
    from concurrent.futures import ThreadPoolExecutor

    hosts = [g.Solver(g.Spot(_flop((0.08 + 0.01 * k, 0.1))), storage="f32", use_iso=False) for k in range(7)]
    gpus = [g.GpuSolver(h) for h in hosts]
    for k, gpu in enumerate(gpus):
        assert hosts[k].spot.data_size[0] * 4 >= 8 << 20
        gpu.iterate(k + 1)
    alone = [[gpu.export_arena(1, p) for p in (0, 1)] for gpu in gpus]
    with ThreadPoolExecutor(7) as pool:
        for _ in range(2):
            both = list(pool.map(lambda gpu: [gpu.export_arena(1, p) for p in (0, 1)], gpus))
            for a, b in zip(alone, both):
                np.testing.assert_array_equal(a[0], b[0])
                np.testing.assert_array_equal(a[1], b[1])


@pytest.mark.parametrize("storage,fmt", [("f32", None), ("compressed", "i16sr"), ("f32", "fp8")])
def test_read_back_between_iterations(tmp_path, storage, fmt):
    """The read-back image and the sweeps' fold summaries share memory: an
    engine read back, synced, saved and queried after every iteration goes on
    as one that is left alone, bit for bit."""
    cfg = W.small_flop_spot()
    ends = []
    for busy in (True, False):
        host = g.Solver(g.Spot(cfg), storage=storage)
        gpu = g.GpuSolver(host, device_format=fmt)
        for _ in range(4):
            gpu.iterate(1)
            if busy:
                for which in (0, 1):
                    for p in (0, 1):
                        gpu.export_arena(which, p)
                gpu.sync_to_cpu(host)
                gpu.save(str(tmp_path / "busy.gto"))
                g.node_strategy(gpu, 0, int(host.spot.tree()["nchild"][0]), int(host.spot.tree()["player"][0]))
        ends.append([gpu.exploitability()] + [gpu.root_cfv(p, 1) for p in (0, 1)]
                    + [gpu.export_arena(which, p) for which in (0, 1) for p in (0, 1)])
    for a, b in zip(*ends):
        np.testing.assert_array_equal(a, b)


def test_sync_of_an_engine_that_holds_few_nodes_leaves_zeros():
    """A depth-limited solve with 16-bit arenas on both sides: the nodes it does
    not hold are zeros in the host's arenas, whatever was read back before."""
    spot = g.Spot(W.flop_spot(g.evaluate7, seed=6, bet=("50",), raise_=(), max_raises=0, pot=100, stack=330,
                              frac=(0.05, 0.08)))
    host = g.Solver(spot, storage="compressed", use_iso=False)
    gpu = g.dl_gpu_solver(host, g.LeafNet(2705, 128, 1, 2652, seed=2), device_format="i16")
    gpu.iterate(3)
    for p in (0, 1):
        gpu.export_arena(1, p)
    gpu.sync_to_cpu(host)
    t = spot.tree()
    visited = g.dl_plan(spot)[3].astype(bool)
    for p in (0, 1):
        held = np.zeros(spot.data_size[p], bool)
        for n in np.nonzero(visited & (t["kind"] == 0) & (t["player"] == p))[0]:
            held[int(t["data_off"][n]):int(t["data_off"][n]) + int(t["nchild"][n]) * spot.nh[p]] = True
        for which in (0, 1):
            a = host.arena(which, p)
            assert not a[~held].any()
            np.testing.assert_array_equal(a[held], gpu.export_arena(which, p)[held])
