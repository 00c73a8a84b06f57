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
