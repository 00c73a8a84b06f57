"""The default engine's chance kernel (64 hands a CTA, children loaded by four
threads a hand) against the plain engine's own (one CTA a node, hands strided,
children one after the other): sums in card order on both sides, so every arena
entry is equal bit for bit.  Sizes around the 64-hand chunks, and a flop whose
suit permutations reach across chunks."""
import pytest

from test_gpu_vector_kernels import _config, _equal

from gtopen_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n0,n1", [(63, 65), (64, 129), (192, 128)])
def test_chunk_edges(n0, n1):
    _equal(_config(4, n0, n1, ("75",), ("2.5x",), 1, seed=7 + n0))


@pytest.mark.parametrize("board", ["KsQs2d", "7h7d2h", "JcTc4c"])
def test_permutations_across_chunks(board):
    """Suit-symmetric ranges of over 150 hands a side on two-tone, paired and
    monotone flops: the children of isomorphic cards are read through hand
    permutations."""
    st = {"bet": W.sizes("50"), "raise": [], "donk": []}
    cfg = {"board": board, "range_oop": "22+,A2s+,K8s+,Q9s+,J9s+,T8s+,97s+,ATo+,KJo+",
           "range_ip": "22+,A5s+,K9s+,QTs+,J9s+,T9s,98s,87s,A9o+,KTo+,QJo",
           "tree": {"starting_pot": 100.0, "effective_stack": 150.0, "rake_pct": 0.0, "rake_cap": 0.0,
                    "oop": [st, st, st], "ip": [st, st, st], "allin_threshold": 0.85, "add_allin": False,
                    "max_raises": 0}}
    _equal(cfg, iters=2)
    _equal(cfg, "compressed", "i16sr", iters=2)
