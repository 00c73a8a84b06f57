"""Training of the turn-leaf network against the same training in 64 bits, at
the real dimensions: several networks trained in turn, the first one again
with its moments kept, losses and every parameter.

What a training may be off: operands and gradients are rounded to bf16 (2^-9
relative) in front of each product, sums are taken in f32 and Adam divides by
its own running scale, so the way a parameter tensor has gone differs by a few
2^-9 of that way, and by more after a single step, where an entry moves by the
learning rate times its gradient's sign.  A CPU emulation of that arithmetic
stays within 0.0152 of the way after one step and 0.0018 after 90, and within
1.6e-6 of a loss.  The bounds are 2^-5 of the way and 1e-4 of a loss.  A first
step that reads row 0 in the place of every row is off by 0.33 to 2 of the way
and by 8e-3 to 4e-2 of a loss."""
import numpy as np
import pytest
import torch

import gtopen_b200 as g

pytestmark = pytest.mark.gpu
DIMS = (2705, 1024, 3, 2652)
LR, SEED = 3e-4, 3


def _rows(n, seed):
    """Inputs as large as the generator's: four one-hot cards, a ratio, two
    normalised reach vectors; targets of a few tenths, a mask."""
    rng = np.random.default_rng(seed)
    x = np.zeros((n, DIMS[0]), np.float32)
    for i in range(n):
        x[i, rng.permutation(52)[:4]] = 1.0
    x[:, 52] = rng.random(n, np.float32)
    reach = rng.random((n, 2, 1326), np.float32) * (rng.random((n, 2, 1326)) < 0.5)
    x[:, 53:] = (reach / reach.sum(2, keepdims=True)).reshape(n, -1)
    m = (rng.random((n, DIMS[3])) < 0.85).astype(np.float32)
    return x, (rng.standard_normal((n, DIMS[3]), np.float32) * np.float32(0.3)) * m, m


class Exact:
    """The network and its optimiser in 64 bits."""

    def __init__(self, net):
        self.ps = [torch.from_numpy(a).cuda().double().requires_grad_()
                   for layer in range(DIMS[2] + 1) for a in net.params(layer)]
        self.opt = torch.optim.Adam(self.ps, lr=LR)

    def train(self, rows, epochs, batch):
        x, t, m = (torch.from_numpy(a).cuda().double() for a in rows)
        n, top, losses = len(x), (1 << 64) - 1, []
        order, s = list(range(n)), (SEED * 0x9E3779B97F4A7C15 + 1) & top
        for _ in range(epochs):
            for i in range(n - 1, 0, -1):  # Fisher-Yates, xorshift64
                s ^= (s << 13) & top
                s ^= s >> 7
                s ^= (s << 17) & top
                j = s % (i + 1)
                order[i], order[j] = order[j], order[i]
            total, nb = 0.0, max(1, n // batch)
            for k in range(nb):
                pick = torch.tensor(order[k * batch:min(n, (k + 1) * batch)]).cuda()
                h = x[pick]
                for layer in range(DIMS[2] + 1):
                    h = h @ self.ps[2 * layer].T + self.ps[2 * layer + 1]
                    if layer < DIMS[2]:
                        h = torch.nn.functional.gelu(h)
                loss = ((h - t[pick]) * m[pick]).square().mean()
                self.opt.zero_grad()
                loss.backward()
                self.opt.step()
                total += loss.item()
            losses.append(total / nb)
        return np.array(losses)


@pytest.mark.parametrize("n,batch,epochs", [(896, 256, 30), (300, 512, 2), (200, 128, 1)])
def test_training_follows_64_bits(n, batch, epochs):
    nets = [g.LeafNet(*DIMS, seed=k) for k in (21, 22)]
    exact = [Exact(net) for net in nets]
    rows = [_rows(n, k) for k in (31, 32)]
    start = [[p.detach().cpu().numpy().copy() for p in e.ps] for e in exact]
    for k in (0, 1, 0):  # the first network again, its moments and step count kept
        got = nets[k].train(*rows[k], epochs=epochs, batch=batch, lr=LR, seed=SEED)
        want = exact[k].train(rows[k], epochs, batch)
        assert np.max(np.abs(got - want) / want) <= 1e-4
        params = [a for layer in range(DIMS[2] + 1) for a in nets[k].params(layer)]
        for a, e, b in zip(params, exact[k].ps, start[k]):
            e = e.detach().cpu().numpy()
            assert np.linalg.norm(a - e) <= 2.0 ** -5 * np.linalg.norm(e - b)


def test_a_failed_product_leaves_the_last_good_step():
    """A product whose wait gave up: the call ends with an error, and weights,
    moments and step count are those of the last whole step -- the training
    goes on as if the failed call had not been made."""
    dims, n = (70, 130, 2, 40), 256
    rng = np.random.default_rng(8)
    x, t = rng.normal(0, 1, (n, 70)).astype(np.float32), rng.normal(0, 1, (n, 40)).astype(np.float32)
    m = np.ones((n, 40), np.float32)
    a, b = g.LeafNet(*dims, seed=3), g.LeafNet(*dims, seed=3)
    params = lambda net: [p for layer in range(dims[2] + 1) for p in net.params(layer)]  # noqa: E731
    for net in (a, b):
        net.train(x, t, m, epochs=2, batch=128, lr=1e-2, seed=1)
    before = params(a)
    a.inject_error()
    with pytest.raises(g.GtobError, match="timeout"):
        a.train(x, t, m, epochs=2, batch=128, lr=1e-2, seed=2)
    assert all(np.array_equal(p, q) for p, q in zip(before, params(a)))
    for net in (a, b):
        net.train(x, t, m, epochs=2, batch=128, lr=1e-2, seed=3)
    assert all(np.array_equal(p, q) for p, q in zip(params(a), params(b)))
