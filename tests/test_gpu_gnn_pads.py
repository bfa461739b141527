"""The terminals' pin lists of a training pass, by list length: counted while
short, walked when one terminal has many of the pins."""
import numpy as np
import pytest

from eplace_b200 import placer
from tests.test_gpu_gnn_forms import F, H, Model, degrees, design

pytestmark = pytest.mark.gpu


def reference(nl, g, e, target):
    """Loss and weight gradient in float64 on the engine's features."""
    import torch
    m, x = Model(nl), torch.tensor(g.features(e).astype(np.float64))
    w, n, side = g.get_weights(), nl.num_nodes, float(nl.core()[2])
    parts, at = [], 0
    for rows, cols in [(H, F), (H, 1)] + 3 * [(H, 2 * H), (H, 1)] + [(4, H), (4, 1)]:
        p = torch.tensor(w[at:at + rows * cols]).reshape(rows, cols)
        parts.append((p.bfloat16() if cols > 1 else p).double().requires_grad_(True))
        at += rows * cols
    h = torch.relu(x @ parts[0].T + parts[1].T)
    for l in (2, 4, 6):
        h = torch.relu(torch.cat([h, m.mean(h)], 1) @ parts[l].T + parts[l + 1].T)
    pred = torch.cat([x[:, 7:9], x[:, 7:9]], 1) + 0.25 * torch.tanh(h @ parts[8].T + parts[9].T)
    loss = ((pred[:n] - torch.tensor(target.astype(np.float64) / side)) ** 2).sum() / (2 * n)
    loss.backward()
    return loss.item(), torch.cat([p.grad.reshape(-1) for p in parts]).numpy()


# one pin in every tenth net is a pad's: with np = 3.9 pins a net, a list of L
# pins is walked from L^2 > 10 np on, 1 / pads of the nets' tenth
@pytest.mark.parametrize("n,pads", [(2_000, 1), (5_000, 1), (40_000, 1), (40_000, 2), (40_000, 7)])
def test_gradient_by_terminal_pins(n, pads):
    nl = design(n, degrees(n + n // 5, n, [33, 700]), pads, seed=n + pads)
    e = placer.Engine(nl, placer.default_params(target_density=1.0, bins_x=32, bins_y=32))
    g = placer.Gnn(seed=4)
    w = g.get_weights()
    w[-(4 * H + 4):] = np.random.default_rng(1).uniform(-0.5, 0.5, 4 * H + 4).astype(np.float32)
    g.set_weights(w)
    target = np.random.default_rng(7).uniform(0.05, 0.95, (n, 4)).astype(np.float32) * np.float32(nl.core()[2])
    loss, grad = g.loss_grad(e, target)
    ref, rg = reference(nl, g, e, target)
    # the bounds of the gradient by row count
    assert loss == pytest.approx(ref, rel=1e-5)
    assert np.abs(grad - rg).max() < 1e-3 * np.abs(rg).max()
    # the order of a terminal's pins is fixed
    g.release(e)
    again = g.loss_grad(e, target)
    assert again[0] == loss and np.array_equal(again[1], grad)
    g.close()
    e.close()


def test_a_terminal_on_most_nets_costs_no_square():
    """60k pins on one terminal: the pass takes no longer than 40 times the
    pass with these pins on 600 terminals (counting alone: over 100 times)."""
    import time
    best = []
    for pads in (600, 1):
        nl = design(5_000, [3] * 600_000, pads, seed=3)
        e = placer.Engine(nl, placer.default_params(target_density=1.0, bins_x=32, bins_y=32))
        g = placer.Gnn(seed=4)
        target = np.full((5_000, 4), 0.5, np.float32)
        times = []
        for _ in range(4):
            g.release(e)
            t = time.perf_counter()
            g.loss_grad(e, target)
            times.append(time.perf_counter() - t)
        best.append(min(times[1:]))
        g.close()
        e.close()
    assert best[1] < 40 * best[0], best
