"""One network and several engines: its workspace is shared by calls that run on
the engines' own streams, some of which return with work pending."""
import numpy as np
import pytest

from eplace_b200 import placer, synth

pytestmark = pytest.mark.gpu


def engines(sizes):
    return [placer.Engine(synth.blob_start(synth.standard_cell(n, seed=n, every_cell_pinned=True, local_pads=True)),
                          placer.default_params(target_density=1.0)) for n in sizes]


@pytest.mark.parametrize("order", [(0, 1, 2), (2, 1, 0), (0, 1, 0, 1)])
def test_proposals_one_after_another(order):
    """Proposals for engine after engine with nothing between them give what
    each gives when it is waited for."""
    es = engines((20_000, 2_000, 9_000))
    g = placer.Gnn(seed=3)
    start, ref = [], []
    for e in es:
        start.append(e.get_positions())
        g.propose(e, 0.5)
        ref.append(e.get_positions())  # waits for the engine's stream
    for e, p in zip(es, start):
        e.set_positions(p)
    for k in order:
        g.propose(es[k], 0.5)
    for k in set(order):
        assert np.array_equal(es[k].get_positions(), ref[k])
        assert not np.array_equal(ref[k], start[k])
    g.close()
    for e in es:
        e.close()


def test_weights_set_behind_a_proposal():
    """New weights wait for the pass that still reads the old ones."""
    (e,) = engines((20_000,))
    g = placer.Gnn(seed=3)
    g.propose(e, 1.0)
    ref = e.get_positions()
    w = g.get_weights()
    for _ in range(3):
        g.release(e)
        g.propose(e, 1.0)
        g.set_weights(np.zeros_like(w))
        assert np.array_equal(e.get_positions(), ref)
        g.set_weights(w)
    g.close()
    e.close()


@pytest.mark.parametrize("cells", [60, 2_000, 40_000])  # one CTA, a few, one per SM
def test_diffusion_wait_gives_up_and_recovers(cells):
    """The diffusion's grid barrier, bounded: with no polls allowed the call
    reports EP_ERR_TIMEOUT, and with the default limit restored the next call
    computes the features anew instead of keeping what was left."""
    (e,) = engines((cells,))
    g = placer.Gnn(seed=3)
    ref, pred = g.features(e), g.forward(e)
    target = np.full((e.info.num_nodes, 4), 0.5, np.float32)
    loss = g.loss_grad(e, target)
    # 20 times: the CTAs give up one after another, the report comes once
    for call in 20 * (g.features, g.forward, lambda e: g.loss_grad(e, target)):
        g.release(e)
        g.set_wait_limit(0)
        with pytest.raises(placer.EPError) as err:
            call(e)
        assert err.value.status == placer.EP_ERR_TIMEOUT
        g.set_wait_limit()
        assert np.array_equal(g.features(e), ref)
    # a proposal returns before its pass is over: the next call reports it
    g.propose(e, 0.5)
    xy = e.get_positions()
    g.release(e)
    g.set_wait_limit(0)
    g.propose(e, 0.5)
    e.synchronize()
    g.set_wait_limit()
    with pytest.raises(placer.EPError) as err:
        g.propose(e, 0.5)
    assert err.value.status == placer.EP_ERR_TIMEOUT
    g.propose(e, 0.5)
    assert np.array_equal(e.get_positions(), xy)
    assert np.array_equal(g.forward(e), pred)
    again = g.loss_grad(e, target)
    assert again[0] == loss[0] and np.array_equal(again[1], loss[1])
    g.close()
    e.close()
