"""The host's side of a run: step limits around the replay's eight steps, a stop
inside and at the end of a replay, a stage that is over before its first step,
runs one after another and several at once -- each against the same steps taken
one call at a time."""
import numpy as np
import pytest

from eplace_b200 import placer, synth

pytestmark = pytest.mark.gpu


def engine(target=0.1, seed=3, cells=400):
    nl = synth.blob_start(synth.standard_cell(cells, seed=seed, every_cell_pinned=True, local_pads=True), sigma_frac=0.15)
    e = placer.Engine(nl, placer.default_params(target_density=1.0, bins_x=32, bins_y=32, precision=placer.PREC_FP64,
                                                target_overflow=target))
    e.save_positions()
    return e


def stepwise(e, limit=0):
    e.load_positions()
    e.initialize()
    e.nesterov_begin()
    taken = 0
    while (not limit or taken < limit) and not e.nesterov_step():
        taken += 1
    s = e.query()
    e.nesterov_end()
    return taken, s["overflow"], e.get_positions_f64()


def run(e, limit=0):
    e.load_positions()
    e.initialize()
    st = e.nesterov_run(limit)
    return st["iterations"], st["overflow"], e.get_positions_f64()


def same(a, b):
    assert a[0] == b[0] and a[1] == b[1] and np.array_equal(a[2], b[2])


@pytest.mark.parametrize("limit", [1, 6, 7, 8, 9, 15, 16, 17, 24])
def test_limited_run_takes_the_same_steps(limit):
    e = engine(target=1e-3)
    ref = stepwise(e, limit)
    assert ref[0] == limit
    same(run(e, limit), ref)
    same(run(e, limit), ref)  # a second run on the same graph
    e.close()


@pytest.mark.parametrize("target", [0.9, 0.6, 0.5, 0.4, 0.3, 0.25, 0.2, 0.15])
def test_run_stops_where_the_steps_do(target):
    e = engine(target=target)
    ref = stepwise(e)
    same(run(e), ref)
    same(run(e, 1000), ref)  # a limit that is not reached
    e.close()


def test_stage_that_is_over_takes_no_step():
    e = engine(target=50.0)
    e.initialize()
    before = e.get_positions_f64()
    assert e.nesterov_run()["iterations"] == 0
    assert np.array_equal(e.get_positions_f64(), before)
    e.close()


def test_batch_of_runs_with_different_ends():
    es = [engine(target=t, seed=s, cells=n) for t, s, n in ((0.5, 1, 200), (0.3, 2, 900), (50.0, 3, 300), (0.2, 4, 400))]
    ref = [run(e) for e in es]
    for e in es:
        e.load_positions()
        e.initialize()
    st = placer.run_batch(es)
    for e, s, r in zip(es, st, ref):
        same((s["iterations"], s["overflow"], e.get_positions_f64()), r)
        e.close()
