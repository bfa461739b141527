"""The quadratic systems' storage by row length: rows of 0, 1, 8, 9, 31, 32 and
more entries, windows that are not full and an odd number of rows, checked by
the residual of the solution in the model written out in float64."""
import numpy as np
import pytest

from eplace_b200 import placer, synth

pytestmark = pytest.mark.gpu


def star_design(n, degrees, seed):
    """Nets of the given degrees on seeded cells (a net's pins on cells of its
    own part of the index), a third of them with a pad, and a last cell on no
    net."""
    rng = np.random.default_rng(seed)
    nt, side = 16, 400.0
    owners = []
    for k, d in enumerate(degrees):
        o = rng.choice(n - 1, size=min(d, n - 1), replace=False)
        if k % 3 == 0 or d == 2:
            o[-1] = n + k % nt
        owners.append(o)
    deg = np.array([len(o) for o in owners])
    owner = np.concatenate(owners)
    f = lambda a: np.ascontiguousarray(a, np.float32)  # noqa: E731
    q = lambda lo, hi, k: np.round(rng.uniform(lo, hi, k) * 8) / 8  # noqa: E731
    rows = int(side)
    t = np.arange(nt) / nt * 2 * np.pi
    return synth.Netlist(
        name="stars", node_w=f(np.ones(n)), node_h=f(np.ones(n)), node_cx=f(q(50, 350, n)), node_cy=f(q(50, 350, n)),
        term_llx=f(np.round(200 + 190 * np.cos(t))), term_lly=f(np.round(200 + 190 * np.sin(t))), term_w=f(np.ones(nt)),
        term_h=f(np.ones(nt)), term_is_ni=np.ones(nt, np.uint8),
        net_start=np.concatenate([[0], np.cumsum(deg)]).astype(np.int32), pin_owner=owner.astype(np.int32),
        pin_dx=f(q(-0.5, 0.5, owner.size)), pin_dy=f(q(-0.5, 0.5, owner.size)), row_llx=f(np.zeros(rows)),
        row_lly=f(np.arange(rows)), row_urx=f(np.full(rows, side)), row_h=f(np.ones(rows)), row_site_w=f(np.ones(rows)), bins=32)


def model(nl, axis):
    """(A, b) of createSparseMatrix at the netlist's centres, in float64."""
    n = nl.num_nodes
    c = np.concatenate([[nl.node_cx, nl.node_cy][axis], ([nl.term_llx, nl.term_lly][axis] + 0.5)]).astype(np.float64)
    off = [nl.pin_dx, nl.pin_dy][axis].astype(np.float64)
    A, b = np.zeros((n, n)), np.zeros(n)
    for k in range(nl.num_nets):
        p = np.arange(nl.net_start[k], nl.net_start[k + 1])
        if len(p) < 2:
            continue
        x = c[nl.pin_owner[p]] + off[p]
        lo, hi = int(np.argmin(x)), int(np.argmax(x))
        for j in range(len(p)):
            for m in range(j + 1, len(p)):
                counts = {j, m} & {lo, hi} if axis == 0 else (m == lo or j == hi or m == hi)
                u, v = nl.pin_owner[p[j]], nl.pin_owner[p[m]]
                if not counts or u == v:
                    continue
                w = 1.0 / (len(p) - 1) / max(abs(x[j] - x[m]), 25.0)
                for s, t, ps, pt in ((u, v, j, m), (v, u, m, j)):
                    if s >= n:
                        continue
                    A[s, s] += w
                    if t < n:
                        A[s, t] -= w
                        b[s] -= w * (off[p[ps]] - off[p[pt]])
                    else:
                        b[s] += w * (x[pt] - off[p[ps]])
    return A, b


@pytest.mark.parametrize("jacobi", [False, True])
@pytest.mark.parametrize("n,degrees", [
    (7, [2, 3, 5]),
    (33, [2] * 60 + [9, 10, 33, 34]),
    (255, [2] * 300 + [3, 4] * 40 + [8, 9, 10, 32, 33, 34, 40]),
    (257, [2] * 300 + [3] * 50 + [17, 31, 32, 33, 64, 65, 200]),
    (1001, [2] * 900 + [3, 4, 5] * 100 + [9, 33, 34, 129, 500, 900]),
], ids=lambda v: str(v) if isinstance(v, int) else "")
def test_solution_satisfies_the_model(n, degrees, jacobi):
    nl = star_design(n, degrees, seed=n)
    e = placer.Engine(nl, placer.default_params(target_density=1.0, bins_x=32, bins_y=32))
    st = e.quadratic_refine(1, 100, jacobi)
    xy = e.get_positions()[:n].astype(np.float64)
    for axis, err in ((0, st["error_x"]), (1, st["error_y"])):
        A, b = model(nl, axis)
        rows = np.diag(A) > 0
        inside = (np.abs(xy - 200.0) < 198.0).all()
        assert inside  # no clamp, so the centres are the solution
        r = np.linalg.norm(b - A @ xy[:, axis]) / np.linalg.norm(b)
        # the engine's own residual, plus float entries, vectors and sums of up
        # to 900 terms (a tree of 32 sums of 29): under 64 roundings of 2^-24 of
        # |A| |x|, which is the size of 2 |b| row by row here
        scale = np.linalg.norm(np.abs(A) @ np.abs(xy[:, axis])) / np.linalg.norm(b)
        assert r <= err + 64 * 2.0 ** -24 * scale, (r, err, scale)
        assert np.isfinite(xy[rows]).all()
    e.close()
