"""The plain path's cooperative Jacobi-PCG (one warp per interior node, rows
of a node gathered together) against the FP64 assembled solve of the oracle,
at the sizes where its split changes: one interior node, fewer nodes than a
block's warps, one and several blocks, more nodes than blocks hold warps, and
vectors beyond shared memory; and beside a serving loop, where the graph of
small kernels runs."""
import numpy as np
import pytest

import madmax_b200 as mb
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def solve(n, nrhs, ln=None, seed=3):
    rng = np.random.default_rng(seed)
    ln = ln or [v / 8.0 for v in n]
    d = mb.rve_desc(n, 0.2, (1e9, 2e10), (0.3, 0.2), ln)
    r = mb.Rve(d)
    eps = rng.normal(0, 1e-3, (nrhs, 6))
    if nrhs > 2:
        eps[1] = 0.0  # a load case without a right-hand side
    sa, st, u, info = r.homogenize(eps, rtol=1e-10, want_u=True)
    return d, r, eps, sa, st, u, info


@pytest.mark.parametrize("n,nrhs", [((2, 2, 2), 1), ((2, 3, 2), 6), ((3, 3, 5), 8), ((5, 3, 4), 1),
                                    ((6, 6, 6), 6), ((4, 9, 7), 7), ((11, 5, 13), 2)])
def test_matches_oracle(n, nrhs):
    d, r, eps, sa, st, u, info = solve(n, nrhs)
    assert info.status == 0 and info.relres <= 1e-10
    cols, _ = r.ell()
    rows = cols.reshape(-1, 3, cols.shape[1])
    assert (rows[:, 0] == rows[:, 1]).all() and (rows[:, 0] == rows[:, 2]).all()
    m = O.mesh(3, [v + 1 for v in n], [v / 8.0 for v in n])
    et = O.fiber_types(m, [v / 8.0 for v in n[:2]], d.radius)
    assert np.array_equal(mb.classify(d), et)
    _, ref, uref, _ = O.homogenize(m, et, tuple(d.E), tuple(d.nu), eps, want_u=True,
                                rtol=1e-12, lin_rtol=1e-13)
    scale = np.abs(ref).max()
    # solves to 1e-10 of the right-hand side's norm; stress and displacement
    # errors are that times the operator's condition, below 100 here
    assert np.abs(st - ref).max() <= 1e-8 * scale
    assert np.abs(sa - eps).max() <= 1e-15
    uref = np.asarray(uref).reshape(nrhs, -1)
    assert np.abs(u - uref).max() <= 1e-8 * np.abs(uref).max()
    _, _, uf, res = r.fields(nrhs - 1)
    assert (uf == u[nrhs - 1]).all() and np.isfinite(res).all()


@pytest.mark.parametrize("n,nrhs", [(20, 6), (33, 8), (44, 8)])
def test_large_matches_graph(n, nrhs):
    """Vectors all on chip, then p only: against the same solve beside a
    started serving loop, which takes the graph of small kernels."""
    d, r, eps, sa, st, u, info = solve((n, n, n), nrhs)
    assert info.status == 0 and info.relres <= 1e-10
    s = mb.Server([mb.rve_desc(3, 0.2, (1e9, 2e9), (0.3, 0.3))], max_inflight=1)
    s.start()
    sg, stg, ug, ig = r.homogenize(eps, rtol=1e-10, want_u=True)
    s.stop()
    s.close()
    assert ig.status == 0 and ig.pad > 3 * ig.inner_its > info.pad
    assert np.abs(st - stg).max() <= 1e-7 * np.abs(stg).max()
    assert np.abs(u - ug).max() <= 1e-7 * np.abs(ug).max()
    again = r.homogenize(eps, rtol=1e-10)
    assert (again[1] == st).all()
