"""Gradients through the reverse grid solve on both sides of its size rule
(one cluster launch for the whole solve up to 384 cells per block of the
cluster, a launch per substep above) and at grids that fill its blocks
unevenly: against central differences of the plain forward, at the tolerance
of the other gradient tests."""
import numpy as np
import pytest

from test_gpu_adjoint import TOL, adjoint_grads, compare, fd_grads, gpu_loss_fn, loss_scale, make, weights, STEPS

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("grid", [(1, 1, 2), (3, 2, 5), (1, 33, 1), (7, 11, 13), (16, 16, 24), (17, 19, 20)])
def test_grid_gradient_matches_finite_differences(built, tmp_path, grid):
    fix, adj, at, words = make(tmp_path, grid=grid)
    E, T = adj.forward(STEPS)
    wE, wT = weights(E, T)
    g = adjoint_grads(adj, wE, wT)
    cols = tuple(c.copy() for c in adj.columns[0])
    fd, noise = fd_grads(gpu_loss_fn(adj, wE, wT), cols, adj.C_e, adj.kappa_e, scale=loss_scale(E, T, wE, wT))
    errs = compare(g, fd, noise)
    assert max(errs.values()) <= TOL, errs


def test_batch_of_uneven_grids_gives_the_gradients_of_each(built, tmp_path):
    """record kernels and cluster solves of several adjoints at once"""
    from ephgb.adjoint import AdjointBatch

    grids = [(3, 2, 5), (7, 11, 13), (16, 16, 24)]
    alone, adjs = [], []
    for k, grid in enumerate(grids):
        for out in (alone, adjs):
            d = tmp_path / f"{k}{len(out)}{out is adjs}"
            d.mkdir()
            out.append(make(d, grid=grid, seed=40 + k)[1])
    batch = AdjointBatch(adjs)
    E, T = batch.forward(STEPS)
    wE, wT = np.ones((len(grids), STEPS)), np.full((len(grids), STEPS), 1e-3)
    batch.backward(wE, wT)
    for k, a in enumerate(alone):
        Ek, Tk = a.forward(STEPS)
        assert np.array_equal(E[k], Ek) and np.array_equal(T[k], Tk)
        g = adjoint_grads(a, wE[k], wT[k])
        gb = batch.gradients(k) if hasattr(batch, "gradients") else adjs[k].gradients(0)
        for name in g:
            assert np.array_equal(np.asarray(g[name]), np.asarray(gb[name])), name
