"""The Lanczos iteration's vector kernel at the edges of its forms: vectors just above
the dense branch (100), of one cluster (up to 16384 components) and of a cooperative
grid beyond, short runs and ones whose basis no longer fits shared memory; as a
captured loop and launch by launch.

H = L (x) R on one block, symmetric with a spread spectrum, against numpy's Lanczos
with full reorthogonalisation from the same vector.  Both Ritz values carry rounding
errors of a few eps ||H|| per step (orthogonality kept to rounding): 1e-12 ||H|| is
above 60 steps' worth; the returned vector has unit norm and that Rayleigh quotient to
the same bound."""
import numpy as np
import pytest

from dmrgcc_b200 import capi

pytestmark = pytest.mark.gpu

SHAPES = [(10, 10), (101, 1), (13, 17), (127, 129), (128, 128), (113, 145), (150, 160)]


def _symmetric(rng, n):
    q, _ = np.linalg.qr(rng.standard_normal((n, n)))
    return (q * np.linspace(-1.0, 1.3, n)) @ q.T


def _lowest(L, R, x, steps):
    V, alpha, beta = [x / np.linalg.norm(x)], [], []
    for i in range(steps):
        w = (L @ V[-1].reshape(L.shape[0], -1) @ R).ravel()
        alpha.append(V[-1] @ w)
        for _ in range(2):
            w -= np.array(V).T @ (np.array(V) @ w)
        beta.append(np.linalg.norm(w))
        V.append(w / beta[-1])
    return np.linalg.eigvalsh(np.diag(alpha) + np.diag(beta[:-1], 1) + np.diag(beta[:-1], -1))[0]


@pytest.mark.parametrize("m,n", SHAPES)
@pytest.mark.parametrize("niter", [2, 9, 60])
@pytest.mark.parametrize("graph", [True, False])
def test_lanczos_step_forms(ctx, m, n, niter, graph):
    niter = min(niter, m * n // 4)
    rng = np.random.default_rng(m * n)
    L, R, x = _symmetric(rng, m), _symmetric(rng, n), rng.standard_normal(m * n)
    site = capi.SiteProblem(1, 1, np.zeros((1, 1)), capi.BlockSpec([0], [0], [m], [n]), np.ones((1, 1, 1, 1)))
    h = capi.Heff(ctx, site, [capi.BlockSpec([0], [0], [m], [m])], [capi.BlockSpec([0], [0], [n], [n])])
    h.set_graph(graph)
    dl, dr, psi = (capi.DeviceArray.from_host(ctx, v) for v in (L, R, x / np.linalg.norm(x)))
    h.set_env(dl, dr)
    e, dim = h.lanczos(psi, niter, 0.0, 0.0)
    v = psi.download()
    h.close()
    norm = np.abs(np.linalg.eigvalsh(L)).max() * np.abs(np.linalg.eigvalsh(R)).max()
    assert dim == niter
    assert abs(e - _lowest(L, R, x, niter)) <= 1e-12 * norm
    assert abs(np.linalg.norm(v) - 1.0) <= 1e-12
    assert abs(v @ (L @ v.reshape(m, n) @ R).ravel() - e) <= 1e-12 * norm


@pytest.mark.parametrize("m,n", [(13, 17), (113, 145), (150, 160), (640, 640)])
@pytest.mark.parametrize("niter", [3, 100])
def test_converged_loop(ctx, m, n, niter):
    """A solve that converges before `niter`, and one that ends there, in both captured
    forms (the convergence test beside the next matvec; after the vector work, above 1
    GFLOP: the last shape) and both vector kernels: the captured loop launches the same
    kernels as launch by launch, so dimension, energy and vector are the same bits."""
    rng = np.random.default_rng(m)
    u, v = (rng.standard_normal(k) for k in (m, n))
    L, R = (np.eye(k) * 0.1 + np.outer(x, x) / (x @ x) for k, x in ((m, u), (n, v)))  # of -L (x) R: -1.21, -0.11, -0.01
    site = capi.SiteProblem(1, 1, np.zeros((1, 1)), capi.BlockSpec([0], [0], [m], [n]), -np.ones((1, 1, 1, 1)))
    start = rng.standard_normal(m * n)
    got = []
    for graph in (True, True, False):
        h = capi.Heff(ctx, site, [capi.BlockSpec([0], [0], [m], [m])], [capi.BlockSpec([0], [0], [n], [n])])
        h.set_graph(graph)
        dl, dr, psi = (capi.DeviceArray.from_host(ctx, x) for x in (L, R, start / np.linalg.norm(start)))
        h.set_env(dl, dr)
        got.append((*h.lanczos(psi, niter, 1e-11, 1e-12), psi.download()))
        h.close()
    e, dim, vec = got[0]
    assert dim == 3
    for other in got[1:]:
        assert other[:2] == (e, dim) and np.array_equal(other[2], vec)
    assert abs(e + 1.21) <= 1e-10 and abs(abs(vec @ np.outer(u, v).ravel()) ** 2 / (u @ u) / (v @ v) - 1) <= 1e-9
