"""The grouped FP64 block GEMM at the edges of its tiles (8-wide DMMA units, at
most 64 x 64 output tiles, k-steps of 16) in the three transpose forms that the
sweep uses: H_eff*psi (A B), the left environment (A^T B) and the right one
(A B^T), against numpy on the same blocks.

One sector, so every operand is one block; several MPO terms per output, enough
of them in the last case for split-K chunks.  Tolerance: a sum of `terms`
products of length k has an error of at most ~(k + terms) eps times the sum of
magnitudes; two chained products, 8x slack."""
import numpy as np
import pytest

from dmrgcc_b200 import capi

pytestmark = pytest.mark.gpu

EDGES = [(1, 1, 1), (7, 9, 1), (8, 8, 2), (9, 17, 1), (16, 15, 2), (33, 40, 1), (63, 65, 2), (64, 64, 1), (66, 129, 1),
         (131, 72, 2), (200, 1, 1), (3, 200, 1), (190, 185, 5), (70, 450, 14)]


def _problem(m, n, bond, seed):
    rng = np.random.default_rng(seed)
    W = rng.standard_normal((bond, bond, 1, 1))
    site = capi.SiteProblem(1, 1, np.zeros((1, 1)), capi.BlockSpec([0], [0], [m], [n]), W)
    L = [capi.BlockSpec([0], [0], [m], [m]) for _ in range(bond)]
    R = [capi.BlockSpec([0], [0], [n], [n]) for _ in range(bond)]
    return site, L, R, W[:, :, 0, 0], rng


def _bound(exact_abs, k, terms):
    return 8 * (k + terms) * np.finfo(float).eps * exact_abs


@pytest.mark.parametrize("m,n,bond", EDGES)
@pytest.mark.parametrize("accumulate", [False, True])
def test_heff_tiles(ctx, m, n, bond, accumulate):
    site, L, R, W, rng = _problem(m, n, bond, 3)
    K, Ld, Rd = rng.standard_normal((m, n)), rng.standard_normal((bond, m, m)), rng.standard_normal((bond, n, n))
    h = capi.Heff(ctx, site, L, R)
    dl, dr, dk = (capi.DeviceArray.from_host(ctx, x) for x in (Ld, Rd, K))
    start = rng.standard_normal((m, n))
    out = capi.DeviceArray.from_host(ctx, start)
    h.set_env(dl, dr)
    for _ in range(2):  # the split-K counters are left ready for the next launch
        out.upload(start)
        h.apply(dk, out, accumulate)
    ctx.sync()
    T = np.einsum("ab,obc->oac", K, Rd)
    want = np.einsum("xo,xab,obc->ac", W, Ld, T, optimize=True) + (start if accumulate else 0.0)
    mag = np.einsum("xo,xab,obc->ac", abs(W), abs(Ld), np.einsum("ab,obc->oac", abs(K), abs(Rd)), optimize=True)
    assert np.all(np.abs(out.download().reshape(m, n) - want) <= _bound(mag + abs(start), m + n, bond * bond))
    h.close()


@pytest.mark.parametrize("m,n,bond", EDGES)
@pytest.mark.parametrize("side", [0, 1])
def test_env_tiles(ctx, m, n, bond, side):
    site, L, R, W, rng = _problem(m, n, bond, 5)
    K = rng.standard_normal((m, n))
    k = m if side == 0 else n
    E = rng.standard_normal((bond, k, k))
    env = capi.Env(ctx, side, site, L if side == 0 else R)
    dk, de = capi.DeviceArray.from_host(ctx, K), capi.DeviceArray.from_host(ctx, E)
    out = capi.DeviceArray.from_host(ctx, np.full(env.out_size, 7.0))  # overwritten
    for _ in range(2):
        env.apply(dk, de, out)
    ctx.sync()

    def update(W, K, E):
        if side == 0:
            return np.einsum("xo,xij->oij", W, np.einsum("ki,xkl,lj->xij", K, E, K, optimize=True))
        return np.einsum("ox,xji->oji", W, np.einsum("jl,xlk,ik->xji", K, E, K, optimize=True))

    got = out.download().reshape(bond, *([n, n] if side == 0 else [m, m]))
    assert np.all(np.abs(got - update(W, K, E)) <= _bound(update(abs(W), abs(K), abs(E)), 2 * k, bond))
    env.close()
