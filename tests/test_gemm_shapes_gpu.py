"""The packed FP64 block GEMM at the edges of its units (8 x 8), tiles (32 or 64),
slices (32 k indices) and split tiles, through H_eff*psi and both environment
updates, real and complex, against numpy on the same blocks.

One sector, so every operand is one block; several MPO terms per output, enough
work in the last case for 64-wide tiles cut into parts.  Tolerance: a sum of
`terms` products of length k has an error of at most ~(k + terms) eps times the
sum of magnitudes; two chained products, 8x slack (a complex product is four real
ones, whose magnitudes are at most twice the complex one's)."""
import numpy as np
import pytest

from dmrgcc_b200 import capi

pytestmark = pytest.mark.gpu

EDGES = [(1, 1, 1), (7, 9, 1), (8, 8, 2), (9, 17, 1), (16, 15, 2), (33, 40, 1), (63, 65, 2), (64, 64, 1), (66, 129, 1),
         (131, 72, 2), (200, 1, 1), (3, 200, 1), (190, 185, 5), (70, 450, 14)]


def _problem(m, n, bond, seed, cplx=False):
    rng = np.random.default_rng(seed)
    W = _values(rng, (bond, bond, 1, 1), cplx)
    site = capi.SiteProblem(1, 1, np.zeros((1, 1)), capi.BlockSpec([0], [0], [m], [n]), W.real)
    L = [capi.BlockSpec([0], [0], [m], [m]) for _ in range(bond)]
    R = [capi.BlockSpec([0], [0], [n], [n]) for _ in range(bond)]
    return site, L, R, W[:, :, 0, 0], rng


def _values(rng, shape, cplx):
    x = rng.standard_normal(shape)
    return x + 1j * rng.standard_normal(shape) if cplx else x


def _upload(ctx, x):
    return capi.DeviceArray.from_host(ctx, np.ascontiguousarray(x).view(np.float64))


def _download(d, shape, cplx):
    x = d.download()
    return (x.view(np.complex128) if cplx else x).reshape(shape)


def _bound(exact_abs, k, terms):
    return 8 * (k + terms) * np.finfo(float).eps * exact_abs


@pytest.mark.parametrize("m,n,bond", EDGES)
@pytest.mark.parametrize("accumulate", [False, True])
@pytest.mark.parametrize("cplx", [False, True])
def test_heff_tiles(ctx, m, n, bond, accumulate, cplx):
    site, L, R, W, rng = _problem(m, n, bond, 3, cplx)
    K, Ld, Rd, start = (_values(rng, x, cplx) for x in ((m, n), (bond, m, m), (bond, n, n), (m, n)))
    h = capi.ZHeff(ctx, site, L, R, W[:, :, None, None]) if cplx else capi.Heff(ctx, site, L, R)
    dl, dr, dk, out = (_upload(ctx, x) for x in (Ld, Rd, K, start))
    h.set_env(dl, dr)
    for _ in range(2):  # the queue and the split tiles' counters are left ready for the next launch
        out.upload(np.ascontiguousarray(start).view(np.float64))
        h.apply(dk, out, accumulate)
    ctx.sync()
    T = np.einsum("ab,obc->oac", K, Rd)
    want = np.einsum("xo,xab,obc->ac", W, Ld, T, optimize=True) + (start if accumulate else 0.0)
    mag = np.einsum("xo,xab,obc->ac", abs(W), abs(Ld), np.einsum("ab,obc->oac", abs(K), abs(Rd)), optimize=True)
    bound = _bound(mag + abs(start), m + n, bond * bond) * (2 if cplx else 1)
    assert np.all(np.abs(_download(out, (m, n), cplx) - want) <= bound)
    h.close()


@pytest.mark.parametrize("m,n,bond", EDGES)
@pytest.mark.parametrize("side", [0, 1])
@pytest.mark.parametrize("cplx", [False, True])
def test_env_tiles(ctx, m, n, bond, side, cplx):
    site, L, R, W, rng = _problem(m, n, bond, 5, cplx)
    k = m if side == 0 else n
    K, E = _values(rng, (m, n), cplx), _values(rng, (bond, k, k), cplx)
    env = capi.Env(ctx, side, site, L if side == 0 else R, Wc=W[:, :, None, None] if cplx else None)
    dk, de = _upload(ctx, K), _upload(ctx, E)
    shape = (bond, n, n) if side == 0 else (bond, m, m)
    out = _upload(ctx, np.full(shape, 7.0 + (3j if cplx else 0.0)))  # overwritten
    for _ in range(2):
        env.apply(dk, de, out)
    ctx.sync()

    def update(W, K, E):
        if side == 0:
            return np.einsum("xo,xij->oij", W, np.einsum("ki,xkl,lj->xij", K.conj(), E, K, optimize=True))
        return np.einsum("ox,xji->oji", W, np.einsum("jl,xlk,ik->xji", K, E, K.conj(), optimize=True))

    bound = _bound(update(abs(W), abs(K), abs(E)), 2 * k, bond) * (2 if cplx else 1)
    assert np.all(np.abs(_download(out, shape, cplx) - update(W, K, E)) <= bound)
    env.close()
