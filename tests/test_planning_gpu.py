"""The planning of environment updates and H_eff on block structures without quantum-number
regularity: several output blocks per output index and first sector, environment lists in
any order, MPO indexes that reach nothing, a block of no rows.  Block maps exact (row-major
by sectors, where some weight is not zero), values against the same loops in numpy.

Tolerance: as in test_gemm_shapes_gpu.py, (k + terms) eps of the sum of magnitudes, 8x slack."""
import numpy as np
import pytest

from dmrgcc_b200 import capi

pytestmark = pytest.mark.gpu
EPS = np.finfo(float).eps


def _structure(seed, cplx):
    rng = np.random.default_rng(seed)
    ns, d, lb, rb = 4, 3, 5, 6
    dl, dr = rng.integers(1, 12, ns), rng.integers(1, 12, ns)
    dl[1], dr[2] = 0, 9
    phys = np.where(rng.random((ns, ns)) < 0.8, rng.integers(0, d, (ns, ns)), -1).astype(np.int32)
    phys[0, 0] = 0
    ket = [(l, r) for l in range(ns) for r in range(ns) if phys[l, r] >= 0]
    rng.shuffle(ket)
    W = rng.standard_normal((lb, rb, d, d)) + (1j * rng.standard_normal((lb, rb, d, d)) if cplx else 0)
    W[rng.random((lb, rb, d, d)) < 0.7] = 0
    W[2] = 0
    W[:, 4] = 0

    def env(bond, dims):
        out = []
        for _ in range(bond):
            blocks = [(x, y) for x in range(ns) for y in range(ns) if rng.random() < 0.6]
            rng.shuffle(blocks)
            out.append([tuple(b) for b in blocks])
        return out

    return rng, ns, phys, [tuple(k) for k in ket], dl, dr, W, env(lb, dl), env(rb, dr)


def _spec(blocks, rows, cols):
    return capi.BlockSpec([a for a, _ in blocks], [b for _, b in blocks], [rows[a] for a, _ in blocks],
                          [cols[b] for _, b in blocks])


def _fill(ctx, rng, lists, rows, cols, cplx):
    """Random values of the lists' blocks: on the device, and by (list, block)."""
    at, flat = {}, []
    for o, blocks in enumerate(lists):
        for a, b in blocks:
            x = rng.standard_normal((rows[a], cols[b])) + (1j * rng.standard_normal((rows[a], cols[b])) if cplx else 0)
            at[o, a, b] = x
            flat.append(x.ravel())
    flat = np.concatenate(flat)
    return capi.DeviceArray.from_host(ctx, np.ascontiguousarray(flat).view(np.float64)), at


def _check(got, want, mag, terms, k):
    assert np.all(np.abs(got - want) <= 16 * (k + terms) * EPS * mag)


@pytest.mark.parametrize("seed", range(6))
@pytest.mark.parametrize("side", [0, 1])
@pytest.mark.parametrize("cplx", [False, True])
def test_environment(ctx, seed, side, cplx):
    rng, ns, phys, ket, dl, dr, W, Lb, Rb = _structure(seed, cplx)
    site = capi.SiteProblem(ns, ns, phys, _spec(ket, dl, dr), W.real)
    lists, dims, odims = (Lb, dl, dr) if side == 0 else (Rb, dr, dl)
    env = capi.Env(ctx, side, site, [_spec(b, dims, dims) for b in lists], Wc=W if cplx else None)
    dk, K = _fill(ctx, rng, [ket], dl, dr, cplx)
    de, E = _fill(ctx, rng, lists, dims, dims, cplx)
    want, mag = {}, {}
    for o, blocks in enumerate(lists):
        for x, y in blocks:
            if dims[x] == 0:
                continue  # the reference skips blocks without rows
            for u in ket:
                for v in ket:
                    if side == 0 and (u[0] != x or v[0] != y) or side == 1 and (u[1] != x or v[1] != y):
                        continue
                    for q in range(W.shape[1 - side]):
                        w = W[o, q, phys[u], phys[v]] if side == 0 else W[q, o, phys[v], phys[u]]
                        if w == 0:
                            continue
                        ku, kv, e = K[0, *u], K[0, *v], E[o, x, y]
                        key = (q, u[1 - side], v[1 - side])
                        f = (lambda a, b, c: a.conj().T @ b @ c) if side == 0 else (lambda a, b, c: a @ b @ c.conj().T)
                        want[key] = want.get(key, 0) + w * f(ku, e, kv)
                        mag[key] = mag.get(key, 0) + abs(w) * f(abs(ku), abs(e), abs(kv))
    got_blocks = [(o, int(a), int(b)) for o, s in enumerate(env.out_blocks()) for a, b in zip(s.left, s.right)]
    assert got_blocks == sorted(want)
    out = capi.DeviceArray(ctx, max(1, env.out_size * (2 if cplx else 1)))
    env.apply(dk, de, out)
    ctx.sync()
    flat = out.download()
    flat = flat.view(np.complex128) if cplx else flat
    pos = 0
    for key in sorted(want):
        n = odims[key[1]] * odims[key[2]]
        _check(flat[pos:pos + n].reshape(want[key].shape), want[key], mag[key], 400, 24)
        pos += n
    env.close()


@pytest.mark.parametrize("seed", range(6))
@pytest.mark.parametrize("cplx", [False, True])
def test_heff(ctx, seed, cplx):
    rng, ns, phys, ket, dl, dr, W, Lb, Rb = _structure(seed, cplx)
    site = capi.SiteProblem(ns, ns, phys, _spec(ket, dl, dr), W.real)
    Ls, Rs = [_spec(b, dl, dl) for b in Lb], [_spec(b, dr, dr) for b in Rb]
    h = capi.ZHeff(ctx, site, Ls, Rs, W) if cplx else capi.Heff(ctx, site, Ls, Rs)
    dk, K = _fill(ctx, rng, [ket], dl, dr, cplx)
    dL, L = _fill(ctx, rng, Lb, dl, dl, cplx)
    dR, R = _fill(ctx, rng, Rb, dr, dr, cplx)
    h.set_env(dL, dR)
    want = {k: np.zeros_like(K[0, *k]) for k in ket}
    mag = {k: np.zeros(K[0, *k].shape) for k in ket}
    for o2, rblocks in enumerate(Rb):
        for l, j in rblocks:
            for k in ket:
                if k[1] != l:
                    continue
                for out in ket:
                    if out[1] != j:
                        continue
                    for o1, lblocks in enumerate(Lb):
                        w = W[o1, o2, phys[out], phys[k]]
                        if w != 0 and (out[0], k[0]) in lblocks:
                            a, b, c = L[o1, out[0], k[0]], K[0, *k], R[o2, l, j]
                            want[out] += w * (a @ b @ c)
                            mag[out] += abs(w) * (abs(a) @ abs(b) @ abs(c))
    out = capi.DeviceArray.from_host(ctx, np.full(dk.n, 3.0))  # overwritten
    h.apply(dk, out)
    ctx.sync()
    flat = out.download()
    flat = flat.view(np.complex128) if cplx else flat
    pos = 0
    for k in ket:
        _check(flat[pos:pos + want[k].size].reshape(want[k].shape), want[k], mag[k], 400, 24)
        pos += want[k].size
    h.close()
