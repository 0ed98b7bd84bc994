"""QR preconditioner of the batched Jacobi SVD at its edges: 16-column panels, the
row counts at which a panel's columns change their register layout (64, 128, 256,
512) or leave the registers (more than 1024), square and single-column sectors, and
sectors whose columns repeat, vanish or lie far below rounding of the largest.  All
sectors of a call are factored together.  Against numpy's SVD with the bounds of the
other SVD tests: both are backward stable, so singular values agree to a modest
multiple of eps of the largest (1e-13), U (S V^T) reproduces the input to 1e-12 and
U's columns are orthogonal to 1e-13 of s_max^2 when weighted with their values."""
import numpy as np
import pytest

from dmrgcc_b200 import capi

pytestmark = pytest.mark.gpu

ROWS = [(64, 16), (65, 17), (128, 15), (129, 32), (256, 33), (257, 31), (512, 16), (513, 47), (1024, 48), (1025, 33),
        (1500, 20), (1025, 1), (16, 16), (17, 17), (2, 1), (97, 97)]


def _graded(rng, m, n, decades):
    k = min(m, n)
    u, _ = np.linalg.qr(rng.standard_normal((m, k)))
    v, _ = np.linalg.qr(rng.standard_normal((n, k)))
    return (u * 10.0 ** -np.linspace(0, decades, k)) @ v.T


def _degenerate(rng):
    a = rng.standard_normal((70, 40))
    a[:, 5:20] = a[:, :15]                       # repeated columns
    b = rng.standard_normal((90, 33))
    b[:, ::3] = 0.0                              # vanishing columns
    c = rng.standard_normal((40, 20))
    c[:, 10:] *= 1e-150                          # squares that underflow
    d = rng.standard_normal((50, 35)) * 10.0 ** -np.arange(35.0)[rng.permutation(35)]
    e = np.zeros((30, 18))
    e[7, 3] = -2.0                               # one entry
    f = np.outer(rng.standard_normal(300), rng.standard_normal(48))
    return [a, b, c, d, e, f]


@pytest.mark.parametrize("which", ["well", "graded", "degenerate"])
@pytest.mark.parametrize("side", [0, 1])
def test_svd_with_qr_at_panel_and_row_edges(ctx, which, side):
    rng = np.random.default_rng(23)
    mats = _degenerate(rng) if which == "degenerate" else [
        rng.standard_normal(s) if which == "well" else _graded(rng, *s, 13) for s in ROWS]
    if side:
        mats = [a.T for a in mats]
    ns = len(mats)
    idx = np.arange(ns, dtype=np.int32)
    rows = np.array([a.shape[0] for a in mats], dtype=np.int32)
    cols = np.array([a.shape[1] for a in mats], dtype=np.int32)
    c = capi.Canonical(ctx, side, rows, cols, capi.BlockSpec(idx, idx, rows, cols))
    kdev = capi.DeviceArray.from_host(ctx, np.concatenate([a.ravel() for a in mats]))
    res = c.run(kdev, 10**6, 1e-300)
    newk = capi.DeviceArray(ctx, res["ket_size"])
    can = capi.DeviceArray(ctx, res["canonical_size"])
    c.write(kdev, newk, can)
    ctx.sync()
    K, Cn = newk.download(), can.download()
    kp = cp = 0
    for s, a in enumerate(mats):
        what = f"sector {s} {a.shape}"
        ref = np.linalg.svd(a, compute_uv=False)
        got = np.sort(c.singular_values(s))[::-1]
        assert np.max(np.abs(got - ref[:got.size])) <= 1e-13 * ref[0], what
        kr, kc = int(res["ket_rows"][s]), int(res["ket_cols"][s])
        cr, cc = int(res["canon_rows"][s]), int(res["canon_cols"][s])
        k, can_s = K[kp:kp + kr * kc].reshape(kr, kc), Cn[cp:cp + cr * cc].reshape(cr, cc)
        kp += kr * kc
        cp += cr * cc
        if side:                                 # ket V^T, canonical U S
            k, can_s = k.T, can_s.T
            a = a.T
        assert np.linalg.norm(k @ can_s - a) <= 1e-12 * np.linalg.norm(a), what
        sig = np.linalg.norm(can_s, axis=1)
        w = k * sig
        assert np.max(np.abs(w.T @ w - np.diag(sig * sig))) <= 1e-13 * sig.max() ** 2, what
