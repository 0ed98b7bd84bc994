"""The split-precision H_eff*psi at the edges of its image rows (8, 128), MMA widths
(16) and k slices (16 TF32, 32 BF16), against numpy on the same blocks: one sector,
one block per operand, up to 14 x 14 terms (long term lists are cut and summed).

Tolerance, relative to the sum of magnitudes of an output element: per stage, an
operand is kept to 2^-22 (TF32X3: two 11-bit parts of an FP32 value) or 2^-16
(BF16X3: two 8-bit parts), the dropped lo*lo product is as large, and the FP32
accumulator adds three products per k, each addition within 2^-23 of its magnitude;
two stages, the intermediate split again."""
import numpy as np
import pytest

from dmrgcc_b200 import capi

pytestmark = pytest.mark.gpu

EDGES = [(1, 1, 1), (7, 9, 2), (8, 16, 1), (15, 17, 2), (31, 33, 1), (32, 48, 2), (64, 127, 1), (128, 128, 2),
         (129, 130, 1), (5, 257, 3), (200, 1, 2), (140, 60, 14)]


@pytest.mark.parametrize("m,n,bond", EDGES)
@pytest.mark.parametrize("accumulate", [False, True])
@pytest.mark.parametrize("precision,bits", [(capi.DMRG_PREC_TF32X3, 22), (capi.DMRG_PREC_BF16X3, 16)])
def test_split_heff_tiles(ctx, m, n, bond, accumulate, precision, bits):
    rng = np.random.default_rng(9)
    W = rng.standard_normal((bond, bond, 1, 1))
    site = capi.SiteProblem(1, 1, np.zeros((1, 1)), capi.BlockSpec([0], [0], [m], [n]), W)
    L = [capi.BlockSpec([0], [0], [m], [m]) for _ in range(bond)]
    R = [capi.BlockSpec([0], [0], [n], [n]) for _ in range(bond)]
    K, Ld, Rd, start = (rng.standard_normal(s) for s in ((m, n), (bond, m, m), (bond, n, n), (m, n)))
    h = capi.Heff(ctx, site, L, R, precision)
    dl, dr, dk, out = (capi.DeviceArray.from_host(ctx, x) for x in (Ld, Rd, K, start))
    h.set_env(dl, dr)
    for _ in range(2):  # the second call on used images
        out.upload(start)
        h.apply(dk, out, accumulate)
    ctx.sync()
    W2 = W[:, :, 0, 0]
    want = np.einsum("xo,xab,obc->ac", W2, Ld, np.einsum("ab,obc->oac", K, Rd), optimize=True)
    mag = np.einsum("xo,xab,obc->ac", abs(W2), abs(Ld), np.einsum("ab,obc->oac", abs(K), abs(Rd)), optimize=True)
    rel = sum(4 * 2.0 ** -bits + 3 * (k + 16) * 2.0 ** -23 for k in (m, n))
    got = out.download().reshape(m, n) - (start if accumulate else 0.0)
    assert np.all(np.abs(got - want) <= rel * mag + 4 * np.finfo(float).eps * np.abs(start))
    h.close()


def test_split_operator_memory(ctx):
    """A split operator that only applies holds the split images (hi and lo, 8 bytes an
    element in TF32X3) and no FP64 ones beside them; its dense or FP64 solve makes those."""
    torch = pytest.importorskip("torch")
    m, n, bond = 1500, 1400, 8
    W = np.ones((bond, bond, 1, 1))
    site = capi.SiteProblem(1, 1, np.zeros((1, 1)), capi.BlockSpec([0], [0], [m], [n]), W)
    L, R = ([capi.BlockSpec([0], [0], [k], [k])] * bond for k in (m, n))
    ctx.sync()
    free = torch.cuda.mem_get_info()[0]
    h = capi.Heff(ctx, site, L, R, capi.DMRG_PREC_TF32X3)
    used = free - torch.cuda.mem_get_info()[0]
    h.close()
    elements = bond * (m * m + n * n) + (bond + 1) * m * n  # environments, products, psi
    # rows in panels of 128 rounded to 8, k to 16; the sums of cut tiles; allocation granularity
    assert used <= 1.5 * 8 * elements + (64 << 20), used
