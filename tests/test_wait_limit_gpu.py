"""A bounded wait of the packed FP64 products that gives up: the kernels end, the status
reaches the caller, and nothing of it is left for the next application.

The limit is lowered on the host (Context.set_wait_polls); one sector, enough work for
64-wide tiles that are cut into parts, and a small case of one tile."""
import numpy as np
import pytest

from dmrgcc_b200 import capi

pytestmark = pytest.mark.gpu

SHAPES = [(9, 17, 1), (190, 185, 5), (70, 450, 14)]


@pytest.fixture()
def own_ctx():
    c = capi.Context(0)
    yield c
    c.close()


def _case(ctx, kind, m, n, bond):
    """An operator and its buffers: apply(which of two inputs) and the output's download()."""
    rng = np.random.default_rng(11)
    cplx = kind[0] == "z"

    def values(*shape):
        x = rng.standard_normal(shape)
        return x + 1j * rng.standard_normal(shape) if cplx else x

    def upload(x):
        return capi.DeviceArray.from_host(ctx, np.ascontiguousarray(x).view(np.float64))

    W = values(bond, bond, 1, 1)
    site = capi.SiteProblem(1, 1, np.zeros((1, 1)), capi.BlockSpec([0], [0], [m], [n]), W.real)
    L = [capi.BlockSpec([0], [0], [m], [m])] * bond
    R = [capi.BlockSpec([0], [0], [n], [n])] * bond
    dk, dl, dr = [upload(values(m, n)) for _ in range(2)], upload(values(bond, m, m)), upload(values(bond, n, n))
    if kind.endswith("env"):
        op, out = capi.Env(ctx, 0, site, L, Wc=W if cplx else None), upload(values(bond, n, n))
        return op, (lambda i=0: op.apply(dk[i], dl, out)), out.download
    op = capi.ZHeff(ctx, site, L, R, W) if cplx else capi.Heff(ctx, site, L, R)
    op.set_env(dl, dr)
    out = upload(values(m, n))
    return op, (lambda i=0: op.apply(dk[i], out)), out.download


@pytest.mark.parametrize("kind", ["heff", "zheff", "env", "zenv"])
@pytest.mark.parametrize("m,n,bond", SHAPES)
def test_give_up_reports(own_ctx, kind, m, n, bond):
    op, apply, _ = _case(own_ctx, kind, m, n, bond)
    own_ctx.set_wait_polls(0)
    apply()
    with pytest.raises(capi.DmrgError) as err:
        own_ctx.sync()
    assert err.value.code == capi.E_NUMERIC
    own_ctx.sync()  # the status is read once
    own_ctx.set_wait_polls(-1)
    op.close()


@pytest.mark.parametrize("kind", ["heff", "zheff", "env", "zenv"])
@pytest.mark.parametrize("m,n,bond", SHAPES)
def test_next_application_is_whole(own_ctx, kind, m, n, bond):
    """However far a launch came before it gave up (some parts of a cut tile done, some
    not), the operator's next application gives what it gave before, bit for bit."""
    op, apply, download = _case(own_ctx, kind, m, n, bond)
    apply()
    own_ctx.sync()
    want = download()
    for polls in range(6):
        own_ctx.set_wait_polls(polls)
        apply(1)
        try:
            own_ctx.sync()
        except capi.DmrgError as err:
            assert err.code == capi.E_NUMERIC
        own_ctx.set_wait_polls(-1)
        apply()
        own_ctx.sync()
        assert np.array_equal(download(), want)
    op.close()


@pytest.mark.parametrize("kind", ["heff", "zheff"])
@pytest.mark.parametrize("m,n", [(5, 7), (13, 17)])
def test_lanczos_reports(own_ctx, kind, m, n):
    """The eigensolver, in its dense branch (below 100 components) and beyond: its own call
    fails, and the next one is not blamed for it."""
    op, _, _ = _case(own_ctx, kind, m, n, 1)
    x = np.random.default_rng(5).standard_normal(m * n * (2 if kind == "zheff" else 1))
    psi = capi.DeviceArray.from_host(own_ctx, x / np.linalg.norm(x))
    own_ctx.set_wait_polls(0)
    with pytest.raises(capi.DmrgError) as err:
        op.lanczos(psi, 4)
    assert err.value.code == capi.E_NUMERIC and "gave up waiting" in str(err.value)
    own_ctx.sync()
    own_ctx.set_wait_polls(-1)
    op.close()


def test_profile_reports(own_ctx):
    op, _, _ = _case(own_ctx, "heff", 9, 17, 1)
    psi, out = capi.DeviceArray(own_ctx, 9 * 17), capi.DeviceArray(own_ctx, 9 * 17)
    psi.zero()
    out.zero()
    own_ctx.set_wait_polls(0)
    with pytest.raises(capi.DmrgError) as err:
        op.profile(psi, out)
    assert err.value.code == capi.E_NUMERIC
    own_ctx.sync()
    op.close()
