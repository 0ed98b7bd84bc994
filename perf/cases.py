"""Performance cases: the site steps of a DMRG sweep, and a whole run, through
the Python binding of the C ABI (dmrgcc_b200.capi).

One site step of a sweep applies H_eff to the site tensor many times (Heff.apply,
ZHeff.apply, inside Heff.lanczos / ZHeff.lanczos), canonicalises the tensor
(Canonical.run + write) and updates an environment (Env.apply).  Sizes follow the
repository's inputs and fixtures: open chains of 16 sites with 3 bosons per site
at most (MPO bond 4), the 8x4 Bose-Hubbard cylinder with 4 (MPO bond 10) up to
bond dimension 1024, the 6x6 Hofstadter cylinder with 2 (complex, MPO bond 14) up
to 256, and the chains of the seeded U/t scan for a whole run.

A site in the middle of the lattice: the boson number left of a bond is its
sector, the bond dimension is spread over the sectors like a Gaussian, every
block allowed by the quantum numbers is present, and the environments are
Hermitian with an identity on the index that carries no operator, as in canonical
form.
"""
from __future__ import annotations

import functools
import math
import os
import tempfile

import numpy as np
import torch

from dmrgcc_b200 import capi, scan

PRECISION = {"fp64": capi.DMRG_PREC_FP64, "tf32x3": capi.DMRG_PREC_TF32X3, "bf16x3": capi.DMRG_PREC_BF16X3}


# ------------------------------------------------------------------ the cases
def listed() -> list[dict]:
    return [
        # H_eff * psi, the inner call of every Lanczos iteration: the mid-chain
        # site of the 16-site chain at D = 64 (launch latency) ...
        dict(name="heff_chain_D64", kind="heff", width=1, d=4, bosons=16, D=64, precision="fp64"),
        # ... an early sweep of the 8x4 cylinder's ramp, at a ragged bond dimension ...
        dict(name="heff_cylinder_D300", kind="heff", width=4, d=5, bosons=16, D=300, precision="fp64"),
        # ... its largest bond dimension, in FP64 and in the split precisions
        dict(name="heff_cylinder_D1024", kind="heff", width=4, d=5, bosons=16, D=1024, precision="fp64"),
        dict(name="heff_cylinder_D1024_tf32x3", kind="heff", width=4, d=5, bosons=16, D=1024, precision="tf32x3"),
        dict(name="heff_cylinder_D600_bf16x3", kind="heff", width=4, d=5, bosons=16, D=600, precision="bf16x3"),
        # the complex H_eff * psi of the 6x6 Hofstadter cylinder at its largest bond dimension
        dict(name="zheff_hofstadter_D256", kind="zheff", width=6, d=3, bosons=4, D=256),
        # the Lanczos solve of one site: small (recurrence, reorthogonalisation and
        # launches) and mid-ramp on the cylinder (matvecs)
        dict(name="lanczos_chain_D64", kind="lanczos", width=1, d=4, bosons=16, D=64, niter=20),
        dict(name="lanczos_cylinder_D512", kind="lanczos", width=4, d=5, bosons=16, D=512, niter=12),
        # the environment update that follows a site on the way right
        dict(name="env_left_cylinder_D1024", kind="env", width=4, d=5, bosons=16, D=1024, side=0, precision="fp64"),
        # the canonicalisation of a tensor widened by the subspace expansion: on the
        # way left at D = 64 of the chain, on the way right at D = 1024 of the cylinder
        dict(name="canon_right_chain_D64", kind="canon", d=4, bosons=16, D=64, expand=3.0, side=1),
        dict(name="canon_left_cylinder_D1024", kind="canon", d=5, bosons=16, D=1024, expand=3.0, side=0),
        # a whole two-site run: one chain of the U/t scan, its first half-sweeps
        dict(name="run_chain_L12_D32", kind="run", L=12, D=32, half_sweeps=3),
    ]


def _log(rng, lo: int, hi: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng) -> dict:
    kind = rng.choice(["heff", "heff", "heff", "zheff", "lanczos", "env", "zenv", "canon", "canon"])
    width = rng.choice([1, 4, 4])
    d = 4 if width == 1 else 5
    top = 256 if width == 1 else 1024
    if kind == "heff":
        return dict(kind=kind, width=width, d=d, bosons=16, D=_log(rng, 32, top),
                    precision=rng.choice(["fp64", "fp64", "tf32x3", "bf16x3"]))
    if kind == "zheff":
        return dict(kind=kind, width=6, d=3, bosons=rng.choice([4, 6]), D=_log(rng, 24, 256))
    if kind == "lanczos":
        return dict(kind=kind, width=width, d=d, bosons=16, D=_log(rng, 32, min(top, 640)), niter=rng.randint(6, 24))
    if kind == "env":
        return dict(kind=kind, width=width, d=d, bosons=16, D=_log(rng, 32, top), side=rng.randint(0, 1),
                    precision=rng.choice(["fp64", "fp64", "fp64", "tf32x3"]))
    if kind == "zenv":
        return dict(kind=kind, width=6, d=3, bosons=rng.choice([4, 6]), D=_log(rng, 24, 256), side=rng.randint(0, 1))
    return dict(kind="canon", d=d, bosons=16, D=_log(rng, 24, min(top, 900)), expand=round(rng.uniform(1.0, 3.0), 2),
                side=rng.randint(0, 1))


# ------------------------------------------------- block structure of one site
def _dims(total: float, bosons: int, spread: float = 1.9) -> list[int]:
    """Sector dimensions of a bond of dimension `total`, every sector 0..bosons present."""
    g = [math.exp(-0.5 * ((q - bosons / 2) / spread) ** 2) for q in range(bosons + 1)]
    return [max(1, int(round(total * x / sum(g)))) for x in g]


class Site:
    """Sectors, ket blocks, MPO tensor and environment blocks of one site."""

    def __init__(self, width: int, d: int, bosons: int, D: int, cplx: bool):
        self.d, self.ns = d, bosons + 1
        self.left = self.right = _dims(D, bosons)
        self.phys = np.full((self.ns, self.ns), -1, np.int32)
        for l in range(self.ns):
            for r in range(l, min(self.ns, l + d)):
                self.phys[l, r] = r - l
        self.ket = [(l, r) for l in range(self.ns) for r in range(self.ns) if self.phys[l, r] >= 0]
        # MPO bond: 0 the completed terms, 1 + 2a / 2 + 2a a pending b+ / b of the
        # site that is a + 1 steps from its partner, last nothing yet
        self.bond = 2 * width + 2
        self.charge = [0] + [1, -1] * width + [0]
        self.partner = [0] + [2 * (i // 2) + (2 if i % 2 == 0 else 1) for i in range(2 * width)] + [self.bond - 1]
        b = np.diag(np.sqrt(np.arange(1, d)), 1)
        n = np.arange(d)
        W = np.zeros((self.bond, self.bond, d, d), np.complex128)
        W[0, 0] = W[-1, -1] = np.eye(d)
        W[-1, 0] = np.diag(4.0 * n * (n - 1))
        for a in range(1, width):
            W[2 * a + 1, 2 * a - 1] = W[2 * a + 2, 2 * a] = np.eye(d)
        W[-1, 2 * width - 1], W[-1, 2 * width] = b.T, b
        for a in sorted({0, width - 1}):  # the bonds along y and x
            t = -np.exp(2j * np.pi * (a + 1) / 6) if cplx else -1.0
            W[2 * a + 1, 0] += t * b
            W[2 * a + 2, 0] += np.conj(t) * b.T
        self.W = W if cplx else np.ascontiguousarray(W.real)
        self.L = [[(i, i - c) for i in range(self.ns) if 0 <= i - c < self.ns] for c in self.charge]  # (bra, ket)
        self.R = [[(l, l + c) for l in range(self.ns) if 0 <= l + c < self.ns] for c in self.charge]  # (ket, bra)

    def spec(self, blocks, rows, cols) -> capi.BlockSpec:
        return capi.BlockSpec([l for l, _ in blocks], [r for _, r in blocks], [rows[l] for l, _ in blocks],
                              [cols[r] for _, r in blocks])

    @property
    def ket_spec(self):
        return self.spec(self.ket, self.left, self.right)

    def env_spec(self, side: int):
        lists, dims = (self.L, self.left) if side == 0 else (self.R, self.right)
        return [self.spec(b, dims, dims) for b in lists]

    def problem(self) -> capi.SiteProblem:
        return capi.SiteProblem(self.ns, self.ns, self.phys, self.ket_spec, self.W.real)

    def w(self, o1, o2, p1, p2):
        return self.W[o1, o2, p1, p2]


@functools.lru_cache(maxsize=64)
def _site(width: int, d: int, bosons: int, D: int, cplx: bool) -> Site:
    return Site(width, d, bosons, D, cplx)


def _site_of(case: dict) -> Site:
    return _site(case["width"], case["d"], case["bosons"], case["D"], case["kind"].startswith("z"))


def _views(flat: torch.Tensor, shapes) -> list[torch.Tensor]:
    out, pos = [], 0
    for r, c in shapes:
        out.append(flat[pos:pos + r * c].view(r, c))
        pos += r * c
    return out


def _shapes(spec: capi.BlockSpec):
    return list(zip(spec.rows.tolist(), spec.cols.tolist()))


# ------------------------------------------------------------------ the values
class Buf:
    """A device buffer of the calling program, as the binding takes it."""

    def __init__(self, t: torch.Tensor):
        self.t, self.ptr, self.n = t, t.data_ptr(), t.numel() * (2 if t.is_complex() else 1)


def _randn(n: int, gen, cplx: bool) -> torch.Tensor:
    dt = torch.complex128 if cplx else torch.float64
    return torch.randn(n, generator=gen, device=gen.device, dtype=dt)


def _environment(site: Site, side: int, gen, cplx: bool) -> torch.Tensor:
    """Blocks of a Hermitian environment: an identity for no operator, a Hamiltonian
    of the block's states for the completed terms, an operator and its adjoint
    for the pending ones."""
    lists, dims = (site.L, site.left) if side == 0 else (site.R, site.right)
    specs = site.env_spec(side)
    flat = _randn(sum(s.size for s in specs), gen, cplx)
    none, done = (site.bond - 1, 0) if side == 0 else (0, site.bond - 1)
    views, at = _views(flat, [x for s in specs for x in _shapes(s)]), {}
    for o, blocks in enumerate(lists):
        for b in blocks:
            at[o, b] = views[len(at)]
    for o, blocks in enumerate(lists):
        for b in blocks:
            v = at[o, b]
            n = v.shape[0]
            if o == none:
                v.copy_(torch.eye(n, dtype=v.dtype, device=v.device))
            elif o == done:
                h = (v + v.conj().T) / (2 * math.sqrt(n))
                v.copy_(h + torch.diag(torch.linspace(-6.0, 2.0, n, dtype=torch.float64, device=v.device)).to(v.dtype))
            elif site.partner[o] > o:
                v.div_(math.sqrt(max(v.shape)))
                at[site.partner[o], (b[1], b[0])].copy_(v.conj().T)
    return flat


_runtime = None


def _rt():
    """The program's context and the stream its calls run on."""
    global _runtime
    if _runtime is None:
        ctx, stream = capi.Context(0), torch.cuda.Stream()
        ctx.set_stream(stream.cuda_stream)
        _runtime = (ctx, stream)
    return _runtime


def _inputs(case: dict, seed: int, device: str) -> dict:
    """The case's input tensors, from the seed alone."""
    gen = torch.Generator(device=device).manual_seed(seed)
    kind = case["kind"]
    cplx = kind.startswith("z")
    if kind == "canon":
        return {"ket": _canon_ket(case, gen)}
    site = _site_of(case)
    psi = _randn(site.ket_spec.size, gen, cplx)
    psi /= torch.linalg.norm(psi)
    if kind in ("env", "zenv"):
        return {"ket": psi * math.sqrt(sum(site.right)), "env": _environment(site, case["side"], gen, cplx)}
    return {"psi": psi, "L": _environment(site, 0, gen, cplx), "R": _environment(site, 1, gen, cplx)}


# The canonicalised tensor: right (left) bond widened by the expansion.
def _canon_shape(case: dict):
    ns, d = case["bosons"] + 1, case["d"]
    thin = _dims(case["D"], case["bosons"])
    wide = [int(math.ceil(x * case["expand"])) for x in _dims(case["D"], case["bosons"], 2.4)]
    left, right = (thin, wide) if case["side"] == 0 else (wide, thin)
    ket = [(l, r) for l in range(ns) for r in range(l, min(ns, l + d))]
    return left, right, ket


def _sectors(case: dict):
    """Per sector of the cut bond: its ket blocks and the shape of its matrix."""
    left, right, ket = _canon_shape(case)
    out = []
    for s in range(case["bosons"] + 1):
        members = [k for k, b in enumerate(ket) if b[1 - case["side"]] == s]
        if case["side"] == 0:
            out.append((members, sum(left[ket[k][0]] for k in members), right[s]))
        else:
            out.append((members, left[s], sum(right[ket[k][1]] for k in members)))
    return out


def _canon_ket(case: dict, gen) -> torch.Tensor:
    """Sector matrices whose singular values fall by three decades over the kept
    ones and by six more over the columns that the expansion added.  The values are
    the case's, so that every seed truncates to the same dimensions; the vectors are
    the seed's."""
    left, right, ket = _canon_shape(case)
    shapes = [(left[l], right[r]) for l, r in ket]
    flat = torch.empty(sum(r * c for r, c in shapes), dtype=torch.float64, device=gen.device)
    views = _views(flat, shapes)
    q0 = case["bosons"] / 2
    uneven = np.random.default_rng(7)
    for s, (members, m, n) in enumerate(_sectors(case)):
        k = min(m, n)
        u = torch.linalg.qr(_randn(m * k, gen, False).view(m, k))[0]
        v = torch.linalg.qr(_randn(n * k, gen, False).view(n, k))[0]
        keep = max(1, math.ceil(k / case["expand"]))
        decades = torch.arange(k, dtype=torch.float64, device=gen.device)
        decades = torch.where(decades < keep, 3 * decades / keep, 3 + 6 * (decades - keep) / max(1, k - keep))
        jitter = torch.from_numpy(uneven.uniform(0.0, 0.6 / keep, k)).to(gen.device)
        a = (u * 10.0 ** (-decades - jitter) * 10.0 ** (-0.03 * (s - q0) ** 2)) @ v.T
        pos = 0
        for p in members:
            w = views[p].shape[case["side"]]
            views[p].copy_(a[pos:pos + w] if case["side"] == 0 else a[:, pos:pos + w])
            pos += w
    return flat / torch.linalg.norm(flat)


def prepare(case: dict, seed: int) -> dict:
    ctx, stream = _rt()
    kind = case["kind"]
    if kind == "run":
        rng = np.random.default_rng(seed)
        text = scan.input_text(case["L"], float(rng.uniform(2.0, 12.0)))
        for m, z in sorted(set(scan.SWEEPS)):
            text = text.replace(f"        {m:<5d} 100   100    1E-12   {z}", f"        {case['D']:<5d} 100   100    1E-12   {z}")
        f, path = tempfile.mkstemp(suffix=".in")
        with os.fdopen(f, "w") as out:
            out.write(text)
        return {"case": case, "path": path, "seed": 1 + seed % 1000}
    s = {"case": case, **{k: Buf(v) for k, v in _inputs(case, seed, "cuda").items()}}
    torch.cuda.current_stream().synchronize()
    if kind == "canon":
        left, right, ket = _canon_shape(case)
        spec = capi.BlockSpec([l for l, _ in ket], [r for _, r in ket], [left[l] for l, _ in ket], [right[r] for _, r in ket])
        s["op"] = capi.Canonical(ctx, case["side"], left, right, spec)
        return s
    site = _site_of(case)
    if kind in ("env", "zenv"):
        s["op"] = capi.Env(ctx, case["side"], site.problem(), site.env_spec(case["side"]),
                           PRECISION[case.get("precision", "fp64")], site.W if kind == "zenv" else None)
        dt = torch.complex128 if kind == "zenv" else torch.float64
        s["out"] = Buf(torch.empty(s["op"].out_size, dtype=dt, device="cuda"))
        return s
    if kind == "zheff":
        s["op"] = capi.ZHeff(ctx, site.problem(), site.env_spec(0), site.env_spec(1), site.W)
    else:
        s["op"] = capi.Heff(ctx, site.problem(), site.env_spec(0), site.env_spec(1), PRECISION[case.get("precision", "fp64")])
    s["op"].set_env(s["L"], s["R"])
    s["out"] = Buf(torch.empty_like(s["psi"].t))
    return s


def run(s: dict):
    case = s["case"]
    kind = case["kind"]
    ctx, stream = _rt()
    if kind == "run":
        r = capi.Run(ctx, s["path"], seed=s["seed"], two_site=True, stop_after_half_sweeps=case["half_sweeps"])
        r.execute()
        out = {"half_sweeps": r.half_sweeps()[0], "steps": r.steps()["energy"]}
        r.close()
        return out
    with torch.cuda.stream(stream):
        if kind in ("heff", "zheff"):
            s["op"].apply(s["psi"], s["out"])
            return s["out"].t
        if kind == "lanczos":
            s["out"].t.copy_(s["psi"].t)  # the start vector of this solve
            energy, dim = s["op"].lanczos(s["out"], case["niter"])
            return {"energy": energy, "dim": dim, "psi": s["out"].t}
        if kind in ("env", "zenv"):
            s["op"].apply(s["ket"], s["env"], s["out"])
            return s["out"].t
        res = s["op"].run(s["ket"], case["D"], 1e-12)
        ket = torch.empty(res["ket_size"], dtype=torch.float64, device="cuda")
        canonical = torch.empty(res["canonical_size"], dtype=torch.float64, device="cuda")
        s["op"].write(s["ket"], Buf(ket), Buf(canonical))
        return {"tdim": res["tdim"], "ket": ket, "canonical": canonical}


# ------------------------------------------------------- what a pass amounts to
def _products(site: Site):
    """H_eff * psi as the list of its products: per (o2, R block, ket block) the
    (o1, out block, weight) that T = K R goes into."""
    pos = {b: i for i, b in enumerate(site.ket)}
    for o2 in range(site.bond):
        for l, j in site.R[o2]:
            for k in range(site.ns):
                if (k, l) not in pos:
                    continue
                p2 = site.phys[k, l]
                terms = []
                for i in range(site.ns):
                    if (i, j) not in pos:
                        continue
                    for o1 in range(site.bond):
                        if i - k == site.charge[o1] and site.w(o1, o2, site.phys[i, j], p2) != 0:
                            terms.append((o1, (i, k), (i, j), site.w(o1, o2, site.phys[i, j], p2)))
                if terms:
                    yield o2, (l, j), (k, l), terms


def _heff_work(site: Site):
    flops = 0.0
    for _, (l, j), (k, _l), terms in _products(site):
        flops += 2.0 * site.left[k] * site.right[l] * site.right[j]
        flops += sum(2.0 * site.left[i] * site.left[k] * site.right[j] for _, (i, _k), _b, _w in terms)
    n = site.ket_spec.size
    return flops, n, sum(x.size for x in site.env_spec(0)), sum(x.size for x in site.env_spec(1))


def _env_products(site: Site, side: int):
    """The update as (in index, in block, bra block, ket block, [(out index, out block, weight)])."""
    kets = set(site.ket)
    lists = site.L if side == 0 else site.R
    for o in range(site.bond):
        for x, y in lists[o]:
            for u in range(site.ns):
                for v in range(site.ns):
                    if side == 0:    # L[o1](x bra, y ket), bra block (x, u), ket block (y, v)
                        bra, ket, out = (x, u), (y, v), (u, v)
                    else:            # R[o2](x ket, y bra), ket block (u, x), bra block (v, y)
                        bra, ket, out = (v, y), (u, x), (u, v)
                    if bra not in kets or ket not in kets:
                        continue
                    terms = []
                    for q in range(site.bond):
                        o1, o2 = (o, q) if side == 0 else (q, o)
                        w = site.w(o1, o2, site.phys[bra], site.phys[ket])
                        if w != 0:
                            terms.append((q, out, w))
                    if terms:
                        yield o, (x, y), bra, ket, terms


def work(case: dict) -> dict:
    kind = case["kind"]
    if kind == "run":
        # per bond and half-sweep some ten two-site matvecs over the scan's sectors
        site = _site(1, 4, case["L"], case["D"], False)
        flops, n, l, r = _heff_work(site)
        steps = (case["L"] - 1) * case["half_sweeps"]
        return {"bytes": 8.0 * steps * (8 * n + l + r), "flops": steps * 10 * 8 * flops}
    if kind == "canon":
        left, right, ket = _canon_shape(case)
        size = sum(left[l] * right[r] for l, r in ket)
        flops = sum(6.0 * max(m, n) * min(m, n) ** 2 for _, m, n in _sectors(case))
        out = sum(m * n for _, m, n in _sectors(case)) / case["expand"]
        return {"bytes": 8.0 * (size + out), "flops": flops}
    site = _site_of(case)
    word, mul = (16.0, 4.0) if kind.startswith("z") else (8.0, 1.0)
    if kind in ("env", "zenv"):
        flops, first = 0.0, set()
        for o, (x, y), bra, ket, terms in _env_products(site, case["side"]):
            b = site.left[bra[0]] * site.right[bra[1]]
            k = site.left[ket[0]] * site.right[ket[1]]
            if case["side"] == 0:
                if (o, x, y, bra) not in first:
                    flops += 2.0 * b * site.left[y]
                flops += 2.0 * site.right[bra[1]] * k * len(terms)
                first.add((o, x, y, bra))
            else:
                if (o, x, y, ket) not in first:
                    flops += 2.0 * k * site.right[y]
                flops += 2.0 * site.left[ket[0]] * b * len(terms)
                first.add((o, x, y, ket))
        size = sum(x.size for x in site.env_spec(case["side"])) + sum(x.size for x in site.env_spec(1 - case["side"]))
        return {"bytes": word * (size + site.ket_spec.size), "flops": mul * flops}
    flops, n, l, r = _heff_work(site)
    times = case["niter"] if kind == "lanczos" else 1
    return {"bytes": word * (2 * n + l + r), "flops": mul * flops * times}


# ------------------------------------------------------------- 64-bit reference
def _blocks_of(flat, blocks, rows, cols):
    return dict(zip(blocks, _views(flat, [(rows[a], cols[b]) for a, b in blocks])))


def _env_blocks(site: Site, side: int, flat):
    lists, dims = (site.L, site.left) if side == 0 else (site.R, site.right)
    keys = [(o, b) for o, blocks in enumerate(lists) for b in blocks]
    return dict(zip(keys, _views(flat, [(dims[b[0]], dims[b[1]]) for _, b in keys])))


def _scalar(w, like):
    return complex(w) if like.is_complex() else float(np.real(w))


class _Operator:
    def __init__(self, site: Site, x: dict):
        self.site, self.products = site, list(_products(site))
        self.L, self.R = _env_blocks(site, 0, x["L"]), _env_blocks(site, 1, x["R"])

    def __call__(self, psi):
        s = self.site
        out = torch.zeros_like(psi)
        K, O = _blocks_of(psi, s.ket, s.left, s.right), _blocks_of(out, s.ket, s.left, s.right)
        for o2, r, k, terms in self.products:
            t = K[k] @ self.R[o2, r]
            for o1, l, o, w in terms:
                O[o] += _scalar(w, psi) * (self.L[o1, l] @ t)
        return out


def _exact_lanczos(site: Site, x: dict, niter: int):
    op, v = _Operator(site, x), x["psi"]
    V, alpha, beta = [v], [], []
    h = torch.zeros_like(v)
    for i in range(niter):
        h = h + op(V[i])
        alpha.append(float(torch.dot(V[i], h)))
        h = h - alpha[i] * V[i]
        beta.append(float(torch.linalg.norm(h)))
        if i + 1 == niter:
            break
        v, h = h / beta[i], -beta[i] * V[i]
        basis = torch.stack(V)
        for _ in range(2):
            v = v - basis.T @ (basis @ v)
        V.append(v / torch.linalg.norm(v))
    e, y = np.linalg.eigh(np.diag(alpha) + np.diag(beta[:-1], 1) + np.diag(beta[:-1], -1))
    y = y[:, 0] * (1.0 if y[np.argmax(np.abs(y[:, 0])), 0] > 0 else -1.0)  # its largest component is positive
    y = torch.from_numpy(y).to(V[0])
    psi = torch.stack(V).T @ y
    return e[0], psi


def exact(case: dict, seed: int):
    kind = case["kind"]
    if kind == "run":
        return None
    x = _inputs(case, seed, "cuda")
    if kind == "canon":
        return _exact_canon(case, x["ket"])
    site = _site_of(case)
    if kind in ("heff", "zheff"):
        return _Operator(site, x)(x["psi"])
    if kind == "lanczos":
        e, psi = _exact_lanczos(site, x, case["niter"])
        return {"energy": float(e), "dim": None, "psi": psi}
    side = case["side"]
    env, K = _env_blocks(site, side, x["env"]), _blocks_of(x["ket"], site.ket, site.left, site.right)
    dims = site.right if side == 0 else site.left
    out = {}
    for o, b, bra, ket, terms in _env_products(site, side):
        t = K[bra].conj().T @ env[o, b] @ K[ket] if side == 0 else K[ket] @ env[o, b] @ K[bra].conj().T
        for q, blk, w in terms:
            if (q, blk) not in out:
                out[q, blk] = torch.zeros(dims[blk[0]], dims[blk[1]], dtype=t.dtype, device=t.device)
            out[q, blk] += _scalar(w, t) * t
    return torch.cat([out[k].reshape(-1) for k in sorted(out)])  # by index, then first and second sector


def _exact_canon(case: dict, flat):
    """numpy's thin SVD of every sector; the largest component of each left singular vector positive."""
    left, right, ket = _canon_shape(case)
    views = [v.cpu().numpy() for v in _views(flat, [(left[l], right[r]) for l, r in ket])]
    sectors, factors = _sectors(case), []
    for members, m, n in sectors:
        a = np.concatenate([views[p] for p in members], axis=case["side"])
        u, s, vt = np.linalg.svd(a, full_matrices=False)
        sign = np.array([1.0 if c[np.argmax(np.abs(c))] > 0 else -1.0 for c in u.T])
        factors.append((u * sign, s, vt * sign[:, None]))
    values = np.concatenate([s for _, s, _ in factors])
    cut = np.sort(values)[::-1][case["D"] - 1] if len(values) > case["D"] else 0.0
    tdim = [max(1, int(np.sum(s >= max(cut, 1e-12)))) for _, s, _ in factors]
    new, canonical = [None] * len(ket), []
    for (members, m, n), (u, s, vt), t in zip(sectors, factors, tdim):
        forced = s[:t] * (s[0] >= max(cut, 1e-12))  # a sector that keeps nothing holds one zero
        pos = 0
        for p in members:
            w = views[p].shape[case["side"]]
            new[p] = u[pos:pos + w, :t] if case["side"] == 0 else vt[:t, pos:pos + w]
            pos += w
        canonical.append(forced[:, None] * vt[:t] if case["side"] == 0 else u[:, :t] * forced)
    flat_of = lambda blocks: np.concatenate([np.ascontiguousarray(b).reshape(-1) for b in blocks])  # noqa: E731
    return {"tdim": None, "ket": flat_of(new), "canonical": flat_of(canonical)}
