"""Timing cases of the NEGF hot path, called the way a transport code calls it.

Each case is a dict of plain values; ``kind`` names the public entry point:

``point``   ``EnergyPointSolver.solve``: one batch of energies of a device
            (system matrix, both contacts' Sancho-Rubio, selected solve with
            current, transmission, density), FP64, mixed or emulated;
``replay``  ``EnergyPointSolver.solve_graph``: the same through the captured
            CUDA graph, as a serving lane runs it;
``solve``   ``RGF.selected_solve`` on device-resident ``DSDBCOO`` containers
            with scattering self-energies, preallocated outputs;
``inv``     ``RGF.selected_inv`` on device containers;
``obc``     one contact of an SCBA iteration: ``OBCSystem(SanchoRubio)`` and
            ``contact_self_energy``;
``w``       ``CoulombScreeningSolve.solve``: the screened-interaction step.

Block-tridiagonal inputs are dense blocks, energies are the stack dimension.
``exact`` restates each of them in plain torch complex128.
"""

import math

import numpy as np
import torch

from quatrex_b200 import (DSDBCOO, RGF, CoulombScreeningSolve, EnergyPointSolver, OBCBlocks, OBCSystem,
                          SanchoRubio, contact_self_energy)

C128 = torch.complex128
KT, BIAS = 0.025, 0.1
SR_STEPS = 16  # decimation steps a lead at these broadenings needs at least
_CASES = [
    # The 16 x 64 device on its 32 energies: the smallest energy-point batch
    # of the benchmark, bound by launches and by the serial inverses.
    dict(name="point 16x64", kind="point", n=16, b=64, energies=32, precision="fp64"),
    # The headline device (32 blocks of 256) on a 64-energy batch.
    dict(name="point 32x256", kind="point", n=32, b=256, energies=64, precision="fp64"),
    # The same device in mixed precision.
    dict(name="point mixed 32x256", kind="point", n=32, b=256, energies=64, precision="mixed"),
    # A device of the uneven batch (blocks of 384) with FP64 products emulated
    # on the int8 tensor cores.
    dict(name="point emulated 8x384", kind="point", n=8, b=384, energies=37, precision="emulated"),
    # Wide blocks (512) with few energies in flight: one shard of a sweep.
    dict(name="point 8x512", kind="point", n=8, b=512, energies=21, precision="fp64"),
    # A small request of the serving loop through its captured graph.
    dict(name="replay 8x128", kind="replay", n=8, b=128, energies=16, precision="fp64"),
    # The smallest plugin call: few narrow blocks of uneven size, 4 energies.
    dict(name="solve tiny ragged", kind="solve", n=6, b=28, ragged=True, energies=4, precision="fp64"),
    # An SCBA iteration's electron solve on uneven blocks.
    dict(name="solve ragged 12x200", kind="solve", n=12, b=200, ragged=True, energies=30, precision="fp64"),
    # The same call in mixed precision, many energies of a narrower device.
    dict(name="solve mixed 10x160", kind="solve", n=10, b=160, ragged=False, energies=100, precision="mixed"),
    # Retarded Green's function only, over a full 100-energy batch.
    dict(name="inv 16x100", kind="inv", n=16, b=100, ragged=False, energies=100, precision="fp64"),
    # Boundary conditions of one contact over an energy grid.
    dict(name="obc 256", kind="obc", n=1, b=256, energies=48, precision="fp64"),
    # The screened-interaction step: small blocks in superblocks of three.
    dict(name="w 12x96", kind="w", n=12, b=96, energies=24, precision="fp64"),
]


def listed():
    return [dict(c) for c in _CASES]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    """A case of the listed ranges: kind, precision and log-uniform sizes,
    the energy count cut so that it costs no more than the largest listed."""
    kind = rng.choice(["point", "point", "solve", "solve", "inv", "obc", "w", "replay"])
    lo_b, hi_b = {"point": (48, 512), "replay": (48, 192), "solve": (16, 384), "inv": (16, 384),
                  "obc": (48, 512), "w": (24, 128)}[kind]
    c = dict(kind=kind, b=_log_int(rng, lo_b, hi_b), precision="fp64")
    c["n"] = 1 if kind == "obc" else _log_int(rng, 4, 24)
    if kind == "w":
        c["n"] = 3 * rng.randint(2, 6)
    c["energies"] = rng.randint(2, 8) if rng.random() < 0.25 else _log_int(rng, 8, 120)
    if kind in ("point", "solve"):
        c["precision"] = rng.choice(["fp64", "fp64", "mixed", "emulated"])
    if kind in ("solve", "inv"):
        c["ragged"] = rng.random() < 0.5
    if kind == "replay":
        c["energies"] = min(c["energies"], 32)
    most = work(_CASES[1])["flops"]
    while c["energies"] > 2 and (work(c)["flops"] > 0.7 * most or _resident(c) > 30e9):
        c["energies"] = max(2, int(0.8 * c["energies"]))
    return c


def _resident(c):
    size = 3 * c["b"] if c["kind"] == "w" else c["b"]
    blocks = c["n"] / 3 if c["kind"] == "w" else c["n"]
    return 16.0 * size * size * c["energies"] * (20 * blocks + 40)


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------
def _rand(g, *shape, scale=1.0):
    """Complex standard normal draws."""
    return torch.randn(*shape, dtype=C128, device="cuda", generator=g) * (math.sqrt(2.0) * scale)


def _h(x):
    return x.conj().transpose(-2, -1)


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _device(c, seed):
    """The benchmark's random device: Hermitian diagonal blocks and one
    coupling with N(0, 1) / 8 entries; energies spread over the band (as its
    16 x 64 configuration: |E| <= 2 at b = 64), Fermi occupations."""
    g = _gen(seed)
    n, b, ne = c["n"], c["b"], c["energies"]
    m = _rand(g, n, b, b, scale=0.125)
    h = 0.5 * (m + _h(m))
    t = _rand(g, b, b, scale=0.125)
    half = min(3.0, 0.2 * math.sqrt(b))
    shift = 0.02 * half * float(torch.rand(1, device="cuda", generator=g))
    e = np.linspace(-half, half, ne) + shift if ne > 1 else np.array([shift])
    f = lambda x: 1.0 / (1.0 + np.exp(np.clip(x / KT, -700, 700)))  # noqa: E731
    return h, t, e, f(e), f(e - BIAS)


def _sizes(c):
    """Block sizes: all b, or uneven ones between 0.55 b and 1.2 b."""
    if not c.get("ragged"):
        return [c["b"]] * c["n"]
    return [max(2, int(c["b"] * (0.55 + 0.65 * ((7 * i + 3) % 11) / 10.0))) for i in range(c["n"])]


def _bt_blocks(c, seed):
    """Energy-dependent block-tridiagonal matrix, diagonally dominant like
    the test fixtures' (uniform complex entries, diagonal = row sum + 1 + i),
    and anti-Hermitian lesser / greater self-energies on the same pattern."""
    g = _gen(seed)
    bs, ne = _sizes(c), c["energies"]
    uni = lambda *s: torch.rand(*s, dtype=C128, device="cuda", generator=g)  # noqa: E731
    vary = lambda x: x * (1.0 + 0.1 * torch.rand(ne, 1, 1, device="cuda", generator=g,  # noqa: E731
                                                 dtype=torch.float64))
    d = [vary(uni(ne, k, k)) for k in bs]
    u = [vary(uni(ne, bs[i], bs[i + 1])) for i in range(len(bs) - 1)]
    lo = [vary(uni(ne, bs[i + 1], bs[i])) for i in range(len(bs) - 1)]
    for i in range(len(bs)):
        rows = d[i].sum(-1)
        if i + 1 < len(bs):
            rows = rows + u[i].sum(-1)
        if i > 0:
            rows = rows + lo[i - 1].sum(-1)
        d[i] = d[i] + torch.diag_embed(rows + (1 + 1j))
    sig = []
    for coef in (1.0, 1j):
        sd = [coef * uni(ne, k, k) for k in bs]
        su = [coef * uni(ne, bs[i], bs[i + 1]) for i in range(len(bs) - 1)]
        sig.append(([x - _h(x) for x in sd], su, [-_h(x) for x in su]))
    return bs, (d, u, lo), sig[0], sig[1]


def _container(bs, blocks, like=None):
    """A DSDBCOO of dense blocks in block-sorted order."""
    d, u, lo = blocks
    if like is None:
        offs = np.concatenate(([0], np.cumsum(bs)))
        rows, cols = [], []
        for i in range(len(bs)):
            for j in (i - 1, i, i + 1):
                if 0 <= j < len(bs):
                    r, k = np.divmod(np.arange(bs[i] * bs[j]), bs[j])
                    rows.append(r + offs[i])
                    cols.append(k + offs[j])
        nnz = sum(r.size for r in rows)
        data = torch.zeros((d[0].shape[0], nnz), dtype=C128, device="cuda")
        m = DSDBCOO(data, np.concatenate(rows), np.concatenate(cols), bs)
    else:
        m = DSDBCOO.zeros_like(like)
    pos = 0
    for i in range(len(bs)):
        for blk in ([lo[i - 1]] if i > 0 else []) + [d[i]] + ([u[i]] if i + 1 < len(bs) else []):
            k = blk.shape[-1] * blk.shape[-2]
            m.data[:, pos:pos + k] = blk.reshape(blk.shape[0], k)
            pos += k
    return m


def _contact_obc(bs, ne, seed):
    """Boundary self-energies at both ends (retarded, lesser, greater)."""
    g = _gen(seed + 99)
    out = []
    for k in (bs[0], bs[-1]):
        s = _rand(g, ne, k, k, scale=0.1)
        gam = 1j * (s - _h(s))
        f = torch.rand(ne, 1, 1, device="cuda", generator=g, dtype=torch.float64)
        out.append((s, 1j * f * gam, 1j * (f - 1.0) * gam))
    return out


def _screened(c, seed):
    """Coulomb matrix and polarizations of a screened-interaction step: V
    Hermitian with weak coupling, P^< = i X and P^> = -i Y with X, Y positive
    semidefinite; the end blocks repeat the lead cells."""
    g = _gen(seed)
    n, b, ne = c["n"], c["b"], c["energies"]
    s2 = math.sqrt(0.5)
    cplx = lambda *s: _rand(g, *s) * s2 * math.sqrt(2.0)  # noqa: E731
    uni = lambda: float(torch.rand(1, device="cuda", generator=g, dtype=torch.float64))  # noqa: E731
    mix = lambda i, x: x if i <= 1 or i >= n - 2 else x * (1.0 + 0.3 * uni())  # noqa: E731
    q, _ = torch.linalg.qr(cplx(b, b))
    ev = 0.2 + 0.8 * torch.rand(b, device="cuda", generator=g, dtype=torch.float64)
    v00 = 0.5 * (q * ev) @ _h(q)
    v01 = (0.4 / math.sqrt(b)) * cplx(b, b)
    vu = [mix(i, v01) for i in range(n - 1)]
    v = ([v00.clone() for _ in range(n)], vu, [_h(x).contiguous() for x in vu])
    herm = 0.5 * (cplx(ne, b, b) + _h(cplx(ne, b, b)))
    sc = 2.0 / math.sqrt(b)
    pd = [mix(i, 0.04 * sc * (herm + _h(herm))) for i in range(n)]
    pu = 0.01 * sc * cplx(ne, b, b)
    pus = [mix(i, pu) for i in range(n - 1)]
    prh = (pd, pus, [_h(x).contiguous() for x in pus])
    pol = []
    for sign in (1.0, -1.0):
        q0, q1 = cplx(ne, b, b) * 0.1 * sc, cplx(ne, b, b) * 0.05 * sc
        qd = [mix(i, q0) for i in range(n)]
        qs = [mix(i, q1) for i in range(n)]
        xd = [1j * sign * (qd[i] @ _h(qd[i]) + qs[i] @ _h(qs[i])) for i in range(n)]
        xl = [1j * sign * (qs[i + 1] @ _h(qd[i])) for i in range(n - 1)]
        pol.append((xd, [-_h(x) for x in xl], xl))
    cont = lambda t: tuple([x.contiguous() for x in lst] for lst in t)  # noqa: E731
    return v, cont(pol[0]), cont(pol[1]), cont(prh)


def prepare(case, seed):
    kind, ne = case["kind"], case["energies"]
    st = {"kind": kind}
    if kind in ("point", "replay"):
        h, t, e, fl, fr = _device(case, seed)
        st["solver"] = EnergyPointSolver(h, t, eta=_eta(case), precision=case["precision"])
        st["args"] = (e, fl, fr)
        if kind == "replay":  # a serving lane captures its graph once
            st["solver"].set_inputs(e, fl, fr)
            st["solver"].capture(ne)
    elif kind in ("solve", "inv"):
        bs, a, sl, sg = _bt_blocks(case, seed)
        st["a"] = _container(bs, a)
        st["rgf"] = RGF(max_batch_size=100, precision=case["precision"])
        st["obc"] = OBCBlocks(len(bs))
        ends = _contact_obc(bs, ne, seed)
        for k, (r, lo, gr) in zip((0, -1), ends):
            st["obc"].retarded[k], st["obc"].lesser[k], st["obc"].greater[k] = r, lo, gr
        st["out"] = [DSDBCOO.zeros_like(st["a"]) for _ in range(1 if kind == "inv" else 3)]
        if kind == "solve":
            st["sl"], st["sg"] = (_container(bs, s, like=st["a"]) for s in (sl, sg))
    elif kind == "obc":
        st["system"], st["occ"] = _lead(case, seed)
        st["obc"] = OBCSystem(SanchoRubio(max_iterations=100, convergence_tol=1e-12), memoization_mode="off")
    else:
        v, pl, pg, prh = _screened(case, seed)
        st["w"] = CoulombScreeningSolve(v, 3, np.linspace(0.05, 1.0, ne), filtering_iteration_limit=0)
        st["args"] = (pl, pg, prh)
    return st


def _eta(case):
    """Broadening: at 1e-3 two correct decimations agree to about 1e-8, at
    1e-4 only to the instability of the recursion itself (up to 4e-6)."""
    return 1e-3


def _lead(case, seed):
    """One contact's lead blocks of A(E) over the grid, with occupations."""
    h, t, e, fl, _ = _device(case, seed)
    ne, b = case["energies"], case["b"]
    z = torch.as_tensor(e, device="cuda").to(C128) + 1j * _eta(case)
    a_ii = z[:, None, None] * torch.eye(b, dtype=C128, device="cuda") - h[0]
    a_ij = (-t).expand(ne, b, b).contiguous()
    a_ji = (-_h(t)).expand(ne, b, b).contiguous()
    return (a_ii, a_ij, a_ji), torch.as_tensor(fl, device="cuda")


def _point_outputs(r):
    b = r.blocks
    return {"transmission": r.transmission, "density": r.density, "current": r.current,
            "sigma_left": r.sigma_left, "sigma_right": r.sigma_right,
            **{k: b[k] for k in ("xl_diag", "xl_upper", "xl_lower", "xg_diag", "xg_upper", "xg_lower",
                                 "xr_diag")}}


def run(st):
    kind = st["kind"]
    if kind == "point":
        return _point_outputs(st["solver"].solve(*st["args"]))
    if kind == "replay":
        return _point_outputs(st["solver"].solve_graph(*st["args"]))
    if kind == "solve":
        cur = st["rgf"].selected_solve(st["a"], st["sl"], st["sg"], obc_blocks=st["obc"], out=st["out"],
                                       return_retarded=True, return_current=True)
        return {"current": cur, "lesser": st["out"][0].data, "greater": st["out"][1].data,
                "retarded": st["out"][2].data}
    if kind == "inv":
        st["rgf"].selected_inv(st["a"], obc_blocks=st["obc"], out=st["out"][0])
        return st["out"][0].data
    if kind == "obc":
        x, _, _ = st["obc"](st["system"], contact="left")
        a_ii, a_ij, a_ji = st["system"]
        return (x, *contact_self_energy(a_ij, a_ji, x, st["occ"]))
    return st["w"].solve(*st["args"])


# ---------------------------------------------------------------------------
# What the work cannot do without
# ---------------------------------------------------------------------------
def work(case):
    n, ne = case["n"], case["energies"]
    kind = case["kind"]
    prod = lambda m, k, j: 8.0 * m * k * j  # noqa: E731
    bs = _sizes(case)
    sq = sum(k * k for k in bs)
    off = sum(bs[i] * bs[i + 1] for i in range(n - 1))
    if kind == "inv":
        # one inverse and six products per layer; A in, X out
        fl = 8.0 * sum(k ** 3 for k in bs) + 6 * sum(prod(bs[i], bs[i + 1], max(bs[i], bs[i + 1]))
                                                    for i in range(n - 1))
        return {"bytes": 16.0 * ne * 2 * (sq + 2 * off), "flops": ne * fl}
    if kind == "obc":
        b = case["b"]
        return {"bytes": 16.0 * ne * b * b * 7, "flops": ne * 8.0 * b ** 3 * (7 * SR_STEPS + 6)}
    if kind == "w":
        b = case["b"]
        s, ns = 3 * b, n // 3
        fl = (9 + 48) * n * 8.0 * b ** 3 + 8.0 * s ** 3 * (ns + 4 + 24 * (ns - 1))
        fl += 2 * 8.0 * s ** 3 * (7 * SR_STEPS + 50)
        return {"bytes": 16.0 * ne * (9 * (3 * n - 2) * b * b / 3 + 2 * (3 * ns - 2) * s * s), "flops": ne * fl}
    # selected solve: an inverse and about 31 products per layer
    fl = 8.0 * sum(k ** 3 for k in bs) + 31 * sum(prod(bs[i], bs[i + 1], max(bs[i], bs[i + 1]))
                                                 for i in range(n - 1))
    if kind == "solve":
        # A, Sigma^< and Sigma^> (diagonal, upper) in; X^<, X^> and diag X^R out
        return {"bytes": 16.0 * ne * (sq + 2 * off + 2 * (sq + off) + 2 * (sq + 2 * off) + sq), "flops": ne * fl}
    b = case["b"]
    fl += 2 * 8.0 * b ** 3 * (7 * SR_STEPS + 6)
    elem = 8.0 if case["precision"] == "mixed" else 16.0
    return {"bytes": elem * ne * (3 * n + 4 * (n - 1)) * b * b + 16.0 * (n + 2) * b * b, "flops": ne * fl}


def tolerance(case):
    kind, precision = case["kind"], case["precision"]
    if precision == "mixed":
        # complex64 blocks through a chain of inverses (measured: 4e-3 in the
        # off-diagonal blocks of a point, 2.3e-5 in the current of a solve)
        return {"rel": 1.5e-2, "max": 0.5} if kind == "point" else {"rel": 1e-4, "max": 1e-2}
    if kind in ("point", "replay", "obc"):
        # the decimation amplifies rounding by an amount that depends on the
        # energy (measured against exact: 4e-11 to 8e-9, heavy-tailed)
        return {"rel": 5e-7, "max": 5e-5}
    if precision == "emulated":
        return {"rel": 1e-9, "max": 1e-7}
    return {"rel": 1e-12, "max": 1e-10}  # measured 4e-16 to 2e-14


# ---------------------------------------------------------------------------
# The same results in plain torch, 64 bits
# ---------------------------------------------------------------------------
def _anti(x):
    return 0.5 * (x - _h(x))


def _rgf(d, u, lo, sl, sg, cur=None):
    """Selected blocks by the recursive Green's function: d, u, lo with the
    boundary self-energies subtracted, sl / sg = (diag, upper) with theirs
    added. cur: (lesser, greater) boundary blocks per end for the current."""
    n = len(d)
    gr, gx, st = [torch.linalg.inv(d[0])], [[], []], [[None], [None]]
    for x, s in enumerate((sl, sg)):
        gx[x].append(gr[0] @ s[0][0] @ _h(gr[0]))
    for j in range(1, n):
        i = j - 1
        p = lo[i] @ gr[i]
        gr.append(torch.linalg.inv(d[j] - p @ u[i]))
        for x, s in enumerate((sl, sg)):
            q = p @ s[1][i]
            t = lo[i] @ gx[x][i] @ _h(lo[i]) + _h(q) - q
            st[x].append(t)
            gx[x].append(gr[j] @ (s[0][j] + t) @ _h(gr[j]))
    xr, xd, xu = [None] * n, [[None] * n, [None] * n], [[None] * (n - 1), [None] * (n - 1)]
    current = torch.zeros((d[0].shape[0], n + 1), dtype=C128, device=d[0].device)
    xr[-1] = gr[-1]
    g0n = gr[-1]
    for x in range(2):
        xd[x][-1] = gx[x][-1]
    for i in range(n - 2, -1, -1):
        j = i + 1
        a, v = gr[i] @ u[i], xr[j] @ lo[i]
        for x, s in enumerate((sl, sg)):
            r1 = gr[i] @ s[1][i] @ _h(xr[j])
            t1 = a @ v @ gx[x][i] - r1 @ _h(a)
            t2 = a @ xd[x][j]
            xu[x][i] = -t2 - gx[x][i] @ _h(v) + r1
            xd[x][i] = gx[x][i] + t2 @ _h(a) + t1 - _h(t1)
        if cur is not None:
            current[:, j] = ((st[1][j] * xd[0][j].transpose(-2, -1)).sum((-2, -1))
                             - (xd[1][j] * st[0][j].transpose(-2, -1)).sum((-2, -1)))
        g0n = -a @ g0n
        xr[i] = gr[i] + a @ v @ gr[i]
    if cur is not None:
        tr = lambda p, q: (p * q.transpose(-2, -1)).sum((-2, -1))  # noqa: E731
        (l0, g0), (ln, gn) = cur
        current[:, 0] = tr(g0, xd[0][0]) - tr(xd[1][0], l0)
        current[:, n] = -(tr(gn, xd[0][-1]) - tr(xd[1][-1], ln))
    return xr, [[_anti(y) for y in xd[x]] for x in range(2)], xu, current, g0n, (gr, u, lo)


def _surface(a_ii, a_ij, a_ji):
    """Sancho-Rubio decimation to 1e-12 and one fixed-point step."""
    eps, eps_s, al, be = a_ii.clone(), a_ii.clone(), a_ji.clone(), a_ij.clone()
    for _ in range(100):
        g = torch.linalg.inv(eps)
        ag, bg = al @ g, be @ g
        t = ag @ be
        eps_s = eps_s - t
        eps = eps - t - bg @ al
        al, be = ag @ al, bg @ be
        if float((0.5 * torch.linalg.matrix_norm(al.abs() + be.abs())).max()) < 1e-12:
            break
    x = torch.linalg.inv(eps_s)
    return torch.linalg.inv(a_ii - a_ji @ x @ a_ij)


def _contact(a_ii, a_ij, a_ji, occ):
    x = _surface(a_ii, a_ij, a_ji)
    s = a_ji @ x @ a_ij
    gam = 1j * (s - _h(s))
    f = occ[:, None, None]
    return x, s, 1j * f * gam, 1j * (f - 1.0) * gam


def _exact_point(case, seed):
    h, t, e, fl, fr = _device(case, seed)
    n, b, ne = case["n"], case["b"], case["energies"]
    z = torch.as_tensor(e, device="cuda").to(C128) + 1j * _eta(case)
    d = [z[:, None, None] * torch.eye(b, dtype=C128, device="cuda") - h[i] for i in range(n)]
    up, dn = (-t).expand(ne, b, b), (-_h(t)).expand(ne, b, b)
    occ = [torch.as_tensor(x, device="cuda") for x in (fl, fr)]
    left, right = _contact(d[0], up, dn, occ[0])[1:], _contact(d[-1], dn, up, occ[1])[1:]
    zero = torch.zeros((ne, b, b), dtype=C128, device="cuda")
    s = []
    for k in (1, 2):
        sd = [zero] * n
        sd[0], sd[-1] = left[k], right[k]
        s.append((sd, [zero] * (n - 1)))
    d[0], d[-1] = d[0] - left[0], d[-1] - right[0]
    xr, xd, xu, cur, g0n, _ = _rgf(d, [up] * (n - 1), [dn] * (n - 1), s[0], s[1],
                                   (left[1:], right[1:]))
    gam = [1j * (x[0] - _h(x[0])) for x in (left, right)]
    tr = ((gam[0] @ g0n @ gam[1]) * g0n.conj()).sum((-2, -1)).real
    low = [[-_h(y) for y in xu[x]] for x in range(2)]
    st = torch.stack
    dens = torch.cat([torch.diagonal(y, dim1=-2, dim2=-1).imag for y in xd[0]], dim=-1)
    return {"transmission": tr, "density": dens, "current": cur, "sigma_left": left[0], "sigma_right": right[0],
            "xl_diag": st(xd[0]), "xl_upper": st(xu[0]), "xl_lower": st(low[0]), "xg_diag": st(xd[1]),
            "xg_upper": st(xu[1]), "xg_lower": st(low[1]), "xr_diag": st(xr)}


def _exact_solve(case, seed):
    bs, (d, u, lo), sl, sg = _bt_blocks(case, seed)
    n, ne = len(bs), case["energies"]
    ends = _contact_obc(bs, ne, seed)
    sl, sg = [list(x) for x in sl], [list(x) for x in sg]
    for k, (r, le, gr) in zip((0, -1), ends):
        d[k] = d[k] - r
        if case["kind"] == "solve":
            sl[0][k], sg[0][k] = sl[0][k] + le, sg[0][k] + gr
    xr, xd, xu, cur, _, (gr, _, _) = _rgf(d, u, lo, sl, sg, (ends[0][1:], ends[1][1:]))
    if case["kind"] == "inv":
        # off-diagonal blocks of X^R from the left-connected functions
        lower = [-xr[i + 1] @ lo[i] @ gr[i] for i in range(n - 1)]
        upper = [-gr[i] @ u[i] @ xr[i + 1] for i in range(n - 1)]
        return _packed(bs, (xr, upper, lower))
    z = lambda m: [torch.zeros_like(x) for x in m]  # noqa: E731
    return {"current": cur, "lesser": _packed(bs, (xd[0], xu[0], [-_h(x) for x in xu[0]])),
            "greater": _packed(bs, (xd[1], xu[1], [-_h(x) for x in xu[1]])),
            "retarded": _packed(bs, (xr, z(u), z(lo)))}


def _packed(bs, blocks):
    d, u, lo = blocks
    parts = []
    for i in range(len(bs)):
        parts += ([lo[i - 1]] if i > 0 else []) + [d[i]] + ([u[i]] if i + 1 < len(bs) else [])
    return torch.cat([p.reshape(p.shape[0], -1) for p in parts], dim=1)


def _dense(m, b):
    """Dense (E, n b, n b) of block lists (diag, upper, lower) of size b."""
    d, u, lo = m
    n = len(d)
    x = d[0].reshape(-1, b, b)
    out = torch.zeros((x.shape[0], n * b, n * b), dtype=C128, device="cuda")
    for i in range(n):
        out[:, i * b:(i + 1) * b, i * b:(i + 1) * b] = d[i]
        if i + 1 < n:
            out[:, i * b:(i + 1) * b, (i + 1) * b:(i + 2) * b] = u[i]
            out[:, (i + 1) * b:(i + 2) * b, i * b:(i + 1) * b] = lo[i]
    return out


def _exact_w(case, seed):
    v, pl, pg, prh = _screened(case, seed)
    n, b, ne = case["n"], case["b"], case["energies"]
    s, ns = 3 * b, n // 3
    pr = tuple([x + 0.5 * (g - q) for x, g, q in zip(prh[t], pg[t], pl[t])] for t in range(3))
    vd, prd = _dense(v, b), _dense(pr, b)
    m = torch.eye(n * b, dtype=C128, device="cuda") - vd @ prd
    m[:, :b, :b] -= v[2][0] @ pr[1][0]
    m[:, -b:, -b:] -= v[1][-1] @ pr[2][-1]
    flip = lambda x: torch.flip(x, (-2, -1))  # noqa: E731
    cut = lambda x, i, j: x[:, i * s:(i + 1) * s, j * s:(j + 1) * s]  # noqa: E731
    ls = []
    for p in (pl, pg):
        x = vd @ _dense(p, b) @ vd
        for (v10, v00, v01, p10, p00, p01, i, j) in (
                (v[2][0], v[0][0], v[1][0], p[2][0], p[0][0], p[1][0], 0, 1),
                (v[1][-1], v[0][-1], v[2][-1], p[1][-1], p[0][-1], p[2][-1], n - 1, n - 2)):
            ii, jj = slice(i * b, (i + 1) * b), slice(j * b, (j + 1) * b)
            x[:, ii, ii] += v10 @ p01 @ v00 + v00 @ p10 @ v01 + v10 @ p00 @ v01
            x[:, ii, jj] += v10 @ p01 @ v01
            x[:, jj, ii] += v10 @ p10 @ v01
        ls.append(x)

    def expand(ji, ii, ij):
        lead = ii.shape[:-2]
        o = [torch.zeros(lead + (s, s), dtype=C128, device="cuda") for _ in range(3)]
        for r in range(3):
            o[1][..., r * b:(r + 1) * b, r * b:(r + 1) * b] = ii
            if r < 2:
                o[1][..., r * b:(r + 1) * b, (r + 1) * b:(r + 2) * b] = ij
                o[1][..., (r + 1) * b:(r + 2) * b, r * b:(r + 1) * b] = ji
        o[2][..., -b:, :b] = ij
        o[0][..., :b, -b:] = ji
        return o

    ends = []
    for right in (False, True):
        tri = ((lambda x: expand(flip(x[1][-1]), flip(x[0][-1]), flip(x[2][-1]))) if right
               else (lambda x: expand(x[2][0], x[0][0], x[1][0])))
        (p10, p00, p01), (v10, v00, v01) = tri(pr), tri(v)
        m00 = torch.eye(s, dtype=C128, device="cuda") - v10 @ p01 - v00 @ p00 - v01 @ p10
        m01, m10 = -v00 @ p01 - v01 @ p00, -v10 @ p00 - v00 @ p10
        x = _surface(m00, m01, m10)
        res = [m10 @ x @ m01]
        aa = x @ m10
        for p in (pl, pg):
            q10, q00, q01 = tri(p)
            s1, s2 = q00 @ v01 + q01 @ v00, q10 @ v01 + q00 @ v00
            l00 = v10 @ s1 + v00 @ (s2 + q01 @ v10) + v01 @ (q10 @ v00 + q00 @ v10)
            l01 = v10 @ q01 @ v01 + v00 @ s1 + v01 @ s2
            a00 = m10 @ x @ l01
            an = a00 - _h(a00)
            q = x @ (l00 - an) @ _h(x)
            w, ai = q, aa
            for _ in range(12):
                w, ai = w + ai @ w @ _h(ai), ai @ ai
            w = q + aa @ w @ _h(aa)
            res.append(m10 @ w @ _h(m10) - an)
        ends.append([flip(y) for y in res] if right else res)
    d = [cut(m, i, i).clone() for i in range(ns)]
    sx = [([cut(x, i, i).clone() for i in range(ns)], [cut(x, i, i + 1) for i in range(ns - 1)]) for x in ls]
    for k, e in zip((0, -1), ends):
        d[k] -= e[0]
        sx[0][0][k] += e[1]
        sx[1][0][k] += e[2]
    _, xd, xu, _, _, _ = _rgf(d, [cut(m, i, i + 1) for i in range(ns - 1)],
                              [cut(m, i + 1, i) for i in range(ns - 1)], sx[0], sx[1])
    out = []
    for x in range(2):
        w = (xd[x], [y.clone() for y in xu[x]], [-_h(y) for y in xu[x]])
        for lst in w:
            for y in lst:
                y[0] = 0.0
        out.append(w)
    return out[0], out[1]


def exact(case, seed):
    kind = case["kind"]
    if kind in ("point", "replay"):
        return _exact_point(case, seed)
    if kind in ("solve", "inv"):
        return _exact_solve(case, seed)
    if kind == "obc":
        (a_ii, a_ij, a_ji), occ = _lead(case, seed)
        return _contact(a_ii, a_ij, a_ji, occ)
    return _exact_w(case, seed)
