"""Performance cases of the RGF path: what a user of the library has it do.

Each case goes through a public entry point (``TransportSolver.solve``,
``solve_grouped``, ``RGF.selected_solve`` / ``selected_inv``, ``SanchoRubio``,
``obc.inverse``) on seeded tight-binding devices of
``quatrex_b200.workloads``.  ``exact`` restates each result in plain torch
complex128: dense inverses of the whole matrix instead of the recursion.
"""

from __future__ import annotations

import math

import numpy as np
import torch

from quatrex_b200.datastructures import DSDBCOO
from quatrex_b200.greens_function_solver import RGF, OBCBlocks
from quatrex_b200.obc import SanchoRubio, inverse
from quatrex_b200.transport import TransportSolver, solve_grouped
from quatrex_b200.workloads import make_device

MU_L, MU_R, KT = 0.1, -0.1, 0.025
# Broadening of the devices.  At the generator's default 1e-6 the decimation of the leads meets, at one
# energy in a few hundred, a block so nearly singular that the surface function moves by up to 1e-5 with
# the rounding alone (8e-7 over 148 energies of b = 256, against 3e-9 at 1e-4), and no error could be
# told from that.
ETA = 1e-4
SR_TOL, SR_MAX = 1e-12, 200

OBSERVABLES = ("density", "hole_density", "transmission", "current_left", "current_right", "dos", "layer_current")
DIAGONALS = ("gr_diag", "gl_diag", "gg_diag")
OFF_DIAGONALS = ("gr_upper", "gr_lower", "gl_upper", "gg_upper")
KEYS = {"observables": OBSERVABLES, "diagonals": OBSERVABLES + DIAGONALS,
        "all": OBSERVABLES + DIAGONALS + OFF_DIAGONALS}


def listed():
    return [
        # the smallest call: invert the contact blocks of a few energies
        dict(name="inverse_8x32", kind="inverse", b=32, ne=8),
        # surface Green's function of one lead over a short energy grid (an SCBA iteration's contact)
        dict(name="sancho_rubio_40x64", kind="sancho", b=64, ne=40),
        # G^R alone over unequal transport cells (odd block sizes), stacked as (energy, k-point)
        dict(name="selected_inv_ragged", kind="selinv", sizes="48,112,80,33,96,57,128,40", ne=14),
        # the plugin call of a ballistic device: the only sources are the contacts
        dict(name="solve_ballistic_16x64", kind="solve", nb=16, b=64, ne=32, batch=100, scatter=False, host=False),
        # the plugin call inside an SCBA loop: every self-energy block filled, layer currents asked for
        dict(name="solve_scattering_12x100", kind="solve", nb=12, b=100, ne=24, batch=100, scatter=True, host=False),
        # the plugin call at the large block size, cut into small energy batches by the memory
        dict(name="solve_ballistic_16x256", kind="solve", nb=16, b=256, ne=32, batch=16, scatter=False, host=False),
        # the plugin call on NumPy operands: the stack is streamed through the device
        dict(name="solve_host_16x64", kind="solve", nb=16, b=64, ne=32, batch=32, scatter=False, host=True),
        # generator form, the CPU-runnable configuration, every output
        dict(name="transport_16x64", kind="transport", nb=16, b=64, ne=32, keys="all", precision="fp64"),
        # generator form at the headline block size: one energy per SM, diagonal blocks and observables
        dict(name="transport_16x256", kind="transport", nb=16, b=256, ne=148, keys="diagonals", precision="fp64"),
        # the largest block size of the uneven batch, observables only
        dict(name="transport_8x512", kind="transport", nb=8, b=512, ne=24, keys="observables", precision="fp64"),
        # the precision form the caller can ask for
        dict(name="transport_mixed_12x256", kind="transport", nb=12, b=256, ne=64, keys="observables",
             precision="mixed"),
        # several small devices of one block size solved together (batching and serving)
        dict(name="grouped_6x64", kind="grouped", count=6, b=64, nb_lo=8, nb_hi=40, ne_lo=64, ne_hi=160),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One case of the same kinds and ranges; sizes log-uniform, odd ones among them."""
    most = max(work(c)["flops"] for c in listed())
    kind = rng.choice(["inverse", "sancho", "selinv", "ballistic", "scattering", "host", "transport", "transport",
                       "mixed", "grouped"])
    while True:
        b = _log_int(rng, 24, 512)
        if kind == "inverse":
            case = dict(kind="inverse", b=b, ne=_log_int(rng, 4, 200))
        elif kind == "sancho":
            case = dict(kind="sancho", b=min(b, 256), ne=_log_int(rng, 8, 150))
        elif kind == "selinv":
            sizes = ",".join(str(_log_int(rng, 24, 160)) for _ in range(rng.randint(4, 10)))
            case = dict(kind="selinv", sizes=sizes, ne=2 * _log_int(rng, 2, 30))
        elif kind in ("ballistic", "scattering", "host"):
            b = _log_int(rng, 24, 128 if kind != "ballistic" else 256)
            case = dict(kind="solve", nb=rng.randint(4, 16), b=b, ne=_log_int(rng, 8, 64),
                        batch=rng.choice([16, 32, 100]), scatter=kind == "scattering", host=kind == "host")
        elif kind == "transport":
            case = dict(kind="transport", nb=rng.randint(4, 24), b=_log_int(rng, 32, 512), ne=_log_int(rng, 8, 160),
                        keys=rng.choice(sorted(KEYS)), precision="fp64")
        elif kind == "mixed":
            case = dict(kind="transport", nb=rng.randint(4, 12), b=rng.choice([128, 256, 512]),
                        ne=_log_int(rng, 16, 96), keys="observables", precision="mixed")
        else:
            case = dict(kind="grouped", count=rng.randint(1, 8), b=rng.randint(16, 64), nb_lo=8, nb_hi=40,
                        ne_lo=32, ne_hi=160)
        w = work(case)
        if w["flops"] <= most and w["bytes"] <= 8e9:
            return case


# ---- inputs -----------------------------------------------------------------
def _dev(x):
    return torch.from_numpy(np.ascontiguousarray(x)).cuda()


def _instances(case):
    """(num_blocks, energies) of each device of a grouped case (fixed by the case)."""
    rng = np.random.default_rng(case["count"] * 1000 + case["b"])
    return [(int(rng.integers(case["nb_lo"], case["nb_hi"] + 1)), int(rng.integers(case["ne_lo"], case["ne_hi"] + 1)))
            for _ in range(case["count"])]


def _fermi(e, mu):
    return 1.0 / (1.0 + torch.exp((e - mu) / KT))


def _surface(a_ii, a_ij, a_ji):
    """Sancho-Rubio decimation in plain torch (stops when the whole batch has converged)."""
    eps, eps_s = a_ii.clone(), a_ii.clone()
    alpha, beta = a_ji.expand_as(a_ii), a_ij.expand_as(a_ii)
    for _ in range(SR_MAX):
        inv = torch.linalg.inv(eps)
        ai, bi = alpha @ inv, beta @ inv
        aib = ai @ beta
        eps_s = eps_s - aib
        eps = eps - aib - bi @ alpha
        alpha, beta = ai @ alpha, bi @ beta
        if float((torch.linalg.norm(alpha.abs() + beta.abs(), dim=(-2, -1)) / 2).max()) < SR_TOL:
            break
    return torch.linalg.inv(eps_s)


def _contacts(h_diag, h_upper, e):
    """(Sigma^R, f) of the left and right contact: the leads repeat the end cells."""
    eye = torch.eye(h_diag.shape[-1], dtype=torch.complex128, device=e.device)
    z = (e + 1j * ETA)[:, None, None] * eye
    up, lo = -h_upper, -h_upper.mH
    g_l = _surface(z - h_diag[0], up[0], lo[0])
    g_r = _surface(z - h_diag[-1], lo[-1], up[-1])
    return ((lo[0] @ g_l @ up[0], _fermi(e, MU_L)), (up[-1] @ g_r @ lo[-1], _fermi(e, MU_R)))


def _lead(case, seed):
    dev = make_device(2, case["b"], case["ne"], seed=seed, eta=ETA)
    d, u, lo = dev.system_blocks()
    return _dev(d[0]), _dev(u[0][0]), _dev(lo[0][0])


def _ragged(case, seed):
    """Blocks of A over unequal cells: H as the generator's, broadened like a device under contacts."""
    sizes = [int(s) for s in case["sizes"].split(",")]
    g = torch.Generator().manual_seed(seed)

    def cn(*shape):
        return torch.complex(torch.randn(shape, generator=g, dtype=torch.float64),
                             torch.randn(shape, generator=g, dtype=torch.float64)) / math.sqrt(2.0)

    e = torch.linspace(-2, 2, case["ne"], dtype=torch.float64)
    diag, upper, lower = [], [], []
    for i, b in enumerate(sizes):
        x = cn(b, b)
        h = (x + x.mH) / (2 * math.sqrt(b)) - 0.05j * torch.eye(b, dtype=torch.complex128)
        diag.append((e[:, None, None] * torch.eye(b, dtype=torch.complex128) - h).cuda())
        if i + 1 < len(sizes):
            t = cn(b, sizes[i + 1]) / (2 * math.sqrt(max(b, sizes[i + 1])))
            upper.append((-t).expand(len(e), -1, -1).cuda())
            lower.append((-t.mH).expand(len(e), -1, -1).cuda())
    return sizes, diag, upper, lower


def _system(case, seed):
    """Operands of the plugin call: A, Sigma^<, Sigma^> as block lists and the contact blocks."""
    nb, b, ne = case["nb"], case["b"], case["ne"]
    dev = make_device(nb, b, ne, seed=seed, eta=ETA)
    hd, hu, e = _dev(dev.h_diag), _dev(dev.h_upper), _dev(dev.energies)
    left, right = _contacts(hd, hu, e)
    eye = torch.eye(b, dtype=torch.complex128, device="cuda")
    z = (e + 1j * ETA)[:, None, None] * eye
    d = [z - hd[i] for i in range(nb)]
    u = [(-hu[i]).expand(ne, b, b) for i in range(nb - 1)]
    lo = [(-hu[i].mH).expand(ne, b, b) for i in range(nb - 1)]
    zero = torch.zeros(ne, b, b, dtype=torch.complex128, device="cuda")
    sl, sg = ([zero] * nb, [zero] * (nb - 1), [zero] * (nb - 1)), ([zero] * nb, [zero] * (nb - 1), [zero] * (nb - 1))
    if case["scatter"]:
        # self-energies of a scattering device: i n and i (n - 1) times a positive broadening, with
        # off-diagonal blocks; Sigma^R = (Sigma^> - Sigma^<) / 2 goes into A
        g = torch.Generator(device="cuda").manual_seed(seed)
        f = _fermi(e, 0.0)[:, None, None]

        def cn(count):
            return torch.randn(count, b, b, generator=g, dtype=torch.complex128, device="cuda")

        m, t = cn(nb), cn(nb - 1)
        gam = 0.1 * (m @ m.mH) / b
        off = 0.02 * t / math.sqrt(b)
        parts = []
        for occ in (f, f - 1.0):
            dd = [1j * occ * gam[i] for i in range(nb)]
            uu = [1j * occ * off[i] for i in range(nb - 1)]
            parts.append((dd, uu, [-x.mH for x in uu]))
        sl, sg = parts
        d = [x - 0.5 * (gg - ll) for x, gg, ll in zip(d, sg[0], sl[0])]
        u = [x - 0.5 * (gg - ll) for x, gg, ll in zip(u, sg[1], sl[1])]
        lo = [x - 0.5 * (gg - ll) for x, gg, ll in zip(lo, sg[2], sl[2])]
    obc = []
    for sig, occ in (left, right):
        gamma = 1j * (sig - sig.mH)
        occ = occ[:, None, None]
        obc.append((sig, 1j * occ * gamma, 1j * (occ - 1.0) * gamma))
    return (d, u, lo), sl, sg, obc


def prepare(case, seed):
    kind = case["kind"]
    if kind == "inverse":
        return dict(case=case, a=_lead(case, seed)[0])
    if kind == "sancho":
        return dict(case=case, blocks=_lead(case, seed), solver=SanchoRubio(SR_MAX, SR_TOL))
    if kind == "selinv":
        _, d, u, lo = _ragged(case, seed)
        shape = (case["ne"] // 2, 2)
        stack = [[x.reshape(shape + tuple(x.shape[1:])) for x in part] for part in (d, u, lo)]
        a = DSDBCOO.from_blocks(*stack)
        return dict(case=case, a=a, out=DSDBCOO.zeros_like(a), solver=RGF())
    if kind == "solve":
        a, sl, sg, obc = _system(case, seed)
        mats = [DSDBCOO.from_blocks(*m) for m in (a, sl, sg)]
        blocks = OBCBlocks(case["nb"])
        for at, (r, l_, g) in ((0, obc[0]), (-1, obc[1])):
            for lst, x in ((blocks.retarded, r), (blocks.lesser, l_), (blocks.greater, g)):
                lst[at] = x.cpu().numpy() if case["host"] else x.contiguous()
        if case["host"]:
            mats = [DSDBCOO(m.data.cpu().numpy(), m.rows, m.cols, m.block_sizes, m.stack_shape) for m in mats]
        return dict(case=case, mats=mats, obc=blocks, out=[DSDBCOO.zeros_like(mats[0]) for _ in range(3)],
                    solver=RGF(max_batch_size=case["batch"]))
    if kind == "transport":
        dev = make_device(case["nb"], case["b"], case["ne"], seed=seed, eta=ETA)
        solver = TransportSolver(dev, max_batch_size=case["ne"], precision=case["precision"])
        return dict(case=case, solver=solver, energies=_dev(dev.energies))
    devices, energies, hams = [], [], []
    for q, (nb, ne) in enumerate(_instances(case)):
        d = make_device(nb, case["b"], ne, seed=seed + q, eta=ETA)
        devices.append(d)
        energies.append(_dev(d.energies))
        hams.append((_dev(d.h_diag), _dev(d.h_upper)))
    return dict(case=case, devices=devices, energies=energies, hams=hams)


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "inverse":
        return inverse(state["a"])
    if kind == "sancho":
        return state["solver"](*state["blocks"], contact="left")
    if kind == "selinv":
        state["solver"].selected_inv(state["a"], out=state["out"])
        return state["out"].data
    if kind == "solve":
        a, sl, sg = state["mats"]
        current = state["solver"].selected_solve(a, sl, sg, obc_blocks=state["obc"], out=state["out"],
                                                 return_retarded=True, return_current=case["scatter"])
        got = {"lesser": state["out"][0].data, "greater": state["out"][1].data, "retarded": state["out"][2].data}
        if case["scatter"]:
            got["current"] = current
        return got
    if kind == "transport":
        return state["solver"].solve(state["energies"], keys=KEYS[case["keys"]])
    return solve_grouped(state["devices"], state["energies"], keys=OBSERVABLES, hamiltonians=state["hams"])


# ---- the same results in plain torch ------------------------------------------
def _dense(d, u, lo, e):
    """The whole matrix at one energy from block lists with an energy axis."""
    offs = np.concatenate(([0], np.cumsum([x.shape[-1] for x in d])))
    m = torch.zeros(int(offs[-1]), int(offs[-1]), dtype=torch.complex128, device="cuda")
    for i, x in enumerate(d):
        m[offs[i]:offs[i + 1], offs[i]:offs[i + 1]] = x[e]
    for i, (x, y) in enumerate(zip(u, lo)):
        m[offs[i]:offs[i + 1], offs[i + 1]:offs[i + 2]] = x[e]
        m[offs[i + 1]:offs[i + 2], offs[i]:offs[i + 1]] = y[e]
    return m, offs


def _row(m, offs, off_diagonals=True):
    """The block-tridiagonal part in the storage order of a data row."""
    nb, parts = len(offs) - 1, []
    for i in range(nb):
        for j in range(max(0, i - 1), min(nb, i + 2)):
            blk = m[offs[i]:offs[i + 1], offs[j]:offs[j + 1]]
            parts.append((blk if i == j or off_diagonals else torch.zeros_like(blk)).reshape(-1))
    return torch.cat(parts)


def _exact_solve(case, seed):
    a, sl, sg, obc = _system(case, seed)
    nb = case["nb"]
    d, sl_d, sg_d = list(a[0]), list(sl[0]), list(sg[0])
    for at, (r, l_, g) in ((0, obc[0]), (nb - 1, obc[1])):
        d[at], sl_d[at], sg_d[at] = d[at] - r, sl_d[at] + l_, sg_d[at] + g
    rows = {"lesser": [], "greater": [], "retarded": []}
    for e in range(case["ne"]):
        m, offs = _dense(d, a[1], a[2], e)
        g = torch.linalg.inv(m)
        rows["retarded"].append(_row(g, offs, off_diagonals=False))
        for key, (sd, s) in (("lesser", (sl_d, sl)), ("greater", (sg_d, sg))):
            rows[key].append(_row(g @ _dense(sd, s[1], s[2], e)[0] @ g.mH, offs))
    got = {k: torch.stack(v) for k, v in rows.items()}
    if case["host"]:
        got = {k: v.cpu().numpy() for k, v in got.items()}
    if case["scatter"]:
        # left-connected functions x_i, X_i and the self-energies they exert on the next block
        comps = [(sl_d, sl, []), (sg_d, sg, [])]
        x = torch.linalg.inv(d[0])
        left = [x @ c[0][0] @ x.mH for c in comps]
        for i in range(nb - 1):
            up, lo = a[1][i], a[2][i]
            for q, (sd, s, tilde) in enumerate(comps):
                w = lo @ x @ s[1][i]
                tilde.append(lo @ left[q] @ lo.mH + w.mH - w)
            x = torch.linalg.inv(d[i + 1] - lo @ x @ up)
            left = [x @ (c[2][i] + c[0][i + 1]) @ x.mH for c in comps]
        blk, b = [], case["b"]
        for key in ("lesser", "greater"):
            at, diag = 0, []
            for i in range(nb):
                at += b * b if i > 0 else 0
                diag.append(got[key][:, at:at + b * b].reshape(-1, b, b))
                at += b * b + (b * b if i + 1 < nb else 0)
            blk.append(diag)
        cur = [((comps[1][2][i] @ blk[0][i + 1]) - (blk[1][i + 1] @ comps[0][2][i])).diagonal(0, -2, -1).sum(-1)
               for i in range(nb - 1)]
        got["current"] = torch.stack(cur, dim=-1)
    return got


def _exact_transport(nb, b, ne, seed, keys):
    dev = make_device(nb, b, ne, seed=seed, eta=ETA)
    hd, hu, en = _dev(dev.h_diag), _dev(dev.h_upper), _dev(dev.energies)
    (sig_l, f_l), (sig_r, f_r) = _contacts(hd, hu, en)
    gam_l, gam_r = 1j * (sig_l - sig_l.mH), 1j * (sig_r - sig_r.mH)
    n = nb - 1
    out = {k: [] for k in keys}

    def trace(x, y):
        return (x * y.mT).sum()

    for e in range(ne):
        m = torch.zeros(nb * b, nb * b, dtype=torch.complex128, device="cuda")
        for i in range(nb):
            m[i * b:(i + 1) * b, i * b:(i + 1) * b] = -hd[i]
        for i in range(n):
            m[i * b:(i + 1) * b, (i + 1) * b:(i + 2) * b] = -hu[i]
            m[(i + 1) * b:(i + 2) * b, i * b:(i + 1) * b] = -hu[i].mH
        m.diagonal().add_(en[e] + 1j * ETA)
        m[:b, :b] -= sig_l[e]
        m[n * b:, n * b:] -= sig_r[e]
        g = torch.linalg.inv(m).reshape(nb, b, nb, b).transpose(1, 2)
        del m
        col_l, col_r = g[:, 0], g[:, n]
        x_l = [col_l[i] @ (1j * gam_l[e]) for i in range(nb)]
        x_r = [col_r[i] @ (1j * gam_r[e]) for i in range(nb)]
        occ = {"l": (f_l[e], f_r[e]), "g": (f_l[e] - 1.0, f_r[e] - 1.0)}

        def keldysh(c, i, j):
            return occ[c][0] * (x_l[i] @ col_l[j].mH) + occ[c][1] * (x_r[i] @ col_r[j].mH)

        gl = torch.stack([keldysh("l", i, i) for i in range(nb)])
        gg = torch.stack([keldysh("g", i, i) for i in range(nb)])
        up = torch.stack([keldysh("l", i, i + 1) for i in range(n)])
        gd = torch.stack([g[i, i] for i in range(nb)])
        si_l, si_r = 1j * gam_l[e], 1j * gam_r[e]
        one = {
            "gr_diag": gd, "gl_diag": gl, "gg_diag": gg,
            "dos": -gd.diagonal(0, -2, -1).imag.mean(-1),
            "density": gl.diagonal(0, -2, -1).imag.sum(-1),
            "hole_density": -gg.diagonal(0, -2, -1).imag.sum(-1),
            "transmission": trace(gam_l[e] @ g[0, n] @ gam_r[e], g[0, n].mH).real,
            "current_left": trace((f_l[e] - 1.0) * si_l, gl[0]) - trace(gg[0], f_l[e] * si_l),
            "current_right": trace((f_r[e] - 1.0) * si_r, gl[n]) - trace(gg[n], f_r[e] * si_r),
            "layer_current": torch.stack([(-hu[i] * up[i].conj() - up[i] * hu[i].conj()).sum() for i in range(n)]),
        }
        if "gg_upper" in out:
            one["gl_upper"] = up
            one["gg_upper"] = torch.stack([keldysh("g", i, i + 1) for i in range(n)])
            one["gr_upper"] = torch.stack([g[i, i + 1] for i in range(n)])
            one["gr_lower"] = torch.stack([g[i + 1, i] for i in range(n)])
        for k in keys:
            out[k].append(one[k])
    return {k: torch.stack(v) for k, v in out.items()}


def exact(case, seed):
    kind = case["kind"]
    if kind == "inverse":
        return torch.linalg.inv(_lead(case, seed)[0])
    if kind == "sancho":
        return _surface(*_lead(case, seed))
    if kind == "selinv":
        _, d, u, lo = _ragged(case, seed)
        rows = []
        for e in range(case["ne"]):
            m, offs = _dense(d, u, lo, e)
            rows.append(_row(torch.linalg.inv(m), offs))
        return torch.stack(rows).reshape(case["ne"] // 2, 2, -1)
    if kind == "solve":
        return _exact_solve(case, seed)
    if kind == "transport":
        return _exact_transport(case["nb"], case["b"], case["ne"], seed, KEYS[case["keys"]])
    return [_exact_transport(nb, case["b"], ne, seed + q, OBSERVABLES) for q, (nb, ne) in enumerate(_instances(case))]


# ---- work and tolerance ---------------------------------------------------------
def work(case):
    """Bytes of inputs and outputs once; flops in block products of 8 b^3 (an inverse counts as one)."""
    kind = case["kind"]
    if kind in ("inverse", "sancho"):
        b, ne = case["b"], case["ne"]
        # about 16 decimation steps (7 block operations each) at eta = 1e-4, and the final inverse
        units = 1 if kind == "inverse" else 113
        return {"bytes": 32.0 * b * b * ne, "flops": 8.0 * units * b**3 * ne}
    if kind == "selinv":
        sizes = [int(s) for s in case["sizes"].split(",")]
        pairs = list(zip(sizes, sizes[1:]))
        nnz = sum(s * s for s in sizes) + 2 * sum(x * y for x, y in pairs)
        flops = sum(s**3 for s in sizes) + sum(4 * x * x * y + 3 * x * y * y for x, y in pairs)
        return {"bytes": 32.0 * nnz * case["ne"], "flops": 8.0 * flops * case["ne"]}
    if kind == "solve":
        nb, b, ne = case["nb"], case["b"], case["ne"]
        units = (32 if case["scatter"] else 21) * (nb - 1) + 5
        blocks = (5 * (3 * nb - 2) if case["scatter"] else 3 * (3 * nb - 2)) + nb + 6
        return {"bytes": 16.0 * b * b * blocks * ne, "flops": 8.0 * units * b**3 * ne}
    jobs = [(case["nb"], case["ne"])] if kind == "transport" else _instances(case)
    keys = KEYS[case.get("keys", "observables")]
    b, bytes_, flops = case["b"], 0.0, 0.0
    for nb, ne in jobs:
        units = 18 * (nb - 1) + 11 + 2 * 113 + (2 * (nb - 1) if "gr_upper" in keys else 0)
        blocks = nb * sum(k in DIAGONALS for k in keys) + (nb - 1) * sum(k in OFF_DIAGONALS for k in keys)
        bytes_ += 16.0 * b * b * (2 * nb - 1 + ne * blocks) + 8.0 * ne * (6 * nb)
        flops += 8.0 * units * b**3 * ne
    return {"bytes": bytes_, "flops": flops}


def tolerance(case):
    """About four times the largest relative error the path shows against ``exact`` over several seeds and
    drawn sizes (in brackets).

    Everything is complex128, so the errors are the conditioning of the inputs: the decimation of the leads
    passes through nearly singular blocks at some energies, and a ballistic device is nearly singular at its
    levels; single entries at such an energy are further off than the norm of the whole batch."""
    kind = case["kind"]
    if kind == "inverse":
        return {"rel": 1e-11, "max": 5e-9}  # (1.3e-12, 4e-10)
    if kind == "sancho":
        return {"rel": 2e-8, "max": 2e-6}  # (3e-9 over 148 energies of b = 256)
    if kind == "selinv" or (kind == "solve" and case["scatter"]):
        return {"rel": 1e-13, "max": 5e-12}  # (1.2e-14, 4.3e-13)
    if kind == "solve":
        return {"rel": 2e-11, "max": 2e-9}  # (5e-12, 4e-10)
    return {"rel": 5e-8, "max": 5e-6}  # (1.1e-8, 4e-7)
