"""The calls that the fully-coupled step is used for, as cases that can be
timed and compared: time-marching and steady steps of the built-in flows in
every storage precision, the exchange of a host code that owns the fields, a
bare residual, and the discrete adjoint.

A case is a dict of plain values; `prepare` builds its mesh, context and
seeded initial state, `run` makes one pass through rhodst_b200.Solver.
"""
from __future__ import annotations

import functools

import numpy as np

from rhodst_b200 import Solver, cases

# what `run` does with the context of each kind of case
#   march     n_steps steps, then the fields back (a run between two outputs)
#   restart   primitive fields in, n_steps steps, primitive fields out (one
#             point of a sweep, each from given fields)
#   exchange  fields in, one step, fields out (a host code that owns them)
#   residual  R(W) of the current state
#   adjoint   the adjoint solve of the pressure force on the case's patch
#   products  (dR/dW)^T v and (dR/dW) v


def listed():
    return [
        # a monitor or an outer solver asking for R(W) on the small channel
        {"name": "residual_step2d", "kind": "residual", "flow": "step2d", "refine": 1},
        # the forwardStep run: unsteady, global time step, block Jacobi
        {"name": "march_step2d", "kind": "march", "flow": "step2d", "refine": 1, "flux": "Kurganov",
         "limiter": "OSPRE", "n_steps": 10},
        # the same run on a four times finer grid
        {"name": "march_step2d_fine", "kind": "march", "flow": "step2d", "refine": 4, "flux": "Kurganov",
         "limiter": "OSPRE", "n_steps": 4},
        # laminar airfoil, Sutherland viscosity, a grid of odd size
        {"name": "march_airfoil_laminar", "kind": "march", "flow": "laminar", "ni": 131, "nj": 35,
         "precision": "fp64", "n_steps": 4},
        # steady turbulent airfoil, negative Spalart-Allmaras, GMRES(30) + ILU(0)
        {"name": "march_airfoil_sa", "kind": "march", "flow": "turbulent", "ni": 257, "nj": 65, "model": "SAneg",
         "precision": "fp64", "n_steps": 2},
        # the RAE2822 tutorial: BiCGStab to a tolerance, Kurganov, Spalart-Allmaras
        {"name": "restart_rae2822", "kind": "restart", "flow": "rae2822", "model": "SpalartAllmaras", "n_steps": 6},
        # a host solver that owns the fields, mid-size wing, FP32 Jacobian
        {"name": "exchange_wing_fp32", "kind": "exchange", "flow": "wing", "na": 98, "nn": 33, "ns": 23, "nt": 11,
         "precision": "fp32"},
        # steady inviscid wing in full precision
        {"name": "march_wing_fp64", "kind": "march", "flow": "wing", "na": 128, "nn": 48, "ns": 48, "nt": 24,
         "precision": "fp64", "n_steps": 2},
        # the benchmark's wing: 1.2 M cells, FP32 Jacobian and ILU
        {"name": "march_wing_fp32", "kind": "march", "flow": "wing", "na": 192, "nn": 64, "ns": 64, "nt": 34,
         "precision": "fp32", "n_steps": 2},
        # BF16 storage on a wing grid of uneven sizes
        {"name": "march_wing_bf16", "kind": "march", "flow": "wing", "na": 130, "nn": 51, "ns": 37, "nt": 19,
         "precision": "bf16", "n_steps": 2},
        # unstructured prisms and tetrahedra, Venkatakrishnan limiter
        {"name": "march_hybrid_fp32", "kind": "march", "flow": "hybrid", "nx": 120, "ny": 40, "nz": 28,
         "precision": "fp32", "n_steps": 2},
        # force gradient: transposed products and the transposed GMRES
        {"name": "adjoint_wing_fp64", "kind": "adjoint", "flow": "wing", "na": 96, "nn": 32, "ns": 24, "nt": 12,
         "precision": "fp64", "directions": 4},
    ]


def _log(rng, lo, hi):
    return lo * (hi / lo) ** rng.random()


def _wing_sizes(rng, n_lo, n_hi):
    """Grid sizes of a wing of about n cells, in the default's proportions
    with some scatter."""
    k = (_log(rng, n_lo, n_hi) / 1.2e6) ** (1.0 / 3.0)
    r = [k * rng.uniform(0.85, 1.12) for _ in range(4)]
    return {"na": 2 * max(16, round(96 * r[0])), "nn": max(10, round(64 * r[1])), "ns": max(8, round(64 * r[2])),
            "nt": max(5, round(34 * r[3]))}


def draw(rng):
    kind = rng.choice(["residual", "step2d", "step2d", "laminar", "turbulent", "rae2822", "exchange", "wing", "wing",
                       "hybrid", "adjoint", "products"])
    if kind == "residual":
        return {"kind": "residual", "flow": "step2d", "refine": rng.randint(1, 6)}
    if kind == "step2d":
        return {"kind": "march", "flow": "step2d", "refine": rng.randint(1, 6),
                "flux": rng.choice(["Kurganov", "HLL", "AUSM+"]),
                "limiter": rng.choice(["OSPRE", "vanLeer", "Minmod", "vanAlbada"]), "n_steps": rng.randint(1, 10)}
    if kind == "laminar":
        return {"kind": "march", "flow": "laminar", "ni": rng.randint(97, 260), "nj": rng.randint(25, 66),
                "precision": rng.choice(["fp64", "fp64", "fp32"]), "n_steps": rng.randint(1, 5)}
    if kind == "turbulent":
        return {"kind": "march", "flow": "turbulent", "ni": rng.randint(129, 321), "nj": rng.randint(40, 81),
                "model": rng.choice(["SAneg", "SARC2", "SpalartAllmaras"]),
                "precision": rng.choice(["fp64", "fp64", "fp32"]), "n_steps": rng.randint(1, 3)}
    if kind == "rae2822":
        return {"kind": "restart", "flow": "rae2822", "model": rng.choice(["SpalartAllmaras", "SAneg"]),
                "n_steps": rng.randint(1, 8)}
    if kind == "hybrid":
        k = _log(rng, 0.25, 1.0)
        return {"kind": "march", "flow": "hybrid", "nx": round(150 * k), "ny": round(50 * k * rng.uniform(0.9, 1.1)),
                "nz": max(6, round(32 * k * rng.uniform(0.8, 1.1))), "precision": rng.choice(["fp64", "fp32", "fp32"]),
                "n_steps": rng.randint(1, 2)}
    if kind == "exchange":
        return dict({"kind": "exchange", "flow": "wing", "precision": rng.choice(["fp64", "fp32"])},
                    **_wing_sizes(rng, 2e4, 5e5))
    if kind == "adjoint":
        return dict({"kind": "adjoint", "flow": "wing", "precision": "fp64", "directions": rng.randint(2, 4)},
                    **_wing_sizes(rng, 2e4, 1.2e5))
    if kind == "products":
        return dict({"kind": "products", "flow": "wing", "precision": "fp64"}, **_wing_sizes(rng, 2e4, 4e5))
    return dict({"kind": "march", "flow": "wing", "precision": rng.choice(["fp64", "fp32", "bf16"]), "n_steps": 1},
                **_wing_sizes(rng, 3e4, 7e5))


@functools.lru_cache(maxsize=4)
def _flow(flow, sizes):
    """Mesh, boundary conditions and dictionary entries of a flow: what a
    program loads once from its case directory."""
    c = dict(sizes)
    if flow == "step2d":
        return cases.forward_step_c1(c["refine"])
    if flow == "laminar":
        return cases.naca0012_laminar(c["ni"], c["nj"], sutherland=True)
    if flow == "turbulent":
        return cases.naca0012_turbulent(c["ni"], c["nj"], model=c["model"])
    if flow == "rae2822":
        return cases.rae2822(model=c["model"])
    if flow == "wing":
        return cases.swept_wing_c3(c["na"], c["nn"], c["ns"], c["nt"])
    return cases.forward_step_3d_hybrid_c5(c["nx"], c["ny"], c["nz"])


_SIZES = ("refine", "ni", "nj", "model", "na", "nn", "ns", "nt", "nx", "ny", "nz")


def _case(case):
    c = _flow(case["flow"], tuple((k, case[k]) for k in _SIZES if k in case))
    opts = {}
    if "precision" in case:
        opts["precision"] = case["precision"]
    if "flux" in case:
        opts["fluxScheme"] = case["flux"]
    if "limiter" in case:
        opts["interpolationSchemes"] = {"reconstruct(rho)": case["limiter"], "reconstruct(U)": case["limiter"] + "V",
                                        "reconstruct(T)": case["limiter"]}
    return c.with_options(**opts)


def _state(case, c, seed):
    """Free stream with smooth disturbances of a few per cent, as the flow
    of a previous run or an interpolated start has them."""
    rng = np.random.default_rng(seed)
    x = c.mesh.C - c.mesh.C.min(axis=0)
    x = x / max(float(x.max()), 1e-300)

    def wave(amp):
        out = np.zeros(c.mesh.n_cells)
        for _ in range(4):
            out += rng.uniform(0.3, 1.0) * np.sin(x @ rng.uniform(-40.0, 40.0, 3) + rng.uniform(0.0, 6.28))
        return amp * out / 2.0

    p, T = c.p * (1.0 + wave(0.02)), c.T * (1.0 + wave(0.02))
    U = c.U * (1.0 + wave(0.03))[:, None]
    nut = None if c.nuTilda is None else c.nuTilda * (1.0 + wave(0.05))
    return p, U, T, nut, rng


def prepare(case, seed):
    c = _case(case)
    s = Solver(c.mesh, c.bcs, c.options)
    p, U, T, nut, rng = _state(case, c, seed)
    s.set_primitive(p, U, T, nut)
    state = {"case": case, "solver": s, "patch": c.force_patch}
    if case["kind"] == "restart":
        state["fields"] = p, U, T, nut
    if case["kind"] == "exchange":
        state["fields"] = s.conservative()
    if case["kind"] == "adjoint":
        state["direction"] = c.force_dirs["drag"]
    if case["kind"] == "products":
        state["v"] = rng.standard_normal((c.mesh.n_cells, 5))
    return state


def run(state):
    case, s = state["case"], state["solver"]
    kind = case["kind"]
    if kind == "residual":
        return s.residual()
    if kind == "march":
        reps = s.step(case["n_steps"])
        rho, rhoU, rhoE = s.conservative()
        return {"rho": rho, "rhoU": rhoU, "rhoE": rhoE, "res_l2": np.array([r["res_l2"] for r in reps])}
    if kind == "restart":
        s.set_primitive(*state["fields"])
        reps = s.step(case["n_steps"])
        p, U, T, nut = s.primitive()
        return {"p": p, "U": U, "T": T, "nuTilda": nut, "res_l2": np.array([r["res_l2"] for r in reps])}
    if kind == "exchange":
        s.set_conservative(*state["fields"])
        reps = s.step(1)
        state["fields"] = s.conservative()
        rho, rhoU, rhoE = state["fields"]
        return {"rho": rho, "rhoU": rhoU, "rhoE": rhoE, "res_l2": np.array([r["res_l2"] for r in reps])}
    if kind == "products":
        u, dU = s.adjoint_product(state["v"])
        return {"JTv": u, "JTv_dU": dU, "Jv": s.tangent_product(state["v"])}
    rep, psi = s.adjoint(state["patch"], state["direction"], p_ref=1.0, rel_tol=1e-12, max_cycles=1,
                         n_directions=case["directions"], want_psi=True)
    return {"psi": psi, "J": np.array([rep["J"]]), "dJ_dU": rep["dJ_dU"]}


def _sizes(case):
    """(cells, internal faces) from the grid sizes."""
    f = case["flow"]
    if f == "step2d":
        n = 4032 * case["refine"] ** 2
        return n, 2 * n
    if f in ("laminar", "turbulent"):
        n = case["ni"] * case["nj"]
        return n, 2 * n
    if f == "rae2822":
        return 23552, 46704
    if f == "wing":
        n = case["na"] * case["nn"] * (case["ns"] + case["nt"])
        return n, 3 * n
    n = int(case["nx"] * case["ny"] * case["nz"] * 3.7)
    return n, int(2.07 * n)


def work(case):
    """Compulsory traffic and arithmetic of one pass.  A residual reads each
    cell's state and each face's geometry and writes R.  A step adds the
    matrix (N + 2F blocks of 25 entries) written once and read by every
    product of the Krylov cycle, the preconditioner's blocks read by every
    application, and two passes over the basis per direction."""
    N, F = _sizes(case)
    S = {"fp64": 8, "fp32": 4, "bf16": 2}[case.get("precision", "fp64")]
    vb = 8 if S == 8 else 4
    res_b, res_f = 40.0 * N + 72.0 * F + 40.0 * N, 600.0 * F
    if case["kind"] == "residual":
        return {"bytes": res_b, "flops": res_f}
    if case["kind"] == "products":
        return {"bytes": 2 * (res_b + 40.0 * N), "flops": 8 * res_f}
    Bk = N + 2 * F
    jacobi = case["flow"] == "step2d"
    mat = 25.0 * S * Bk
    prec = 25.0 * S * N if jacobi else mat
    m = {"turbulent": 30}.get(case["flow"], 20)
    if case["flow"] == "rae2822":       # BiCGStab, about ten iterations of two products and two applications
        step_b = res_b + mat + prec + 10 * (2 * mat + 2 * prec + 12 * 40.0 * N)
        step_f = res_f + 10 * 4 * 50.0 * Bk
    else:
        orth = 2 * 5.0 * vb * N * m * (m + 1) / 2.0
        step_b = res_b + 2 * mat + 2 * prec + (m + 2) * mat + (m + 1) * prec + orth
        step_f = res_f + (2 * m + 3) * 50.0 * Bk + 4 * 5.0 * N * m * (m + 1)
    if case["kind"] == "adjoint":
        return {"bytes": case["directions"] * (step_b + res_b), "flops": case["directions"] * (step_f + 4 * res_f)}
    n = case.get("n_steps", 1)
    return {"bytes": n * step_b + 80.0 * N, "flops": n * step_f}


def exact(case, seed):
    """The bare residual in plain numpy: Kurganov fluxes of the OSPRE /
    OSPREV-limited states, Gauss gradients, per unit volume.  The other
    kinds return what a truncated Krylov solve leaves, which has no value of
    its own to compare with."""
    if case["kind"] != "residual":
        return None
    c = _case(case)
    m, th = c.mesh, c.options["thermo"]
    p, U, T, _, _ = _state(case, c, seed)
    R, Cp = th["R"], th["Cp"]
    g = Cp / (Cp - R)
    N, Fi = m.n_cells, m.n_internal_faces
    o, n = np.asarray(m.owner)[:Fi], np.asarray(m.neighbour)[:Fi]

    def record(p, U, T):        # rho, rhoU, RT, e, c
        rho = p / (R * T)
        return np.column_stack([rho, rho[:, None] * U, R * T, Cp * T - p / rho, np.sqrt(g * R * T)])

    q = record(p, U, T)
    # boundary values of the patches that are not empty
    ids, pb, Ub, Tb = [], [], [], []
    for P in m.patches:
        if P.type == 3:
            continue
        f = np.arange(P.start, P.start + P.size)
        oc = np.asarray(m.owner)[f]
        spec = c.bcs[P.name]
        S = m.Sf[f]
        nrm = S / m.magSf[f][:, None]
        out = (q[oc, 1:4] * S).sum(1) >= 0.0

        def value(sp, inner):
            if isinstance(sp, str):
                if sp in ("symmetryPlane", "slip") and inner.ndim == 2:
                    return inner - (nrm * inner).sum(1)[:, None] * nrm
                return inner
            ref = np.broadcast_to(np.asarray(sp[1], dtype=float), inner.shape)
            if sp[0] == "inletOutlet":
                return np.where(out if inner.ndim == 1 else out[:, None], inner, ref)
            return ref
        ids.append(f)
        pb.append(value(spec["p"], p[oc]))
        Ub.append(value(spec["U"], U[oc]))
        Tb.append(value(spec["T"], T[oc]))
    fb = np.concatenate(ids)
    ob = np.asarray(m.owner)[fb]
    qb = record(np.concatenate(pb), np.concatenate(Ub), np.concatenate(Tb))
    S, Sb = m.Sf[:Fi], m.Sf[fb]
    w = np.asarray(m.weights)[:Fi, None]
    V = np.asarray(m.V)
    grad = np.zeros((N, 7, 3))
    t = (w * q[o] + (1 - w) * q[n])[:, :, None] * S[:, None, :]
    np.add.at(grad, o, t)
    np.add.at(grad, n, -t)
    np.add.at(grad, ob, qb[:, :, None] * Sb[:, None, :])
    grad /= V[:, None, None]
    d = m.C[n] - m.C[o]

    def sides(xP, xN, r_o, r_n):
        def lim(r):
            rr = r * (r + 1.0)
            return np.maximum(1.5 * rr / (rr + 1.0), 0.0)
        wo = lim(r_o) * w[:, 0] + (1.0 - lim(r_o))
        wn = lim(r_n) * w[:, 0]
        if xP.ndim == 2:
            wo, wn = wo[:, None], wn[:, None]
        return wo * xP + (1 - wo) * xN, wn * xP + (1 - wn) * xN

    def ratio(gc, gf):
        big = np.abs(gc) >= 1000 * np.abs(gf)
        sg = np.where(gc >= 0, 1.0, -1.0) * np.where(gf >= 0, 1.0, -1.0)
        return np.where(big, 2000 * sg - 1, 2 * (gc / np.where(big, 1.0, gf)) - 1)

    so, sn = np.empty((Fi, 7)), np.empty((Fi, 7))
    for j in (0, 4, 5, 6):
        gf = q[n, j] - q[o, j]
        so[:, j], sn[:, j] = sides(q[o, j], q[n, j], ratio((d * grad[o, j]).sum(1), gf),
                                   ratio((d * grad[n, j]).sum(1), gf))
    gv = q[n, 1:4] - q[o, 1:4]
    gf = (gv * gv).sum(1)
    so[:, 1:4], sn[:, 1:4] = sides(q[o, 1:4], q[n, 1:4],
                                   ratio((gv * np.einsum("fk,fjk->fj", d, grad[o, 1:4])).sum(1), gf),
                                   ratio((gv * np.einsum("fk,fjk->fj", d, grad[n, 1:4])).sum(1), gf))

    def kurganov(a, b, S):
        mag = np.sqrt((S * S).sum(1))
        Ua, Ubb = a[:, 1:4] / a[:, :1], b[:, 1:4] / b[:, :1]
        Ea = a[:, 0] * (a[:, 5] + 0.5 * (Ua * Ua).sum(1))
        Eb = b[:, 0] * (b[:, 5] + 0.5 * (Ubb * Ubb).sum(1))
        pa, pbb = a[:, 0] * a[:, 4], b[:, 0] * b[:, 4]
        va, vb = (Ua * S).sum(1), (Ubb * S).sum(1)
        ap = np.maximum(np.maximum(va + a[:, 6] * mag, vb + b[:, 6] * mag), 0.0)
        am = np.minimum(np.minimum(va - a[:, 6] * mag, vb - b[:, 6] * mag), 0.0)
        aa = ap / (ap - am)
        aS = am * aa
        fa, fb2 = va * aa - aS, vb * (1 - aa) + aS
        mom = fa[:, None] * a[:, 1:4] + fb2[:, None] * b[:, 1:4] + (aa * pa + (1 - aa) * pbb)[:, None] * S
        return np.column_stack([fa * a[:, 0] + fb2 * b[:, 0], mom, fa * (Ea + pa) + fb2 * (Eb + pbb) + aS * (pa - pbb)])

    out = np.zeros((N, 5))
    fl = kurganov(so, sn, S)
    np.add.at(out, o, fl)
    np.add.at(out, n, -fl)
    np.add.at(out, ob, kurganov(qb, qb, Sb))
    return out / V[:, None]
