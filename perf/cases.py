"""The workloads this framework is timed on: its public entry points over the
sizes that its configurations, tests and benchmark use.

Every case is a dict of plain values with a "kind":

* maps       A x and A^T y of a problem (V2RDMProblem.Au / ATu)
* maps_grad  torch.ops.v2rdm.Au with its backward (A x, then A^T w)
* project    PSD projections from scratch (V2RDMProblem.project)
* warm       two successive warm projections, as a host solver's iterations
* solve      boundary-point iterations from the random guess, host arrays
* resume     boundary-point iterations from a checkpoint, then the density
             packing that the orbital step reads
* batch      independent Hubbard rings in one launch (BatchProblem)
* orbital    orbital energy and gradient with density-fitted integrals
"""
import math

import numpy as np
import torch

import hilbert_b200 as hb
import hilbert_b200.torch_ops  # noqa: F401  registers torch.ops.v2rdm
from hilbert_b200 import orbital
from hilbert_b200.synthetic import df_hamiltonian

CG_STEPS = 30   # CG iterations per outer iteration that work() counts


def listed():
    return [
        # the smallest calls: one A x and one A^T y of a small ring, latency and launches only
        dict(name="maps_n6", kind="maps", n=6, na=3, nb=3, pos="DQG"),
        # the same pair at the headline (20e,20o) active space
        dict(name="maps_n20", kind="maps", n=20, na=10, nb=10, pos="DQG"),
        # the differentiable operator with three-index conditions, open shell, odd size
        dict(name="maps_grad_t2_n9", kind="maps_grad", n=9, na=5, nb=4, pos="DQGT2"),
        # one stand-alone projection, odd size: blocks of 11 to 242 rows
        dict(name="project_n11", kind="project", n=11, na=6, nb=6, pos="DQG"),
        # the projections of two neighbouring iterations of a host solver, blocks up to 800 rows
        dict(name="warm_n20", kind="warm", n=20, na=10, nb=10, pos="DQG", step=1e-4),
        # the smallest solve: a half-filled Hubbard ring, latency-bound iterations
        dict(name="solve_ring6", kind="solve", ham="ring", n=6, na=3, nb=3, pos="DQG", outer=60),
        # an ordinary active space, open shell, odd size
        dict(name="solve_df9", kind="solve", ham="df", n=9, na=5, nb=4, pos="DQG", outer=40),
        # three-index conditions: blocks of 306 rows beside many small ones
        dict(name="solve_t2_n6", kind="solve", ham="df", n=6, na=3, nb=3, pos="DQGT2", outer=12),
        # seniority-zero program: thousands of variables, hundreds of tiny blocks
        dict(name="solve_doci10", kind="solve", ham="doci", n=10, na=5, nb=5, pos="DQG", outer=60),
        # the headline active space in the middle of its solve, as after a checkpoint or an orbital step
        dict(name="resume_df20", kind="resume", ham="df", n=20, na=10, nb=10, pos="DQG", before=120, outer=30),
        # many independent rings of uneven size in one launch
        dict(name="batch_rings", kind="batch", count=12, lmin=6, lmax=10, pos="DQG", outer=8),
        # the orbital step's energy and gradient: 40 orbitals, 160 auxiliary functions
        dict(name="orbital_n40", kind="orbital", n=40, naux=160, nact=10, ncore=5),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["maps", "maps", "maps_grad", "project", "warm", "solve", "solve", "solve", "resume",
                       "batch", "orbital"])

    def electrons(n):
        na = rng.randint(max(1, n // 2 - 1), n // 2 + 1)
        return dict(n=n, na=na, nb=max(1, na - rng.randint(0, 1)))

    if kind == "maps":
        if rng.random() < 0.7:
            return dict(kind=kind, **electrons(_log(rng, 4, 20)), pos=rng.choice(["DQG", "DQG", "DQ", "DG"]))
        return dict(kind=kind, **electrons(_log(rng, 4, 9)), pos=rng.choice(["DQGT2", "DQGT1T2", "DQG+D3"]))
    if kind == "maps_grad":
        return dict(kind=kind, **electrons(_log(rng, 4, 9)), pos=rng.choice(["DQGT2", "DQG", "DQGT1"]))
    if kind == "project":
        return dict(kind=kind, **electrons(_log(rng, 4, 13)), pos="DQG")
    if kind == "warm":
        return dict(kind=kind, **electrons(_log(rng, 6, 20)), pos="DQG", step=10.0 ** rng.uniform(-6.0, -3.5))
    if kind == "solve":
        ham = rng.choice(["ring", "df", "df", "doci", "t2"])
        if ham == "ring":
            n = _log(rng, 4, 10)
            half = max(1, n // 2 + rng.randint(-1, 0))
            return dict(kind=kind, ham=ham, n=n, na=half, nb=half, pos="DQG", outer=rng.randint(20, 60))
        if ham == "df":
            return dict(kind=kind, ham=ham, **electrons(_log(rng, 4, 11)), pos="DQG", outer=rng.randint(15, 40))
        if ham == "doci":
            n = rng.randint(6, 16)
            return dict(kind=kind, ham=ham, n=n, na=n // 2, nb=n // 2, pos="DQG", outer=rng.randint(20, 60))
        return dict(kind=kind, ham="df", **electrons(rng.randint(4, 6)), pos="DQGT2", outer=rng.randint(6, 12))
    if kind == "resume":
        return dict(kind=kind, ham="df", **electrons(_log(rng, 8, 16)), pos="DQG", before=rng.randint(80, 120),
                    outer=rng.randint(10, 30))
    if kind == "batch":
        return dict(kind=kind, count=rng.randint(3, 12), lmin=rng.randint(4, 6), lmax=rng.randint(7, 10), pos="DQG",
                    outer=rng.randint(4, 8))
    n = _log(rng, 16, 56)
    return dict(kind=kind, n=n, naux=rng.randint(2 * n, 4 * n), nact=rng.randint(4, min(12, n - 4)),
                ncore=rng.randint(0, 4))


def _problem(case):
    if case.get("ham") == "doci":
        return hb.DOCIProblem(case["n"], case["na"], case["nb"], case["pos"])
    return hb.V2RDMProblem(case["n"], case["na"], case["nb"], case["pos"], True, True,
                           hubbard_multiplicity=case.get("ham") == "ring")


def _objective(case, p, seed):
    """c of the case's Hamiltonian, drawn from the seed"""
    if case["ham"] == "ring":
        return p.c_hubbard(1.0, float(np.random.default_rng(seed).uniform(1.0, 8.0)))
    n = case["n"]
    return p.c_external(*df_hamiltonian(n, 20 * n, seed_b=seed, seed_h=seed + 1))


def _options(outer):
    # the benchmark's thresholds; MAXITER bounds the pass
    return hb.Options({"R_CONVERGENCE": 1e-6, "E_CONVERGENCE": 1e-6, "CG_CONVERGENCE": 1e-9, "MAXITER": outer,
                       "MU_UPDATE_FREQUENCY": 500})


def _normal(seed, *shape):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return torch.randn(*shape, dtype=torch.float64, device="cuda", generator=g)


def _blocks(dims, seed):
    """A packed symmetric matrix per block with the spectrum that the iterations
    project: three tenths of the eigenvalues positive, pairs degenerate."""
    out = []
    for k, n in enumerate(int(d) for d in dims):
        if n == 0:
            continue
        q, _ = torch.linalg.qr(_normal(1000 * seed + 2 * k, n, n))
        w = 0.1 + _normal(1000 * seed + 2 * k + 1, n).abs()
        w[: n // 2 * 2 : 2] = w[1 : n // 2 * 2 : 2]   # spin multiplets
        sign = torch.full((n,), -1.0, dtype=torch.float64, device="cuda")
        sign[: max(1, (3 * n) // 10)] = 1.0
        u = (q * (w * sign)) @ q.T
        out.append((0.5 * (u + u.T)).reshape(-1))
    return torch.cat(out)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "maps":
        p = _problem(case)
        return dict(kind=kind, p=p, x=_normal(2 * seed, p.n_primal), y=_normal(2 * seed + 1, p.n_dual))
    if kind == "maps_grad":
        p = _problem(case)
        return dict(kind=kind, x=_normal(2 * seed, p.n_primal).requires_grad_(), w=_normal(2 * seed + 1, p.n_dual),
                    spec=(case["n"], case["na"], case["nb"], case["pos"], True, True, False))
    if kind == "project":
        p = _problem(case)
        return dict(kind=kind, p=p, U=_blocks(p.dims, seed))
    if kind == "warm":
        p = _problem(case)
        ua = _blocks(p.dims, seed)
        parts = []
        for k, n in enumerate(int(d) for d in p.dims):
            s = _normal(7000 * seed + k, n, n) / math.sqrt(max(n, 1))
            parts.append((0.5 * (s + s.T)).reshape(-1))
        ub = ua + case["step"] * torch.cat(parts)
        p.project(ub, 1.0, warm=True)
        return dict(kind=kind, p=p, ua=ua, ub=ub)
    if kind == "solve":
        p = _problem(case)
        return dict(kind=kind, p=p, x=p.guess("RANDOM"), b=p.b(), c=_objective(case, p, seed),
                    options=_options(case["outer"]))
    if kind == "resume":
        p = _problem(case)
        c = _objective(case, p, seed)
        x = torch.from_numpy(p.guess("RANDOM")).cuda()
        b, dc = torch.from_numpy(p.b()).cuda(), torch.from_numpy(c).cuda()
        p.solve_device(x, b, dc, _options(case["before"]))
        return dict(kind=kind, p=p, x=x, b=b, c=dc, mu=p.get_mu(), y=p.get_y(), z=p.get_z(),
                    options=_options(case["outer"]))
    if kind == "batch":
        rng = np.random.default_rng(seed)
        parts, cs = [], []
        # the sizes are the case's own, the same for every seed; U/t is drawn
        sizes = np.random.default_rng(case["count"]).integers(case["lmin"], case["lmax"] + 1, case["count"])
        for L in (int(v) for v in sizes):
            p = hb.V2RDMProblem(L, L // 2, L // 2, case["pos"], True, True, hubbard_multiplicity=True)
            parts.append(p)
            cs.append(p.c_hubbard(1.0, float(rng.uniform(1.0, 8.0))))
        batch = hb.BatchProblem(parts)
        return dict(kind=kind, p=batch, x=torch.from_numpy(np.concatenate([q.guess("RANDOM") for q in parts])).cuda(),
                    b=torch.from_numpy(np.concatenate([q.b() for q in parts])).cuda(),
                    c=torch.from_numpy(np.concatenate(cs)).cuda(), options=_options(case["outer"]))
    if kind == "orbital":
        n, naux, nact, ncore = case["n"], case["naux"], case["nact"], case["ncore"]
        B = 0.1 * _normal(9 * seed, naux, n, n)
        B = 0.5 * (B + B.transpose(1, 2))
        h = torch.diag(torch.linspace(-1.0, -10.0, n, dtype=torch.float64, device="cuda"))
        m = _normal(9 * seed + 1, n, n)
        h = h + 0.025 * (m + m.T)
        d = _normal(9 * seed + 2, nact, nact)
        D = d @ d.T / nact
        v = _normal(9 * seed + 3, nact, nact)
        v = 0.5 * (v + v.T)
        G = torch.einsum("tu,vw->tuvw", D, D) + 0.01 * torch.einsum("tu,vw->tuvw", v, v)
        D, G = orbital.full_densities(D, G, ncore, n - ncore - nact)
        k = 0.05 * _normal(9 * seed + 4, n, n)
        return dict(kind=kind, kappa=(k - k.T).requires_grad_(), h=h, B=B.contiguous(), D=D, G=G)
    raise ValueError(kind)


def run(state):
    kind = state["kind"]
    if kind == "maps":
        return {"Ax": state["p"].Au(state["x"]), "ATy": state["p"].ATu(state["y"])}
    if kind == "maps_grad":
        ax = torch.ops.v2rdm.Au(state["x"], *state["spec"])
        (gx,) = torch.autograd.grad(ax, state["x"], state["w"])
        return {"Ax": ax, "ATw": gx}
    if kind == "project":
        x, z = state["p"].project(state["U"], 0.5)
        return {"x": x, "z": z}
    if kind == "warm":
        xa, za = state["p"].project(state["ua"], 1.0, warm=True)
        xb, zb = state["p"].project(state["ub"], 1.0, warm=True)
        return {"xa": xa, "za": za, "xb": xb, "zb": zb}
    if kind == "solve":
        p = state["p"]
        x, st = p.solve(state["x"], state["b"], state["c"], state["options"])
        return {"x": x, "y": p.get_y(), "z": p.get_z(), "energy": st["energy"]}
    if kind == "resume":
        p = state["p"]
        p.set_state(state["mu"], state["y"], state["z"])
        x = state["x"].clone()
        st = p.solve_device(x, state["b"], state["c"], state["options"])
        d2, d1 = p.pack_spatial_density(x)
        return {"x": x, "d2": d2, "d1": d1, "energy": st["energy"]}
    if kind == "batch":
        x = state["x"].clone()
        st = state["p"].solve_device(x, state["b"], state["c"], state["options"])
        return {"x": x, "y": state["p"].get_y(), "energy": st["energy"]}
    E = orbital.rotated_energy(state["kappa"], state["h"], state["B"], state["D"], state["G"])
    (g,) = torch.autograd.grad(E, state["kappa"])
    return {"E": E.detach(), "dE": g}


def work(case):
    kind = case["kind"]
    if kind == "orbital":
        n, q = case["n"], case["naux"]
        # B, h, D, G and kappa in, E and the gradient out; B' and its adjoint: 2 + 4 products per factor, one with G
        return {"bytes": 8.0 * (q * n * n + n ** 4 + 4 * n * n), "flops": 2.0 * (q + 1) * 6 * n ** 3 + 2.0 * q * n ** 4}
    if kind == "batch":
        sizes = np.random.default_rng(case["count"]).integers(case["lmin"], case["lmax"] + 1, case["count"])
        parts = [hb.V2RDMProblem(int(L), int(L) // 2, int(L) // 2, case["pos"]) for L in sizes]
    else:
        parts = [_problem(case)]
    npri, ndual = sum(p.n_primal for p in parts), sum(p.n_dual for p in parts)
    cubes = sum(float(d) ** 3 for p in parts for d in p.dims)
    nnz = sum(p.operator_nnz()[0] for p in parts)
    if kind in ("maps", "maps_grad"):
        return {"bytes": 16.0 * (npri + ndual), "flops": 4.0 * nnz}
    if kind in ("project", "warm"):
        k = 1 if kind == "project" else 2
        return {"bytes": 24.0 * npri * k, "flops": 16.0 / 3.0 * cubes * k}
    # per CG iteration r, y, the direction and t; per outer iteration U, x, z, c and the norms
    outer = case["outer"]
    return {"bytes": 8.0 * outer * (CG_STEPS * (2 * npri + 7 * ndual) + 6 * npri + 4 * ndual),
            "flops": outer * (16.0 / 3.0 * cubes + CG_STEPS * 4.0 * nnz)}


def exact(case, seed):
    kind = case["kind"]
    if kind in ("project", "warm"):
        state = prepare(case, seed)
        dims = [int(d) for d in state["p"].dims]

        def split(u, mu):
            u = u.cpu().numpy()
            xs, zs, off = [], [], 0
            for n in dims:
                m = u[off:off + n * n].reshape(n, n)
                off += n * n
                m = 0.5 * (m + m.T)
                w, v = np.linalg.eigh(m)
                pos = (v * np.maximum(w, 0.0)) @ v.T
                xs.append((pos / mu).reshape(-1))
                zs.append((pos - m).reshape(-1))
            return np.concatenate(xs), np.concatenate(zs)

        if kind == "project":
            x, z = split(state["U"], 0.5)
            return {"x": x, "z": z}
        xa, za = split(state["ua"], 1.0)
        xb, zb = split(state["ub"], 1.0)
        return {"xa": xa, "za": za, "xb": xb, "zb": zb}
    if kind == "orbital":
        s = prepare(case, seed)
        n = case["n"]
        k = s["kappa"].detach().cpu().requires_grad_()
        h, B, D, G = (s[v].cpu() for v in ("h", "B", "D", "G"))
        U = torch.linalg.matrix_exp(k)
        b = (U.T @ B @ U).reshape(-1, n * n)
        E = ((U.T @ h @ U) * D).sum() + 0.5 * ((b @ G.reshape(n * n, n * n)) * b).sum()
        (g,) = torch.autograd.grad(E, k)
        return {"E": E.detach(), "dE": g}
    return None   # the constraint maps and the iterations built on them have no form outside this package
