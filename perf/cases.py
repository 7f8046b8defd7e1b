"""The work a user of this framework has it do, as cases that can be timed and compared.

A case is a dict of plain values: an operation on a mesh, and how the mesh is made.

  op       rhs        gh_rhs: prepare and one right-hand side, du of a state vector
           steps      step_batched: `steps` RK4 steps of one chunk of an evolution
           plain      rk4_step: the plain form, one step at a time, the only form of the :pasted interior
           monitors   what a driver asks for between chunks: the constraint monitors, their norms, the
                      diag field set, the masked error and the characteristic speed
           regrid     the refinement indicator, its firing sweeps and the state's transfer to the new forest
           tangent    one tangent-linear RK4 step
           adjoint    one reverse RK4 step
  physics  fourier (flat space and Fourier modes), wave (gauge wave), hole (Kerr-Schild at rest),
           moving (a boosted hole), fitted (harmonic Kerr with the :fitted target cache)
  N, roots, radii   blocks of N^3 cells, roots^3 of them at level 0, refined within the radii (comma separated)
  halfwidth, q, precision, variant

Every state is the physics' analytic state plus a few Fourier modes of small amplitude whose phases
and amplitudes come from the seed: smooth data that satisfy no equation exactly, as the data of a
run under way do. An evolution goes on from pass to pass, in place, its time with it.
"""
import importlib.util
import math
import sys
from pathlib import Path

import torch

AMPLITUDE = 1e-4  # of the modes, as the repository's Fourier workload has it
# adds, multiplies, divides and square roots of one right-hand-side point at q = 4, by gauge source
FLOP_RHS = {"fourier": 7909, "wave": 7909, "hole": 7957, "moving": 8283, "fitted": 7909}
FLOP_MONITORS = 2159 + 13890  # the gauge and the ADM constraints of one point


def package():
    if "tgh_b200" not in sys.modules:
        pkg = Path("treegeneralizedharmonic.jl_b200").resolve()
        spec = importlib.util.spec_from_file_location("tgh_b200", pkg / "__init__.py",
                                                      submodule_search_locations=[str(pkg)])
        mod = importlib.util.module_from_spec(spec)
        sys.modules["tgh_b200"] = mod
        spec.loader.exec_module(mod)
    return sys.modules["tgh_b200"]


def _case(name, op, physics, N, roots, q=4, **more):
    return {"name": name, "op": op, "physics": physics, "N": N, "roots": roots, "q": q, "precision": "fp64", **more}


def listed():
    return [
        # the smallest mesh of the tests: one right-hand side is launches and latency
        _case("rhs_fourier_n8", "rhs", "fourier", 8, 2),
        # high order, an odd block edge, 27 blocks: rows that fill no warp and meet no 16-byte boundary
        _case("rhs_wave_n27_q8", "rhs", "wave", 27, 3, q=8),
        # the mixed-precision option around a hole with the sampled gauge source
        {**_case("rhs_hole_mixed_n24", "rhs", "hole", 24, 4, variant="damped", halfwidth=8.0), "precision": "mixed"},
        # the Fourier-mode workload, 8 blocks of 32^3, a chunk of 4 steps: an ordinary small evolution
        _case("steps_fourier_n32", "steps", "fourier", 32, 2, steps=4),
        # the static hole on 64 blocks of 32^3, no refinement
        _case("steps_hole_n32", "steps", "hole", 32, 4, variant="damped", halfwidth=8.0, steps=2),
        # the moving hole in refinement shells, 232 blocks of 32^3 on four levels: the path's main use at
        # the largest size of which three states fit the card
        _case("steps_moving_levels", "steps", "moving", 32, 2, radii="8,6,3.2,1.9", variant="damped",
              halfwidth=16.0, steps=2),
        # the harmonic chart with the fitted interior on 2472 blocks of 8^3: many small blocks
        _case("steps_fitted_n8", "steps", "fitted", 8, 1, radii="10,1.6,1.3,1", variant="fitted", halfwidth=1.25,
              steps=2),
        # the plain form with the :pasted limiter at sixth order
        _case("plain_pasted_n16_q6", "plain", "hole", 16, 4, q=6, variant="pasted", halfwidth=4.0),
        # the analysis between two chunks of the static hole
        _case("monitors_hole_n32", "monitors", "hole", 32, 4, variant="damped", halfwidth=8.0),
        # the regrid of the moving hole: verdict and transfer, N = 16
        _case("regrid_moving_n16", "regrid", "moving", 16, 4, radii="3,1.6", variant="damped", halfwidth=6.0),
        # the two derivative forms of a step, on the static hole of the gradient study
        _case("tangent_hole_n16", "tangent", "hole", 16, 2, variant="damped", halfwidth=4.0),
        _case("adjoint_hole_n16", "adjoint", "hole", 16, 2, variant="damped", halfwidth=4.0),
    ]


def draw(rng):
    """One more case of the same ranges: block edges 8 to 32 (odd ones on unrefined meshes), orders 2 to
    8, both precisions, every operation, at most the listed hierarchy's work."""
    op = rng.choice(["rhs", "rhs", "steps", "steps", "steps", "plain", "monitors", "regrid", "tangent", "adjoint"])
    physics = rng.choice({"rhs": ["fourier", "wave", "hole", "moving"], "steps": ["fourier", "hole", "moving", "fitted"],
                          "plain": ["wave", "hole"], "monitors": ["wave", "hole", "moving"], "regrid": ["moving"],
                          "tangent": ["wave", "hole"], "adjoint": ["wave", "hole"]}[op])
    q = rng.choice([2, 4, 4, 4, 6, 8])
    smallest = max(8, 2 * (q // 2 + 1))
    N = round(math.exp(rng.uniform(math.log(smallest), math.log(32))))
    if rng.random() < 0.3:
        N = 32
    c = {"op": op, "physics": physics, "N": N, "roots": rng.choice([2, 2, 3, 4]), "q": q, "precision": "fp64"}
    if op in ("rhs", "steps") and rng.random() < 0.15:
        c["precision"] = "mixed"
    if op == "steps":
        c["steps"] = rng.choice([1, 2, 3])
    if physics in ("hole", "moving"):
        c["variant"] = rng.choice(["damped", "frozen"]) if physics == "hole" else "damped"
        if op == "plain":
            c["variant"] = "pasted"
        c["halfwidth"] = round(rng.uniform(3.0, 5.0), 3)
    if physics == "moving":
        c["N"] += c["N"] % 2
        c["roots"] = rng.choice([2, 4])
        c["radii"] = rng.choice(["1.6", "3,1.6", "2.2"])
    if physics == "fitted":
        c.update(N=8, roots=1, radii=rng.choice(["10,1.6,1.3", "10,1.6,1.2"]), variant="fitted",
                 halfwidth=round(rng.uniform(1.25, 1.4), 3), q=4, precision="fp64")
    if op in ("tangent", "adjoint"):
        c["N"], c["roots"] = min(c["N"], 16), 2
        c["q"] = min(c["q"], 4)
    return c


# ---- the mesh and the inputs ----

def _physics(tgh, c):
    kind, hw = c["physics"], c.get("halfwidth", 1.0)
    hole = dict(M=1.0, a=0.7, halfwidth=hw, r0=0.8, rho_max=4.0, variant=c.get("variant"), eps_ko=0.5)
    if kind == "fourier":
        return tgh.perturbed_minkowski_case()
    if kind == "wave":
        return tgh.gauge_wave_case(eps_ko=0.5, gamma0=1.0, gamma2=-0.5)
    if kind == "hole":
        return tgh.kerr_schild_case(r1=1.3, gauge="sampled", **hole)
    if kind == "moving":
        return tgh.kerr_schild_case(r1=1.3, v=0.1, gauge="algebraic", **hole)
    return tgh.harmonic_kerr_case(r1=1.0, **hole)


def _forest(tgh, c, case, radii):
    if not radii:
        return tgh.gh_forest(case, c["N"], c["roots"])
    radii = [float(r) for r in radii.split(",")]
    path = ((0.0, 0.0, 0.0), (0.07, 0.0, 0.0)) if c["physics"] == "moving" else None
    return tgh.hole_forest(case, c["N"], c["roots"], radii, path=path)


def _modes(x, y, z, width, seed, nvars=20, nmodes=3):
    """A sum of a few Fourier modes for each variable, periodic over `width`, at the points (x, y, z)."""
    g = torch.Generator().manual_seed(int(seed))
    k = torch.randint(1, 4, (nvars, nmodes, 3), generator=g).double() * (2.0 * math.pi / width)
    phase = torch.rand(nvars, nmodes, generator=g).double() * 2.0 * math.pi
    amp = AMPLITUDE * (0.5 + torch.rand(nvars, nmodes, generator=g).double())
    for v in range(nvars):
        acc = torch.zeros_like(x)
        for m in range(nmodes):
            acc += float(amp[v, m]) * torch.sin(float(k[v, m, 0]) * x + float(k[v, m, 1]) * y + float(k[v, m, 2]) * z +
                                                float(phase[v, m]))
        yield acc


def _add_modes(u, forest, seed):
    """u plus the modes, block by block of a level at a time: a point's value depends on its position only."""
    n1 = forest.N + 1
    view = u.view(forest.nblocks, 20, n1, n1, n1)
    h = torch.tensor([forest.h0 / 2 ** int(l) for l in forest.level], dtype=torch.float64, device=u.device)
    corner = torch.from_numpy(forest.corner).to(u.device).double()
    i = torch.arange(n1, dtype=torch.float64, device=u.device)
    axis = [forest.lo[d] + (corner[:, d, None] + i) * h[:, None] for d in range(3)]
    x, y, z = axis[0][:, None, None, :], axis[1][:, None, :, None], axis[2][:, :, None, None]
    shape = (forest.nblocks, n1, n1, n1)
    x, y, z = (t.expand(shape).contiguous() for t in (x, y, z))
    for v, f in enumerate(_modes(x, y, z, forest.h0 * forest.cells0[0], seed)):
        view[:, v] += f
    return u


def prepare(case, seed):
    tgh = package()
    physics = _physics(tgh, case)
    forest = _forest(tgh, case, physics, case.get("radii"))
    P = tgh.GHProblem(physics, forest, case["q"], margin_check=False, precision=case["precision"])
    hmin = forest.h0 / 2 ** int(forest.level.max())
    if case["physics"] == "fitted":
        P.fill_target_analytic(0.0, physics.interior["r1"] + hmin, 0.0)
    u = P.initial_state(P.statevector(), 0.0)
    dt = 0.25 * hmin / P.max_speed(u, 0.0)  # one step for every state of this mesh: the unperturbed speed's
    _add_modes(u, forest, seed)
    s = {"op": case["op"], "P": P, "u": u, "t": 0.0, "dt": dt, "steps": case.get("steps", 1)}
    if case["op"] in ("rhs",):
        s["du"] = torch.zeros_like(u)
    elif case["op"] in ("tangent", "adjoint"):
        g = torch.Generator(device="cuda").manual_seed(int(seed))
        s["ut"] = torch.randn(u.shape, dtype=torch.float64, device="cuda", generator=g)
    elif case["op"] == "regrid":
        # the forest one regrid later: the finest shell drawn in by a fifth
        radii = case["radii"].split(",")
        radii[-1] = str(0.8 * float(radii[-1]))
        s["to"] = tgh.GHProblem(physics, _forest(tgh, case, physics, ",".join(radii)), case["q"], margin_check=False)
        s["u2"] = s["to"].statevector()
    return s


def run(s):
    P, u, op = s["P"], s["u"], s["op"]
    if op == "rhs":
        P.gh_rhs(s["du"], u, s["t"])
        return s["du"]
    if op == "steps":
        P.step_batched(u, s["t"], s["dt"], s["steps"])
        s["t"] += s["steps"] * s["dt"]
        return u
    if op == "plain":
        P.rk4_step(u, s["t"], s["dt"])
        s["t"] += s["dt"]
        return u
    if op == "tangent":
        P.tangent_rk4_step(u, s["ut"], s["t"], s["dt"], "state")
        s["t"] += s["dt"]
        return u, s["ut"]
    if op == "adjoint":
        lam, th = s["ut"].clone(), [0.0, 0.0, 0.0]
        P.adjoint_rk4_step(u, s["t"], s["dt"], lam, th)
        return lam, th
    if op == "monitors":
        P.gh_constraint(u, s["t"])
        P.adm_constraint(u, s["t"])
        norms = P.constraint_norms()
        return {"diag": P.diag(), "norms": norms, "error": P.error_norm(u, s["t"]), "speed": P.max_speed(u, s["t"])}
    if op == "regrid":
        verdict = P.tau(u, s["t"])
        counts, boxes = P.firing([0.4, 0.1])
        s["to"].transfer_from(P, u, s["t"], s["u2"])
        return {"verdict": verdict, "counts": counts, "boxes": boxes, "tau": P.diag(), "u": s["u2"]}
    raise ValueError(op)


def _points(c):
    """Owned points of the case's mesh, the closed blocks' face planes counted in every block."""
    tgh = package()
    forest = _forest(tgh, c, _physics(tgh, c), c.get("radii"))
    return forest.nblocks * (forest.N + 1) ** 3


def work(case):
    n, op, f = _points(case), case["op"], FLOP_RHS[case["physics"]]
    state = 160.0 * n
    if op == "rhs":
        return {"bytes": 2 * state, "flops": float(f * n)}
    if op in ("steps", "plain"):
        k = case.get("steps", 1)
        return {"bytes": 2 * state * k, "flops": float(k * (4 * f + 280) * n)}
    if op == "monitors":
        return {"bytes": state + 72.0 * n, "flops": float((FLOP_MONITORS + 300) * n)}
    if op == "regrid":
        return {"bytes": 2 * state + 8.0 * n, "flops": 400.0 * n}
    if op == "tangent":
        return {"bytes": 4 * state, "flops": 3.0 * (4 * f + 280) * n}
    # a reverse pass costs a few forward ones: the step again, and its transpose
    return {"bytes": 3 * state, "flops": 5.0 * (4 * f + 280) * n}


def tolerance(case):
    # Sums in another order: the second derivatives carry eps |u| / h^2, so an increment's error follows
    # the spacing, a state's after a step does not. Measured against exact(): 3e-16 to 9e-13 for the
    # right-hand side (the last at q = 8 on 81^3 points of the gauge wave, and a fine grid has more),
    # 3e-16 to 4e-15 for states after two to four steps; the mixed form's right-hand side 4e-8 to 2e-6.
    if case["precision"] == "mixed":
        return {"rel": 1e-5, "max": 1e-2} if case["op"] == "rhs" else {"rel": 1e-6, "max": 1e-3}
    if case["op"] in ("steps", "plain"):
        return {"rel": 1e-13, "max": 1e-10}
    if case["op"] == "rhs":
        return {"rel": 1e-11, "max": 1e-8}
    if case["op"] == "monitors":
        return {"rel": 1e-8, "max": 1e-5}  # differences of O(1) second derivatives that nearly cancel
    if case["op"] == "regrid":
        # the Loehner ratio next to the analytic ghosts moves by 1e-13 / its noise floor; counts stay
        return {"rel": 1e-11, "max": 1e-9, "differ": 0.0}
    return {"rel": 1e-11, "max": 1e-8}


# ---- the same in plain torch, 64 bits: periodic unrefined meshes without an interior ----

def _weights(q):
    m = q // 2
    f = math.factorial
    d1 = {k: (-1) ** (k + 1) * f(m) ** 2 / (k * f(m - k) * f(m + k)) for k in range(1, m + 1)}
    d2 = {k: 2 * (-1) ** (k + 1) * f(m) ** 2 / (k * k * f(m - k) * f(m + k)) for k in range(1, m + 1)}
    d2[0] = -2.0 * sum(1.0 / k ** 2 for k in range(1, m + 1))
    r = m + 1
    ko = {k: -((-1) ** k) * math.comb(2 * r, r + k) / 4 ** r for k in range(r + 1)}
    return d1, d2, ko


_ROW = [0, 1, 2, 3, 1, 2, 3, 2, 3, 3]
_COL = [0, 0, 0, 0, 1, 1, 1, 2, 2, 3]


def _full(p):
    """[10, ...] packed to [4, 4, ...]."""
    out = p.new_empty((4, 4) + p.shape[1:])
    for n in range(10):
        out[_ROW[n], _COL[n]] = p[n]
        out[_COL[n], _ROW[n]] = p[n]
    return out


def _exact_rhs(u, h, q, eps, g0, g2):
    """d_t of u [20, z, y, x] on a periodic grid: the first-order-in-time harmonic system, no gauge source."""
    w1, w2, wk = _weights(q)

    def shift(f, axis, k):
        return torch.roll(f, -k, dims=3 - axis)

    def first(f, axis):
        return sum(w1[k] * (shift(f, axis, k) - shift(f, axis, -k)) for k in w1) / h

    def second(f, axis):
        return (w2[0] * f + sum(w2[k] * (shift(f, axis, k) + shift(f, axis, -k)) for k in w1)) / h ** 2

    def dissipation(f):
        return eps / h * sum(wk[0] * f + sum(wk[k] * (shift(f, a, k) + shift(f, a, -k)) for k in range(1, len(wk)))
                             for a in range(3))

    e = torch.einsum
    hh, Pi = u[:10], u[10:]
    eta = torch.diag(torch.tensor([-1.0, 1.0, 1.0, 1.0], dtype=u.dtype, device=u.device))
    g = _full(hh) + eta[:, :, None, None, None]
    gu = torch.linalg.inv(g.permute(2, 3, 4, 0, 1)).permute(3, 4, 0, 1, 2)
    alpha = (-gu[0, 0]) ** -0.5
    beta = alpha ** 2 * gu[0, 1:]
    root = torch.linalg.det(g[1:, 1:].permute(2, 3, 4, 0, 1)).sqrt()
    gam = gu[1:, 1:] + beta[:, None] * beta[None] / alpha ** 2
    dh = [first(hh, a) for a in range(3)]
    dt = sum(beta[i] * dh[i] for i in range(3)) + alpha / root * Pi + dissipation(hh)
    D = torch.stack([_full(x) for x in [dt] + dh])  # D[c, a, b] = d_c g_ab
    V = e("abijk,adbijk->dijk", gu, D) - 0.5 * e("abijk,dabijk->dijk", gu, D)  # the lowered contraction of Gamma
    S = -e("cijk,cabijk->abijk", e("cdijk,dijk->cijk", gu, V), D)
    dgu = -e("mpijk,apqijk,qnijk->amnijk", gu, D, gu)
    C2 = -e("amnijk,mnbijk->abijk", dgu, D)
    S = S + C2 + C2.transpose(0, 1)
    low = 0.5 * (e("bxcijk->xbcijk", D) + e("cxbijk->xbcijk", D) - D)
    G = e("axijk,xbcijk->abcijk", gu, low)
    S = S - 2.0 * e("xyaijk,yxbijk->abijk", G, G)
    tC = -alpha * e("xijk,xijk->ijk", gu[0], V)
    Z = -(1.0 + g2) * tC * g
    Z[0] += -alpha * V
    Z[:, 0] += -alpha * V
    S = S + g0 * Z
    # d_i of alpha, beta, sqrt(gamma) and A^{ij} = alpha sqrt(gamma) gamma^{ij}
    dP = torch.zeros_like(Pi)
    dal = [0.5 * alpha ** 3 * dgu[i + 1, 0, 0] for i in range(3)]
    div_b = 0.0
    for i in range(3):
        db = 2 * alpha * dal[i] * gu[0, 1:] + alpha ** 2 * dgu[i + 1, 0, 1:]
        dr = 0.5 * root * e("mnijk,mnijk->ijk", gam, D[i + 1, 1:, 1:])
        dgam = (dgu[i + 1, 1:, 1:] + (db[:, None] * beta[None] + beta[:, None] * db[None]) / alpha ** 2 -
                2 * dal[i] / alpha ** 3 * beta[:, None] * beta[None])
        div_b = div_b + db[i]
        dA = (dal[i] * root + alpha * dr) * gam[i] + alpha * root * dgam[i]
        for j in range(3):
            dP += dA[j] * dh[j]
            dP += alpha * root * gam[i, j] * (second(hh, i) if i == j else first(first(hh, j), i))
        dP += beta[i] * first(Pi, i)
    dP += div_b * Pi + dissipation(Pi)
    for n in range(10):
        dP[n] -= alpha * root * S[_ROW[n], _COL[n]]
    return torch.cat([dt, dP])


def exact(case, seed):
    """The path in plain torch where the mesh is one periodic grid: the right-hand side and the steps of the
    fourier and wave physics. The other cases have refinement faces, a hole's analytic boundary, its gauge source
    and its interior layer, which are not restated here."""
    if case["op"] not in ("rhs", "steps", "plain") or case["physics"] not in ("fourier", "wave"):
        return None
    wave = case["physics"] == "wave"
    width, lo = (1.0, 0.0) if wave else (2.0, -1.0)
    N, R, q = case["N"], case["roots"], case["q"]
    n = N * R
    h = width / n
    p = lo + torch.arange(n, dtype=torch.float64, device="cuda") * h
    z, y, x = torch.meshgrid(p, p, p, indexing="ij")
    u = torch.stack(list(_modes(x, y, z, width, seed)))
    speed = 1.0
    if wave:  # ds^2 = H (dx^2 - dt^2) + dy^2 + dz^2, H = 1 - A sin(2 pi (x - t)), at t = 0
        A = 1 / 20
        H1 = -A * torch.sin(2 * math.pi * x)
        dtH = 2 * math.pi * A * torch.cos(2 * math.pi * x)
        u[0] -= H1
        u[4] += H1
        # Pi = sqrt(gamma) / alpha d_t h, sqrt(gamma) = alpha = sqrt(H)
        u[10] -= dtH
        u[14] += dtH
    par = (0.5, 1.0, -0.5 if wave else 0.0)
    if case["op"] == "rhs":
        u = _exact_rhs(u, h, q, *par)
    else:
        # the step prepare() takes: cfl h / lambda of the unperturbed state, alpha sqrt(tr gamma^ij) + |beta|
        if wave:
            speed = float(torch.sqrt((1 + H1) * (2 + 1 / (1 + H1))).max())
        else:
            speed = math.sqrt(3.0)
        dt = 0.25 * h / speed
        for _ in range(case.get("steps", 1)):
            k1 = _exact_rhs(u, h, q, *par)
            k2 = _exact_rhs(u + 0.5 * dt * k1, h, q, *par)
            k3 = _exact_rhs(u + 0.5 * dt * k2, h, q, *par)
            k4 = _exact_rhs(u + dt * k3, h, q, *par)
            u = u + dt / 6 * (k1 + 2 * k2 + 2 * k3 + k4)
    i = torch.arange(N + 1, device="cuda")
    out = torch.empty((R ** 3, 20, N + 1, N + 1, N + 1), dtype=torch.float64, device="cuda")
    for b in range(R ** 3):
        at = [(b // R ** d % R * N + i) % n for d in range(3)]
        out[b] = u[:, at[2]][:, :, at[1]][:, :, :, at[0]]
    return out.reshape(-1)
