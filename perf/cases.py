"""The work that programs have this framework do, as cases that can be timed one by one.

A case is a system (pairing model, neutron matter or electron gas, in the sizes of the
command line's defaults, the tests and the benchmark) and a way of running it:

  solve    a kept solver: T2 = 0, the whole solve loop, T2 read back
  sweep    a new system per pass, as the command line runs one: basis, solver, solve, T2
  create   a new solver per pass for a basis that the host program has built
  steps    a host program that keeps the iteration loop and asks for one iteration at a time,
           from the first-order amplitudes
  stages   a host program that keeps the reference's loop body (main.cpp:591-665) and calls its
           stages by name
  batch    several systems of a density sweep solved together
  channel  the ladder term of one channel on device buffers that the program owns

The stop threshold is 1e-10 on the correlation energy, so that the amplitudes of a mixed solve
are those of the FP64 fixed point.  The seed moves the density or the coupling by a few percent.
"""
import ctypes
import math
import random

import numpy as np
import torch

from coupled_cluster_doubles_b200 import CCDSolver, System, _native, solve_batch

TOL = 1e-10
MAX_ITERS = 100
MIXING = 0.5
# Typical iterations of a solve to TOL at this mixing, for work().
ITERATIONS = dict(pairing=25, inf_matter=45, electron_gas=31)


def listed():
    eg = dict(model="electron_gas")
    return [
        # The smallest system of the tests: nothing but launches and latency.
        dict(name="pairing8", run="solve", model="pairing", shells=8, filled=8, param=-1.0,
             precision="fp64"),
        # The command line's default system, run as the command line does, once per density.
        dict(name="pnm14_sweep", run="sweep", model="inf_matter", shells=4, filled=2, param=0.08,
             precision="fp64"),
        # N=14, |n|^2 <= 20: many orbitals, thin channels (at most 14 hole pairs).
        dict(name="eg14s19", run="solve", shells=19, filled=2, param=1.0, precision="fp64", **eg),
        # N=54, |n|^2 <= 20: the middle size, mixed precision.
        dict(name="eg54s19_mixed", run="solve", shells=19, filled=4, param=1.0,
             precision="mixed", **eg),
        # The same size from a host program's own loop: ten iterations, each one's energy read.
        dict(name="eg54s19_steps", run="steps", count=10, shells=19, filled=4, param=1.0,
             precision="fp64", **eg),
        # N=38, |n|^2 <= 16 through the stage entry points, ten iterations.
        dict(name="eg38s15_stages", run="stages", count=10, shells=15, filled=3, param=1.0,
             precision="fp64", **eg),
        # The benchmark's workload, N=54, |n|^2 <= 36, in both precisions.
        dict(name="eg54s32_mixed", run="solve", shells=32, filled=4, param=2.0,
             precision="mixed", **eg),
        dict(name="eg54s32", run="solve", shells=32, filled=4, param=2.0, precision="fp64", **eg),
        # The benchmark's workload with a new solver per point, as a parameter scan has it.
        dict(name="eg54s32_create", run="create", shells=32, filled=4, param=2.0,
             precision="mixed", **eg),
        # The largest system: neutron matter, N=66, |n|^2 <= 36.
        dict(name="pnm66s32", run="solve", model="inf_matter", shells=32, filled=5, param=0.08,
             precision="fp64"),
        # A sweep over particle numbers and densities, all systems in flight together.
        dict(name="eg_batch8", run="batch", count=8, shells=19, filled=4, param=1.0,
             precision="mixed", **eg),
        # One of the widest channels of N=54, |n|^2 <= 36 on the program's own buffers.
        dict(name="channel1796x54", run="channel", pp=1796, hh=54),
    ]


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    run = rng.choice(["solve", "solve", "solve", "sweep", "create", "steps", "stages", "batch",
                      "channel"])
    if run == "channel":
        # Every hh up to the entry point's limit, pp up to the largest channel of the tests.
        return dict(run=run, pp=log_int(8, 3000), hh=log_int(1, 72))
    case = dict(run=run, precision=rng.choice(["fp64", "mixed"]))
    if run in ("steps", "stages"):
        # A mixed iteration's own rounding is what the polish of a solve removes; single
        # iterations are compared in FP64.
        case["precision"] = "fp64"
    if run in ("steps", "stages", "batch"):
        case["count"] = rng.randint(2, 10)
    model = "electron_gas" if run == "batch" else rng.choice(
        ["pairing", "inf_matter", "electron_gas", "electron_gas"])
    big = 20 if run in ("batch", "stages", "sweep") else 32
    if model == "pairing":
        case.update(shells=rng.randint(4, 12), param=round(rng.uniform(-1.0, 0.4), 3))
        case["filled"] = 2 * rng.randint(1, case["shells"] // 2)
    elif model == "inf_matter":
        case.update(filled=rng.choice([2, 2, 3, 4, 5]), param=round(rng.uniform(0.06, 0.16), 4))
        case["shells"] = max(case["filled"] + 2, log_int(4, big))
    else:
        case.update(filled=rng.choice([2, 3, 4]), param=round(rng.uniform(0.5, 2.0), 3))
        case["shells"] = max(case["filled"] + 2, log_int(5, big))
    case["model"] = model
    return case


def _members(case, seed):
    """(model, shells, filled, parameter) of each system of a pass."""
    rng = random.Random(1000003 * seed + 7)

    def moved(x):
        return x * (1.0 + 0.05 * (2.0 * rng.random() - 1.0))

    if case["run"] != "batch":
        return [(case["model"], case["shells"], case["filled"], moved(case["param"]))]
    out = []
    for k in range(case["count"]):
        filled = 2 + (case["filled"] - 2 + k) % 3
        shells = max(filled + 2, case["shells"] - 2 * (k % 4))
        out.append((case["model"], shells, filled, moved(case["param"] * (0.75 + k / 16.0))))
    return out


def _system(model, shells, filled, param):
    # No V block and no table on the host: the solver makes them on the device.
    kw = dict(load_v_pppp=False, tables=False, v_blocks=False)
    if model == "pairing":
        return System.pairing(xi=1.0, g=param, n_pair_states=shells, n_particles=filled, **kw)
    if model == "inf_matter":
        return System.inf_matter(density=param, tz_max=1, n_shells=shells,
                                 n_particle_shells=filled, **kw)
    return System.electron_gas(r_s=param, n_shells=shells, n_particle_shells=filled, **kw)


def _solver(case, system):
    return CCDSolver(system, precision=case["precision"], v_mode="on_the_fly",
                     path="tables" if case["run"] == "stages" else "fused")


def prepare(case, seed):
    if case["run"] == "channel":
        pp, hh = case["pp"], case["hh"]
        g = torch.Generator(device="cuda").manual_seed(seed)

        def block(rows, cols, scale):
            return scale * torch.randn(rows, cols, generator=g, dtype=torch.float64,
                                       device="cuda")

        v = block(pp, pp, 0.02)
        return dict(case=case, lib=_native.gpu_lib(), v_pppp=(v + v.T).contiguous(),
                    v_hhpp=block(hh, pp, 0.05), v_hhhh=block(hh, hh, 0.05),
                    t2=block(pp, hh, 0.01),
                    d=torch.empty(pp, hh, dtype=torch.float64, device="cuda"))
    members = _members(case, seed)
    state = dict(case=case, members=members)
    if case["run"] == "sweep":
        return state
    state["systems"] = [_system(*m) for m in members]
    state["t2"] = [np.zeros(s.t2_size()) for s in state["systems"]]
    if case["run"] != "create":
        state["solvers"] = [_solver(case, s) for s in state["systems"]]
    return state


def run(state):
    case = state["case"]
    kind = case["run"]
    if kind == "channel":
        rc = state["lib"].ccdgpu_calc_channel_t2diff_pphh_noalloc(
            state["v_pppp"].data_ptr(), state["v_hhpp"].data_ptr(), state["v_hhhh"].data_ptr(),
            state["t2"].data_ptr(), state["d"].data_ptr(), case["pp"], case["hh"],
            ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
        if rc != 0:
            raise RuntimeError(f"channel ladder: status {rc}")
        return state["d"]
    if kind == "sweep":
        with _system(*state["members"][0]) as system, _solver(case, system) as sol:
            res = sol.solve(tol=TOL, max_iters=MAX_ITERS, mixing=MIXING)
            return dict(e=res.e_corr, t2=sol.t2(), e_ref=system.reference_energy)
    if kind == "create":
        with _solver(case, state["systems"][0]) as sol:
            res = sol.solve(tol=TOL, max_iters=MAX_ITERS, mixing=MIXING)
            return dict(e=res.e_corr, t2=sol.t2(state["t2"][0]))
    if kind == "batch":
        for sol in state["solvers"]:
            sol.reset()
        res = solve_batch(state["solvers"], tol=TOL, max_iters=MAX_ITERS, mixing=MIXING)
        return dict(e=[r.e_corr for r in res],
                    t2=[s.t2(out) for s, out in zip(state["solvers"], state["t2"])])
    sol, t2 = state["solvers"][0], state["t2"][0]
    if kind == "steps":
        e = [sol.mbpt2(init_t2=True)]
        for _ in range(case["count"]):
            e.append(sol.step(MIXING))
        return dict(e=e, t2=sol.t2(t2))
    sol.reset()
    if kind == "stages":
        e = []
        for _ in range(case["count"]):
            sol.calc_t2diff_p2_p1hh()
            sol.calc_t2diff_h2pp_h1()
            sol.calc_t2diff_phhp()
            sol.calc_t2diff_pphh()
            sol.map_from_distributed()
            e.append(sol.calc_t2_pphh(MIXING))
            sol.map_to_distributed()
        return dict(e=e, t2=sol.t2(t2))
    res = sol.solve(tol=TOL, max_iters=MAX_ITERS, mixing=MIXING)
    return dict(e=res.e_corr, t2=sol.t2(t2))


# ---- the channels of a basis, and the iteration in plain torch -----------------------------


def _shell_cutoff(shells):
    """Largest |n|^2 of the first `shells` occupied shells of the cubic lattice."""
    found, e = 1, 0
    while found < shells:
        e += 1
        m = e
        while m % 4 == 0:
            m //= 4
        found += m % 8 != 7
    return e


def _orbitals(model, shells, filled):
    """Quantum numbers (one row per orbital) and the number of holes."""
    if model == "pairing":
        return np.array([(p // 2 + 1, 1 - 2 * (p % 2)) for p in range(2 * shells)]), filled
    cut, fermi = _shell_cutoff(shells), _shell_cutoff(filled)
    n = math.isqrt(cut)
    axis = range(-n, n + 1)
    rows = [(x, y, z, s) for x in axis for y in axis for z in axis
            if x * x + y * y + z * z <= cut for s in (-1, 1)]
    rows = np.array(sorted(rows, key=lambda r: r[0] ** 2 + r[1] ** 2 + r[2] ** 2))
    return rows, int(((rows[:, :3] ** 2).sum(1) <= fermi).sum())


class _Lists:
    """Pairs (p, q), p in P and q in Q, grouped by a key: pairs of group g are
    p[start[g]:start[g+1]], in (p, q) order."""

    def __init__(self, key, P, Q, n_keys):
        sub = key[np.ix_(P, Q)].ravel()
        order = np.argsort(sub, kind="stable")
        self.p = P[order // len(Q)]
        self.q = Q[order % len(Q)]
        self.count = np.bincount(sub, minlength=n_keys)
        self.start = np.concatenate([[0], np.cumsum(self.count)])

    def group(self, g):
        lo, hi = self.start[g], self.start[g + 1]
        return self.p[lo:hi], self.q[lo:hi]


def _channels(qn, np_):
    n = len(qn)
    holes, parts = np.arange(np_), np.arange(np_, n)
    conserved = qn[:, 1:] if qn.shape[1] == 2 else qn  # the pairing model: the spin alone
    span = 4 * int(np.abs(conserved).max()) + 1

    def key(sign):
        k = np.zeros((n, n), dtype=np.int64)
        for col in conserved.T:
            k = k * span + (col[:, None] + sign * col[None, :]) + span // 2
        ids, inv = np.unique(k, return_inverse=True)
        return inv.reshape(n, n), len(ids)

    reg, n_reg = key(+1)
    mod, n_mod = key(-1)
    pairs = dict(pp=_Lists(reg, parts, parts, n_reg), hh=_Lists(reg, holes, holes, n_reg),
                 ph=_Lists(mod, parts, holes, n_mod), hp=_Lists(mod, holes, parts, n_mod))
    pp, hh = pairs["pp"].count.astype(float), pairs["hh"].count.astype(float)
    cross = np.bincount(reg[np.ix_(holes, parts)].ravel(), minlength=n_reg).astype(float)
    cost = (hh * hh + hh * cross + hh * pp + cross * cross + cross * pp + pp * pp +
            cross * cross + cross * cross)
    order = [c for c in np.lexsort((np.arange(n_reg), -cost)) if pp[c] and hh[c]]
    mods = [c for c in range(n_mod) if pairs["ph"].count[c] and pairs["hp"].count[c]]
    return pairs, reg, mod, order, mods


def _model(model, param, qn, np_, dev):
    """Bare energies and the antisymmetrised interaction <pq|v|rs> of conserving quadruples."""
    q = torch.as_tensor(qn, dtype=torch.float64, device=dev)
    if model == "pairing":
        def v(p, r, s, t):
            ok = ((q[p, 0] == q[r, 0]) & (q[s, 0] == q[t, 0]) & (q[p, 1] == -q[r, 1]) &
                  (q[s, 1] == -q[t, 1]))
            return ok.double() * (-0.5 * param * q[p, 1] * q[s, 1])

        return q[:, 0] - 1.0, v
    n, spin = q[:, :3], q[:, 3]
    if model == "electron_gas":
        hartree, fine = 27.21138505, 1.0 / 137.035999139
        hbarc, mass = 0.1973269788 * 10000 / hartree, 0.5109989461 * 1000000 / hartree
        box = (4.0 / 3.0 * math.pi * np_) ** (1.0 / 3.0) * param * hbarc / (mass * fine)

        def direct(p, r, s, t):
            q2 = ((n[p] - n[s]) ** 2).sum(-1) * (2 * math.pi / box) ** 2
            same = (spin[p] == spin[s]) & (spin[r] == spin[t]) & (q2 > 0)
            return same.double() * (4 * math.pi * fine * hbarc / box ** 3) / torch.where(
                q2 > 0, q2, 1.0)
    else:
        hbarc, mass = 197.3269788, 939.565
        box = (np_ / param) ** (1.0 / 3.0)

        def direct(p, r, s, t):
            k = (math.pi / box) * (n[p] - n[r] - n[s] + n[t])
            q2 = (k ** 2).sum(-1)

            def term(v0, kappa):
                return v0 / box ** 3 * (math.pi / kappa) ** 1.5 * torch.exp(-q2 / (4 * kappa))

            vr, vt, vs = term(200.0, 1.487), term(-178.0, 0.639), term(-91.85, 0.465)
            same = ((spin[p] == spin[s]) & (spin[r] == spin[t])).double()
            swap = ((spin[p] == spin[t]) & (spin[r] == spin[s])).double()
            return (0.5 * (vr + 0.5 * vt + 0.5 * vs) - 0.25 * (vt - vs)) * (same - swap)

    eps = (hbarc * hbarc / (2 * mass)) * (2 * math.pi / box) ** 2 * (n ** 2).sum(1)
    return eps, lambda p, r, s, t: direct(p, r, s, t) - direct(p, r, t, s)


def _ccd(model, shells, filled, param, count=None, first_order=False):
    """The iteration in plain torch, FP64: to the stop rule, or `count` iterations; from zero, or
    from the first-order amplitudes.  Returns (energies, T2 in channel order)."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    qn, np_ = _orbitals(model, shells, filled)
    pairs, reg, mod, order, mods = _channels(qn, np_)
    bare, v = _model(model, param, qn, np_, dev)
    every, holes = torch.arange(len(qn), device=dev)[:, None], torch.arange(np_, device=dev)
    eps = bare + v(every, holes, every, holes).sum(1)
    e_ref = float((0.5 * v(holes[:, None], holes, holes[:, None], holes)).sum() +
                  bare[:np_].sum())

    def put(x):
        return torch.as_tensor(x, device=dev)

    def blocks(bra, ket):
        (p, r), (s, t) = (tuple(map(put, x)) for x in (bra, ket))
        return v(p[:, None], r[:, None], s, t)

    # Regular channels: where each block starts, the pair lists, V.
    n = len(qn)
    offset, width = np.zeros(reg.max() + 1, dtype=np.int64), np.zeros(reg.max() + 1, np.int64)
    pos = np.zeros((n, n), dtype=np.int64)
    total, chans, parts = 0, [], []
    for c in order:
        pp, hh = pairs["pp"].group(c), pairs["hh"].group(c)
        offset[c], width[c] = total, len(hh[0])
        pos[pp], pos[hh] = np.arange(len(pp[0])), np.arange(len(hh[0]))
        chans.append((total, len(pp[0]), len(hh[0]), blocks(pp, pp), blocks(hh, hh),
                      blocks(pp, hh)))
        parts.append([x.ravel() for x in np.broadcast_arrays(pp[0][:, None], pp[1][:, None],
                                                             hh[0], hh[1])])
        total += len(pp[0]) * len(hh[0])
    a, b, i, j = (np.concatenate(x) for x in zip(*parts))

    def where(a, b, i, j):
        c = reg[a, b]
        return put(offset[c] + pos[a, b] * width[c] + pos[i, j])

    at_ji, at_ba, at_both = where(a, b, j, i), where(b, a, i, j), where(b, a, j, i)
    a, b, i, j = map(put, (a, b, i, j))
    den = eps[i] + eps[j] - eps[a] - eps[b]
    v_flat = torch.cat([ch[5].reshape(-1) for ch in chans])
    # Modified channels: the amplitude behind each element of the (a i) x (j b) blocks, V.
    rings, ring_at, ring_n = [], [], 0
    for c in mods:
        ph, hp = pairs["ph"].group(c), pairs["hp"].group(c)
        rows, cols = len(ph[0]), len(hp[0])
        ring_at.append(where(ph[0][:, None], hp[1][None, :], ph[1][:, None],
                             hp[0][None, :]).reshape(-1))
        (hk, hc), (pd, pl) = tuple(map(put, hp)), tuple(map(put, ph))
        v_cd = v(hk[:, None], pl, hc[:, None], pd)                 # <kl|v|cd>
        v_cj = v(hk[:, None], hc[None, :], hc[:, None], hk[None])  # <kb|v|cj>
        rings.append((ring_n, rows, cols, v_cd, v_cj))
        ring_n += rows * cols
    ring_at = torch.cat(ring_at)

    t = v_flat / den if first_order else torch.zeros(total, dtype=torch.float64, device=dev)
    energies = [float((0.25 * v_flat * t).sum())] if first_order else []
    last = 100.0
    while True:
        value = v_flat.clone()
        x_h = torch.zeros(n, dtype=torch.float64, device=dev)
        y_p = torch.zeros(n, dtype=torch.float64, device=dev)
        for at, pp, hh, v_pppp, v_hhhh, v_pphh in chans:
            tb = t[at:at + pp * hh].view(pp, hh)
            hh_hh = v_pphh.T @ tb
            value[at:at + pp * hh].view(pp, hh).add_(
                0.5 * (v_pppp @ tb + tb @ (v_hhhh + 0.5 * hh_hh)))
        x_h.index_add_(0, i, v_flat * t)
        y_p.index_add_(0, a, v_flat * t)
        t_ring, r_ring = t[ring_at], torch.empty(ring_n, dtype=torch.float64, device=dev)
        for at, rows, cols, v_cd, v_cj in rings:
            tb = t_ring[at:at + rows * cols].view(rows, cols)
            torch.mm(tb, v_cj + 0.5 * (v_cd @ tb), out=r_ring[at:at + rows * cols].view(rows, cols))
        r = torch.empty_like(t)
        r[ring_at] = r_ring
        value += r - r[at_ji] - r[at_ba] + r[at_both]
        value -= 0.5 * (x_h[i] + x_h[j] + y_p[a] + y_p[b]) * t
        t = MIXING * value / den + (1.0 - MIXING) * t
        e = float(0.25 * (v_flat * t).sum())
        energies.append(e)
        done = len(energies) - first_order
        if (done == count) if count else (abs(e - last) <= TOL or done > MAX_ITERS):
            return energies, t, e_ref
        last = e


def exact(case, seed):
    if case["run"] == "channel":
        s = prepare(case, seed)
        t = s["t2"]
        return 0.5 * (t @ (s["v_hhhh"] + 0.5 * s["v_hhpp"] @ t)) + 0.5 * s["v_pppp"] @ t
    if case["run"] == "batch" and case["count"] > 4 or case["shells"] > 26 and case["filled"] > 4:
        return None  # over 20 seconds
    got = [_ccd(*m, count=case.get("count") if case["run"] in ("steps", "stages") else None,
                first_order=case["run"] == "steps") for m in _members(case, seed)]
    if case["run"] == "batch":
        return dict(e=[g[0][-1] for g in got], t2=[g[1] for g in got])
    energies, t2, e_ref = got[0]
    out = dict(e=energies if case["run"] in ("steps", "stages") else energies[-1], t2=t2)
    if case["run"] == "sweep":
        out["e_ref"] = e_ref
    return out


def work(case):
    """Bytes and operations that the path cannot do without: per iteration V once (V_pppp by its
    antisymmetry a quarter; two 16-bit terms an element in a mixed iteration), T2 read and
    written, the products of the ladders and the ring."""
    if case["run"] == "channel":
        pp, hh = case["pp"], case["hh"]
        return dict(bytes=8.0 * (pp * pp + 3 * pp * hh + hh * hh),
                    flops=2.0 * pp * pp * hh + 4.0 * pp * hh * hh)
    total = dict(bytes=0.0, flops=0.0)
    for model, shells, filled, _ in _members(case, 0):
        qn, np_ = _orbitals(model, shells, filled)
        pairs, _, _, order, mods = _channels(qn, np_)
        pp, hh = pairs["pp"].count[order].astype(float), pairs["hh"].count[order].astype(float)
        ph, hp = pairs["ph"].count[mods].astype(float), pairs["hp"].count[mods].astype(float)
        v4 = float((pp * pp).sum()) / 4
        n_t, rest = float((pp * hh).sum()), float((hh * hh).sum() + (ph * hp + hp * hp).sum())
        v4_bytes = 8.0
        if case["precision"] == "mixed":
            v4_bytes = 0.5 * (4.0 + 8.0)  # about half of a solve to TOL is the FP64 polish
        per = dict(bytes=v4 * v4_bytes + 8.0 * (3 * n_t + rest),
                   flops=float((0.5 * pp * pp * hh + 2 * pp * hh * hh +
                                pp * hh * hh).sum() + (4 * ph * hp * hp).sum()))
        iterations = case["count"] if case["run"] in ("steps", "stages") else ITERATIONS[model]
        for k in total:
            total[k] += iterations * per[k]
        total["bytes"] += 8.0 * n_t  # T2 to the host
        if case["run"] in ("create", "sweep"):
            total["bytes"] += v4 * (12.0 if case["precision"] == "mixed" else 8.0)
    return total
