"""The work users have this engine do, as cases that can be timed and compared.

Every case goes through the package's public entry points: `System` (a driver
that steps one system and reads its state back), `Batch` (many systems advanced
together), `Server` (requests that arrive and are served together),
`System.set_coords` with the analysis of a restarted system, and the field update
on buffers that the caller owns.  A case is a dict of plain values:

  melt     linear AB diblocks of one length: chains, length, f_a, grid, chi, units,
           count_bits, field_rule, sweeps
  blend    A and B homopolymers (N = 64) with AB diblocks (N = 32): chains, grid, sweeps
  comb     a backbone with two-bead side chains at every third bead: chains,
           backbone, grid, sweeps
  batch    uneven diblock systems stepped in one Batch: systems, mix_seed,
           edge_scale, sweeps
  served   requests submitted at once and polled until all are done: requests,
           mix_seed, edge_lo, edge_hi, divide (of the 50 / 100 / 500 sweeps a request asks for)
  restart  host coordinates in, counts, field, energies and chain observables out:
           chains, length, grid
  field    omega and field energy of the caller's device counts: types, cells,
           literal

units "cell" are the synthetic workloads' (cell edge 1, A = 0.5, about one trial in
two hundred accepted); "reference" are those of the reference's own configuration.dat
(box edge 4 per 24 cells, k = 3 (N - 1) / 2, dt N / xi = 0.17, about every second
trial accepted).
"""
import ctypes
import math

import numpy as np
import torch

import new_arch_b200 as nb
from new_arch_b200 import _lib
from new_arch_b200.server import Server
from new_arch_b200.spec import (Arch, SystemSpec, batched_mix, blend_system, cell_units, diblock_arch, diblock_melt,
                                interaction_matrix, linear_bonds, served_request)


def listed():
    return [
        # The smallest call: the plain system (1,000 diblocks on 16^3 cells, 16-bit counts) one sweep at a
        # time, as a driver does that prints the statistics and keeps the state of every sweep.
        dict(name="plain report", kind="melt", chains=1000, length=32, f_a=0.5, nx=16, ny=16, nz=16, chi=20.0,
             units="cell", count_bits=16, field_rule="every", sweeps=1),
        # The plain system between two check points (TCHECK = 1000 sweeps).
        dict(name="plain run", kind="melt", chains=1000, length=32, f_a=0.5, nx=16, ny=16, nz=16, chi=20.0,
             units="cell", count_bits=16, field_rule="every", sweeps=1000),
        # The reference's own input: 12,800 chains of 32 beads on 24^3 cells in its units and with its field
        # rule, between two check points.
        dict(name="reference configuration", kind="melt", chains=12800, length=32, f_a=0.5, nx=24, ny=24, nz=24,
             chi=30.0, units="reference", count_bits=32, field_rule="reference", sweeps=1000),
        # Chains of an odd length on a grid of uneven axes.
        dict(name="odd lengths", kind="melt", chains=60606, length=33, f_a=0.4, nx=72, ny=60, nz=59, chi=22.0,
             units="cell", count_bits=32, field_rule="every", sweeps=500),
        # Long chains, longer than a warp can hold in registers.
        dict(name="long chains", kind="melt", chains=15625, length=128, f_a=0.5, nx=64, ny=64, nz=64, chi=20.0,
             units="cell", count_bits=32, field_rule="every", sweeps=500),
        # A branched architecture: combs of 40 beads.
        dict(name="combs", kind="comb", chains=50000, backbone=24, nx=64, ny=64, nz=64, chi=20.0, sweeps=500),
        # A blend of three architectures in one system, a quarter of the full-size one.
        dict(name="blend", kind="blend", chains=500000, nx=128, ny=128, nz=64, sweeps=300),
        # The large diblock melt, 51.2M beads on 128^3 cells: a production run.
        dict(name="large system", kind="melt", chains=1600000, length=32, f_a=0.3, nx=128, ny=128, nz=128, chi=25.0,
             units="cell", count_bits=32, field_rule="every", sweeps=500),
        # A parameter study: uneven systems (lengths 16 to 64, axes 16 to 64) stepped together.
        dict(name="parameter study", kind="batch", systems=20, mix_seed=2024, edge_scale=1.0, sweeps=1000),
        # The served form: requests of mixed size and sweep count that arrive together.
        dict(name="served burst", kind="served", requests=32, mix_seed=4242, edge_lo=16, edge_hi=64, divide=1),
        # A restart from host coordinates with the analysis that a check point prints.
        dict(name="restart and analysis", kind="restart", chains=100000, length=32, nx=96, ny=72, nz=60),
        # The field update of an application that owns its buffers, two types on 128^3 cells.
        dict(name="field update", kind="field", types=2, cells=2097152, literal=False),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _grid(rng, cells):
    """Three axes of about `cells` cells in all, within a factor of two of each other, odd ones among them."""
    edge = cells ** (1.0 / 3.0)
    if rng.random() < 0.4:
        edge = 2.0 ** max(3, round(math.log2(edge)))
        return (int(edge),) * 3
    return tuple(max(6, int(round(edge * 2.0 ** rng.uniform(-0.5, 0.5)))) for _ in range(3))


_MOST_TRIALS = 51_200_000 * 500      # bead trials of the largest listed case


def _sweeps(rng, beads):
    return max(1, min(_log(rng, 1, 1000), _MOST_TRIALS // max(beads, 200_000) // 4))


def draw(rng):
    kind = rng.choice(("melt", "melt", "melt", "melt", "comb", "blend", "batch", "served", "restart", "field"))
    if kind == "melt":
        units = rng.choice(("cell", "cell", "reference"))
        beads = _log(rng, 32_000, 25_000_000 if units == "cell" else 2_000_000)
        length = rng.choice((8, 16, 32, 32, 48, 64, 20, 33, 128, 200))
        chains = max(1, beads // length)
        nx, ny, nz = _grid(rng, chains * length / (rng.uniform(7.0, 24.0) if units == "cell" else 30.0))
        small = chains * length < 65536
        return dict(kind=kind, chains=chains, length=length, f_a=round(rng.uniform(0.2, 0.8), 3), nx=nx, ny=ny, nz=nz,
                    chi=round(rng.uniform(10.0, 30.0), 2), units=units, count_bits=16 if small else 32,
                    field_rule=rng.choice(("every", "reference")), sweeps=_sweeps(rng, chains * length))
    if kind == "comb":
        chains, backbone = _log(rng, 1000, 100_000), rng.choice((12, 24, 36))
        nx, ny, nz = _grid(rng, chains * backbone * 1.67 / 8.0)
        return dict(kind=kind, chains=chains, backbone=backbone, nx=nx, ny=ny, nz=nz, chi=round(rng.uniform(10.0, 30.0), 2),
                    sweeps=min(500, _sweeps(rng, chains * backbone * 2)))
    if kind == "blend":
        chains = _log(rng, 20_000, 400_000)
        nx, ny, nz = _grid(rng, chains * 2.1)
        return dict(kind=kind, chains=chains, nx=nx, ny=ny, nz=nz, sweeps=min(300, _sweeps(rng, chains * 61)))
    if kind == "batch":
        systems = rng.randint(4, 20)
        return dict(kind=kind, systems=systems, mix_seed=rng.randint(1, 1 << 20), edge_scale=round(rng.uniform(0.4, 1.0), 3),
                    sweeps=_log(rng, 20, 1000))
    if kind == "served":
        return dict(kind=kind, requests=rng.randint(4, 32), mix_seed=rng.randint(1, 1 << 20), edge_lo=rng.randint(8, 20), edge_hi=rng.randint(24, 64),
                    divide=rng.choice((1, 2, 10)))
    if kind == "restart":
        chains, length = _log(rng, 1000, 200_000), rng.choice((16, 32, 33, 48, 64))
        nx, ny, nz = _grid(rng, chains * length / 7.8)
        return dict(kind=kind, chains=chains, length=length, nx=nx, ny=ny, nz=nz)
    return dict(kind=kind, types=rng.choice((1, 2, 2, 3, 4)), cells=_log(rng, 4096, 4_000_000), literal=rng.random() < 0.3)


# ---------------------------------------------------------------- inputs
def _melt_spec(case, seed):
    n, grid = case["length"], (case["nx"], case["ny"], case["nz"])
    rule = nb.FIELD_REFERENCE if case["field_rule"] == "reference" else nb.FIELD_EVERY
    if case["units"] == "cell":
        return diblock_melt(case["chains"], n, case["f_a"], grid, case["chi"], 50.0, seed, field_rule=rule,
                            count_bits=case["count_bits"])
    edge = 4.0 / 24.0
    return SystemSpec(2, *grid, *(edge * g for g in grid), interaction_matrix(2, case["chi"], 50.0), n,
                      1.5 * (n - 1), 0.17 / n, seed, nb.HAM_SCMF0, rule, case["count_bits"],
                      [diblock_arch(n, case["f_a"], case["chains"], 0.0)])


def _comb_spec(case, seed):
    nb_, k_sig = case["backbone"], cell_units()
    bonds, types = linear_bonds(nb_), [0] * nb_
    for b in range(0, nb_, 3):
        j = len(types)
        types += [1, 1]
        bonds += [[b, j], [j, j + 1]]
    grid = (case["nx"], case["ny"], case["nz"])
    return SystemSpec(2, *grid, *(float(g) for g in grid), interaction_matrix(2, case["chi"], 50.0), 32, k_sig[0], 0.5,
                      seed, nb.HAM_SCMF0, nb.FIELD_EVERY, 32, [Arch(len(types), case["chains"], types, bonds, k_sig[1])])


def _restart_spec(case, seed):
    return diblock_melt(case["chains"], case["length"], 0.5, (case["nx"], case["ny"], case["nz"]), 20.0, 50.0, seed)


def _restart_coords(case, seed):
    """Random walks of the synthetic bond length, started anywhere in the box."""
    rng = np.random.default_rng(seed)
    walk = rng.standard_normal((case["chains"], case["length"], 3), dtype=np.float32)
    walk *= np.float32(cell_units()[1])
    walk[:, 0] = rng.random((case["chains"], 3), dtype=np.float32) * np.float32([case["nx"], case["ny"], case["nz"]])
    return np.cumsum(walk, axis=1, dtype=np.float32).reshape(-1, 3)


def _batch_specs(case, seed):
    specs = batched_mix(case["systems"], case["mix_seed"], case["edge_scale"])
    for i, sp in enumerate(specs):
        sp.seed = 1000 * seed + i
    return specs


def _served_requests(case, seed):
    rng = np.random.default_rng(case["mix_seed"])
    reqs = [served_request(rng, 50_000 + 100 * seed + i, case["edge_lo"], case["edge_hi"])
            for i in range(case["requests"])]
    return [(sp, max(1, k // case["divide"])) for sp, k in reqs]


def _field_inputs(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    mean = torch.full((case["types"], case["cells"]), 24.0 / case["types"], device="cuda")
    counts = torch.poisson(mean, generator=g).to(torch.int32)
    chi = 10.0 + (seed % 20)
    return counts, interaction_matrix(case["types"], chi, 50.0), 24.0


def _started(spec):
    s = nb.System(spec)
    s.init_coords()
    return s


def prepare(case, seed):
    kind = case["kind"]
    if kind == "melt":
        return kind, case, _started(_melt_spec(case, seed))
    if kind == "comb":
        return kind, case, _started(_comb_spec(case, seed))
    if kind == "blend":
        return kind, case, _started(blend_system(seed, case["chains"], (case["nx"], case["ny"], case["nz"])))
    if kind == "batch":
        systems = [_started(sp) for sp in _batch_specs(case, seed)]
        return kind, case, systems, nb.Batch(systems)
    if kind == "served":
        return kind, case, _served_requests(case, seed), Server(100 * 10**9)
    if kind == "restart":
        return kind, case, nb.System(_restart_spec(case, seed)), _restart_coords(case, seed)
    counts, xn, density = _field_inputs(case, seed)
    omega = torch.empty(counts.shape, dtype=torch.float32, device="cuda")
    energy = torch.zeros(1, dtype=torch.float64, device="cuda")
    return kind, case, counts, np.ascontiguousarray(xn, dtype=np.float64), density, omega, energy


# ---------------------------------------------------------------- one pass
def run(state):
    kind, case = state[:2]
    if kind in ("melt", "comb", "blend"):
        s = state[2]
        st = s.step_stats(case["sweeps"])
        return {"coords": s.coords(), "counts": s.counts(), "omega": s.omega(), "accepts": st["total_accepts"],
                "e_field": st["e_field"]}
    if kind == "batch":
        _, _, systems, batch = state
        batch.step(case["sweeps"])
        return {"coords": [s.coords() for s in systems], "counts": [s.counts() for s in systems],
                "omega": [s.omega() for s in systems]}
    if kind == "served":
        _, _, requests, server = state
        ids = [server.submit(sp, k) for sp, k in requests]
        done = {}
        while len(done) < len(ids):
            for r in server.poll(64, 200):
                done[r["id"]] = r
        return {"counts": [done[i]["counts"] for i in ids], "accepts": np.array([done[i]["accepts"] for i in ids]),
                "e_field": np.array([done[i]["e_field"] for i in ids]), "e_bond": np.array([done[i]["e_bond"] for i in ids])}
    if kind == "restart":
        _, _, s, xyz = state
        s.set_coords(xyz)
        st, obs = s.stats(), s.analyze()[0]
        return {"counts": s.counts(), "omega": s.omega(), "e_bond": st["e_bond"], "e_field": st["e_field"],
                "re2": obs["re2"], "rg2": obs["rg2"], "bond2": obs["bond2"]}
    _, _, counts, xn, density, omega, energy = state
    _lib.check(_lib.lib().scmf_update_omega_noalloc(
        counts.data_ptr(), omega.data_ptr(), case["types"], case["cells"], 1.0 / density,
        xn.ctypes.data_as(ctypes.POINTER(ctypes.c_double)), 32, nb.HAM_LITERAL if case["literal"] else nb.HAM_SCMF0,
        energy.data_ptr(), torch.cuda.current_stream().cuda_stream))
    return {"omega": omega, "energy": energy}


# ---------------------------------------------------------------- the least work
_ON_CHIP = 64 << 20       # state below this may stay on the chip from sweep to sweep
_TRIAL_OPS = 160          # Philox4x32-10 (about 60), three normals (24), forces, energy, Metropolis (76)


def _sweep_work(beads, cells, types, sweeps):
    state = 24 * beads + 8 * cells * types       # positions read and written, counts read, omega written
    passes = sweeps if state > _ON_CHIP else 1
    return state * passes, (_TRIAL_OPS * beads + 12 * cells * types) * sweeps


def work(case):
    kind = case["kind"]
    if kind in ("melt", "comb", "blend"):
        cells = case["nx"] * case["ny"] * case["nz"]
        if kind == "melt":
            beads = case["chains"] * case["length"]
        elif kind == "comb":
            beads = case["chains"] * (case["backbone"] + 2 * ((case["backbone"] + 2) // 3))
        else:
            beads = blend_system(0, case["chains"]).n_beads
        b, f = _sweep_work(beads, cells, 2, case["sweeps"])
        return {"bytes": b, "flops": f}
    if kind == "batch":
        w = [_sweep_work(sp.n_beads, sp.n_cells, 2, case["sweeps"]) for sp in _batch_specs(case, 0)]
        return {"bytes": sum(x[0] for x in w), "flops": sum(x[1] for x in w)}
    if kind == "served":
        w = [_sweep_work(sp.n_beads, sp.n_cells, 2, k) for sp, k in _served_requests(case, 0)]
        return {"bytes": sum(x[0] for x in w), "flops": sum(x[1] for x in w)}
    if kind == "restart":
        beads, cells = case["chains"] * case["length"], case["nx"] * case["ny"] * case["nz"]
        return {"bytes": 24 * beads + 16 * cells, "flops": 40 * beads + 24 * cells}
    return {"bytes": 8 * case["types"] * case["cells"], "flops": 12 * case["types"] * case["cells"]}


# ---------------------------------------------------------------- the values in 64 bits
def _omega64(counts, scaling, xn, nref, literal):
    """[types, cells] omega and the field energy sum_T omega_T n_T."""
    n = counts.shape[0]
    xn = np.asarray(xn, dtype=np.float64).reshape(n, n)
    phi = counts.astype(np.float64) * scaling
    tot = phi.sum(axis=0)
    omega = np.empty_like(phi)
    for t in range(n):
        w = (tot - 1.0) * xn[t, t] / nref
        for u in range(n):
            if u != t:
                w = w + (xn[u, t] * phi[u] if literal else -0.5 * xn[u, t] * (phi[t] - phi[u])) / nref
        omega[t] = w
    return omega, float((omega * counts).sum())


def exact(case, seed):
    """Sweeps have no value in 64 bits: every trial is decided by the 32-bit value that its random stream and
    its field give, and one trial decided the other way changes all that follow."""
    if case["kind"] == "field":
        counts, xn, density = _field_inputs(case, seed)
        omega, energy = _omega64(counts.cpu().numpy(), 1.0 / density, xn, 32, case["literal"])
        return {"omega": omega, "energy": np.array([energy])}
    if case["kind"] != "restart":
        return None
    spec, n, nc = _restart_spec(case, seed), case["length"], case["nx"] * case["ny"] * case["nz"]
    r = _restart_coords(case, seed).astype(np.float64)
    cell = [np.floor(r[:, a]).astype(np.int64) % g for a, g in enumerate((case["nx"], case["ny"], case["nz"]))]
    at = cell[0] + case["nx"] * (cell[1] + case["ny"] * cell[2])
    kinds = np.tile(np.asarray(spec.archs[0].mono_type, dtype=np.int64), case["chains"])
    counts = np.bincount(kinds * nc + at, minlength=2 * nc).reshape(2, nc)
    omega, e_field = _omega64(counts, nc / spec.n_beads, spec.xn, spec.nref, False)
    c = r.reshape(case["chains"], n, 3)
    bond, ends = (c[:, 1:] - c[:, :-1]) ** 2, (c[:, -1] - c[:, 0]) ** 2
    spread = ((c - c.mean(axis=1, keepdims=True)) ** 2).mean(axis=1)

    def four(v):
        m = v.reshape(-1, 3).mean(axis=0)
        return np.append(m, m.sum())

    return {"counts": counts.reshape(-1).astype(np.uint32), "omega": omega.reshape(-1),
            "e_bond": spec.harmonic_normb * float(bond.sum()), "e_field": e_field, "re2": four(ends), "rg2": four(spread),
            "bond2": four(bond)}
