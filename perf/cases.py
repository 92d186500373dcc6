"""Timed cases of the docking path: what a program that docks on this framework has it do.

Every case is a dict of plain values. ``prepare`` makes what such a program has in hand before the
call (the system's evaluation context, the chromosomes or the ensemble, drawn from the seed),
``run`` makes one pass through the public entry points (``flexaidds_gb300.evaluator``, the C ABI
of ``include/fxe.h``), ``work`` counts what the pass cannot do without and ``exact`` restates, in
plain numpy, the outputs that have a closed form.

A case's system (receptor, ligand, energy matrix) follows from the case alone, as a program keeps
one system over many calls; its chromosomes, energies and GA seeds follow from the seed.
"""
import ctypes as C
import functools

import numpy as np
import torch

from flexaidds_gb300 import evaluator, prepare as setup, synth, system

KB = 0.001987206   # kcal/(mol K), LIB/statmech.h:26
FIELDS = ("com", "con", "wal", "sas", "elec", "gist", "hbond", "gist_desolv", "metal_coord", "totsas", "evalue")

# The systems of the repository's benchmark and tests: receptor atoms, cleft radius (A), the
# receptor cube's edge (0: from the density), ligand atoms, torsions, seed, flexible side chains and
# their rotamers.
SMALL = dict(n_rec=2000, cleft=8.0, edge=0.0, n_lig=24, n_tor=6, system=11, side_chains=0, rotamers=8)
PLAIN = dict(n_rec=6000, cleft=12.0, edge=60.032427451306646, n_lig=48, n_tor=12, system=7, side_chains=3, rotamers=8)
MANY = dict(n_rec=4000, cleft=10.0, edge=51.92391670510951, n_lig=30, n_tor=7, system=31, side_chains=0, rotamers=8)


def listed():
    return [
        # one pose scored from its internal coordinates, as a local search or a re-scoring step
        # calls ic2cf: the smallest call, all latency
        dict(SMALL, name="pose_ic", kind="score_ic", n=1, source="scored"),
        # a small job's population, genes in host memory, records back to it: the call that takes
        # the place of the reference's batch evaluator in its GA loop
        dict(SMALL, name="population_small", kind="score_host", n=500, source="evolved", precision=0),
        # the benchmark's population: every pose passes the clash pre-filter (a converged search),
        # genes and records resident on the device
        dict(PLAIN, name="population_plain", kind="score_device", n=2000, source="scored", precision=0),
        # the same population in single-precision geometry
        dict(PLAIN, name="population_fast", kind="score_device", n=2000, source="scored", precision=1),
        # uniform chromosomes, most of which clash: an initial screen of a cleft, more poses than
        # the context holds at once and an odd number of them
        dict(MANY, name="screen_uniform", kind="score_host", n=30011, source="uniform", precision=0),
        # many ligands of 10-70 atoms on one receptor, uneven populations, one launch of each kernel
        dict(MANY, name="batch_ligands", kind="batch", jobs=24, atoms_lo=10, atoms_hi=70, tors_hi=15,
             pop_lo=200, pop_hi=2000, precision=0),
        # whole genetic algorithms on the device: admission, generations, ensemble, thermodynamics
        dict(SMALL, name="ga_small", kind="ga", population=500, generations=25, fitness="PSHARE", precision=0),
        dict(PLAIN, name="ga_large", kind="ga", population=1999, generations=10, fitness="PSHARE", precision=0),
        # downstream of a run: clustering of its ensemble (the reference's defaults), the ensemble's
        # sort and near-duplicate removal, its thermodynamics and the Boltzmann weights
        dict(PLAIN, name="cluster", kind="cluster", centres=500, per=400, temperature=0, rmsd=2.0, results=10),
        dict(name="ensemble", kind="ensemble", n=250007, genes=19, distinct=60000),
        dict(name="thermo_device", kind="thermo_device", n=1000000, multiplicity=0, temperature=300.0),
        dict(name="weights_host", kind="weights", n=50000, multiplicity=1, temperature=310.0),
    ]


def _log(rng, lo, hi):
    return int(round(float(np.exp(rng.uniform(np.log(lo), np.log(hi))))))


def _draw_system(rng):
    n_rec = _log(rng, 600, 6000)
    side = rng.choice((0, 0, 1, 2, 3))
    return dict(n_rec=n_rec, cleft=round(rng.uniform(8.0, 12.0) if n_rec >= 1500 else rng.uniform(6.0, 7.5), 2), edge=0.0,
                n_lig=rng.randint(10, 48), n_tor=rng.randint(0, 12), system=rng.randint(1, 10 ** 6),
                side_chains=side, rotamers=rng.randint(4, 10))


def draw(rng):
    kind = rng.choice(("score_ic", "score_host", "score_host", "score_device", "score_device", "screen", "batch", "ga",
                       "ga", "cluster", "ensemble", "thermo_device", "weights"))
    if kind == "score_ic":
        return dict(_draw_system(rng), kind=kind, n=_log(rng, 1, 64), source="evolved")
    if kind in ("score_host", "score_device"):
        return dict(_draw_system(rng), kind=kind, n=_log(rng, 16, 2000), source="evolved",
                    precision=rng.choice((0, 0, 1)))
    if kind == "screen":
        return dict(_draw_system(rng), kind="score_host", n=_log(rng, 2000, 25000), source="uniform", precision=0)
    if kind == "batch":
        lo = rng.randint(10, 30)
        hi = rng.randint(lo, 60)
        pop = _log(rng, 100, 1000)
        return dict(MANY, system=rng.randint(1, 10 ** 6), edge=0.0, kind=kind, jobs=rng.randint(2, 20), atoms_lo=lo,
                    atoms_hi=hi, tors_hi=rng.randint(0, 15), pop_lo=pop, pop_hi=rng.randint(pop, 1500),
                    precision=rng.choice((0, 0, 1)))
    if kind == "ga":
        return dict(_draw_system(rng), kind=kind, population=_log(rng, 50, 1500), generations=rng.randint(3, 10),
                    fitness=rng.choice(("PSHARE", "PSHARE", "LINEAR", "SMFREE")), precision=0)
    if kind == "cluster":
        return dict(_draw_system(rng), kind=kind, centres=_log(rng, 20, 500), per=_log(rng, 20, 400),
                    temperature=rng.choice((0, 0, 300)), rmsd=round(rng.uniform(1.0, 3.0), 2), results=rng.randint(5, 30))
    if kind == "ensemble":
        n = _log(rng, 3000, 250000)
        return dict(kind=kind, n=n, genes=rng.randint(5, 20), distinct=max(1, n // rng.randint(2, 8)))
    return dict(kind=kind, n=_log(rng, 1000, 1000000), multiplicity=rng.randint(0, 1), temperature=round(rng.uniform(250.0, 350.0), 1))


# ---------------------------------------------------------------------------------------------
# systems and populations
# ---------------------------------------------------------------------------------------------

_SHAPE = ("n_rec", "cleft", "edge", "n_lig", "n_tor", "system", "side_chains", "rotamers")


@functools.lru_cache(maxsize=8)
def _inputs(n_rec, cleft, edge, n_lig, n_tor, seed, side_chains, rotamers):
    return system.make_inputs(n_rec, cleft, n_lig, n_tor, seed=seed, edge=edge or None, side_chains=side_chains,
                              rotamers=rotamers)


@functools.lru_cache(maxsize=8)
def _descriptor(*shape):
    return setup.prepare(_inputs(*shape))


def _of(case):
    return _descriptor(*(case[k] for k in _SHAPE))


@functools.lru_cache(maxsize=1)
def _stream():
    """The one stream this program queues device calls on."""
    return torch.cuda.Stream()


def _scored(d, n, seed):
    """The first n chromosomes of a seeded uniform stream that pass the clash pre-filter (as many
    as 40 blocks of it hold, repeated when they are fewer)."""
    ev = evaluator.GPUEvaluator(d, max_poses=16384, precision=evaluator.GPUEvaluator.FAST)
    keep, have = [], 0
    for k in range(40):
        g = synth.random_genes(16384 if n <= 64 else 65536, d.n_genes, seed=seed * 1000 + k)
        # (a clash is found before the polyhedra, whatever their precision)
        keep.append(g[ev.eval_genes(g)["status"] != 2])
        have += len(keep[-1])
        if have >= n:
            break
    ev.close()
    g = np.concatenate(keep)
    if len(g) == 0:
        g = synth.random_genes(n, d.n_genes, seed=seed)
    return np.ascontiguousarray(g[np.arange(n) % len(g)])


def _evolved(evs, pops, seed, generations=4):
    """Each context's population after a few GA generations with the default operators."""
    eng = evaluator.GAEngine(max_jobs=len(evs), precision=0)
    slots = [eng.admit(eng.job(ev, max(2, p), generations + 1, seed * 7919 + k), ev) for k, (ev, p) in enumerate(zip(evs, pops))]
    for _ in range(generations):
        eng.step()
    got = [eng.read_population(s, max(2, p))[0][:p] for s, p in zip(slots, pops)]
    eng.close()
    # a population is kept sorted by energy; a program's own order is another
    rng = np.random.default_rng(seed)
    return [np.ascontiguousarray(g[rng.permutation(len(g))]) for g in got]


def _population(d, case, seed):
    n = case["n"]
    if case["source"] == "uniform":
        return synth.random_genes(n, d.n_genes, seed=seed)
    if case["source"] == "scored":
        return _scored(d, n, seed)
    ev = evaluator.GPUEvaluator(d, max_poses=max(2, n))
    g = _evolved([ev], [n], seed)[0]
    ev.close()
    return g


@functools.lru_cache(maxsize=4)
def _batch_descriptors(*key):
    (n_rec, cleft, edge, seed, jobs, lo, hi, tors, pop_lo, pop_hi) = key
    base = _inputs(n_rec, cleft, edge, 12, 3, seed, 0, 8)
    rng = np.random.default_rng(seed + 1)
    out = []
    for k in range(jobs):
        n, t, p = (int(rng.integers(a, b + 1)) for a, b in ((lo, hi), (0, tors), (pop_lo, pop_hi)))
        lig = synth.random_ligand(n, t, seed=seed * 1000 + k)
        out.append((setup.prepare(system.SystemInputs(receptor=base.receptor, ligand=lig, grid_xyz=base.grid_xyz,
                                                      emat=base.emat)), p))
    return out


def _batch_of(case):
    return _batch_descriptors(*(case[k] for k in ("n_rec", "cleft", "edge", "system", "jobs", "atoms_lo", "atoms_hi",
                                                  "tors_hi", "pop_lo", "pop_hi")))


def _ensemble_inputs(case, seed):
    """A GA's snapshots: chromosomes on their bins, the survivors repeated over the generations and
    many within a bin of another, energies around their family's."""
    rng = np.random.default_rng(seed)
    m, ng = case["distinct"], case["genes"]
    fam = rng.integers(0, 37, size=(max(1, m // 12), ng))
    member = rng.integers(0, len(fam), size=m)
    step = (rng.random((m, ng)) < 0.03) * rng.integers(-1, 2, size=(m, ng))
    ic = (fam[member] + step) * 5.0 - 90.0
    e = rng.normal(-25.0, 6.0, size=len(fam))[member] + np.abs(step).sum(1) * rng.normal(0.4, 0.2, size=m)
    pick = rng.integers(0, m, size=case["n"])
    return np.ascontiguousarray(ic[pick]), np.ascontiguousarray(e[pick])


def _energies(case, seed):
    rng = np.random.default_rng(seed)
    e = rng.normal(-30.0, 5.0, case["n"])
    mult = rng.integers(1, 9, case["n"]).astype(np.int32) if case["multiplicity"] else None
    return e, mult


# ---------------------------------------------------------------------------------------------
# the interface
# ---------------------------------------------------------------------------------------------

def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case, "kind": kind}
    if kind in ("score_ic", "score_host", "score_device"):
        d = _of(case)
        genes = _population(d, case, seed)
        s["ev"] = evaluator.GPUEvaluator(d, max_poses=min(case["n"], 8192), precision=case.get("precision", 0))
        if kind == "score_ic":
            s["ic"] = d.genes_to_ic(genes)
        elif kind == "score_host":
            s["genes"] = genes
        else:
            s["genes"] = torch.from_numpy(genes).cuda()
            s["out"] = torch.zeros(case["n"], 12, dtype=torch.float64, device="cuda")
    elif kind == "batch":
        jobs = _batch_of(case)
        evs = []
        for d, p in jobs:
            evs.append(evaluator.GPUEvaluator(d, max_poses=max(2, p), precision=case["precision"],
                                              share_receptor_with=evs[0] if evs else None))
        pops = _evolved(evs, [p for _, p in jobs], seed)
        s["evs"] = evs
        first = np.concatenate([[0], np.cumsum([len(g) for g in pops])])
        s["genes"] = [torch.from_numpy(g).cuda() for g in pops]
        s["out"] = torch.zeros(int(first[-1]), 12, dtype=torch.float64, device="cuda")
        s["batch"] = evaluator.Batch(max_jobs=len(evs), max_poses=int(first[-1]))
        s["table"] = [(ev, g.shape[0], g.data_ptr(), s["out"][int(k):].data_ptr()) for ev, g, k in zip(evs, s["genes"], first)]
    elif kind == "ga":
        s["ev"] = evaluator.GPUEvaluator(_of(case), max_poses=case["population"], precision=case["precision"])
        s["engine"] = evaluator.GAEngine(max_jobs=1, precision=case["precision"])
        s["job"] = evaluator.GAEngine.job(s["ev"], case["population"], case["generations"], seed, fitness=case["fitness"])
    elif kind == "cluster":
        d = _of(case)
        s["ic"], s["e"] = synth.clustered_ensemble(d, case["centres"], case["per"], seed=seed)
        s["ev"] = evaluator.GPUEvaluator(d, max_poses=2)
    elif kind == "ensemble":
        s["ic"], s["e"] = _ensemble_inputs(case, seed)
        # the program's arrays for the kept chromosomes: as long as the snapshots, -1 and 0 past them
        s["index"], s["energy"] = np.full(case["n"], -1, np.int64), np.zeros(case["n"])
        s["kept"] = 0
    else:
        e, mult = _energies(case, seed)
        if kind == "thermo_device":
            lib = evaluator.load_library()
            lib.fxe_thermo_compute_device_fixed.argtypes = [C.c_void_p, C.c_void_p, C.c_int64, C.c_double, C.c_void_p, C.c_void_p]
            s["lib"] = lib
            s["e"] = torch.from_numpy(e).cuda()
            s["mult"] = torch.from_numpy(mult).cuda() if mult is not None else None
            s["out"] = torch.zeros(8, dtype=torch.float64, device="cuda")
        else:
            s["e"], s["mult"] = e, mult
    if torch.cuda.is_available():
        torch.cuda.synchronize()
    return s


def _records(out):
    """The fields of a device buffer of records (11 doubles, two int32 each)."""
    r = {f: out[:, k] for k, f in enumerate(FIELDS)}
    r["rclash"], r["status"] = (out.view(torch.int32)[:, 22 + k] for k in range(2))
    return r


def run(state):
    case, kind = state["case"], state["kind"]
    if kind == "score_ic":
        r = state["ev"].eval_ic(state["ic"])
        return {f: r[f] for f in r.dtype.names}
    if kind == "score_host":
        r = state["ev"].eval_genes(state["genes"])
        return {f: r[f] for f in r.dtype.names}
    if kind == "score_device":
        state["ev"].eval_genes_device(state["genes"].data_ptr(), case["n"], state["out"].data_ptr(), _stream().cuda_stream)
        return _records(state["out"])
    if kind == "batch":
        state["batch"].eval_genes_device(state["table"], _stream().cuda_stream)
        return _records(state["out"])
    if kind == "ga":
        eng = state["engine"]
        slot = eng.admit(state["job"], state["ev"])
        for _ in range(case["generations"]):
            eng.step()
        eng.finished()
        genes, energies = eng.read_population(slot, case["population"])
        best_genes, best, thermo = eng.collect(slot, 300.0)
        return {"genes": genes, "energies": energies, "best_genes": best_genes, "best": best, "thermo": thermo}
    if kind == "cluster":
        return state["ev"].cluster(state["ic"], state["e"], case["temperature"], case["rmsd"], case["results"])
    if kind == "ensemble":
        r = evaluator.ensemble_dedup(state["ic"], state["e"])
        k, old = len(r["index"]), state["kept"]
        state["index"][:k], state["energy"][:k], state["kept"] = r["index"], r["energy"], k
        state["index"][k:old], state["energy"][k:old] = -1, 0.0
        return {"index": state["index"], "energy": state["energy"]}
    if kind == "thermo_device":
        rc = state["lib"].fxe_thermo_compute_device_fixed(
            state["e"].data_ptr(), state["mult"].data_ptr() if state["mult"] is not None else None, case["n"],
            case["temperature"], state["out"].data_ptr(), _stream().cuda_stream)
        if rc != 0:
            raise RuntimeError(state["lib"].fxe_last_error().decode())
        return state["out"]
    return {"weights": evaluator.boltzmann_weights(state["e"], state["mult"], case["temperature"]),
            "thermo": evaluator.thermo(state["e"], state["mult"], case["temperature"])}


def _score_work(n, atoms, scored, n_genes, n_rec):
    """Bytes and operations of scoring n poses: per scored atom the candidates' distances, the
    contact planes, the hull's plane tests, vertices, faces and areas (about 9,900 operations on the
    benchmark's systems); a pose the clash pre-filter rejects needs its build and its distances."""
    flops = n * atoms * (60 + 8 * 143 + scored * 8800)
    return {"bytes": n * (4 * n_genes + 96 + 16) + 20 * n_rec + 40 * 40 * 8, "flops": flops}


def work(case):
    kind = case["kind"]
    if kind in ("score_ic", "score_host", "score_device", "ga"):
        atoms = case["n_lig"] + 5 * case["side_chains"]
        ng = 4 + case["n_tor"] + case["side_chains"]
        if kind == "ga":
            P, G = case["population"], case["generations"]
            w = _score_work(P * (G + 1), atoms, 0.5, ng, case["n_rec"])
            w["bytes"] += G * P * (4 * ng + 8)
            if case["fitness"] != "LINEAR":
                w["flops"] += (G + 1) * P * P * (3 * ng + 4)
            return w
        return _score_work(case["n"], atoms, {"scored": 1.0, "evolved": 0.5, "uniform": 0.02}[case["source"]], ng, case["n_rec"])
    if kind == "batch":
        n = case["jobs"] * (case["pop_lo"] + case["pop_hi"]) // 2
        return _score_work(n, (case["atoms_lo"] + case["atoms_hi"]) // 2, 0.5, 4 + case["tors_hi"] // 2, case["n_rec"])
    if kind == "cluster":
        n, ng = case["centres"] * case["per"], 4 + case["n_tor"] + case["side_chains"]
        return {"bytes": n * (8 * ng + 8 + 8), "flops": n * case["n_lig"] * 60}
    if kind == "ensemble":
        return {"bytes": case["n"] * (8 * case["genes"] + 8) + case["distinct"] * 16, "flops": case["n"] * case["genes"]}
    n, per = case["n"], 8 + 4 * case["multiplicity"]
    return {"bytes": n * (per + (8 if kind == "weights" else 0)), "flops": n * (20 if kind == "thermo_device" else 33)}


def _thermo_record(e, mult, T):
    """log Z and the moments of a canonical ensemble, max-shifted, and the weights."""
    e = e.astype(np.longdouble)
    kT = np.longdouble(KB) * np.longdouble(T)
    lw = -e / kT + (np.log(mult.astype(np.longdouble)) if mult is not None else 0.0)
    m = lw.max()
    w = np.exp(lw - m)
    z = w.sum()
    p = w / z
    log_z = m + np.log(z)
    mean, sq = (p * e).sum(), (p * e * e).sum()
    var = sq - mean * mean
    f = -kT * log_z
    rec = dict(temperature=T, log_Z=log_z, free_energy=f, mean_energy=mean, mean_energy_sq=sq,
               heat_capacity=var / (kT * kT), entropy=(mean - f) / np.longdouble(T), std_energy=np.sqrt(max(var, 0.0)))
    return {k: float(v) for k, v in rec.items()}, p.astype(np.float64)


def exact(case, seed):
    kind = case["kind"]
    if kind in ("thermo_device", "weights"):
        e, mult = _energies(case, seed)
        rec, p = _thermo_record(e, mult, case["temperature"])
        return np.array(list(rec.values())) if kind == "thermo_device" else {"weights": p, "thermo": rec}
    if kind == "ensemble":
        # sorted by energy (equal energies in input order), then every chromosome within 0.1 of the
        # last one kept, on every gene, dropped
        ic, e = _ensemble_inputs(case, seed)
        order = np.argsort(e, kind="stable")
        rows = ic[order]
        same = np.concatenate([[False], (rows[1:] == rows[:-1]).all(1)])
        kept, last = [], None
        for p in np.flatnonzero(~same):
            if last is None or not (np.abs(rows[p] - last) < 0.1).all():
                kept.append(p)
                last = rows[p]
        index, energy = np.full(case["n"], -1, np.int64), np.zeros(case["n"])
        index[:len(kept)], energy[:len(kept)] = order[kept], e[order[kept]]
        return {"index": index, "energy": energy}
    return None
