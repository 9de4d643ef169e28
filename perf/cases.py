"""The calls a program makes of this library, at the sizes it makes them.

Six kinds of call, each through the public entry points of `gpu`, `avalanche`,
`ensemble` and `adjoint`:

  run       whole kinetic steps over resident tiles: stage the tiles, advance
            them (transport phases, newborn FIFO, commit, compaction, and
            with feedback the field or the coupled carrier fluid), fetch them
  apply     the drop-in step on host tiles (rrea_gpu_apply_step): what an
            overlay calls once per step
  photons   a photon tile on its own: the phase and the newborn legs of its
            secondaries
  fluid     the coupled carrier-fluid + Maxwell update of a field grid
  field     the Maxwell update of a field grid and the particle diagnostics
            beside it (charge grid, census)
  ensemble  the batched uniform-field instances, stepped to their ends
  adjoint   the pathwise field gradient (forward and reverse)

Geometries, distributions and step are those of `workloads` and the
benchmark; every array comes from the seed.  A pass starts from the same
staged inputs each time, so a state can be run again.  Grids cross to and
from the host through the C-ABI into buffers the program keeps, as an overlay
does; outputs whose number depends on the run come in buffers of a fixed
size, zero behind the last one.
"""
import ctypes
import math

import numpy as np
import torch

from rrea_feedback_warpx_amrex_geant4_gb300 import DEFAULT_CLOSURE, DEFAULT_TABLES, adjoint, avalanche, ensemble, gpu
from rrea_feedback_warpx_amrex_geant4_gb300 import workloads

DT_S = 5.0e-10
CORE = ("r", "z", "theta", "ux", "uy", "uz")
FETCHED = CORE + ("w", "id")
QE = 1.602176634e-19

# Arithmetic one particle cannot do without in one step, in FP64 operations
# (a multiply-add counts two): a handful of substeps of chord, field work,
# two half kicks, table drag, one hazard draw and one elastic deflection for
# the charged species; one flight and on average less than one interaction
# for photons; a charged substep without discrete events in the adjoint.
FLOPS_CHARGED = 5 * 900.0
FLOPS_PHOTON = 700.0
FLOPS_ADJOINT_SUBSTEP = 300.0
FLOPS_FLUID_CELL = 400.0
FLOPS_MAXWELL_CELL = 40.0


def listed():
    return [
        # the plain uniform-field case at its own seed count: every kernel is
        # a fraction of a wave, so latency and launches count
        dict(name="run_c0_10k", kind="run", grid="uniform_c0", electrons=10_000, photons=4_000, positrons=6, steps=4,
             feedback="none", cap=0, target=0),
        # the scale-up case early in its run: its 1e5 seeds with the field
        # following through the coupled carrier fluid
        dict(name="run_scaleup_100k", kind="run", grid="scaleup_c1", electrons=100_000, photons=50_001,
             positrons=6_251, steps=2, feedback="fluid", cap=0, target=0),
        # the benchmark's population: 2^21 e-, half as many photons and a
        # sixteenth as many e+, coupled fluid and field
        dict(name="run_scaleup_2m", kind="run", grid="scaleup_c1", electrons=1 << 21, photons=1 << 20,
             positrons=1 << 17, steps=2, feedback="fluid", cap=0, target=0),
        # the profiled atmosphere's 512 x 4096 grid, density profile bound,
        # an entering column of e- and e+ with the kinetic field feedback
        dict(name="run_profiled_400k", kind="run", grid="profiled_c2", electrons=400_000, photons=0,
             positrons=100_003, steps=2, feedback="field", cap=0, target=0),
        # a run held at its macroparticle cap: the weight-doubling merge
        # after every commit, an odd population
        dict(name="run_capped_300k", kind="run", grid="scaleup_c1", electrons=300_007, photons=60_013,
             positrons=9_001, steps=2, feedback="none", cap=250_000, target=0),
        # the drop-in step over small host tiles: the smallest call
        dict(name="apply_2k", kind="apply", grid="scaleup_c1", electrons=2_311, photons=1_155, positrons=144),
        # and over ordinary ones, odd in every species (chunked upload)
        dict(name="apply_600k", kind="apply", grid="scaleup_c1", electrons=600_011, photons=300_005,
             positrons=37_500),
        # photons alone, 50 keV to 100 MeV, with their newborn legs
        dict(name="photons_1m", kind="photons", grid="scaleup_c1", photons=1_000_003),
        # the coupled fluid + field update of the scale-up grid, no particles
        dict(name="fluid_256x2048", kind="fluid", nr=256, nz=2048, steps=8),
        # the field update of the largest grid with the diagnostics of a
        # 5e5-particle tile
        dict(name="field_512x4096", kind="field", nr=512, nz=4096, steps=10, particles=500_009),
        # twelve batched uniform-field instances run to their ends
        dict(name="ensemble_12", kind="ensemble", instances=12, scale=0.003),
        # one field gradient: 1e5 electrons, 96 steps in 4 substeps
        dict(name="adjoint_100k", kind="adjoint", electrons=100_003, steps=96, nodes=256),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["run", "run", "run", "apply", "apply", "photons", "fluid", "field", "ensemble", "adjoint"])
    if kind == "run":
        grid = rng.choice(["uniform_c0", "scaleup_c1", "scaleup_c1", "profiled_c2"])
        n = _log(rng, 1_000, 1_500_000)
        steps = rng.randint(1, 4) if n < 300_000 else rng.randint(1, 2)
        feedback = rng.choice(["none", "field", "field" if grid == "profiled_c2" else "fluid"])
        # a controlled run sheds what one step added: the thinning target sits
        # just below the population, for the plain case's small ones
        control = rng.choice(["none", "none", "cap", "target" if grid == "uniform_c0" and n < 40_000 else "cap"])
        return dict(kind=kind, grid=grid, electrons=n, photons=int(n * rng.uniform(0.0, 0.5)),
                    positrons=int(n * rng.uniform(0.0, 0.2 if grid == "profiled_c2" else 0.0625)), steps=steps,
                    feedback=feedback, cap=int(0.8 * n) if control == "cap" else 0,
                    target=int(0.995 * n) if control == "target" else 0)
    if kind == "apply":
        n = _log(rng, 1_000, 1_200_000)
        return dict(kind=kind, grid=rng.choice(["uniform_c0", "scaleup_c1"]), electrons=n,
                    photons=int(n * rng.uniform(0.0, 0.5)), positrons=int(n * rng.uniform(0.0, 0.0625)))
    if kind == "photons":
        return dict(kind=kind, grid=rng.choice(["uniform_c0", "scaleup_c1"]), photons=_log(rng, 2_000, 2_000_000))
    if kind == "fluid":
        return dict(kind=kind, nr=_log(rng, 24, 512), nz=_log(rng, 40, 3000), steps=rng.randint(2, 8))
    if kind == "field":
        return dict(kind=kind, nr=_log(rng, 24, 512), nz=_log(rng, 40, 4096), steps=rng.randint(2, 10),
                    particles=_log(rng, 1_000, 1_000_000))
    if kind == "ensemble":
        return dict(kind=kind, instances=rng.randint(2, 14), scale=round(rng.uniform(0.001, 0.003), 5))
    return dict(kind=kind, electrons=_log(rng, 1_000, 100_000), steps=rng.randint(17, 96),
                nodes=rng.choice([64, 129, 256, 400]))


# ---------------------------------------------------------------- inputs
def _tile(n, k, r, theta, z, mu, phi):
    s = np.sqrt(1.0 - mu * mu)
    u = workloads.proper_velocity(k)
    t = {"r": r, "z": z, "theta": theta, "ux": u * s * np.cos(phi), "uy": u * s * np.sin(phi), "uz": u * mu,
         "w": np.ones(n), "id": np.arange(1, n + 1, dtype=np.int64), "cpu": np.zeros(n, dtype=np.int32)}
    for f in CORE:
        t[f] = np.ascontiguousarray(t[f], dtype=np.float64)
        t["prev_" + f] = t[f].copy()
    return t


def _charged(grid, n, seed):
    """A charged tile of the grid's workload.  In the uniform-field case a
    run's particles have spread along the axis (its seeds all start at one
    point with one energy); the scale-up case's own seed distribution; and
    the profiled case's entering column (K from E^-1.5 on 1-100 MeV, zenith
    density ~ cos^2)."""
    rng = np.random.default_rng(seed)
    if grid == "scaleup_c1":
        return workloads.make_electrons(grid, n, seed=seed)
    theta = rng.uniform(-np.pi, np.pi, n)
    phi = rng.uniform(0.0, 2.0 * np.pi, n)
    if grid == "profiled_c2":
        a = -0.5
        k = (1.0e6 ** a + rng.uniform(0.0, 1.0, n) * (1.0e8 ** a - 1.0e6 ** a)) ** (1.0 / a)
        r = 1000.0 * np.sqrt(rng.uniform(0.0, 0.98, n))
        z = 6000.0 - 10.0 * rng.uniform(0.0, 1.0, n)
        return _tile(n, k, r, theta, z, -rng.uniform(0.0, 1.0, n) ** (1.0 / 3.0), phi)
    k = np.minimum(1.2e4 + rng.exponential(7.0e6, n), 1.0e8)
    r = np.minimum(np.abs(rng.normal(0.0, 2.0, n)), 49.0)
    return _tile(n, k, r, theta, rng.uniform(0.0, 60.0, n), 1.0 - 0.3 * rng.uniform(0.0, 1.0, n) ** 2, phi)


def _photons(grid, n, seed, e_hi=1.0e8):
    t = workloads.make_photons(grid, n, DT_S, seed=seed, e_lo=5.0e4, e_hi=e_hi)
    return t


def _at_start(photons):
    """Resident photons are staged where they are: the step pushes them."""
    for f in ("r", "z", "theta"):
        photons[f][:] = photons["prev_" + f]
    return photons


def _context(grid, capacity, seed):
    ctx = gpu.RreaGpuContext(workloads.make_config(gpu, grid, rng_seed=1 + seed % 1_000_003), capacity)
    ctx.load_tables(DEFAULT_TABLES)
    if grid == "profiled_c2":
        alt, dens, alt0, field = workloads.profiled_atmosphere()
        ctx.set_density_profile(alt, dens, alt0, workloads.TABLE_DENSITY)
    else:
        field = workloads.make_field(grid)
    ctx.set_field(**field)
    ctx.set_launch(128, 16, diagnostics=False)
    return ctx, field


def _pointers(arrays):
    return [a.ctypes.data_as(ctypes.POINTER(ctypes.c_double)) if a is not None else None for a in arrays]


def _call(ctx, name, *arrays):
    """One C-ABI call of the context over host arrays."""
    ctx._check(getattr(ctx.lib, name)(ctx.handle, *_pointers(arrays)))


def _buffers(n):
    b = {f: np.zeros(n) for f in FETCHED[:-1]}
    b["id"] = np.zeros(n, dtype=np.int64)
    b["cpu"] = np.zeros(n, dtype=np.int32)
    for f in CORE:
        b["prev_" + f] = b[f]
    return b


def _tile_buffers(n_e, n_g, n_p):
    """Room for the tiles after a few steps' births."""
    return [_buffers(n_e + n_e // 4 + n_g // 8 + 16_384), _buffers(n_g + n_e // 4 + 16_384),
            _buffers(n_p + n_e // 32 + n_g // 16 + 16_384)]


RECORD_KEYS = ("species", "process", "parent_index", "root_key", "lineage")
RECORD_REALS = ("x", "y", "z", "dir_x", "dir_y", "dir_z", "weight", "energy_eV", "birth_fraction")


def _record_buffers(n):
    return dict(keys=np.zeros((len(RECORD_KEYS), n), dtype=np.int64), reals=np.zeros((len(RECORD_REALS), n)), n=0)


def _grid_buffers(cfg):
    nr, nz = cfg.nr, cfg.nz
    return dict(field=[np.zeros((nr + 1) * nz), np.zeros(nr * (nz + 1)), np.zeros((nr + 1) * (nz + 1))],
                current=[np.zeros((nr + 1) * nz), np.zeros(nr * (nz + 1))], sources=np.zeros(5 * nr * nz),
                fluid=[np.zeros(nr * nz) for _ in range(5)])


def _grid_field(nr, nz, rng):
    er = rng.normal(0.0, 2.0e3, (nz, nr + 1))
    er[:, 0] = 0.0
    bt = rng.normal(0.0, 1.0e-6, (nz + 1, nr + 1))
    bt[:, 0] = 0.0
    return dict(er=er.ravel(), ez=rng.normal(0.0, 2.0e3, nr * (nz + 1)), bt=bt.ravel(),
                amb_er=np.zeros((nr + 1) * nz), amb_ez=np.full(nr * (nz + 1), -5.0e5))


def _grid_config(nr, nz, seed):
    # cells of the scale-up grid: 0.78 m x 0.98 m
    return gpu.default_config(r_hi=200.0 / 256 * nr, z_lo=0.0, z_hi=2000.0 / 2048 * nz, nr=nr, nz=nz,
                              rng_seed=1 + seed % 1_000_003)


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("run", "apply", "photons"):
        grid = case["grid"]
        n_e, n_g, n_p = (int(case.get(s, 0)) for s in ("electrons", "photons", "positrons"))
        capacity = max(n_e, n_g, n_p) + max(n_e, n_g, n_p) // 4 + 65_536
        ctx, field = _context(grid, capacity, seed)
        tiles = [_charged(grid, n_e, seed + 1), _photons(grid, n_g, seed + 2), _charged(grid, n_p, seed + 3)]
        s = dict(case=case, ctx=ctx, field=field, tiles=tiles)
        if kind == "apply":
            s["restore"] = ([{"id": t["id"].copy()} for t in tiles])
            s["restore"][1].update({f: tiles[1][f].copy() for f in CORE})
        else:
            _at_start(tiles[1])
            s["out"] = _tile_buffers(n_e, n_g, n_p)
        s["records"] = _record_buffers((n_e + n_g + n_p) // 4 + 8_192)
        s["grids"] = _grid_buffers(ctx.config)
        if case.get("feedback") == "fluid":
            ctx.fluid_configure(**workloads.fluid_overrides())
            ctx.fluid_load_closure(DEFAULT_CLOSURE)
            s["empty"] = np.zeros(ctx.config.nr * ctx.config.nz)
        return s
    if kind in ("fluid", "field"):
        nr, nz = int(case["nr"]), int(case["nz"])
        rng = np.random.default_rng(seed)
        cfg = _grid_config(nr, nz, seed)
        n = int(case.get("particles", 16))
        ctx = gpu.RreaGpuContext(cfg, n)
        s = dict(case=case, ctx=ctx, field=_grid_field(nr, nz, rng), grids=_grid_buffers(cfg))
        if kind == "fluid":
            ctx.fluid_configure(**workloads.fluid_overrides())
            ctx.fluid_load_closure(DEFAULT_CLOSURE)
            i, j = np.arange(nr * nz) % nr, np.arange(nr * nz) // nr
            # carriers and ionization along the axis behind an avalanche
            blob = np.exp(-(i * 4.0 / nr) ** 2 - ((j - 0.4 * nz) * 4.0 / nz) ** 2)
            ne, pos = (1.0e12 * blob * rng.uniform(0.5, 1.5, nr * nz) for _ in range(2))
            neg = 0.3e12 * blob * rng.uniform(0.5, 1.5, nr * nz)
            s["fluid"] = [pos, neg, ne, QE * (pos - neg - ne)]
            s["rates"] = [a * blob * rng.uniform(0.0, 1.0, nr * nz) for a in (1.0e20, 1.0e20, 1.0e18)]
            return s
        k = np.exp(rng.uniform(np.log(1.0e4), np.log(1.0e8), n))
        t = _tile(n, k, cfg.r_hi * rng.uniform(0.0, 0.999, n) ** 2, rng.uniform(-np.pi, np.pi, n),
                  cfg.z_hi * rng.uniform(0.0, 0.999, n), rng.uniform(-1.0, 1.0, n), rng.uniform(0.0, 2.0 * np.pi, n))
        t["w"][:] = rng.uniform(0.5, 3.0, n)
        s["tile"] = t
        s["edges"], s["thresholds"] = avalanche.SPECTRUM_EDGES_EV, avalanche.THRESHOLDS_EV
        return s
    if kind == "ensemble":
        inst = ensemble.batched_instances(int(case["instances"]), duration_scale=float(case["scale"]))
        total = sum(i.n_seeds for i in inst)
        return dict(case=case, run=ensemble.EnsembleRun(inst, capacity=2 * total + 65_536, rng_seed=1 + seed % 1_000_003),
                    seeds=ensemble.seed_tile(inst), empty=workloads.make_electrons(ensemble.CASE, 0))
    n, nodes = int(case["electrons"]), int(case["nodes"])
    rng = np.random.default_rng(seed)
    k = np.exp(rng.uniform(np.log(3.0e5), np.log(2.0e7), n))
    mu = rng.uniform(0.6, 1.0, n)
    phi = rng.uniform(0.0, 2.0 * np.pi, n)
    sn = np.sqrt(1.0 - mu * mu)
    seeds = dict(z=rng.uniform(0.0, 5.0, n), dir=np.stack([sn * np.cos(phi), sn * np.sin(phi), mu], 1), k=k,
                 w=rng.uniform(0.5, 2.0, n), id=np.arange(1, n + 1, dtype=np.uint64))
    cfg = adjoint.default_config(steps=int(case["steps"]), n_nodes=nodes, k_threshold_eV=8.0e6, z_plane_m=12.0,
                                 density_ratio=workloads.AIR_DENSITY / workloads.TABLE_DENSITY,
                                 rng_seed=1 + seed % 1_000_003)
    prob = adjoint.PushAdjoint(cfg, seeds)
    e = torch.tensor(adjoint.adjoint_field_profile(n_nodes=nodes, z_hi=cfg.z_hi, seed=seed % 1_000_003),
                     dtype=torch.float64, device="cuda")
    return dict(case=case, prob=prob, nodes=e)


# ---------------------------------------------------------------- a pass
def _fetch(ctx, species, fetch, buf):
    n = ctx.resident_count(species)
    fetch({f: a[:n] for f, a in buf.items() if f != "n"})
    for f in FETCHED:
        buf[f][n:buf.get("n", n)] = 0
    buf["n"] = n
    return {f: buf[f] for f in FETCHED}


def _records(buf, sec):
    n = len(sec)
    for row, f in zip(buf["keys"], RECORD_KEYS):
        row[:n] = sec[f].view(np.int64) if f == "root_key" or f == "lineage" else sec[f]
    for row, f in zip(buf["reals"], RECORD_REALS):
        row[:n] = sec[f]
    for a in (buf["keys"], buf["reals"]):
        a[:, n:buf["n"]] = 0
    buf["n"] = n
    return {"keys": buf["keys"], "reals": buf["reals"], "n": n}


def _field(s):
    _call(s["ctx"], "rrea_gpu_download_field", *s["grids"]["field"])
    return s["grids"]["field"]


def _sources(s):
    _call(s["ctx"], "rrea_gpu_download_sources", s["grids"]["sources"])
    return s["grids"]["sources"]


def _fluid(s):
    # the relaxation time is 1/sigma scaled, without bound where sigma is small
    _call(s["ctx"], "rrea_gpu_fluid_get_state", *s["grids"]["fluid"], None)
    return s["grids"]["fluid"]


def _run_steps(s):
    case, ctx = s["case"], s["ctx"]
    feedback = case["feedback"]
    if feedback != "none":
        ctx.set_field(**s["field"])
    if feedback == "fluid":
        _call(ctx, "rrea_gpu_fluid_set_state", *[s["empty"]] * 4)
    run = avalanche.AvalancheRun(ctx, s["tiles"][0], photons=s["tiles"][1], positrons=s["tiles"][2],
                                 feedback=feedback != "none", fluid=feedback == "fluid",
                                 merge_cap=case["cap"] or None, population_target=case["target"] or None)
    moved = 0
    for _ in range(case["steps"]):
        moved += run.advance(DT_S)[0]
    out = {"moved": moved, "sources": _sources(s)}
    for name, sp, fetch, buf in (("electrons", gpu.SPECIES_ELECTRON, ctx.fetch_electrons, s["out"][0]),
                                 ("photons", gpu.SPECIES_PHOTON, ctx.fetch_photons, s["out"][1]),
                                 ("positrons", gpu.SPECIES_POSITRON, ctx.fetch_positrons, s["out"][2])):
        out[name] = _fetch(ctx, sp, fetch, buf)
    if feedback != "none":
        out["field"] = _field(s)
    if feedback == "fluid":
        out["fluid"] = _fluid(s)
    return out


def _run_apply(s):
    ctx, tiles = s["ctx"], s["tiles"]
    # the overlay gathers its tiles anew each step: ids, and the photons'
    # pushed end points (a charged phase starts from the captured prev_*)
    for t, keep in zip(tiles, s["restore"]):
        for f, a in keep.items():
            np.copyto(t[f], a)
    ctx.reset_current()
    ctx.reset_sources()
    surv = ctx.apply_step(tiles[0], tiles[1], tiles[2], 1, DT_S)
    _call(ctx, "rrea_gpu_download_current", *s["grids"]["current"])
    return {"tiles": [{f: t[f] for f in CORE + ("id",)} for t in tiles], "survivors": _records(s["records"], surv),
            "current": s["grids"]["current"], "sources": _sources(s)}


def _run_photons(s):
    ctx = s["ctx"]
    ctx.reset_sources()
    ctx.stage_photons(s["tiles"][1])
    ctx.step_photons_resident(1, DT_S)
    ctx.drain_resident(1, DT_S)
    surv = ctx.fetch_survivors()
    return {"photons": _fetch(ctx, gpu.SPECIES_PHOTON, ctx.fetch_photons, s["out"][1]),
            "survivors": _records(s["records"], surv), "sources": _sources(s)}


def _run_fluid(s):
    ctx = s["ctx"]
    ctx.set_field(**s["field"])
    _call(ctx, "rrea_gpu_fluid_set_state", *s["fluid"])
    ctx.reset_current()
    for _ in range(s["case"]["steps"]):
        _call(ctx, "rrea_gpu_fluid_set_source_rates", *s["rates"])
        diag = ctx.advance_field_coupled(DT_S)
    return {"field": _field(s), "fluid": _fluid(s), "substeps": int(diag["substeps"])}


def _run_field(s):
    ctx = s["ctx"]
    ctx.set_field(**s["field"])
    ctx.reset_current()
    for _ in range(s["case"]["steps"]):
        ctx.advance_field(DT_S, 2)
    ctx.stage_electrons(s["tile"])
    return {"field": _field(s), "charge": ctx.deposit_charge(),
            "census": ctx.census(gpu.SPECIES_ELECTRON, s["edges"], s["thresholds"])}


def _run_ensemble(s):
    run = s["run"]
    run.ctx.stage_electrons(s["seeds"])
    run.ctx.stage_photons(s["empty"])
    run.ctx.stage_positrons(s["empty"])
    run.step, run.results, run.active = 0, {}, list(range(len(run.instances)))
    res = run.run()["results"]
    return {"electron_count": np.array([r["electron_count"] for r in res]),
            "photon_count": np.array([r["photon_count"] for r in res]),
            "multiplication": np.array([r["multiplication"] for r in res]),
            "weights": np.array([[r["electron_weight"], r["photon_weight"], r["positron_weight"]] for r in res]),
            "electrons": np.stack([r["spectra"]["electron"] for r in res]),
            "photons": np.stack([r["spectra"]["photon"] for r in res])}


def _run_adjoint(s):
    loss = s["prob"].forward(s["nodes"])
    grad = s["prob"].backward(s["nodes"])
    return {"loss": loss, "grad": grad, "state": s["prob"].final_state()}


def run(state):
    return {"run": _run_steps, "apply": _run_apply, "photons": _run_photons, "fluid": _run_fluid, "field": _run_field,
            "ensemble": _run_ensemble, "adjoint": _run_adjoint}[state["case"]["kind"]](state)


# ---------------------------------------------------------------- what a pass needs
def _grid_of(case):
    p = workloads.CASES[case["grid"]]
    return p["nr"] * p["nz"]


def work(case):
    kind = case["kind"]
    if kind in ("run", "apply", "photons"):
        n_c = case.get("electrons", 0) + case.get("positrons", 0)
        n_g = case.get("photons", 0)
        steps = case.get("steps", 1)
        cells = _grid_of(case)
        # a particle's state read and written every step, the sources and
        # current grids, and with feedback the field and fluid grids
        b = 112.0 * (n_c + n_g) * steps + 8.0 * 7 * cells
        f = steps * (FLOPS_CHARGED * n_c + FLOPS_PHOTON * n_g)
        if case.get("feedback", "none") != "none":
            b += 8.0 * 10 * cells * steps
            f += 2 * FLOPS_MAXWELL_CELL * cells * steps
        if case.get("feedback") == "fluid":
            b += 8.0 * 16 * cells * steps
            f += 2 * FLOPS_FLUID_CELL * cells * steps
        return {"bytes": b, "flops": f}
    if kind == "fluid":
        cells = case["nr"] * case["nz"]
        return {"bytes": 8.0 * 26 * cells * case["steps"],
                "flops": 2.0 * (FLOPS_FLUID_CELL + FLOPS_MAXWELL_CELL) * cells * case["steps"]}
    if kind == "field":
        cells = case["nr"] * case["nz"]
        return {"bytes": 8.0 * 10 * cells * case["steps"] + 72.0 * case["particles"],
                "flops": 2.0 * FLOPS_MAXWELL_CELL * cells * case["steps"] + 60.0 * case["particles"]}
    if kind == "ensemble":
        inst = ensemble.batched_instances(int(case["instances"]), duration_scale=float(case["scale"]))
        moved = float(sum(i.n_seeds * i.steps for i in inst))
        return {"bytes": 112.0 * moved, "flops": FLOPS_CHARGED * moved}
    substeps = float(case["electrons"]) * case["steps"] * 4
    # forward, then recomputation and adjoint of every substep
    return {"bytes": 2 * 48.0 * case["electrons"] * (2 + case["steps"] / 32.0),
            "flops": 3.0 * FLOPS_ADJOINT_SUBSTEP * substeps}


# ---------------------------------------------------------------- in 64 bits, by numpy
def _maxwell(nr, nz, dr, dz, dt, substeps, er, ez, bt):
    """The TM-RZ leapfrog with zero current: B restaggered by (dt - dts)/2,
    per substep B, Silver-Mueller, E, then B restaggered back."""
    c, eps0, mu0 = 299792458.0, 8.8541878128e-12, 1.25663706212e-6
    er, ez, bt = er.reshape(nz, nr + 1).copy(), ez.reshape(nz + 1, nr).copy(), bt.reshape(nz + 1, nr + 1).copy()

    def advance_b(h):
        if nr > 1 and nz > 1:
            bt[1:-1, 1:-1] += h * ((ez[1:-1, 1:] - ez[1:-1, :-1]) / dr - (er[1:, 1:-1] - er[:-1, 1:-1]) / dz)

    def open_faces():
        bt[:, nr] = -ez[:, nr - 1] / c
        bt[0, :] = -er[0, :] / c
        bt[nz, :] = er[nz - 1, :] / c
        bt[:, 0] = 0.0

    def advance_e(h):
        c2 = h / (eps0 * mu0)
        er[:, 1:] += -c2 * (bt[1:, 1:] - bt[:-1, 1:]) / dz
        er[:, 0] = 0.0
        i = np.arange(nr)
        ez[:, :] += c2 * ((i + 1) * bt[:, 1:] - i * bt[:, :-1]) / ((i + 0.5) * dr)

    dts = dt / substeps
    advance_b(0.5 * (dt - dts))
    for _ in range(substeps):
        advance_b(dts)
        open_faces()
        advance_e(dts)
    advance_b(-0.5 * (dt - dts))
    open_faces()
    return er.ravel(), ez.ravel(), bt.ravel()


def _charge(cfg, t):
    """Cell-centred CIC charge: folded at the axis, clamped at the edges."""
    nr, nz = cfg.nr, cfg.nz
    fr = t["r"] / (cfg.r_hi / nr) - 0.5
    fz = t["z"] / (cfg.z_hi / nz) - 0.5
    i0, j0 = np.floor(fr).astype(np.int64), np.floor(fz).astype(np.int64)
    tr, tz = fr - i0, fz - j0
    out = np.zeros(nr * nz)
    for a, wr in ((0, 1.0 - tr), (1, tr)):
        for b, wz in ((0, 1.0 - tz), (1, tz)):
            i = np.clip(i0 + a, 0, nr - 1)
            j = np.clip(j0 + b, 0, nz - 1)
            out += np.bincount(i + nr * j, weights=-t["w"] * wr * wz, minlength=nr * nz)
    return out.reshape(nz, nr)


def exact(case, seed):
    """Only the field update and the diagnostics beside it have a plain
    numpy form; the stochastic transport, the closure fluid and the gradient
    need the physics tables and their samplers."""
    if case["kind"] != "field":
        return None
    nr, nz = int(case["nr"]), int(case["nz"])
    rng = np.random.default_rng(seed)
    cfg = _grid_config(nr, nz, seed)
    f = _grid_field(nr, nz, rng)
    n = int(case["particles"])
    k = np.exp(rng.uniform(np.log(1.0e4), np.log(1.0e8), n))
    t = _tile(n, k, cfg.r_hi * rng.uniform(0.0, 0.999, n) ** 2, rng.uniform(-np.pi, np.pi, n),
              cfg.z_hi * rng.uniform(0.0, 0.999, n), rng.uniform(-1.0, 1.0, n), rng.uniform(0.0, 2.0 * np.pi, n))
    t["w"][:] = rng.uniform(0.5, 3.0, n)
    er, ez, bt = f["er"], f["ez"], f["bt"]
    for _ in range(case["steps"]):
        er, ez, bt = _maxwell(nr, nz, cfg.r_hi / nr, cfg.z_hi / nz, DT_S, 2, er, ez, bt)
    ke = workloads.kinetic_energy(t["ux"], t["uy"], t["uz"])
    w, edges, thr = t["w"], avalanche.SPECTRUM_EDGES_EV, avalanche.THRESHOLDS_EV
    inside = (ke >= edges[0]) & (ke < edges[-1])
    hist = np.bincount(np.searchsorted(edges, ke[inside], side="right") - 1, weights=w[inside],
                       minlength=len(edges) - 1)
    census = {"count": n, "max_weight": float(w.max()), "sum_w": float(w.sum()), "sum_w2": float((w * w).sum()),
              "sum_wk": float((w * ke).sum()), "under": float(w[ke < edges[0]].sum()),
              "over": float(w[ke >= edges[-1]].sum()), "above": np.array([w[ke >= x].sum() for x in thr]),
              "hist": hist}
    return {"field": [er, ez, bt], "charge": _charge(cfg, t), "census": census}
