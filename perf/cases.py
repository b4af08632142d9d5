"""The work that users of the framework have it do, as cases to be timed.

A case is a dict of plain values; `listed` has the named ones, `draw` more of
the same ranges.  Three kinds, each through the package's public entry points:

shower     primaries transported to completion: `transport` (device tensors),
           `transport_host` (host arrays), with the beam-spot gun in front
           where the primaries are generated on the device;
stages     one step of a host-driven loop over a batch of tracks in flight:
           `gpil`, `propagate`, `along_step`, `post_step`;
functions  the reference's per-track functions called one by one on a batch:
           streams and draws, tables, step limits, losses, the helix;
models     interaction sampling, a batch for each of the reference's models.

The sizes and set-ups are those of geantexascalepilot_b200/configs.py, the
tests and bench.py, from a smoke-sized call to the full batch.
"""
import math

import numpy as np
import torch

import geantexascalepilot_b200 as gx
from geantexascalepilot_b200 import api, geometry

GAMMA, ELECTRON, POSITRON = 0, 1, 2
M1, M2 = 4294967087, 4294944443  # the two moduli of MRG32k3a
KB2C = -0.299792458e-3           # GeV / kilogauss / cm, the helix stepper's default

# track-steps per MeV of primary energy, and floating-point operations a step
# cannot do without (cross sections, step limit, move, loss), for work()
STEPS_PER_MEV, FLOPS_PER_STEP = 5.8, 250.0


def listed():
    return [
        # a smoke test or a single event: the call's latency is what counts
        _shower("two_electrons_fp64", n=2, beam="electron", energy=1000.0, field=0.0, precision=0),
        # photons of a source in a lead block, FP64, step count of each primary
        _shower("photons_in_lead_fp64", n=10000, beam="gamma", energy=10.0, field=0.0, precision=0, geometry="box",
                primary_steps=True),
        # test-beam electrons in the calorimeter, FP64 reference run
        _shower("calorimeter_fp64", n=10000, beam="electron", energy=1000.0, field=0.0, precision=0),
        # one bunch of 10 GeV e- and photons in the 4 T calorimeter: a small batch, an odd number
        _shower("field_batch_61", n=61, beam="electron+gamma", energy=10000.0),
        # the same at the size of a production batch
        _shower("field_batch_20000", n=20000, beam="electron+gamma", energy=10000.0),
        # a beam spot with a continuous spectrum, generated on the device and transported
        _shower("beam_spot_16384", n=16384, beam="spot", energy=1.0e5),
        # events of about 100 primaries handed over from the host, scored per event and layer
        _shower("host_events_256", n=25600, beam="electron", energy=10000.0, events=256, host=True),
        # the calorimeter as a volume tree, as a detector description gives it
        _shower("volume_tree_1001", n=1001, beam="electron+gamma", energy=10000.0, geometry="tree"),
        # multiple scattering with lateral displacement
        _shower("scattering_3000", n=3000, beam="electron", energy=1000.0, msc=2),
        # a host's own step loop over the tracks in flight
        {"name": "stages_100003", "kind": "stages", "n": 100003, "field": 4.0},
        # the per-track functions on a batch
        {"name": "functions_300007", "kind": "functions", "n": 300007, "draws": 8},
        # interaction sampling on a batch
        {"name": "models_200003", "kind": "models", "n": 200003},
    ]


def _shower(name, n, beam, energy, field=4.0, precision=1, geometry="layers", events=1, msc=0, host=False,
            primary_steps=False):
    c = {"kind": "shower", "n": n, "beam": beam, "energy": energy, "field": field, "precision": precision,
         "geometry": geometry, "events": events, "msc": msc, "host": host, "primary_steps": primary_steps}
    return dict(c, name=name) if name else c


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["field", "field", "fp64", "box", "spot", "events", "tree", "scattering", "stages", "functions",
                       "models"])
    if kind == "stages":
        return {"kind": kind, "n": size(1000, 400000), "field": rng.choice([0.0, 4.0])}
    if kind == "functions":
        return {"kind": kind, "n": size(1000, 600000), "draws": rng.randint(1, 16)}
    if kind == "models":
        return {"kind": kind, "n": size(1000, 400000)}
    energy = round(math.exp(rng.uniform(math.log(100.0), math.log(2.0e4))), 3)
    # primaries up to a total energy (MeV) that keeps a pass below the largest listed one
    upto = lambda total: max(2, min(20000, int(total / energy)))  # noqa: E731
    if kind == "box":
        return _shower(None, n=size(2, 20000), beam="gamma", energy=round(rng.uniform(1.0, 20.0), 3), field=0.0,
                       precision=rng.choice([0, 0, 1]), geometry="box", primary_steps=rng.random() < 0.5)
    if kind == "fp64":
        return _shower(None, n=size(1, upto(2.0e7)), beam=rng.choice(["electron", "electron+gamma"]), energy=energy,
                       field=rng.choice([0.0, 4.0]), precision=0)
    if kind == "spot":
        return _shower(None, n=size(32, 16384), beam="spot", energy=rng.choice([1.0e4, 1.0e5]))
    if kind == "events":
        ev = size(2, 256)
        return _shower(None, n=ev * rng.randint(20, 100), beam="electron", energy=rng.choice([1000.0, 10000.0]),
                       events=ev, host=rng.random() < 0.5)
    if kind == "tree":
        return _shower(None, n=size(2, upto(2.0e7)), beam="electron+gamma", energy=energy, geometry="tree")
    if kind == "scattering":
        return _shower(None, n=size(2, upto(2.0e7)), beam="electron", energy=energy, field=rng.choice([0.0, 4.0]),
                       msc=rng.choice([1, 2]))
    return _shower(None, n=size(1, upto(2.0e8)), beam="electron+gamma", energy=energy)


# ------------------------------------------------------------------ prepare
_manager = None


def _data_manager():
    """The physics data: loaded once by a program and kept."""
    global _manager
    if _manager is None:
        _manager = gx.ProxyDataManager(device=0)
    return _manager


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) % (1 << 62))


def _uniform(g, n, lo, hi):
    return lo + (hi - lo) * torch.rand(n, generator=g, device="cuda", dtype=torch.float64)


def _directions(g, n):
    d = torch.randn((n, 3), generator=g, device="cuda", dtype=torch.float64)
    return d / d.norm(dim=1, keepdim=True)


def _stream_seed(seed):
    """Six MRG32k3a state words from a seed."""
    return [float(1 + (int(seed) * 7919 + k * 104729) % 4294944000) for k in range(6)]


def _config(case, seed):
    cfg = api.default_config()
    cfg.seed[:] = _stream_seed(seed)
    cfg.precision = case.get("precision", 0)
    cfg.Bz = case["field"]
    cfg.axis = 0 if case.get("beam") == "electron+gamma" or case["kind"] == "stages" else 2
    cfg.nevents = case.get("events", 1)
    cfg.msc = case.get("msc", 0)
    if case.get("geometry") == "box":
        cfg.geometry, cfg.axis, cfg.box_mat, cfg.charged_local = 0, 2, 1, 1
        cfg.box_half[:] = [50.0, 50.0, 50.0]
        cfg.box_centre[:] = [0.0, 0.0, 50.0]
    return cfg


def prepare(case, seed):
    if case["kind"] == "stages":
        return _prepare_stages(case, seed)
    if case["kind"] == "functions":
        return dict(_function_inputs(case, seed), case=case, dm=_data_manager())
    if case["kind"] == "models":
        return _prepare_models(case, seed)
    dm, n, cfg = _data_manager(), case["n"], _config(case, seed)
    s = {"case": case, "dm": dm, "cfg": cfg, "nvol": 1 if case["geometry"] == "box" else 100}
    if case["geometry"] == "tree":
        tree = geometry.calorimeter(nlayers=50, axis=cfg.axis)
        s["nvol"], s["tree"] = dm.load_geometry(tree), tree
        cfg.geometry = 2
    if case["beam"] == "spot":
        s["gun"] = dict(energy=(10.0, case["energy"]), seed=list(cfg.seed))
        return s
    if case["events"] > 1:
        # Poisson multiplicities with the case's mean, at least one primary
        mult = torch.poisson(torch.full((case["events"],), n / case["events"], device="cuda"),
                             generator=_generator(seed)).long().clamp_(min=1)
        s["events"] = torch.repeat_interleave(torch.arange(case["events"], device="cuda"), mult).int()
        n = s["events"].numel()
        _, E, pos, d = api.spot_gun(n, types=(ELECTRON,), energy=(case["energy"], case["energy"]), cone_deg=10.0,
                                    half=(0.0, 0.0), seed=list(cfg.seed))
        t = torch.full((n,), ELECTRON, dtype=torch.int32, device="cuda")
    else:
        t = torch.full((n,), GAMMA if case["beam"] == "gamma" else ELECTRON, dtype=torch.int32, device="cuda")
        if case["beam"] == "electron+gamma":
            t[n - n // 2:] = GAMMA
        E = torch.full((n,), case["energy"], dtype=torch.float64, device="cuda")
        pos, d = torch.zeros((2, n, 3), dtype=torch.float64, device="cuda")
        pos[:, cfg.axis] = 0.0 if case["geometry"] == "box" else -200.0
        d[:, cfg.axis] = 1.0
    s.update(types=t, E=E, pos=pos, dir=d)
    if case["host"]:
        for k in ("types", "E", "pos", "dir", "events"):
            if k in s:
                s[k] = s[k].cpu().pin_memory().numpy()
    return s


def _prepare_stages(case, seed):
    """Tracks of a developed shower, anywhere in the calorimeter."""
    n, g, cfg = case["n"], _generator(seed), _config(case, seed)
    t = api.TrackSoA(n)
    t.n = n
    t.type.copy_(torch.randint(0, 3, (n,), generator=g, device="cuda", dtype=torch.int32))
    t.primary.copy_(torch.arange(n, dtype=torch.int32))
    t.volume.fill_(-2)
    for f in ("x", "y", "z"):
        getattr(t, f).copy_(_uniform(g, n, -199.0, 199.0))
    d = _directions(g, n)
    for k, f in enumerate(("dx", "dy", "dz")):
        getattr(t, f).copy_(d[:, k])
    t.ekin.copy_(torch.exp(_uniform(g, n, math.log(0.1), math.log(1.0e4))))
    for f in ("nil0", "nil1", "nil2", "msc_range"):
        getattr(t, f).fill_(-1.0)
    t.rng.copy_(gx.MRG32k3a.substreams(list(cfg.seed), 0, n).view(-1))
    work = api.TrackSoA(n)
    work.n = n
    return {"case": case, "dm": _data_manager(), "cfg": cfg, "tracks": t, "work": work,
            "secondaries": api.TrackSoA(2 * n)}


def _function_inputs(case, seed):
    n, g = case["n"], _generator(seed)
    s = {"seed": _stream_seed(seed), "E": torch.exp(_uniform(g, n, math.log(0.01), math.log(1.0e5))),
         "mat": torch.randint(1, 3, (n,), generator=g, device="cuda", dtype=torch.int32)}
    s["pstep"] = _uniform(g, n, 0.0, 2.0)
    s["nil"] = _uniform(g, n, -0.2, 3.0)  # some are spent, to be drawn anew
    s["saved"] = _uniform(g, n, 1.0, 50.0)
    s["step"] = torch.exp(_uniform(g, n, math.log(1e-3), math.log(10.0)))
    s["pos"], s["dir"] = 100.0 * torch.randn((n, 3), generator=g, device="cuda", dtype=torch.float64), _directions(g, n)
    s["charge"] = 2.0 * torch.randint(0, 2, (n,), generator=g, device="cuda").double() - 1.0
    s["momentum"] = torch.exp(_uniform(g, n, math.log(1e-3), math.log(100.0)))
    return s


def _prepare_models(case, seed):
    n, g, dm = case["n"], _generator(seed), _data_manager()
    E = torch.exp(_uniform(g, n, math.log(0.1), math.log(1.0e4)))
    lead = dict(mode=api.MODE_PHYSICS, Z=82, density_factor=1.4e-8, sb_table=2)
    return {"case": case, "seed": _stream_seed(seed), "E": E, "pair_E": 1.1 + E, "dir": _directions(g, n),
            "models": [gx.ProxyKleinNishina(dm, **lead), gx.ProxySauterGavrila(dm, **lead),
                       gx.ProxyBetheHeitler(dm, **lead), gx.ProxySeltzerBerger(dm, cut=0.0949, **lead),
                       gx.ProxyMollerScattering(dm, cut=0.951, **lead)]}


# ---------------------------------------------------------------------- run
def run(state):
    return {"shower": _run_shower, "stages": _run_stages, "functions": _run_functions,
            "models": _run_models}[state["case"]["kind"]](state)


def _run_shower(s):
    c, ps = s["case"], None
    if c["host"]:
        edep, stats = api.transport_host(s["dm"], s["cfg"], s["types"], s["E"], s["pos"], s["dir"], s.get("events"),
                                         nvol=s["nvol"])
    else:
        if c["beam"] == "spot":
            prims = api.spot_gun(c["n"], **s["gun"])
        else:
            prims = s["types"], s["E"], s["pos"], s["dir"]
        edep, stats, ps = api.transport(s["dm"], s["cfg"], *prims, s.get("events"), nvol=s["nvol"],
                                        primary_steps=c["primary_steps"])
    return {"edep": edep, "primary_steps": ps, "escaped": stats["escaped"],
            "counts": [stats[k] for k in ("steps", "substeps", "tracks", "sec_gamma", "sec_electron", "sec_positron",
                                          "n_pair", "n_annih", "errors")]}


STAGE_INT = ("type", "status", "volume", "next_volume", "process", "boundary", "rng")
STAGE_DBL = ("x", "y", "z", "dx", "dy", "dz", "ekin", "nil0", "nil1", "nil2", "pstep", "step", "snext", "safety")


def _run_stages(s):
    t, sec = s["work"], s["secondaries"]
    fields = api.TrackSoA.INT_FIELDS + api.TrackSoA.DBL_FIELDS + ("rng",)
    torch._foreach_copy_([getattr(t, f) for f in fields], [getattr(s["tracks"], f) for f in fields])
    edep = torch.zeros((1, 100), dtype=torch.float64, device="cuda")
    api.gpil(s["dm"], s["cfg"], t)
    api.propagate(s["dm"], s["cfg"], t)
    api.along_step(s["dm"], s["cfg"], t, edep)
    api.post_step(s["dm"], s["cfg"], t, sec, edep)
    return {"edep": edep, "tracks": {f: getattr(t, f) for f in STAGE_INT + STAGE_DBL},
            "secondaries": {f: getattr(sec, f) for f in STAGE_INT + STAGE_DBL}}


def _run_functions(s):
    c, dm = s["case"], s["dm"]
    states = gx.MRG32k3a.substreams(s["seed"], 0, c["n"])
    draws = gx.MRG32k3a.uniform(states, c["draws"])
    tables = [dm.table_value(api.TABLES.index(t), 1, s["E"]) for t in ("Lambda.compt.gamma", "Range.eIoni.e-")]
    nil, saved = s["nil"].clone(), s["saved"].clone()
    limit = gx.ProxyCompton(dm).PostStepGPIL(s["E"], s["pstep"], nil, saved, states, mat=1)
    ioni = gx.ProxyIonization(dm)
    along = ioni.AlongStepGPIL(s["mat"], s["E"], mode=api.MODE_PHYSICS)
    loss = ioni.AlongStepDoIt(s["mat"], s["step"], s["E"], mode=api.MODE_PHYSICS)
    moved = gx.ConstFieldHelixStepper([0.0, 0.0, 40.0]).DoStepArr(s["pos"], s["dir"], s["charge"], s["momentum"],
                                                                  s["step"])
    return {"draws": draws, "states": states, "tables": tables, "limit": limit, "nil": nil, "saved": saved,
            "along": along, "loss": loss, "moved": moved}


def _run_models(s):
    n, out = s["case"]["n"], []
    for k, m in enumerate(s["models"]):
        states = gx.MRG32k3a.substreams(s["seed"], k * n, n)
        o = m.SampleSecondaries(s["pair_E"] if k == 2 else s["E"], s["dir"], states)
        out.append([o[f] for f in ("E", "dir", "edep", "status", "nsec", "sec_type", "sec_E", "sec_dir")] + [states])
    return out


# --------------------------------------------------------------------- work
def work(case):
    n, k = float(case["n"]), case["kind"]
    if k == "stages":
        # per track: 29 fields read and 25 written, and two secondaries' records written
        return {"bytes": n * (8 * 18 + 4 * 14) * 4.0, "flops": n * FLOPS_PER_STEP}
    if k == "functions":
        # states, draws, energies and the functions' own inputs and outputs
        return {"bytes": n * (24 + 8 * case["draws"] + 8 * 42), "flops": n * (30 * case["draws"] + 500)}
    if k == "models":
        # per model: energy, direction and stream in; final state, two secondaries and stream out
        return {"bytes": 5 * n * (32 + 48 + 32 + 16 + 16 + 8 + 64), "flops": 5 * n * 300}
    energy = case["energy"] / math.log(case["energy"] / 10.0) if case["beam"] == "spot" else case["energy"]
    per_mev = 0.5 if case["geometry"] == "box" else STEPS_PER_MEV
    return {"bytes": n * 68.0 + case["events"] * 100 * 8.0, "flops": n * energy * per_mev * FLOPS_PER_STEP}


# -------------------------------------------------------------------- exact
def _jump_host(k):
    """A^(2^(76 + b)) mod m of MRG32k3a's component k, for b = 0, 1, ..."""
    m = (M1, M2)[k]
    a = [[0, 1, 0], [0, 0, 1], [-810728, 1403580, 0] if k == 0 else [-1370589, 0, 527612]]
    b = 0
    while True:
        if b >= 76:
            yield a
        a = [[sum(a[i][j] * a[j][c] for j in range(3)) % m for c in range(3)] for i in range(3)]
        b += 1


def _substreams_host(seed, n):
    """The states of substreams 0 .. n - 1: a (6, n) array of whole numbers."""
    out = np.empty((6, n), np.uint64)
    idx = np.arange(n, dtype=np.uint64)
    for k in range(2):
        m = np.uint64((M1, M2)[k])
        v = [np.full(n, int(w), np.uint64) for w in seed[3 * k:3 * k + 3]]
        for b, a in zip(range(max(1, (n - 1).bit_length())), _jump_host(k)):
            on = (idx >> np.uint64(b)) & np.uint64(1) == 1
            old = [w[on] for w in v]
            for i in range(3):
                v[i][on] = sum((np.uint64(a[i][j]) * old[j]) % m for j in range(3)) % m
        out[3 * k:3 * k + 3] = v
    return out


def _draws_host(s, k):
    """k draws of each stream."""
    s, out = s.astype(np.int64), np.empty((k, s.shape[1]))
    for j in range(k):
        p1 = (1403580 * s[1] - 810728 * s[0]) % M1
        p2 = (527612 * s[5] - 1370589 * s[3]) % M2
        s = np.stack([s[1], s[2], p1, s[4], s[5], p2])
        out[j] = np.where(p1 > p2, p1 - p2, p1 - p2 + M1) / (M1 + 1.0)
    return out


def exact(case, seed):
    """The draws and the helix; sampled and tabulated values have no closed form."""
    if case["kind"] != "functions":
        return None
    s = _function_inputs(case, seed)
    draws = _draws_host(_substreams_host(s["seed"], case["n"]), case["draws"])
    B, d, step = 40.0, s["dir"], s["step"]
    radius = s["momentum"] / (KB2C * s["charge"] * B)  # of a track across the field, signed
    phi = -step / radius
    sin, cosm1 = torch.sin(phi), -2.0 * torch.sin(0.5 * phi) ** 2
    pos = s["pos"] + torch.stack([radius * (cosm1 * d[:, 1] - sin * d[:, 0]),
                                  radius * (-cosm1 * d[:, 0] - sin * d[:, 1]), step * d[:, 2]], 1)
    moved = torch.stack([d[:, 0] + cosm1 * d[:, 0] + sin * d[:, 1], d[:, 1] + cosm1 * d[:, 1] - sin * d[:, 0],
                         d[:, 2]], 1)
    return {"draws": torch.from_numpy(draws), "states": None, "tables": [None, None], "limit": None, "nil": None,
            "saved": None, "along": None, "loss": (None, None), "moved": (pos, moved)}
