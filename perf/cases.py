"""Performance cases of the spray update: what is timed, on which sizes.

Each case is one piece of work that a flow solver (or the program around it)
has this library do, through its public entry points:

* ``call`` -- one ``updateParticles`` call as a flow solver that keeps its own
  particle container makes it: describe the level (``set_geometry``,
  ``set_grids``), hand over every tile's droplets from device memory
  (``pmp_spray_set_particles``, the AMReX record or one array per component),
  ``pmp_spray_update``, ``pmp_spray_sync``, write the droplets back
  (``pmp_spray_get_particles``).  Gas state and sources are device arrays.
* ``step`` -- one time step with the droplets kept in the library:
  time-step estimate, moveKickDrift, moveKick, transferSource, re-binning, and
  the droplets read out for the step's output; ``views`` says whether the flow
  solver's arrays are in device memory or (a CPU flow solver) in page-locked
  host memory, where the sources are the result.
* ``fields`` -- the plot-file fields (computeDerivedVars) and the time-step
  estimate.
* ``train`` -- the learned form's surrogate trained for one pass over tuples
  labelled at the case's state (forward, backward and Adam).

Distributions are those of pelemp_b200/workloads.py: single-fuel n-heptane
droplets (median 20 um, 300 K) in 800-1000 K air, or two-fuel
n-decane / n-heptane droplets (median 15 um, 290-350 K) in a sinusoidal
temperature field; 1e-4 m cells, 3 ghost cells of state and 2 of source.

``exact`` restates the whole path (gather, droplet physics, deposits, move,
re-binning order) in plain 64-bit torch.
"""
import ctypes as C
import math

import torch

from pelemp_b200 import capi, spray, workloads

DX = 1e-4
STATE_GHOSTS, SOURCE_GHOSTS = 3, 2
MODES = {"fp64": capi.PMP_MODE_FP64, "mixed": capi.PMP_MODE_MIXED, "learned": capi.PMP_MODE_LEARNED}
DT = {1: 1e-6, 2: 5e-7}  # flow time step by fuel count (the configurations' own)
SPECIES = {1: ["N2", "O2", "NC7H16"], 2: ["N2", "O2", "NC10H22", "NC7H16", "CO2"]}
FUELS = {1: ["NC7H16"], 2: ["NC10H22", "NC7H16"]}
REF_T = {1: 300.0, 2: 298.15}
TUPLE_BYTES = 64


def _case(name, kind, n, boxes, box, **more):
    c = dict(name=name, kind=kind, n=n, nbx=boxes[0], nby=boxes[1], nbz=boxes[2], bx=box[0], by=box[1], bz=box[2],
             form="fp64", fuels=1, pelec=False, cfl=0.1, move=True, aos=True, uneven=False, views="device")
    c.update(more)
    return c


def listed():
    return [
        # a nearly empty level: call overhead and the latency of one droplet
        _case("call_fp64_small", "call", 800, (1, 1, 1), (16, 16, 16), aos=False),
        # the small reference configuration (100k droplets, one box)
        _case("call_fp64_100k", "call", 100_000, (1, 1, 1), (32, 32, 32)),
        # two fuels, eight boxes, four sub-cycles: the configuration at scale, an eighth of it
        _case("call_fp64_2fuel", "call", 2_000_000, (2, 2, 2), (32, 32, 32), fuels=2, cfl=2.0),
        # many boxes with very uneven droplet counts (a spray near its nozzle)
        _case("call_fp64_uneven", "call", 777_777, (4, 4, 4), (32, 32, 32), uneven=True),
        # the PeleC coupling (CGS, temperature from the energy), two sub-cycles
        _case("call_fp64_pelec", "call", 300_007, (2, 2, 1), (32, 32, 17), pelec=True, cfl=1.0, aos=False),
        # the kick without a drift, mixed precision, an odd count
        _case("call_mixed_kick", "call", 99_991, (1, 1, 1), (33, 31, 32), form="mixed", move=False),
        # the largest level: two fuels, four sub-cycles, mixed precision
        _case("call_mixed_2fuel", "call", 8_000_000, (2, 2, 2), (64, 64, 32), form="mixed", fuels=2, cfl=2.0),
        # the surrogate's inference inside the update
        _case("call_learned", "call", 1_000_000, (2, 2, 1), (32, 32, 32), form="learned", aos=False),
        # a whole time step with the droplets resident
        _case("step_mixed_2fuel", "step", 4_000_000, (2, 2, 2), (64, 32, 32), form="mixed", fuels=2, cfl=2.0),
        # a time step of a flow solver whose arrays are in host memory
        _case("step_host_views", "step", 1_000_000, (2, 2, 2), (32, 32, 32), form="mixed", fuels=2, cfl=2.0,
              views="host"),
        # plot-file fields of a loaded level
        _case("fields_2fuel", "fields", 2_000_000, (2, 2, 2), (32, 32, 32), fuels=2),
        # one pass of the surrogate's training
        _case("train_surrogate", "train", 65_536, (1, 1, 1), (32, 32, 32)),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case: kinds by how often they are used, sizes over the whole range."""
    kind = rng.choice(["call"] * 7 + ["step"] * 2 + ["fields", "train"])
    fuels = rng.choice([1, 2])
    form = rng.choice(["fp64", "fp64", "mixed", "mixed", "learned"])
    views, pelec = "device", False
    if kind == "step":
        form, views = rng.choice(["fp64", "mixed"]), rng.choice(["device", "device", "host"])
    elif kind == "fields":
        form = "fp64"
    elif kind == "train":
        form = "fp64"
    elif form != "learned":
        pelec = rng.random() < 0.15
    cfl = rng.choice([0.1, 1.0, 2.0]) if kind in ("call", "step") else 0.1
    most = {"call": 1_500_000 if form != "mixed" else 6_000_000, "step": 1_000_000 if form == "fp64" else 3_000_000,
            "fields": 4_000_000, "train": 120_000}[kind]
    # a step's droplets age while it is repeated: not so few that they evaporate meanwhile
    least = {"call": 500 if form != "learned" else 20_000, "step": 150_000, "fields": 2_000, "train": 20_000}[kind]
    if views == "host":
        most = 800_000
    n = _log_int(rng, least, most)
    nb = [rng.choice([1, 1, 2, 2, 3]) for _ in range(3)] if kind != "train" else [1, 1, 1]
    # 3-9 droplets per cell where the box sizes allow it
    cells = max(512.0, n / rng.uniform(3.0, 9.0) / (nb[0] * nb[1] * nb[2]))
    side = min(72.0, max(8.0, cells ** (1.0 / 3.0)))
    box = [max(8, min(72, int(side * rng.uniform(0.8, 1.25)))) for _ in range(3)]
    case = _case("", kind, n, nb, box, form=form, fuels=fuels, pelec=pelec, cfl=cfl,
                 move=True if kind != "call" else rng.random() < 0.7, aos=rng.random() < 0.6,
                 uneven=kind == "call" and rng.random() < 0.25, views=views)
    del case["name"]
    return case


# --------------------------------------------------------------------------
# inputs

def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _unit(case):
    """Metres to the coupling's length unit."""
    return 100.0 if case["pelec"] else 1.0


def _subcycles(case):
    return math.ceil(case["cfl"] / 0.5) if case["move"] and case["cfl"] > 0.5 else 1


def _problem(case):
    """The level (grids, geometry, liquid properties) without state and droplets."""
    import numpy as np
    nf, u = case["fuels"], _unit(case)
    nb, bs = (case["nbx"], case["nby"], case["nbz"]), (case["bx"], case["by"], case["bz"])
    nc = [nb[d] * bs[d] for d in range(3)]
    boxes = []
    for k in range(nb[2]):
        for j in range(nb[1]):
            for i in range(nb[0]):
                lo = (i * bs[0], j * bs[1], k * bs[2])
                boxes.append((lo, tuple(lo[d] + bs[d] - 1 for d in range(3))))
    dx = np.full(3, DX * u)
    return workloads.Problem(
        name="case", species=SPECIES[nf], fuels=FUELS[nf], ref_T=REF_T[nf], plo=np.zeros(3), phi=np.array(nc) * dx,
        dx=dx, domain_lo=(0, 0, 0), domain_hi=tuple(n - 1 for n in nc), bndry_lo=(0, 0, 0), bndry_hi=(0, 0, 0),
        boxes=boxes, state_ghosts=STATE_GHOSTS, source_ghosts=SOURCE_GHOSTS, state=[], parts=[], flow_dt=DT[nf],
        spray_cfl_lev=case["cfl"], steps=1, pelec=case["pelec"])


def _counts(case, nbox, seed):
    """Droplets per box: even, or Zipf with the largest box capped at a fifth of all."""
    n = case["n"]
    if not case["uneven"] or nbox == 1:
        return [n // nbox + (1 if b < n % nbox else 0) for b in range(nbox)]
    w = [(k + 1) ** -1.2 for k in range(nbox)]
    s = sum(w)
    c = [min(int(n * x / s), max(n // 5, n // nbox)) for x in w]
    c[-1] += n - sum(c)
    g = torch.Generator().manual_seed(seed)
    return [c[i] for i in torch.randperm(nbox, generator=g).tolist()]


def _gas(case, prob, g):
    """One (components, nz, ny, nx) state per box over the grown box, all in one buffer."""
    dev = _device()
    ns = prob.nspec
    nx, ny, nz = (prob.domain_hi[d] + 1 for d in range(3))
    if case["fuels"] == 1:
        T = 800.0 + 200.0 * torch.rand((nz, ny, nx), generator=g, device=dev, dtype=torch.float64)
    else:
        ax = [torch.sin(2 * math.pi * (torch.arange(n, device=dev, dtype=torch.float64) + 0.5) / n) for n in (nx, ny, nz)]
        T = 900.0 + 100.0 * ax[2][:, None, None] * ax[1][None, :, None] * ax[0][None, None, :]
    vel = 10.0 * torch.rand((3, nz, ny, nx), generator=g, device=dev, dtype=torch.float64) - 5.0
    Y = [0.767, 0.233] + [0.0] * (ns - 2)
    W = [MW[s] * 1e-3 for s in prob.species]
    wbar = 1.0 / sum(y / w for y, w in zip(Y, W))
    rho = 101325.0 * wbar / (8.31446261815324 * T)
    full = torch.zeros((prob.n_state_comp, nz, ny, nx), device=dev, dtype=torch.float64)
    if case["pelec"]:
        vel, rho = vel * 100.0, rho * 1e-3
        e = torch.zeros_like(T)
        for s, y in zip(prob.species, Y):
            if y > 0.0:
                e += y * (_h(s, T) - RU / MW[s] * T)
        full[0:3] = rho * vel
        full[4 + ns] = rho * (e + 0.5 * (vel * vel).sum(0))
        full[5 + ns] = T - 7.0  # the stored temperature: only where the inversion starts
    else:
        full[0:3] = vel
        full[5 + ns] = T
    full[3] = rho
    for k in range(ns):
        full[4 + k] = rho * Y[k]
    shapes, los = [], []
    for b in range(len(prob.boxes)):
        lo, hi = prob.grown(b, STATE_GHOSTS)
        los.append(lo)
        shapes.append((prob.n_state_comp,) + tuple(hi[d] - lo[d] + 1 for d in (2, 1, 0)))
    flat, parts = _flat(shapes, dev)
    for lo, t in zip(los, parts):
        ix = [torch.remainder(torch.arange(lo[d], lo[d] + t.shape[3 - d], device=dev), (nx, ny, nz)[d]) for d in range(3)]
        t.copy_(full[:, ix[2]][:, :, ix[1]][:, :, :, ix[0]])
    return flat, parts, los


def _flat(shapes, dev, pin=False):
    sizes = [math.prod(s) for s in shapes]
    flat = torch.zeros(sum(sizes), dtype=torch.float64, device=dev, pin_memory=pin)
    out, o = [], 0
    for s, m in zip(shapes, sizes):
        out.append(flat[o:o + m].view(s))
        o += m
    return flat, out


def _src_shapes(prob, ghosts):
    out = []
    for b in range(len(prob.boxes)):
        lo, hi = prob.grown(b, ghosts)
        out.append((prob.n_src_comp,) + tuple(hi[d] - lo[d] + 1 for d in (2, 1, 0)))
    return out


def _droplets(case, prob, g, counts):
    """pos (3, n), rdata (10 + F, n), id (n,) of all boxes, box by box."""
    dev = _device()
    n, nf, u = case["n"], case["fuels"], _unit(case)
    box = torch.repeat_interleave(torch.arange(len(counts), device=dev), torch.tensor(counts, device=dev))
    lo = torch.tensor([b[0] for b in prob.boxes], device=dev, dtype=torch.float64)
    ext = torch.tensor([case["bx"], case["by"], case["bz"]], device=dev, dtype=torch.float64)
    r = torch.rand((3, n), generator=g, device=dev, dtype=torch.float64).clamp_(1e-7, 1.0 - 1e-7)
    pos = (lo[box].T.contiguous() + r * ext[:, None]) * (DX * u)
    rd = torch.zeros((10 + nf, n), device=dev, dtype=torch.float64)
    rd[0:3] = (20.0 * torch.rand((3, n), generator=g, device=dev, dtype=torch.float64) - 10.0) * u
    z = torch.randn(n, generator=g, device=dev, dtype=torch.float64)
    med, sig = (20e-6, 0.3) if nf == 1 else (15e-6, 0.4)
    rd[4] = (med * torch.exp(sig * z)).clamp_(2e-6, 80e-6) * u
    if nf == 1:
        rd[3], rd[5] = 300.0, 1.0
    else:
        rd[3] = 290.0 + 60.0 * torch.rand(n, generator=g, device=dev, dtype=torch.float64)
        rd[5] = torch.rand(n, generator=g, device=dev, dtype=torch.float64)
        rd[6] = 1.0 - rd[5]
    rd[5 + nf] = rd[6 + nf] = 1.0
    return pos, rd, torch.arange(1, n + 1, device=dev, dtype=torch.int32)


def _inputs(case, seed):
    g = torch.Generator(device=_device()).manual_seed(int(seed))
    prob = _problem(case)
    counts = _counts(case, len(prob.boxes), int(seed) % 97)
    gas = _gas(case, prob, g)
    return prob, counts, gas, _droplets(case, prob, g, counts)


def _record(pos, rd, ids):
    """AMReX's particle record {pos[3], rdata[10 + F], id, cpu} as rows of doubles."""
    rec = torch.empty((ids.shape[0], 4 + rd.shape[0]), device=ids.device, dtype=torch.float64)
    rec[:, :3] = pos.T
    rec[:, 3:-1] = rd.T
    tail = rec.view(torch.int32)
    tail[:, -2] = ids
    tail[:, -1] = 0
    return rec


def _particles(aos, bufs, a, b):
    """pmp_particles of rows (AoS) or columns (SoA) [a, b) of device buffers."""
    p = capi.Particles()
    p.where, p.n = capi.PMP_WHERE_DEVICE, b - a
    if aos:
        p.layout = capi.PMP_LAYOUT_AOS
        p.aos = bufs[0][a:].data_ptr()
        return p
    p.layout = capi.PMP_LAYOUT_SOA
    pos, rd, ids = bufs
    for d in range(3):
        p.pos[d] = pos[d, a:].data_ptr()
    for r in range(rd.shape[0]):
        p.rdata[r] = rd[r, a:].data_ptr()
    p.id = ids[a:].data_ptr()
    return p


def _out_buffers(case, n):
    dev = _device()
    nr = 10 + case["fuels"]
    if case["aos"]:
        return (torch.zeros((n, 4 + nr), device=dev, dtype=torch.float64),)
    return (torch.zeros((3, n), device=dev, dtype=torch.float64), torch.zeros((nr, n), device=dev, dtype=torch.float64),
            torch.zeros(n, device=dev, dtype=torch.int32))


def _droplet_outputs(case, bufs, n):
    """The droplets as outputs: reals and ids apart."""
    if case["aos"]:
        rec = bufs[0][:n]
        return {"reals": rec[:, :-1], "id": rec.view(torch.int32)[:, -2]}
    return {"pos": bufs[0][:, :n], "rdata": bufs[1][:, :n], "id": bufs[2][:n]}


class _State:
    pass


def prepare(case, seed):
    prob, counts, (gas_flat, gas, gas_lo), drops = _inputs(case, seed)
    s = _State()
    s.case, s.prob, s.n = case, prob, case["n"]
    s.sp = spray.from_problem(prob, mode=MODES[case["form"]] if case["form"] != "learned" else capi.PMP_MODE_FP64,
                              set_droplets=False)
    s.keep = [gas_flat, gas]
    s.first = [0]
    for c in counts:
        s.first.append(s.first[-1] + c)
    host = case["views"] == "host"
    s.src_flat, src = _flat(_src_shapes(prob, SOURCE_GHOSTS), "cpu" if host else _device(), pin=host)
    s.keep.append(src)
    src_lo = [prob.grown(b, SOURCE_GHOSTS)[0] for b in range(len(prob.boxes))]
    if host:
        h_flat, h_gas = _flat([t.shape for t in gas], "cpu", pin=True)
        h_flat.copy_(gas_flat)
        s.keep += [h_flat, h_gas]
        s.st = spray.views([t.numpy() for t in h_gas], gas_lo)
        s.sr = spray.views([t.numpy() for t in src], src_lo)
    else:
        s.st, s.sr = spray.views(gas, gas_lo), spray.views(src, src_lo)
    s.stream = torch.cuda.current_stream().cuda_stream
    s.bufs = (_record(*drops),) if case["aos"] else drops
    s.parts = [_particles(case["aos"], s.bufs, a, b) for a, b in zip(s.first, s.first[1:])]
    torch.cuda.current_stream().synchronize()
    if case["kind"] == "call":
        s.out = _out_buffers(case, s.n)
        s.outs = [_particles(case["aos"], s.out, a, b) for a, b in zip(s.first, s.first[1:])]
        s.boxes, s.geom = prob.box_array(), prob.geometry()
        if case["form"] == "learned":
            _hand_over(s)
            s.sp.learn_generate(s.st, prob.flow_dt, STATE_GHOSTS, case["move"], case["cfl"],
                                sample_stride=max(1, s.n // 40_000), augment=2, seed=1)
            s.sp.learn_train(epochs=10, batch=8192, seed=1)
            s.sp.set_mode(capi.PMP_MODE_LEARNED)
        return s
    _hand_over(s)
    if case["kind"] == "step":
        s.out = _out_buffers(case, s.n)
        if host:
            s.sp.set_host_source_in(False)
        else:
            s.act_flat, act = _flat(_src_shapes(prob, 0), _device())
            s.keep.append(act)
            s.act = spray.views(act, [b[0] for b in prob.boxes])
    elif case["kind"] == "fields":
        nvar = 15 + (2 if case["fuels"] > 1 else 0)
        shapes = [(nvar,) + tuple(hi[d] - lo[d] + 1 for d in (2, 1, 0)) for lo, hi in prob.boxes]
        s.var_flat, var = _flat(shapes, _device())
        s.keep.append(var)
        s.var = spray.views(var, [b[0] for b in prob.boxes])
    else:
        s.sp.learn_generate(s.st, prob.flow_dt, STATE_GHOSTS, True, 0.1, sample_stride=1, augment=1, seed=1)
    return s


def _check(s, rc):
    if rc != capi.PMP_OK:
        info = s.sp.last_error()
        raise spray.SprayError(rc, info)


def _hand_over(s):
    L, h = spray.lib(), s.sp._h
    for b, p in enumerate(s.parts):
        _check(s, L.pmp_spray_set_particles(h, b, C.byref(p)))


def run(s):
    c, sp, prob = s.case, s.sp, s.prob
    L, h = spray.lib(), sp._h
    if c["kind"] == "call":
        s.src_flat.zero_()  # the temporary source is zero before the call
        _check(s, L.pmp_spray_set_geometry(h, C.byref(s.geom)))
        _check(s, L.pmp_spray_set_grids(h, len(s.boxes), s.boxes))
        _hand_over(s)
        sp.update_particles(s.st, s.sr, prob.flow_dt, 0.0, STATE_GHOSTS, SOURCE_GHOSTS, False, False, c["move"],
                            c["cfl"], s.stream)
        for b, p in enumerate(s.outs):
            _check(s, L.pmp_spray_get_particles(h, b, C.byref(p)))
        return {"source": s.src_flat, **_droplet_outputs(c, s.out, s.n)}
    if c["kind"] == "step":
        dt = sp.est_timestep(0.5, 0.0, s.stream)
        if c["views"] == "host":
            sp.update_particles_host(s.st, s.sr, prob.flow_dt, 0.0, STATE_GHOSTS, SOURCE_GHOSTS, False, False, True,
                                     c["cfl"], s.stream)
            lost = sp.redistribute(s.stream)
        else:
            s.act_flat.zero_()
            sp.move_kick_drift(s.st, s.sr, prob.flow_dt, 0.0, False, False, STATE_GHOSTS, SOURCE_GHOSTS, True, c["cfl"],
                               s.stream, sync=False)
            sp.move_kick(s.st, s.sr, prob.flow_dt, 0.0, False, False, STATE_GHOSTS, SOURCE_GHOSTS, c["cfl"], s.stream)
            sp.transfer_source(s.sr, s.act, SOURCE_GHOSTS, 0, s.stream)
            lost = sp.redistribute(s.stream)
        counts, a = [], 0
        for b in range(len(prob.boxes)):
            counts.append(sp.num_particles(b))
            p = _particles(c["aos"], s.out, a, a + counts[-1])
            _check(s, L.pmp_spray_get_particles(h, b, C.byref(p)))
            a += counts[-1]
        src = s.src_flat if c["views"] == "host" else s.act_flat
        return {"dt": dt, "dropped": lost, "counts": torch.tensor(counts), "source": src,
                **_droplet_outputs(c, s.out, a)}
    if c["kind"] == "fields":
        s.var_flat.zero_()
        sp.compute_derived_vars(s.var, 0, True, s.stream)
        return {"fields": s.var_flat, "dt": sp.est_timestep(0.5, 0.0, s.stream)}
    sp.learn_train(epochs=1, batch=8192, seed=1)
    return torch.from_numpy(sp.learn_weights())


def work(case):
    n, nf, ns = case["n"], case["fuels"], len(SPECIES[case["fuels"]])
    nb = case["nbx"] * case["nby"] * case["nbz"]

    def cells(g):
        return nb * (case["bx"] + 2 * g) * (case["by"] + 2 * g) * (case["bz"] + 2 * g)

    rec = 8 * (13 + nf) + 8  # a droplet's record
    # operations of one sub-step: the exponentials, logarithms and cube roots
    # at about 20 each, the rest of the expressions
    sub = 20.0 * (2 * ns + nf * (ns - 1) + nf + 40) + 300.0 + 40.0 * ns
    mesh = 8 * cells(1) * (5 + ns) + 8 * cells(0) * (5 + nf)
    if case["kind"] == "call":
        return {"bytes": 2 * n * rec + mesh, "flops": n * _subcycles(case) * sub}
    if case["kind"] == "step":
        subs = _subcycles(case) + (1 if case["views"] == "device" else 0)
        return {"bytes": 3 * n * rec + 2 * mesh, "flops": n * subs * sub}
    if case["kind"] == "fields":
        return {"bytes": n * 8 * (10 + nf) + 8 * cells(0) * (15 + (nf if nf > 1 else 0)), "flops": 60.0 * n}
    rows = 2.0 * n
    return {"bytes": rows * TUPLE_BYTES, "flops": rows * 6.0 * (10 * 64 + 2 * 64 * 64 + 64 * 5)}


# --------------------------------------------------------------------------
# exact: the path in plain 64-bit torch

RU, PATM = 8.31446261815324e7, 1013250.0
MW = {"N2": 28.0134, "O2": 31.9988, "NC7H16": 100.2019, "NC10H22": 142.2817, "CO2": 44.0095}
# cp/R = a0 + a1 T + ... + a4 T^4, h/(R T) adds a5/T
CP = {
    "N2": (3.5492490645113044, -0.0006767968577349293, 1.915101363324171e-06, -1.0468274772510976e-09,
           1.775012341228676e-13, -1043.0618443046233),
    "O2": (3.074942613080369, 0.0016206589546061579, -5.166026191705722e-07, -2.2311028896590883e-11,
           2.8959341376681204e-14, -984.2327320517037),
    "NC7H16": (-0.7086344389527767, 0.08249179609541833, -4.976340802458444e-05, 1.4378093217507722e-08,
               -1.618632740202551e-12, -25630.363277610413),
    "NC10H22": (-0.6189015779283004, 0.11571929746580203, -7.111460102705e-05, 2.126769733049748e-08,
                -2.5242710645737724e-12, -34379.33070177772),
    "CO2": (2.5286461871111885, 0.008130486870124458, -5.918198545407305e-06, 2.0812051208170463e-09,
            -2.813322220494283e-13, -48395.35810336827)}
# cubics in ln T: ln mu, ln lambda, ln(P D) (CGS)
MU = {
    "N2": (-18.4504115932678, 3.214711462401816, -0.3546388748593225, 0.01630476771536381),
    "O2": (-19.70467885233813, 3.7568748066153184, -0.42310661902084845, 0.019174123298156643),
    "NC7H16": (-19.935050208200714, 2.639458873637377, -0.16499072887197586, 0.0032539519196954987),
    "NC10H22": (-17.04192150782738, 1.249330458673676, 0.04317292454119765, -0.006893748834668457),
    "CO2": (-23.214440621596648, 4.8195287516294965, -0.5269126383512059, 0.022187427247711722)}
LAM = {
    "N2": (3.9161525187921273, 0.5634638320507468, 0.03007898182573429, -0.0014898037117685662),
    "O2": (-3.5820860173071267, 3.68895745389154, -0.398050639342719, 0.017989899488740087),
    "NC7H16": (-9.555795030807138, 3.5146401540840713, -0.03593577248878505, -0.012308424120103346),
    "NC10H22": (-4.963892061492923, 1.3319239073207676, 0.2935184079906858, -0.028617025362708687),
    "CO2": (-4.439945451531272, 2.9229221991164525, -0.14850683830458794, 0.0002640057565739968)}
DBIN = {
    "NC7H16": {"N2": (-7.418891131323367, 5.257157718419377, -0.4631429142875803, 0.019916209551153842),
               "O2": (-7.882800856054706, 5.388437435387331, -0.4750560351029627, 0.020223871642538662),
               "NC10H22": (-5.677336940536171, 3.421090043821817, -0.14015087730452366, 0.0024483525605443683),
               "CO2": (-8.084578280264296, 5.139824619254318, -0.4135031000221628, 0.01634996449515813)},
    "NC10H22": {"N2": (-7.936507835939606, 5.352167665739831, -0.47225695429289716, 0.02018046453047065),
                "O2": (-8.294443171352023, 5.431111139960571, -0.4763491362615458, 0.020105961977646997),
                "NC7H16": (-5.677336940536171, 3.421090043821817, -0.14015087730452366, 0.0024483525605443683),
                "CO2": (-7.946581787472698, 4.935029339550768, -0.37875683516078035, 0.014507518314061456)}}
# critical and boiling temperature, latent heat, cp, density (MKS), Antoine a b c
LIQUID = {"NC7H16": (540.0, 371.6, 3.63e5, 2248.3, 681.4, 4.02832, 1268.636, -56.199),
          "NC10H22": (617.8, 447.27, 3.5899e5, 2192.1, 640.0, 4.07857, 1501.268, -78.67)}


def _poly(c, x):
    r = torch.full_like(x, c[-1])
    for a in c[-2::-1]:
        r = r * x + a
    return r


def _cp(s, T):
    return _poly(CP[s][:5], T) * (RU / MW[s])


def _h(s, T):
    c = [CP[s][n] / (n + 1) for n in range(5)]
    return (_poly(c, T) * T + CP[s][5]) * (RU / MW[s])


def _cbrt(x):
    return torch.sign(x) * torch.exp(torch.log(x.abs().clamp_min(1e-300)) / 3.0) * (x != 0)


def _heat_coeff(ratio, B_M, Nu_0):
    """The B_T fixed point: each droplet stops when its own change is below 1e-7."""
    ln1 = torch.log(1.0 + B_M)

    def step(B):
        inv = B / (torch.log1p(B) * (1.0 + B) ** 0.7)
        return 2.0 + (Nu_0 - 2.0) * inv

    old = torch.exp(ratio / Nu_0 * ln1) - 1.0
    B = torch.exp(ratio / step(old) * ln1) - 1.0
    go = (B - old).abs() > 1e-7
    for _ in range(100):
        if not bool(go.any()):
            break
        new = torch.exp(ratio / step(B) * ln1) - 1.0
        new = torch.where(go, new, B)
        go = go & ((new - B).abs() > 1e-7)
        B = new
    return torch.where(B_M <= 1e-15, torch.zeros_like(B), step(B) * torch.log1p(B) / B)


class _Model:
    def __init__(self, case):
        p = case["pelec"]
        self.pelec, self.sp, self.fu = p, SPECIES[case["fuels"]], FUELS[case["fuels"]]
        self.u_ru, self.u_eng, self.u_mass, self.u_rhod, self.u_mu, self.u_lam, self.u_pres = \
            (1.0,) * 7 if p else (1e-7, 1e-4, 1e-3, 0.1, 0.1, 1e-5, 0.1)
        eng, rho, pres = (1e4, 1e-3, 10.0) if p else (1.0, 1.0, 1.0)
        ref = REF_T[case["fuels"]]
        self.ref_T, self.indx = ref, [self.sp.index(f) for f in self.fu]
        self.mw = [MW[s] * self.u_mass for s in self.sp]
        self.liq = []
        for f in self.fu:
            tc, tb, lat, cp, rl, a, b, c = LIQUID[f]
            h_ref = float(_h(f, torch.tensor(ref, dtype=torch.float64))) * self.u_eng
            self.liq.append(dict(tc=tc, tb=tb, cp=cp * eng, rho=rl * rho, a=a, b=b, c=c, d=1e5 * pres,
                                 lat=lat * eng - h_ref, hb=lat * eng * ((tc - ref) / (tc - tb)) ** -0.38))

    def source(self, dt0, T_g, rho_g, u_g, Y_g, vel, T, dia, Y, num):
        """calculateSpraySource: the new droplet state and the source rates."""
        mw, nf, ns = self.mw, len(self.fu), len(self.sp)
        W = sum(Y_g[k] / mw[k] for k in range(ns))
        p = rho_g * RU * W * T_g * self.u_ru
        W = 1.0 / W
        boil = []
        for f, q in enumerate(self.liq):
            cc = 1.0 / (torch.log(PATM * self.u_pres / p) * RU * self.u_ru / (q["hb"] * mw[self.indx[f]]) + 1.0 / q["tb"])
            boil.append(cc.clamp_max(q["tc"]))
        vel, Y = vel.clone(), [y.clone() for y in Y]
        Y0 = [y.clone() for y in Y]

        def rho_liquid():
            return 1.0 / sum(Y[f] / self.liq[f]["rho"] for f in range(nf))

        rho_p = rho_liquid()
        m = math.pi / 6.0 * rho_p * dia ** 3
        m0 = m.clone()
        alive = torch.ones_like(T, dtype=torch.bool)
        nsub, isub = torch.ones_like(T), 1
        mom, eng = torch.zeros_like(vel), torch.zeros_like(T)
        dt, h_dep, mi = None, None, [torch.zeros_like(T) for _ in range(nf)]
        while True:
            on = alive & (isub <= nsub)
            if not bool(on.any()):
                break
            Tb = sum(Y[f] * boil[f] for f in range(nf))
            cp_p = sum(Y[f] * self.liq[f]["cp"] for f in range(nf))
            mw_p = 1.0 / sum(Y[f] / mw[self.indx[f]] for f in range(nf))
            dT = (T_g - T).clamp_min(0.0)
            Ts = T + dT / 3.0
            h_now = [_h(f, T) * self.u_eng for f in self.fu]
            h_dep = h_now if h_dep is None else [torch.where(on, a, b) for a, b in zip(h_now, h_dep)]
            L, Xv = [], []
            mbar, sumX = torch.zeros_like(T), torch.zeros_like(T)
            for f, q in enumerate(self.liq):
                i = self.indx[f]
                Tp = torch.minimum(T, 0.99 * boil[f])
                L.append(h_now[f] + q["lat"] - q["cp"] * (Tp - self.ref_T))
                ps = q["d"] * torch.exp((q["a"] - q["b"] / (Tp + q["c"])) * math.log(10.0))
                x = Y[f] * mw_p / mw[i] * ps / p
                x = torch.where(ps > Y_g[i] * W / mw[i] * p, x, torch.zeros_like(x))
                mbar, sumX = mbar + x * mw[i], sumX + x
                Xv.append(x)
            tot = mbar + (1.0 - sumX) * W
            sumYs, sumYf, sumYv, Ys = torch.zeros_like(T), torch.zeros_like(T), torch.zeros_like(T), [None] * ns
            for f in range(nf):
                i = self.indx[f]
                wet = Xv[f] > 0.0
                yv = Xv[f] * mw[i] / tot
                ys = torch.where(wet, yv + (Y_g[i] - yv) / 3.0, torch.zeros_like(T))
                sumYv, sumYf, sumYs = sumYv + yv, sumYf + torch.where(wet, Y_g[i], torch.zeros_like(T)), sumYs + ys
                Ys[i] = ys
            renorm = (1.0 - sumYs) / (1.0 - sumYf)
            for k in range(ns):
                y = Y_g[k] * renorm
                Ys[k] = y if Ys[k] is None else torch.where(Ys[k] == 0.0, y, Ys[k])
            cps = [_cp(s, Ts) * self.u_eng for s in self.sp]
            cp_s = sum(Ys[k] * cps[k] for k in range(ns))
            mw_s = 1.0 / sum(Ys[k] / mw[k] for k in range(ns))
            B_M = ((sumYv - sumYf) / (1.0 - sumYv).clamp_min(1e-15)).clamp_max(20.0)
            rho_s = mw_s * p / (RU * self.u_ru * Ts)
            lnT = torch.log(Ts)
            wbar = 1.0 / sum(Ys[k] / MW[s] for k, s in enumerate(self.sp))
            X = [Ys[k] * wbar / MW[s] for k, s in enumerate(self.sp)]
            mu = sum(X[k] * torch.exp(6.0 * _poly(MU[s], lnT)) for k, s in enumerate(self.sp)) ** (1.0 / 6.0) * self.u_mu
            lam = sum(X[k] * torch.exp(0.25 * _poly(LAM[s], lnT)) for k, s in enumerate(self.sp)) ** 4 * self.u_lam
            D = []
            for f, i in enumerate(self.indx):
                rest = [k for k in range(ns) if k != i]
                t1 = sum(Ys[k] for k in rest)
                t2 = sum(X[k] * torch.exp(-_poly(DBIN[self.fu[f]][self.sp[k]], lnT)) for k in rest)
                D.append(MW[self.fu[f]] * t1 / (t2 * RU * Ts))
            du = u_g - vel
            mag = (du * du).sum(0).sqrt()
            Re = rho_s * mag * dia / mu
            Rs = Re.clamp_min(1e-300)
            cd = torch.where(Re > 1000.0, torch.full_like(Re, 0.424),
                             torch.where(Re > 1.0, 24.0 / Rs * (1.0 + _cbrt(Re * Re) / 6.0),
                                         torch.where(Re > 0.0, 24.0 / Rs, torch.zeros_like(Re))))
            force = 0.125 * rho_s * cd * math.pi * dia * dia * mag
            tau = 0.75 * rho_s * cd * mag / (dia * rho_p)
            mom = mom + on * num * force * du
            if self.pelec:
                eng = eng + on * num * force * (du * vel).sum(0)
            Pr = mu * cp_s / lam
            powR = torch.where(Re > 0.0, Rs.clamp_max(400.0) ** 0.077, torch.zeros_like(Re)).clamp_min(1.0)
            Nu_0 = 1.0 + powR * _cbrt(1.0 + Re * Pr)
            wet = sumX > 0.0
            safe = torch.where(wet, sumX, torch.ones_like(sumX))
            rhoD, cpf, ysum = torch.zeros_like(T), torch.zeros_like(T), torch.zeros_like(T)
            for f, i in enumerate(self.indx):
                D[f] = D[f] * mw_s / mw[i] * self.u_rhod * (Xv[f] / safe)
                rhoD, cpf, ysum = rhoD + D[f], cpf + Ys[i] * cps[i], ysum + Ys[i]
            cpf = cpf / torch.where(wet, ysum, torch.ones_like(T))
            rD = torch.where(wet, rhoD, torch.ones_like(T))
            BM = torch.where(wet, B_M, torch.ones_like(T))
            logB = torch.log1p(BM)
            Sh = 2.0 + (powR * _cbrt(1.0 + Re * mu / rD) - 1.0) * BM / (logB * (1.0 + BM) ** 0.7)
            Nu = torch.where(wet, _heat_coeff(cpf * Sh * rD / lam, BM, Nu_0), Nu_0)
            mdot, sumL = torch.zeros_like(T), torch.zeros_like(T)
            for f in range(nf):
                r = -(D[f] * math.pi * dia * Sh * logB).clamp_min(0.0)
                mi[f] = torch.where(wet & (Xv[f] > 0.0), r, mi[f])
                r = torch.where(wet & (Xv[f] > 0.0), r, torch.zeros_like(r))
                mdot, sumL = mdot + r, sumL + r * L[f]
            conv = math.pi * lam * dia * dT * Nu
            eng = eng + on * num * conv
            Tdot = (sumL + conv) / m.clamp_min(1e-300) / cp_p
            if isub == 1:
                nsub = (dt0 * tau).floor() + 1.0
                heat = dT > 1e-15
                cand = torch.maximum((dt0 * -mdot / (0.2 * m)).floor(),
                                     torch.where(heat, (dt0 * conv / m / (cp_p * dT.clamp_min(1e-15))).floor(), torch.zeros_like(T)))
                nsub = torch.where(heat, torch.maximum(nsub, cand + 1.0), nsub).clamp(1.0, 100.0)
                dt = dt0 / nsub
            h = 0.5 * dt
            vel = torch.where(on, vel + h * tau * du, vel)
            newT, newm = T + h * Tdot, m + mdot * h
            live = on & (newm > 1e-13 * self.u_mass) & (newT < Tb)
            dead = on & ~live
            if nf > 1:
                frac = [((Y[f] * m + mi[f] * h) / newm).clamp(0.0, 1.0) for f in range(nf)]
                frac = [torch.where(y <= 1e-12, torch.zeros_like(y), y) for y in frac]
                s = sum(frac)
                Y = [torch.where(live, y / s, Y[f]) for f, y in enumerate(frac)]
            T = torch.where(live, newT, T)
            m = torch.where(live, newm, torch.where(dead, torch.zeros_like(m), m))
            rho_p = torch.where(live, rho_liquid(), rho_p)
            dia = torch.where(live, _cbrt(6.0 * m / (math.pi * rho_p)), dia)
            nsub = torch.where(dead, torch.full_like(nsub, float(isub)), nsub)
            alive = alive & ~dead
            isub += 1
        mom, eng = mom / nsub, eng / nsub
        rate = (m - m0) / (0.5 * dt0)
        mass = num * rate
        if self.pelec:
            eng = eng + num * 0.5 * (vel * vel).sum(0) * rate
        mom = mom + num * vel * rate
        yd = []
        for f in range(nf):
            r = num * (Y[f] * m - Y0[f] * m0) / (0.5 * dt0)
            yd.append(r)
            eng = eng + r * h_dep[f]
        return vel, T, dia, Y, alive, torch.stack([*mom, mass, *yd, eng])

    def cell_fields(self, st):
        """(rho, T, u, Y) per cell, flattened, of one box's state."""
        ns = len(self.sp)
        q = st.reshape(st.shape[0], -1)
        rho = q[3]
        Y = q[4:4 + ns] / rho
        if not self.pelec:
            return torch.cat([rho[None], q[5 + ns][None], q[0:3], Y])
        u = q[0:3] / rho
        e = q[4 + ns] / rho - 0.5 * (u * u).sum(0)
        T = q[5 + ns].clone()
        for _ in range(20):
            em = sum(Y[k] * (_h(s, T) - RU / MW[s] * T) for k, s in enumerate(self.sp))
            cv = sum(Y[k] * (_cp(s, T) - RU / MW[s]) for k, s in enumerate(self.sp))
            T = T + (e - em) / cv
        return torch.cat([rho[None], T[None], u, Y])


def _update(case, M, st, st_lo, src, src_lo, pos, rd, ids, move):
    """updateParticles for one box, in place on (clones of) the droplets."""
    nf, dx = case["fuels"], DX * _unit(case)
    dxi = 1.0 / dx
    subs = math.ceil(case["cfl"] / 0.5) if move and case["cfl"] > 0.5 else 1
    dt = DT[nf] / subs
    F = M.cell_fields(st)
    nx, ny = st.shape[3], st.shape[2]
    S, sx, sy = src.view(src.shape[0], -1), src.shape[3], src.shape[2]
    for _ in range(subs):
        live = (ids > 0).nonzero()[:, 0]
        if not live.numel():
            return
        x = pos[:, live]
        l = x * dxi + 0.5
        i = l.floor()
        hi = l - i
        i, w = i.long(), torch.stack([1.0 - hi, hi])
        g = torch.zeros((F.shape[0], live.numel()), device=x.device, dtype=torch.float64)
        for kk in (0, 1):
            for jj in (0, 1):
                for ii in (0, 1):
                    at = ((i[2] - 1 + kk - st_lo[2]) * ny + (i[1] - 1 + jj - st_lo[1])) * nx + (i[0] - 1 + ii - st_lo[0])
                    g += w[ii, 0] * w[jj, 1] * w[kk, 2] * F[:, at]
        r = rd[:, live]
        vel, T, dia, Y, alive, rate = M.source(dt, g[1], g[0], g[2:5], g[5:], r[0:3], r[3], r[4], list(r[5:5 + nf]),
                                               r[5 + nf])
        c = (x * dxi).floor().long()
        at = ((c[2] - src_lo[2]) * sy + (c[1] - src_lo[1])) * sx + (c[0] - src_lo[0])
        S.index_add_(1, at, -(1.0 / dx ** 3) * dt / DT[nf] * rate)
        r[0:3], r[3], r[4] = vel, T, dia
        for f in range(nf):
            r[5 + f] = Y[f]
        rd[:, live] = r
        if move:
            pos[:, live] = torch.where(alive, x + dt * vel, x)
        ids[live] = torch.where(alive, ids[live], torch.full_like(ids[live], -1))


def _as_outputs(case, pos, rd, ids):
    if case["aos"]:
        return {"reals": torch.cat([pos, rd]).T, "id": ids}
    return {"pos": pos, "rdata": rd, "id": ids}


def exact(case, seed):
    """What run() returns for these inputs on a first pass, in plain 64-bit torch.

    A trained surrogate's weights have no such value."""
    if case["kind"] == "train":
        return None
    prob, counts, (_, gas, gas_lo), (pos, rd, ids) = _inputs(case, seed)
    M, dev, nf = _Model(case), _device(), case["fuels"]
    first = [0]
    for c in counts:
        first.append(first[-1] + c)
    spans = list(zip(first, first[1:]))
    mv = torch.maximum(torch.maximum(rd[0].abs(), rd[1].abs()), rd[2].abs()) / (DX * _unit(case))
    dt = float((0.5 / mv).min())
    src_lo = [prob.grown(b, SOURCE_GHOSTS)[0] for b in range(len(prob.boxes))]
    if case["kind"] == "fields":
        return {"fields": _fields(case, prob, M, spans, pos, rd), "dt": dt}

    def update(flat_ghosts, move):
        flat, src = _flat(_src_shapes(prob, flat_ghosts), dev)
        for b, (a, e) in enumerate(spans):
            for lo in range(a, e, 2_000_000):
                s = slice(lo, min(e, lo + 2_000_000))
                p, r, i = pos[:, s].clone(), rd[:, s].clone(), ids[s].clone()
                _update(case, M, gas[b], gas_lo[b], src[b], src_lo[b], p, r, i, move)
                pos[:, s], rd[:, s], ids[s] = p, r, i
        return flat, src

    flat, src = update(SOURCE_GHOSTS, case["move"])
    if case["kind"] == "call":
        return {"source": flat, **_as_outputs(case, pos, rd, ids)}
    n = [prob.domain_hi[d] + 1 for d in range(3)]
    dx = DX * _unit(case)
    order = _cell_order(case, prob, spans, _inputs(case, seed)[3][0])
    if case["views"] == "device":
        src2 = update(SOURCE_GHOSTS, False)[1]
        total = torch.zeros((prob.n_src_comp, n[2], n[1], n[0]), device=dev, dtype=torch.float64)
        for group in (src, src2):
            for lo, t in zip(src_lo, group):
                ix = [torch.remainder(torch.arange(lo[d], lo[d] + t.shape[3 - d], device=dev), n[d]) for d in range(3)]
                at = (ix[2][:, None, None] * n[1] + ix[1][None, :, None]) * n[0] + ix[0][None, None, :]
                total.view(prob.n_src_comp, -1).index_add_(1, at.reshape(-1), t.reshape(t.shape[0], -1))
        flat = torch.cat([total[:, lo[2]:hi[2] + 1, lo[1]:hi[1] + 1, lo[0]:hi[0] + 1].reshape(-1) for lo, hi in prob.boxes])
    # re-binning: periodic wrap, then box, then cell, stable in the order the droplets were in
    pos, rd, ids = pos[:, order], rd[:, order], ids[order]
    keep = ids > 0
    lost = int((~keep).sum())
    pos, rd, ids = pos[:, keep], rd[:, keep], ids[keep]
    for d in range(3):
        Ld = float(prob.phi[d])
        pos[d] = torch.where(pos[d] >= Ld, pos[d] - Ld, pos[d])
        pos[d] = torch.where(pos[d] < 0.0, pos[d] + Ld, pos[d])
    c = (pos * (1.0 / dx)).floor().long()
    bs = (case["bx"], case["by"], case["bz"])
    bi = [c[d] // bs[d] for d in range(3)]
    box = (bi[2] * case["nby"] + bi[1]) * case["nbx"] + bi[0]
    loc = [c[d] - bi[d] * bs[d] for d in range(3)]
    key = ((box * bs[2] + loc[2]) * bs[1] + loc[1]) * bs[0] + loc[0]
    order = torch.sort(key, stable=True)[1]
    return {"dt": dt, "dropped": lost, "counts": torch.bincount(box, minlength=len(prob.boxes)), "source": flat,
            **_as_outputs(case, pos[:, order], rd[:, order], ids[order])}


def _cell_order(case, prob, spans, pos):
    """The order of droplets handed over: box by box, by cell, stable."""
    out = []
    for (lo, _), (a, e) in zip(prob.boxes, spans):
        c = (pos[:, a:e] * (1.0 / (DX * _unit(case)))).floor().long()
        key = ((c[2] - lo[2]) * case["by"] + (c[1] - lo[1])) * case["bx"] + (c[0] - lo[0])
        out.append(a + torch.sort(key, stable=True)[1])
    return torch.cat(out)


def _fields(case, prob, M, spans, pos, rd):
    nf, dx = case["fuels"], DX * _unit(case)
    nvar = 15 + (nf if nf > 1 else 0)
    out = []
    for (lo, hi), (a, e) in zip(prob.boxes, spans):
        p, r = pos[:, a:e], rd[:, a:e]
        c = (p * (1.0 / dx)).floor().long()
        nx, ny, nz = (hi[d] - lo[d] + 1 for d in range(3))
        at = ((c[2] - lo[2]) * ny + (c[1] - lo[1])) * nx + (c[0] - lo[0])
        rho = 1.0 / sum(r[5 + f] / M.liq[f]["rho"] for f in range(nf))
        d, num = r[4], r[5 + nf]
        vol, surf = math.pi / 6.0 * d ** 3, math.pi * d * d
        m = vol * rho
        zero = torch.zeros_like(d)
        v = [num * m, num * m / dx ** 3, num, num * vol, num * surf, num * vol / dx ** 3, num * d, num * vol * 6.0, zero, zero,
             num * m * r[3], torch.ones_like(d), num * m * r[0], num * m * r[1], num * m * r[2]]
        if nf > 1:
            v += [r[5 + f] * m for f in range(nf)]
        V = torch.zeros((nvar, nz * ny * nx), device=p.device, dtype=torch.float64)
        V.index_add_(1, at, torch.stack(v))
        for den, num_ in ((2, 6), (4, 7), (0, 10), (0, 12), (0, 13), (0, 14)):
            V[num_] = torch.where(V[den] != 0.0, V[num_] / V[den], V[num_])
        out.append(V.reshape(-1))
    return torch.cat(out)
