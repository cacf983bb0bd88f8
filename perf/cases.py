"""What programs on this framework spend their time on, one call each, with the sizes they use.

A case is one of these calls, made on lattices built from a seed:

  update     Magnets.update(): one step, its switches returned to the host. Interactive use, hand-written
             loops and every program taken over from Hotspice step like this.
  run        Magnets.run(steps): a fixed number of steps on the device (sweeps, benchmarks).
  progress   Magnets.progress(): steps until a Monte Carlo step limit, the call of most experiments.
  resync     Magnets.run(steps), then Magnets.resync_energies(): long runs that recompute the energies from
             the spins now and then, to bound the drift of the increments.
  batch      BatchEngine.run_from_host(): a parameter sweep, many small simulations in one launch, start
             states from host memory and results back to it.
  recompute  Magnets.update_energy(): the full sum of the interaction over every pair of magnets, made at
             each construction, each change of the state, the geometry or a material parameter.
  relax      a start state is set and Magnets.relax() quenches it to a metastable state.

Lattice constants, moments, barriers and temperatures are those of the benchmark's workloads.
"""
import math

import numpy as np
import torch

import hotspice_b200 as hs
from hotspice_b200.engine import BatchEngine

# class name, lattice constant (m), moment (A m^2)
LATTICES = {
    "square": ("OOP_Square", 200e-9, 1.1e-15),
    "pinwheel": ("IP_Pinwheel", 300e-9, 1e-15),
    "kagome": ("IP_Kagome", 500e-9, 1e-15),
}


def listed():
    return [
        # the smallest call: a step of a small lattice, driven from Python
        {"name": "update_neel_square_32", "call": "update", "lattice": "square", "nx": 32, "ny": 32, "scheme": "Neel",
         "cutoff": 0, "zeeman": False, "pbc": False, "T": 300.0},
        # the same for an in-plane lattice of odd sides under Metropolis multisampling
        {"name": "update_metropolis_pinwheel_151x113", "call": "update", "lattice": "pinwheel", "nx": 151, "ny": 113,
         "scheme": "Metropolis", "cutoff": 16, "zeeman": True, "pbc": False, "T": 300.0},
        # a kinetic run of one 64 x 64 lattice with the uncut interaction
        {"name": "run_neel_square_64", "call": "run", "lattice": "square", "nx": 64, "ny": 64, "scheme": "Neel",
         "cutoff": 0, "zeeman": False, "pbc": False, "T": 300.0, "steps": 1000, "graphs": False},
        # an experiment's progress() on a sparse in-plane lattice with two reversal channels
        {"name": "progress_neel_kagome_200", "call": "progress", "lattice": "kagome", "nx": 200, "ny": 111, "scheme": "Neel",
         "cutoff": 16, "zeeman": True, "pbc": False, "T": 300.0, "mcsteps": 0.04},
        # one 512 x 512 pinwheel under Metropolis multisampling, the step kernels replayed from graphs
        {"name": "run_metropolis_pinwheel_512", "call": "run", "lattice": "pinwheel", "nx": 512, "ny": 512,
         "scheme": "Metropolis", "cutoff": 20, "zeeman": True, "pbc": False, "T": 300.0, "steps": 256, "graphs": True},
        # a large one of ragged sides: hundreds of switches per step
        {"name": "run_metropolis_pinwheel_1500x1201", "call": "run", "lattice": "pinwheel", "nx": 1500, "ny": 1201,
         "scheme": "Metropolis", "cutoff": 20, "zeeman": True, "pbc": False, "T": 300.0, "steps": 128, "graphs": True},
        # Poisson-disc multisampling of the uncut interaction, recomputed every 100 steps
        {"name": "resync_poisson_square_1024", "call": "resync", "lattice": "square", "nx": 1024, "ny": 1024,
         "scheme": "Metropolis", "cutoff": 0, "zeeman": False, "pbc": False, "T": 300.0, "steps": 100},
        # Wolff clusters of the exchange-only Ising lattice somewhat above its critical temperature
        {"name": "run_wolff_ising_300", "call": "run", "lattice": "square", "nx": 300, "ny": 300, "scheme": "Wolff",
         "cutoff": 0, "zeeman": False, "pbc": True, "T": 300.0, "steps": 200, "graphs": False},
        # the parameter sweep: 256 uneven simulations of mixed lattices, 200 steps each
        {"name": "batch_256_mixed", "call": "batch", "count": 256, "n_min": 32, "n_max": 256, "steps": 200},
        # the full sum for a small lattice: construction and state changes in a loop
        {"name": "recompute_square_96", "call": "recompute", "lattice": "square", "nx": 96, "ny": 96, "scheme": "Neel",
         "cutoff": 0, "zeeman": False, "pbc": False, "T": 300.0},
        # and for a large in-plane one of ragged sides, both energy channels
        {"name": "recompute_pinwheel_640x571", "call": "recompute", "lattice": "pinwheel", "nx": 640, "ny": 571,
         "scheme": "Neel", "cutoff": 0, "zeeman": False, "pbc": False, "T": 300.0},
        # a quench of a random 512 x 512 pinwheel
        {"name": "relax_pinwheel_512", "call": "relax", "lattice": "pinwheel", "nx": 512, "ny": 512, "scheme": "Neel",
         "cutoff": 8.3, "zeeman": True, "pbc": False, "T": 300.0},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    call = rng.choice(("update", "run", "run", "progress", "resync", "batch", "recompute", "recompute", "relax"))
    if call == "batch":
        lo = rng.randint(32, 64)
        return {"call": call, "count": _log_int(rng, 24, 256), "n_min": lo, "n_max": rng.randint(2 * lo, 256),
                "steps": rng.randint(50, 200)}
    scheme = rng.choice(("Neel", "Metropolis"))
    if call == "run":
        scheme = rng.choice(("Neel", "Metropolis", "Metropolis", "Wolff"))
    elif call == "resync":
        scheme = "Metropolis"
    if scheme == "Wolff":
        nx = 2 * _log_int(rng, 16, 256)
        return {"call": call, "lattice": "square", "nx": nx, "ny": max(32, 2 * int(nx * rng.uniform(0.3, 0.5))),
                "scheme": scheme, "cutoff": 0, "zeeman": False, "pbc": True, "T": rng.uniform(250.0, 400.0),
                "steps": rng.randint(50, 200), "graphs": False}
    lattice = "square" if call == "resync" else rng.choice(("square", "pinwheel", "pinwheel", "kagome"))
    big = {"update": 256, "run": 1500 if scheme == "Metropolis" else 320, "progress": 256, "resync": 600,
           "recompute": 512, "relax": 512}[call]
    nx = _log_int(rng, 250 if call == "resync" else 32, big)
    ny = max(32, int(nx * rng.uniform(0.7, 1.0)))
    if call == "resync" and rng.random() < 0.5:
        nx = rng.randint(850, 1024)
        ny = int(nx * rng.uniform(0.9, 1.0))
    pbc = rng.random() < 0.25
    if lattice == "kagome":
        pbc = False
        nx, ny = nx // 4 * 4, max(31, ny // 4 * 4 - 1)
    if pbc:
        nx, ny = nx // 2 * 2, ny // 2 * 2
    full = call == "resync" or call == "recompute" and rng.random() < 0.7 or max(nx, ny) <= 128 and rng.random() < 0.4
    case = {"call": call, "lattice": lattice, "nx": nx, "ny": ny, "scheme": scheme,
            "cutoff": 0 if full else rng.choice((8.3, 16, 20)), "zeeman": not full or rng.random() < 0.5, "pbc": pbc,
            "T": rng.uniform(200.0, 400.0)}
    if call == "run":
        case["graphs"] = scheme == "Metropolis" and max(nx, ny) >= 400
        case["steps"] = rng.randint(64, 128) if case["graphs"] else rng.randint(200, 1000)
    elif call == "progress":
        case["mcsteps"] = rng.choice((0.02, 0.04)) if scheme == "Neel" else rng.choice((0.25, 0.5))
    elif call == "resync":
        case["steps"] = rng.randint(25, 100)
    return case


def _lattice(case, seed, g):
    cls, a, moment = LATTICES[case["lattice"]]
    nx, ny = case["nx"], case["ny"]
    pattern = g.integers(0, 2, size=(ny, nx)) * 2 - 1
    if case["scheme"] == "Wolff":
        energies, barrier = [hs.ExchangeEnergy(J=1e-21)], 0.0
        params = hs.SimParams(UPDATE_SCHEME="Wolff", MULTISAMPLING_SCHEME="cluster")
    else:
        energies = [hs.DipolarEnergy(cutoff_range=case["cutoff"] * a if case["cutoff"] else math.inf)]
        if case["zeeman"]:
            energies.append(hs.ZeemanEnergy(float(g.uniform(0, 2e-3)), float(g.uniform(0, 2 * math.pi))))
        barrier = 5.5e-20 * g.lognormal(-0.05 ** 2 / 2, 0.05, size=(ny, nx))
        params = hs.SimParams(UPDATE_SCHEME=case["scheme"],
                              MULTISAMPLING_SCHEME="Poisson" if case["call"] == "resync" else "grid")
    engine = hs.EngineConfig(persistent=not (case.get("graphs") or case["call"] == "resync"))
    return getattr(hs.ASI, cls)(a, nx=nx, ny=ny, T=case["T"], E_B=barrier, moment=moment, pattern=pattern, PBC=case["pbc"],
                                energies=energies, params=params, engine=engine, seed=seed)


def _sweep(case, seed, g):
    """Mixed lattices as in the benchmark's batch; even instances Néel, odd ones Metropolis. The
    lattices are the case's own, their states, barriers, fields and temperatures the seed's."""
    out = []
    sizes = np.random.default_rng(case["count"])
    for i in range(case["count"]):
        kind = ("square", "pinwheel", "kagome")[int(sizes.integers(0, 3))]
        n = int(sizes.integers(case["n_min"], case["n_max"] + 1))
        ny = max(int(n / math.sqrt(3)) // 4 * 4 - 1, 3) if kind == "kagome" else n
        out.append(_lattice({"call": "batch", "lattice": kind, "nx": n, "ny": ny, "scheme": "Neel" if i % 2 == 0 else "Metropolis",
                             "cutoff": 16, "zeeman": True, "pbc": False, "T": float(g.uniform(200, 400))},
                            seed * 1000 + i, g))
    return out


def prepare(case, seed):
    g = np.random.default_rng(seed)
    if case["call"] == "batch":
        engine = BatchEngine(_sweep(case, seed, g))
        host_in = engine.pack_host()
        layout, total = engine.state_layout(("m", "C"))
        return {"case": case, "engine": engine, "host_in": host_in, "layout": layout,
                "host_out": torch.empty(total, dtype=torch.uint8, pin_memory=True)}
    mm = _lattice(case, seed, g)
    state = {"case": case, "mm": mm}
    if case["call"] == "relax":
        state["start"] = mm.m.cpu().numpy()
    return state


def _state_of(mm):
    out = {"m": mm.m, "attempted": mm.attempted_switches, "switches": mm.switches, "t": mm.t}
    dip = mm.get_energy("dipolar", verbose=False)
    if dip is not None:
        out["E"] = dip.E
        if mm.in_plane:
            out["E_perp"] = dip.E_perp
    return out


def run(state):
    case = state["case"]
    call = case["call"]
    if call == "batch":
        engine, host_out = state["engine"], state["host_out"]
        engine.run_from_host(case["steps"], state["host_in"], host_out=host_out, out_fields=("m", "C"))
        torch.cuda.current_stream().synchronize()
        raw = host_out.numpy()
        spins = np.concatenate([raw[off:off + size] for _, field, off, size in state["layout"] if field == "m"])
        counters = np.stack([raw[off:off + size] for _, field, off, size in state["layout"] if field == "C"])
        counters = counters.view(hs._lib.COUNTERS_DTYPE).ravel()
        return {"m": spins.view(np.int8), "t": counters["t"], "attempted": counters["attempted"],
                "switches": counters["switches"]}
    mm = state["mm"]
    if call == "update":
        switched = mm.update()
        return {"n": 0 if switched is None else int(np.asarray(switched).reshape(2, -1).shape[1]), "m": mm.m}
    if call == "run":
        mm.run(case["steps"])
        return _state_of(mm)
    if call == "progress":
        dt, mcsteps = mm.progress(t_max=math.inf, MCsteps_max=case["mcsteps"])
        return {"dt": dt, "mcsteps": mcsteps, **_state_of(mm)}
    if call == "resync":
        mm.run(case["steps"])
        mm.resync_energies()
        return _state_of(mm)
    if call == "recompute":
        mm.update_energy()
        dip = mm.get_energy("dipolar")
        return {"E": dip.E, "E_perp": dip.E_perp} if mm.in_plane else {"E": dip.E}
    mm.m = state["start"]
    mm.update_energy()
    mm.relax()
    return _state_of(mm) | {"sweeps": mm.relax_sweeps}


# ------------------------------------------------------------------------------------------------
# What a pass cannot do without
# ------------------------------------------------------------------------------------------------
def _window(case):
    """Cells of a switch's interaction window."""
    if not case["cutoff"] and case["scheme"] == "Metropolis":
        return min(case["nx"] * case["ny"], 41 * 41)   # SimParams.REDUCED_KERNEL_SIZE, when many switch at once
    if not case["cutoff"]:
        return case["nx"] * case["ny"]     # the part of the uncut window that lies on the lattice
    pitch = {"square": 1.0, "pinwheel": 0.5, "kagome": 0.25}[case["lattice"]]   # column spacing / a
    rows = {"square": 1.0, "pinwheel": 0.5, "kagome": 0.25 * math.sqrt(3)}[case["lattice"]]
    w = 2 * int(case["cutoff"] / pitch) + 1, 2 * int(case["cutoff"] / rows) + 1
    return min(w[0], case["nx"]) * min(w[1], case["ny"])


def _step_bytes(case):
    """One step: a Néel step reads every magnet's energy (8), spin (1), Zeeman factor (4) and
    barrier (4), and both energies in-plane; a Metropolis step its candidates'. Each switch
    reads the interaction (4) and the moments (4) and updates the energies (16) in its window."""
    two = case["lattice"] != "square"
    cells = case["nx"] * case["ny"]
    magnets = cells * {"square": 1.0, "pinwheel": 0.5, "kagome": 0.375}[case["lattice"]]
    window = _window(case) * (44 if two else 24)
    if case["scheme"] == "Neel":
        return magnets * (29 if two else 17) + window
    if case["scheme"] == "Wolff":
        return 64.0 * 16               # a cluster of some tens of spins: spin and stamps
    # candidates lie at least about 40 cells apart (calc_r of these moments: some 10 lattice constants)
    picks = max(1.0, cells / 40.0 ** 2 / 2)
    return picks * 29 + 0.4 * picks * window


def work(case):
    if case["call"] == "batch":
        n = 0.5 * (case["n_min"] + case["n_max"])
        per = [_step_bytes({"lattice": k, "nx": int(n), "ny": int(n * (0.57 if k == "kagome" else 1.0)), "scheme": s, "cutoff": 16})
               for k in LATTICES for s in ("Neel", "Metropolis")]
        total = case["count"] * case["steps"] * sum(per) / len(per)
        return {"bytes": total, "flops": total / 4}
    cells = case["nx"] * case["ny"]
    channels = 1 if case["lattice"] == "square" else 2
    kernels = {"square": 1, "pinwheel": 2, "kagome": 3}[case["lattice"]]
    # the full sum: spins and moments in, energies out, every kernel window once; by a fast
    # convolution, two transforms of the doubled lattice for each kernel and channel
    padded = 4 * cells
    full = {"bytes": cells * (5 + 8 * channels) + channels * kernels * 4 * padded,
            "flops": 2 * channels * kernels * 2.5 * padded * math.log2(padded)}
    call = case["call"]
    if call == "recompute":
        return full
    if call == "relax":
        # a sweep decides every magnet (13 bytes) and updates the energies of every cell once or more
        sweeps = 0.1 * math.hypot(case["nx"], case["ny"])
        return {"bytes": sweeps * cells * (6.5 + 20 * channels), "flops": sweeps * cells * 40.0}
    if call == "update":
        steps = 1
    elif call == "progress":
        picks = 1.0 if case["scheme"] == "Neel" else max(1.0, cells / 3200.0)
        steps = max(1.0, case["mcsteps"] * cells * 0.5 / picks)
    else:
        steps = case["steps"]
    total = steps * _step_bytes(case)
    out = {"bytes": total, "flops": total / 4}
    if call == "resync":
        out = {k: out[k] + full[k] for k in out}
    return out


# ------------------------------------------------------------------------------------------------
# The full sum in 64 bits
# ------------------------------------------------------------------------------------------------
def _convolve(kernel, source):
    """out[y, x] = sum over (y', x') of kernel[y - y' + ny - 1, x - x' + nx - 1] source[y', x']."""
    ny, nx = source.shape
    shape = (3 * ny, 3 * nx)
    full = torch.fft.irfft2(torch.fft.rfft2(kernel, shape) * torch.fft.rfft2(source, shape), shape)
    return full[ny - 1:2 * ny - 1, nx - 1:2 * nx - 1]


def _with_images(kernel, ny, nx):
    """The kernel plus its eight neighbouring periodic images, each where it lies in the window."""
    out = kernel.clone()
    height, width = kernel.shape
    for sy in (-ny, 0, ny):
        for sx in (-nx, 0, nx):
            if sy or sx:
                ys, xs = slice(max(0, sy), min(height, height + sy)), slice(max(0, sx), min(width, width + sx))
                yo, xo = slice(max(0, -sy), min(height, height - sy)), slice(max(0, -sx), min(width, width - sx))
                out[ys, xs] += kernel[yo, xo]
    return out


def exact(case, seed):
    """The energies of an uncut recompute; the other calls' outputs are those of a random walk."""
    if case["call"] != "recompute" or case["cutoff"]:
        return None
    g = np.random.default_rng(seed)
    ny, nx = case["ny"], case["nx"]
    _, a, moment = LATTICES[case["lattice"]]
    spins = torch.from_numpy((g.integers(0, 2, size=(ny, nx)) * 2 - 1).astype(np.float64))
    ix, iy = (torch.from_numpy(v) for v in np.meshgrid(np.arange(nx), np.arange(ny)))
    if case["lattice"] == "square":
        pitch, occupied, angle = (a, a), torch.ones_like(spins), None
    elif case["lattice"] == "pinwheel":
        pitch, occupied = (a / 2, a / 2), ((ix + iy) % 2 == 1).double()
        angle = (iy % 2 == 1).double() * (math.pi / 2) - math.pi / 4
    else:
        pitch = a / 4, a / 4 * math.sqrt(3)
        occupied = (((ix + iy) % 4 == 1) | ((ix - iy) % 4 == 3)).double()
        angle = torch.full_like(spins, math.pi / 2)
        angle[((ix - iy) % 4 == 1) & (ix % 2 == 1)] = -math.pi / 6
        angle[((ix + iy) % 4 == 3) & (ix % 2 == 1)] = math.pi / 6
    mm = spins * occupied * moment
    rx = ((torch.arange(2 * nx - 1) - (nx - 1)).double() * pitch[0])[None, :]
    ry = ((torch.arange(2 * ny - 1) - (ny - 1)).double() * pitch[1])[:, None]
    r2 = rx * rx + ry * ry
    r2[ny - 1, nx - 1] = math.inf
    r3 = 1e-7 * r2 ** -1.5

    def summed(kernel, source):
        return _convolve(_with_images(kernel, ny, nx) if case["pbc"] else kernel, source)

    if angle is None:      # E_i = sum_j mu0 / 4 pi m_i m_j / r^3
        return {"E": mm * summed(r3, mm)}
    ox, oy = torch.cos(angle), torch.sin(angle)
    mx, my = mm * ox, mm * oy
    xx, xy, yy = r3 * (3 * rx * rx / r2 - 1), r3 * (3 * rx * ry / r2), r3 * (3 * ry * ry / r2 - 1)
    fx, fy = summed(xx, mx) + summed(xy, my), summed(xy, mx) + summed(yy, my)    # the field at every site
    # E_i = -m_i . B_i, and the same with the magnet turned by 90 degrees
    return {"E": -mm * (ox * fx + oy * fy), "E_perp": -mm * (ox * fy - oy * fx)}
