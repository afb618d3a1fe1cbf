"""What a user of this framework runs, as cases to be timed and compared.

Each case is one pass through public entry points: the time step of a model
(fesomc.model.GpuModel, an ensemble of members packed per level count), the
learned closure's network (fesomc.closure.Closure) and the energy of a state
in the caller's device arrays (fesomc_energy_device).  The mesh of a case is
fixed by its sizes; the initial temperature and salinity, the wind stress and
the tide come from the seed.
"""
import collections
import ctypes as C
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "fesom-c_b200"))

from fesomc import abi, cases, closure, ensemble, model  # noqa: E402

HIDDEN = 256   # width of the closure network's three hidden layers

ETA, UV2D, UV3D, TS, MIX, WVEL = abi.F_ETA, abi.F_UV2D, abi.F_UV3D, abi.F_TS, abi.F_MIX, abi.F_WVEL
RESULT = ETA | UV2D | UV3D | TS | MIX | WVEL      # the prognostic state and the mixing fields
SURFACE = ETA | UV2D | TS                          # what an output file of a large run holds
FIELDS = {ETA: ("eta_n",), UV2D: ("U_n_2D",), UV3D: ("U_n", "V_n"), TS: ("TF", "SF"), MIX: ("bt", "Kv", "Av"),
          WVEL: ("Wvel",)}


def listed():
    return [
        # the reference's own test case, a lock exchange with upwind
        # tracers on 39 layers: its energy written every 100 steps
        {"name": "lock-exchange-100", "kind": "lock", "steps": 100},
        # the smallest call: one step of a small mesh with the forcing from
        # the host and the state read back, as a driver that couples another
        # model does every step
        dict(STEP, name="small-1", nx=40, ny=16, nsigma=11, dx=300.0, h1=25.0, steps=1, host=True, out=RESULT),
        # the 16,281-node benchmark mesh as the Fortran driver runs it: the
        # forcing of every step pushed from the host, output after ten
        dict(STEP, name="estuary-16k-host", nx=200, ny=80, nsigma=11, dx=300.0, h1=25.0, steps=10, host=True,
             out=RESULT),
        # a mid-size mesh in its file order (numbered at random) with 21
        # levels, temperature by Miura's scheme and the biharmonic viscosities
        dict(STEP, name="estuary-42k-miura-bih", nx=300, ny=140, nsigma=21, dx=150.0, h1=40.0, steps=20, adv=4,
             bih=True, shuffle=True, out=RESULT),
        # upwind tracers, atmospheric fluxes and tidal potential on the
        # device, and a level count no kernel is specialised for
        dict(STEP, name="estuary-40k-atm-upwind", nx=271, ny=147, nsigma=31, dx=150.0, h1=40.0, steps=20, adv=1,
             atm=True, out=RESULT),
        # the FP32 form along the space-filling curve at a quarter of the
        # benchmark's nodes: the production form for long runs
        dict(STEP, name="estuary-232k-fp32", nx=700, ny=330, nsigma=21, dx=170.0, h1=40.0, steps=60, fp32=True,
             sfc=True, out=SURFACE),
        # the benchmark workload: 1.05 M nodes, 21 levels, FP64, MUSCL
        # tracers, stored along the curve, output every twenty minutes
        dict(STEP, name="estuary-1052k-fp64", nx=1500, ny=700, nsigma=21, dx=80.0, h1=40.0, steps=60, sfc=True,
             out=SURFACE),
        # a perturbed ensemble of twelve members of 4k to 40k nodes, packed
        # by level count, FP32 form
        {"name": "ensemble-12-packed", "kind": "ensemble", "members": 12, "lo": 4000, "hi": 40000, "steps": 10},
        # the closure's network on a column set: inference on the tensor
        # cores, as the closure is evaluated off-line
        {"name": "closure-forward-48k", "kind": "forward", "nsigma": 21, "columns": 48000},
        # one training batch: loss and gradients of the largest minibatch
        {"name": "closure-grad-8192", "kind": "grad", "nsigma": 21, "columns": 8192},
        # the energy diagnostic over a caller's own device arrays
        {"name": "energy-262k", "kind": "energy", "nodes": 262144},
    ]


# a time-step case without options: MUSCL tracers, FP64, the mesh's own order,
# forcing evaluated on the device
STEP = {"kind": "step", "nx": 40, "ny": 16, "nsigma": 11, "dx": 300.0, "h1": 25.0, "steps": 1, "adv": 2, "fp32": False,
        "sfc": False, "host": False, "bih": False, "atm": False, "shuffle": False, "out": RESULT}


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step"] * 7 + ["ensemble", "forward", "grad", "energy"])
    if kind == "ensemble":
        lo = _log(rng, 1000, 6000)
        return {"kind": kind, "members": rng.randint(3, 10), "lo": lo, "hi": lo * rng.randint(2, 7),
                "steps": rng.randint(3, 12)}
    if kind == "forward":
        return {"kind": kind, "nsigma": rng.randint(8, 32), "columns": _log(rng, 100, 60000)}
    if kind == "grad":
        return {"kind": kind, "nsigma": rng.randint(8, 32), "columns": _log(rng, 64, 8192)}
    if kind == "energy":
        return {"kind": kind, "nodes": _log(rng, 1000, 1000000)}
    nodes = _log(rng, 700, 250000)
    aspect = rng.uniform(1.5, 3.0)
    ny = max(12, int(math.sqrt(nodes / aspect)))
    nx = max(24, int(nodes / ny))
    small = nodes < 60000
    adv = rng.choice([2, 2, 2, 1, 4])
    fp32 = rng.random() < 0.3
    return dict(STEP, nx=nx, ny=ny, nsigma=rng.choice([11, 21, 21, rng.randint(9, 36)]), dx=170.0, h1=40.0,
                steps=rng.randint(1, 24) if small else rng.randint(20, 60), adv=adv, fp32=fp32,
                sfc=rng.random() < 0.5, host=rng.random() < 0.3, bih=small and adv == 4 and not fp32,
                atm=adv == 1 and not fp32, shuffle=rng.random() < 0.2, out=RESULT if small else SURFACE)


# --------------------------------------------------------------------------
# cases with a mesh: the last few are kept, as a program keeps its mesh while
# it starts runs from other states
# --------------------------------------------------------------------------
_bases = collections.OrderedDict()


def _keep(key, make):
    if key in _bases:
        _bases.move_to_end(key)
    else:
        while len(_bases) >= 2:
            _bases.popitem(last=False)
        _bases[key] = make()
    return _bases[key]


def _estuary(c):
    over = {"fp32_form": int(c["fp32"]), "sfc_order": int(c["sfc"])}
    if c["bih"]:
        over.update(bih_3D=1, bih_2D=1, Abh0=10.0)
    if c["atm"]:
        over.update(T_potential=1, atm={"qns": -50.0, "qsr": 100.0})
    if c["shuffle"]:
        over["shuffle"] = 7
    return cases.estuary_case("estuary", c["nx"], c["ny"], c["dx"], c["nsigma"], 2.0, c["h1"], stress=(0.0, 0.1),
                              tracer_adv=c["adv"], **over)


def _seeded(base, seed, salt=True):
    """The case on the same mesh with temperature, salinity, wind stress and
    tide of this seed."""
    rng = np.random.default_rng(seed)
    m = base.mesh
    x, y = m.coord_nod2D[:, 0], m.coord_nod2D[:, 1]
    span = max(float(np.ptp(x)), 1e-30)
    p1, p2, k = rng.uniform(0.0, 6.28, 3), rng.uniform(0.0, 6.28, 3), rng.uniform(2.0, 12.0, 6)
    wave = sum(np.sin(k[i] * x / span + p1[i]) * np.sin(k[3 + i] * y / span + p2[i]) for i in range(3)) / 3.0
    state = dict(base.state0)
    state["TF"] = (base.state0["TF"].reshape(m.N, m.L) + 0.2 * wave[:, None]).reshape(-1)
    if salt:
        state["SF"] = (base.state0["SF"].reshape(m.N, m.L) + 0.1 * wave[:, None]).reshape(-1)
    state["T_old"], state["Tclim"] = state["TF"].copy(), state["TF"].copy()
    state["S_old"], state["Sclim"] = state["SF"].copy(), state["SF"].copy()
    f0 = base.forcing_fn(1, cases.advance_time(base.params.time_jd0, base.params.dt))
    factor = {"taux": rng.uniform(0.7, 1.2), "ampt": rng.uniform(0.8, 1.1)}
    factor["tauy"] = factor["taux"]
    held = {n: f0[n] * v for n, v in factor.items() if n in f0}

    def forcing(step, time_jd):
        f = base.forcing_fn(step, time_jd)
        f.update(held)
        return f

    return cases.Case(base.name, m, base.params, state, forcing, meta=base.meta)


def _device_forcing(g):
    case = g.case
    f = case.forcing_fn(1, case.params.time_jd0 + 20.0)   # past the ramp: the full runoff
    g.set_forcing(f)
    base = np.ascontiguousarray(f["runoff_rivers"])
    abi.check(g.lib.fesomc_gpu_set_device_forcing(g.h, abi.dptr(base), 1), "fesomc_gpu_set_device_forcing")


def _fields(g, groups):
    """The fields of an output file.  The FP32 form holds all but the
    elevation in FP32: a program that runs it writes them so."""
    st = g.state(groups)
    out = {n: st[n] for bit, names in FIELDS.items() if bit & groups for n in names}
    if g.case.params.fp32_form:
        out = {n: v if n == "eta_n" else v.astype(np.float32) for n, v in out.items()}
    return out


def prepare(case, seed):
    kind = case["kind"]
    if kind == "lock":
        base = _keep(kind, cases.le_medium)
        return {"kind": kind, "model": model.GpuModel(_seeded(base, seed, salt=False)), "steps": case["steps"]}
    if kind == "step":
        sizes = {k: v for k, v in case.items() if k not in ("name", "steps", "host", "out")}
        base = _keep(repr(sorted(sizes.items())), lambda: _estuary(case))
        g = model.GpuModel(_seeded(base, seed))
        g.arrays = None            # the model has its own copy on the device
        if case["atm"] and not case["fp32"]:
            g.set_atm_fields(*cases.atm_coefficients(g.case.mesh, g.case.params.time_jd0))
        if not case["host"]:
            _device_forcing(g)
        return {"kind": kind, "model": g, "steps": case["steps"], "host": case["host"], "out": case["out"]}
    if kind == "ensemble":
        members = _keep(repr(("ensemble", case["members"], case["lo"], case["hi"])), lambda: [
            cases.ensemble_member(i, nodes_range=(case["lo"], case["hi"]), fp32_form=1)
            for i in range(case["members"])])
        ens = ensemble.PackedEnsemble([_seeded(m, [seed, i]) for i, m in enumerate(members)])
        return {"kind": kind, "ensemble": ens, "steps": case["steps"]}
    gen = torch.Generator().manual_seed(seed)
    if kind in ("forward", "grad"):
        net = closure.Closure(case["nsigma"])
        p, X, T = _network(case, gen)
        net.params(p.numpy())
        return {"kind": kind, "net": net, "X": X.numpy(), "T": T.numpy()}
    en, arrays = _energy_arrays(case, gen)
    dev = [a.to("cuda") for a in arrays]
    return {"kind": kind, "nodes": en.to("cuda"), "arrays": dev, "lib": abi.load()}


def run(state):
    kind = state["kind"]
    if kind == "lock":
        g = state["model"]
        g.run(state["steps"])
        return dict(_fields(g, ETA | UV2D | UV3D | MIX | WVEL), T=_fields(g, TS)["TF"], energy=g.energy())
    if kind == "step":
        g = state["model"]
        if state["host"]:
            g.step(state["steps"])
        else:
            g.run(state["steps"])
        return _fields(g, state["out"])
    if kind == "ensemble":
        ens = state["ensemble"]
        _, status = ens.run(state["steps"])
        out = [_fields(g, SURFACE) for g in ens.models]
        return {"status": status, "packs": out}
    if kind == "forward":
        return state["net"].forward(state["X"], bf16=True)
    if kind == "grad":
        loss, g = state["net"].grad(state["X"], state["T"])
        return {"loss": loss, "gradients": g}
    eta, depth, area, w_cv, u2, earea = state["arrays"]
    e = C.c_double()
    rc = state["lib"].fesomc_energy_device(
        eta.numel(), earea.numel(), 1.0, eta.data_ptr(), depth.data_ptr(), area.data_ptr(), state["nodes"].data_ptr(),
        w_cv.data_ptr(), u2.data_ptr(), earea.data_ptr(), torch.cuda.current_stream().cuda_stream, C.byref(e))
    abi.check(rc, "fesomc_energy_device")
    return e.value


# --------------------------------------------------------------------------
# the network and the energy: inputs, and their results in 64 bits
# --------------------------------------------------------------------------
def _dims(case):
    return [3 * case["nsigma"] + 3, HIDDEN, HIDDEN, HIDDEN, case["nsigma"]]


def _network(case, gen):
    d = _dims(case)
    parts = []
    for l in range(4):   # weights of a trained network's size, small biases
        parts.append(torch.randn(d[l + 1] * d[l], generator=gen) / math.sqrt(d[l]))
        parts.append(0.1 * torch.randn(d[l + 1], generator=gen))
    n = case["columns"]
    X = torch.randn(n, d[0], generator=gen)
    return torch.cat(parts), X, torch.randn(n, d[4], generator=gen)


def _forward64(case, p, X):
    d, o, a = _dims(case), 0, X
    for l in range(4):
        W = p[o:o + d[l + 1] * d[l]].view(d[l + 1], d[l])
        o += d[l + 1] * d[l]
        z = a @ W.T + p[o:o + d[l + 1]]
        o += d[l + 1]
        a = torch.nn.functional.silu(z) if l < 3 else z
    return a


def _energy_arrays(case, gen):
    """A mesh of rows of quads and triangles, with the elevation, depth and
    velocities of a shallow sea."""
    n = case["nodes"]
    row = max(4, int(math.sqrt(n)))
    e = max(1, n - row - 1)
    i = torch.arange(e, dtype=torch.int32)
    tri = torch.rand(e, generator=gen) < 0.4
    en = torch.stack([i, i + row, i + row + 1, torch.where(tri, i, i + 1)], dim=1) + 1
    f = lambda *s: torch.rand(*s, generator=gen, dtype=torch.float64)  # noqa: E731
    w = 0.25 + 0.1 * f(e, 4)
    return en.contiguous(), [2.4 * f(n) - 1.2, 40.0 * f(n), 6400.0 * (0.8 + 0.4 * f(n)), w / w.sum(1, keepdim=True),
                             1.0 * f(e, 2) - 0.5, 6400.0 * (0.8 + 0.4 * f(e))]


def exact(case, seed):
    kind = case["kind"]
    if kind in ("lock", "step", "ensemble"):
        return None      # a whole model: its own arithmetic is the only one
    gen = torch.Generator().manual_seed(seed)
    if kind == "energy":
        en, (eta, depth, area, w, u2, earea) = _energy_arrays(case, gen)
        idx = (en - 1).long()
        h = (w * torch.clamp(depth + eta, min=1.0)[idx]).sum(1)
        pe = math.fsum((0.5 * 9.8 * area * eta * eta).tolist())
        ke = math.fsum((0.5 * h * earea * (u2 * u2).sum(1)).tolist())
        return (pe + ke) / math.fsum(area.tolist())
    p, X, T = (t.double() for t in _network(case, gen))
    if kind == "forward":
        return _forward64(case, p, X)
    p.requires_grad_(True)
    loss = ((_forward64(case, p, X) - T) ** 2).mean()
    return {"loss": loss.item(), "gradients": torch.autograd.grad(loss, p)[0]}


# --------------------------------------------------------------------------
def _step_bytes(nodes, layers, form_bytes):
    """The prognostic fields of one step, read and written once: per node
    layer T and S at two time levels, their climatology (read), Kv, bt and W;
    per element layer (1.3 elements a node) the velocities, their AB
    right-hand sides, the filtered velocities and Av."""
    per_node = (4 * 2 + 2 + 2 * 2 + 2) * form_bytes
    per_elem = 1.3 * (7 * 2) * form_bytes
    return nodes * layers * (per_node + per_elem)


def work(case):
    kind = case["kind"]
    if kind == "lock":
        return {"bytes": _step_bytes(4515, 39, 8) * case["steps"], "flops": 0}
    if kind == "step":
        n = (case["nx"] + 1) * (case["ny"] + 1)
        return {"bytes": _step_bytes(n, case["nsigma"] - 1, 4 if case["fp32"] else 8) * case["steps"], "flops": 0}
    if kind == "ensemble":
        total = 0.0
        for i in range(case["members"]):
            d = cases.ensemble_draw(i, nodes_range=(case["lo"], case["hi"]))
            total += _step_bytes((d["nx"] + 1) * (d["ny"] + 1), d["nsigma"] - 1, 4)
        return {"bytes": total * case["steps"], "flops": 0}
    if kind == "energy":
        n = case["nodes"]
        return {"bytes": n * 24 + n * (16 + 32 + 16 + 8), "flops": 30 * n}
    d, n = _dims(case), case["columns"]
    params = sum(d[l] * d[l + 1] for l in range(4))
    if kind == "forward":
        return {"bytes": 4 * n * (d[0] + d[4]) + 4 * params, "flops": 2 * params * n}
    return {"bytes": 4 * n * (d[0] + d[4]) + 8 * params, "flops": 6 * params * n}
