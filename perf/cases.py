"""What a program that uses this library has it do, as cases that can be timed and compared.

Two users are behind them.  One links the library under the reference solver's host code:
the reference-named launchers over arrays that the program owns (hash, sort, cell tables,
walls, drag, the explicit particle operators, heat and turbulence), one by one or as the
whole explicit step.  The other runs the library's own semi-implicit step (`Solver`), its
pressure solve alone (`CalcPoisson`), and trains and evaluates the network of the learned
start.  Sizes are those of the scenes in `simulation_project_gb300.scenes` and of the
benchmark: 2,000 to 882,080 particles, batches of 512 to 16,384 rows, 1,000 to 884,736 rows
of inference.
"""
import ctypes as C
import math

import numpy as np
import torch

from simulation_project_gb300 import lib, scenes
from simulation_project_gb300.learned import Mlp
from simulation_project_gb300.lib import call
from simulation_project_gb300.refpath import RefStep
from simulation_project_gb300.solver import Solver

DEV = "cuda"
LARGEST = 884_736
LAYERS = (("in", 12), ("h1", 128), ("h2", 128), ("h3", 128), ("out", 2))


# ---------------------------------------------------------------------------
# cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # the native step on the smallest dam break: launches and host waits count
        {"name": "step_dam_2k", "kind": "step", "scene": "dam", "l0": 0.02, "drag": 0},
        # ... on the rotating bucket with drag spheres, an ordinary size
        {"name": "step_bucket_108k", "kind": "step", "scene": "bucket", "l0": 0.004, "drag": 64},
        # ... and at the size of the benchmark
        {"name": "step_bucket_882k", "kind": "step", "scene": "bucket", "l0": 0.002, "drag": 64},
        # the pressure solve alone, started from zero, as a program that keeps its own step calls it
        {"name": "poisson_103k", "kind": "poisson", "side": 47},
        # the reference's explicit step through its launchers, dam break
        {"name": "explicit_step_16k", "kind": "explicit_step", "scene": "dam", "l0": 0.01, "drag": 0},
        # its layers: the viscous predictor at the largest size
        {"name": "viscous_885k", "kind": "viscous", "side": 96},
        # pressure and its gradient at an ordinary, odd size
        {"name": "pressure_gradient_103k", "kind": "pressure_gradient", "side": 47},
        # heat, turbulence and the turbulent predictor on a small block
        {"name": "heat_turbulence_16k", "kind": "heat_turbulence", "side": 25},
        # hash, sort and reorder: twice in every explicit step
        {"name": "topology_882k", "kind": "topology", "scene": "bucket", "l0": 0.002, "drag": 0},
        # triangle cells, wall distance and drag of the rotating bucket
        {"name": "walls_108k", "kind": "walls", "scene": "bucket", "l0": 0.004, "drag": 64},
        # the network over every particle of the benchmark's scene
        {"name": "mlp_infer_882k", "kind": "mlp_infer", "rows": 882_080},
        # loss and gradients of one training batch (the default batch)
        {"name": "mlp_grad_8192", "kind": "mlp_grad", "rows": 8192},
    ]


def draw(rng):
    def spread(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["step", "step", "poisson", "explicit_step", "viscous", "pressure_gradient", "heat_turbulence",
                       "topology", "walls", "mlp_infer", "mlp_grad"])
    if kind in ("step", "explicit_step", "topology", "walls"):
        bucket = kind == "walls" or rng.random() < 0.6
        most = {"step": 800_000, "explicit_step": 400_000, "topology": 850_000, "walls": 300_000}[kind]
        n = spread(14_000 if bucket else 2_000, most if bucket else 64_000)
        # particles of a scene are about its fluid volume over l0^3
        l0 = round(((0.00692 if bucket else 0.016) / n) ** (1.0 / 3.0), 6)
        return {"kind": kind, "scene": "bucket" if bucket else "dam", "l0": l0,
                "drag": rng.choice({"walls": [1, 16, 64], "topology": [0]}.get(kind, [0, 64]) if bucket else [0])}
    if kind == "mlp_infer":
        return {"kind": kind, "rows": spread(1_000, 880_000)}
    if kind == "mlp_grad":
        return {"kind": kind, "rows": spread(512, 16_384)}
    hi = {"viscous": 94, "pressure_gradient": 80, "heat_turbulence": 60, "poisson": 60}[kind]
    return {"kind": kind, "side": max(12, round(spread(12 ** 3, hi ** 3) ** (1.0 / 3.0)))}


# ---------------------------------------------------------------------------
# what a program has in hand
# ---------------------------------------------------------------------------
def _scene(case, seed):
    seed = int(seed) & 0x7FFFFFFF
    if case["kind"] == "poisson":   # fluid at rest density, as inside a vessel
        return scenes.random_block(case["side"], l0=0.004, seed=seed, jitter=0.02, with_box=False,
                                   explicit_pressure=False)
    if "side" in case:
        sc = scenes.random_block(case["side"], l0=0.004, seed=seed, jitter=0.3, with_box=False)
        if case["kind"] == "heat_turbulence":
            p = sc.param
            p.bUpdateTemperature = p.bTurbulance = True
            p.FruidThermalConductivity, p.FruidThermalResistance = 0.6, 2e-4
            p.MaxWallTemperature, p.MinWallTemperature = 330.0, 290.0
            p.ViscosityUpdateParameterA, p.ViscosityUpdateParameterB = -2e-8, 7e-6
            p.SmagorinskyConstant, p.FilterWidth = 0.12, 0.004
            p.TurbulanViscosityRatio, p.Cnue, p.Cepsilon, p.TurbulanceIntensity = 1e-2, 0.094, 1.048, 0.5
        return sc
    l0 = case["l0"]
    if case["scene"] == "dam":
        return scenes.dam_break(l0=l0, dt=1e-4, seed=seed)
    sc = scenes.rotating_bucket(l0=l0, dt=5e-5, seed=seed, n_drag=case["drag"], drag_seed=seed + 1)
    if case["kind"] == "walls":
        sc.vel = np.random.default_rng(seed).normal(0.0, 0.05, sc.pos.shape)
    return sc


class _View:
    """A device array of the library's caller as a torch tensor, without a copy."""

    def __init__(self, array, shape=None, dtype=None):
        self.array = array
        dtype = np.dtype(dtype or array.dtype)
        self.__cuda_array_interface__ = {"shape": tuple(shape or array.shape), "typestr": dtype.str, "strides": None,
                                         "data": (array.ptr, False), "version": 3}


def _view(g, key):
    a = g.d[key]
    if key == "stl_distance":   # CDistance: magnitude and direction
        return torch.as_tensor(_View(a, (a.shape[0], 4), np.float32), device=DEV)
    return torch.as_tensor(_View(a), device=DEV)


def _bind(g):
    """The binding calls of a program that holds several particle sets: the launchers use
    the set that was bound last."""
    d, p = g.p, call
    p("InitializeDeviceMemConst", g.param, g.n, d("triangles"), g.t, g.tp.ptr, g.capacity, d("stl_distance"),
      d("stl_id"), d("cells"), g.cells, d("cell_start"), d("cell_end"), d("index"), g.box)
    p("InitializeDeviceConstOutPutParticles", d("out_id"), d("out_pos"), d("out_vel"), d("out_pressure"),
      d("out_density"), d("out_temperature"), d("out_kin_visc"), d("out_solid_rate"), d("out_type"))
    p("InitializeDeviceConstInputParticles", *[d(k) for k in RefStep.IN + ["turb_visc", "strain"]])
    p("DragParametersToConst", g.dp.ptr, d("drag_acc"), d("drag_temperature"), g.drag_num, d("magnifier_count"), None)


def _topology(g):
    s, d = g.stream.ref(), g.p
    call("CaculateCellIDandInitializeHash", s, g.n, g.cells, d("hash"), d("index"), d("out_pos"))
    g.stream.sync()   # SortUsingThrust runs on the legacy default stream
    call("SortUsingThrust", g.n, d("hash"), d("index"))
    call("reorderDataAndFindCellStart", s, g.n, g.cells, d("hash"), d("index"), d("cell_start"), d("cell_end"))


OUT = {
    "explicit_step": ("out_id", "out_pos", "out_vel", "out_pressure", "out_density", "stl_id", "stl_distance"),
    "viscous": ("out_pos", "out_vel"),
    "pressure_gradient": ("out_pressure", "out_density", "out_pos", "out_vel"),
    "heat_turbulence": ("out_temperature", "out_kin_visc", "turb_visc", "strain", "out_pos", "out_vel"),
    "topology": ("hash", "index", "cell_start", "cell_end", "id", "pos", "vel", "pressure", "density", "temperature",
                 "kin_visc", "solid_rate", "type"),
    "walls": ("stl_id", "stl_distance", "drag_acc", "out_type"),
}


def _weights(seed):
    """Network parameters as a training run starts from, in the order of the parameter vector."""
    g = torch.Generator().manual_seed(int(seed) + 17)
    parts = []
    for (_, a), (name, b) in zip(LAYERS[:-1], LAYERS[1:]):
        s = 1.0 / math.sqrt(a)
        parts += [torch.empty(a, b).uniform_(-s, s, generator=g), torch.empty(b).uniform_(-s, s, generator=g)]
    return parts


def _rows(case, seed):
    g = torch.Generator(device=DEV).manual_seed(int(seed))
    x = torch.randn(case["rows"], 12, device=DEV, generator=g)
    t = torch.randn(case["rows"], 2, device=DEV, generator=g) * 0.3
    return x, t


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("mlp_infer", "mlp_grad"):
        x, t = _rows(case, seed)
        m = Mlp(max_batch=case["rows"] if kind == "mlp_grad" else 1024, seed=1)
        m.set_params(torch.cat([p.reshape(-1) for p in _weights(seed)]).numpy())
        y = torch.empty(case["rows"], 2, device=DEV)
        grad = torch.empty(sum(p.numel() for p in _weights(0)), device=DEV)
        return {"kind": kind, "net": m, "x": x, "t": t, "y": y, "grad": grad}
    sc = _scene(case, seed)
    if kind == "step":
        n = sc.n
        host = [torch.empty(n, 3, dtype=torch.float64, pin_memory=True),
                torch.empty(n, 3, dtype=torch.float64, pin_memory=True),
                torch.empty(n, dtype=torch.float64, pin_memory=True)]
        return {"kind": kind, "solver": Solver(sc, precision="fp32_ir"), "i": 0, "host": host,
                "np": [h.numpy() for h in host], "state": [torch.empty_like(h, dtype=torch.float32) for h in host]}
    if kind == "poisson":
        out = [torch.zeros(sc.n, device=DEV) for _ in range(3)]
        return {"kind": kind, "solver": Solver(sc, precision="fp32_ir"), "n": sc.n, "out": out,
                "zero": torch.zeros(sc.n, device=DEV)}
    g = RefStep(sc)
    if kind == "heat_turbulence":
        warm = np.random.default_rng(seed).uniform(295, 325, sc.n).astype(np.float32)
        g.d["out_temperature"].upload(warm)
    if kind not in ("explicit_step", "topology"):
        _bind(g)
        _topology(g)
        g.sync()
        if kind != "walls":   # no wall near any particle
            s = g.stream.ref()
            call("ResetTriangleTopology", s, g.cells, g.p("cells"))
            call("CalcSTLDistance", s, g.n)
            g.sync()
    return {"kind": kind, "g": g, "i": 0, "out": {k: _view(g, k) for k in OUT[kind]}}


def run(state):
    kind = state["kind"]
    if kind == "step":
        # one step, and its state as the reference's own particle records hold it (float)
        state["solver"].step(state["i"])
        state["i"] += 1
        state["solver"].download_state(*state["np"])
        for a, b in zip(state["state"], state["host"]):
            a.copy_(b)
        return dict(zip(("pos", "vel", "press"), state["state"]))
    if kind == "poisson":
        a, b, x = state["out"]
        state["solver"].calc_poisson(state["n"], a.data_ptr(), b.data_ptr(), x.data_ptr(), state["zero"].data_ptr())
        return {"diagonal": a, "rhs": b, "pressure": x}
    if kind == "mlp_infer":
        state["net"].forward(state["x"].data_ptr(), state["y"].data_ptr(), state["x"].shape[0])
        return state["y"]
    if kind == "mlp_grad":
        loss = state["net"].loss_grad(state["x"].data_ptr(), state["t"].data_ptr(), state["x"].shape[0],
                                      state["grad"].data_ptr())
        return {"loss": loss, "grad": state["grad"]}
    g = state["g"]
    _bind(g)
    s, n = g.stream.ref(), g.n
    if kind == "explicit_step":
        g.step(state["i"])
        state["i"] += 1
    elif kind == "topology":
        _topology(g)
    elif kind == "viscous":
        call("CalcExplicitly", s, n)
    elif kind == "pressure_gradient":
        call("CalcExplicitPressure", s, n)
        call("CalcExplicitPressureGradient", s, n)
    elif kind == "heat_turbulence":
        call("CalcTemperatureFactor", s, n)
        call("CalcTurbulenceViscosity", s, n)
        call("CalcExplicitly", s, n)
    else:
        call("ResetTriangleTopology", s, g.cells, g.p("cells"))
        call("RegisterTriangleTopology", s, g.p("triangles"), g.t, g.p("cells"), g.cells)
        call("CalcSTLDistance", s, n)
        call("CalcDragEffect", s, n)
    return state["out"]


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def _count(case):
    if "rows" in case:
        return case["rows"]
    if "side" in case:
        return case["side"] ** 3
    return (0.00706 if case["scene"] == "bucket" else 0.016) / case["l0"] ** 3


def work(case):
    n, kind = _count(case), case["kind"]
    near, far = 33.0, 250.0   # neighbours within 2.1 and 4 particle distances
    if kind == "mlp_infer":
        return {"bytes": n * 56.0, "flops": n * 2.0 * (12 * 128 + 2 * 128 * 128 + 128 * 2)}
    if kind == "mlp_grad":
        return {"bytes": n * 56.0 + 8 * 34946, "flops": n * 6.0 * (12 * 128 + 2 * 128 * 128 + 128 * 2)}
    if kind == "topology":   # positions to keys; nine arrays to sorted order; keys and indices
        return {"bytes": n * (12 + 8 + 2 * 48.0), "flops": n * 6.0}
    if kind == "viscous":
        return {"bytes": n * (12 + 12 + 8 + 24.0), "flops": n * far * 20}
    if kind == "pressure_gradient":
        return {"bytes": n * (12 + 12 + 20 + 8 + 32.0), "flops": n * near * 40}
    if kind == "heat_turbulence":
        return {"bytes": n * (12 + 12 + 8 + 48.0), "flops": n * (near * 80 + far * 20)}
    if kind == "walls":   # positions, velocities; distance, id, drag, type; the triangles
        return {"bytes": n * (12 + 12 + 20 + 20.0) + 9216 * 52.0, "flops": n * 100.0}
    if kind == "poisson":   # positions and start in; three arrays out; a hundred products with the matrix
        return {"bytes": n * (24 + 4 + 12.0), "flops": n * far * (20 + 100 * 2)}
    if kind == "explicit_step":
        return {"bytes": n * 2 * 60.0, "flops": n * (far * 20 + near * 40)}
    return {"bytes": n * 2 * 56.0, "flops": n * far * (2 * 20 + 25 * 2)}   # step


# ---------------------------------------------------------------------------
# the same in 64 bits
# ---------------------------------------------------------------------------
def _neighbours(pos, re, chunk):
    """(targets, candidates, difference, distance, inside) of all pairs closer than re, by
    chunks of targets: pos[candidate] - pos[target], padded."""
    lo = pos.min(0).values
    c = ((pos - lo) / re).long() + 1
    dims = c.max(0).values + 2
    key = (c[:, 0] * dims[1] + c[:, 1]) * dims[2] + c[:, 2]
    skey, order = torch.sort(key, stable=True)
    cells = int(dims.prod())
    start = torch.searchsorted(skey, torch.arange(cells + 1, device=pos.device))
    most = int((start[1:] - start[:-1]).max())
    off = torch.tensor([[i, j, k] for i in (-1, 0, 1) for j in (-1, 0, 1) for k in (-1, 0, 1)], device=pos.device)
    off = (off[:, 0] * dims[1] + off[:, 1]) * dims[2] + off[:, 2]
    slot = torch.arange(most, device=pos.device)
    for t in torch.split(order, chunk):
        cell = key[t][:, None] + off[None]
        s, e = start[cell], start[cell + 1]
        at = s[..., None] + slot
        ok = (at < e[..., None]).flatten(1)
        j = order[at.clamp(max=pos.shape[0] - 1)].flatten(1)
        diff = pos[j] - pos[t][:, None]
        r = diff.square().sum(-1).sqrt()
        ok &= (r < re) & (j != t[:, None])
        yield t, j, diff, torch.where(ok, r, torch.ones_like(r)), ok


def _exact_layers(case, seed):
    sc = _scene(case, seed)
    p, kind = sc.param, case["kind"]
    l0 = float(p.InitialParticleDistance)
    pos = torch.tensor(sc.pos.astype(np.float32), device=DEV).double()
    vel = torch.tensor(sc.vel.astype(np.float32), device=DEV).double()
    n, dt, rho, n0 = sc.n, float(p.Dt), float(p.Density), float(p.ConstantParticleDensity)
    reg, rel = float(p.GradientInfluenceRadiusCoefficient) * l0, float(p.LaplacianInfluenceRadiusCoefficient) * l0
    new = lambda *s: torch.zeros(*s, dtype=torch.float64, device=DEV)  # noqa: E731
    out = {k: None for k in OUT[kind]}

    def w_of(re, r, ok):
        return torch.where(ok, re / r - 1, torch.zeros_like(r))

    visc = torch.tensor(sc.visc.astype(np.float32), device=DEV).double()
    if kind == "heat_turbulence":
        temp = torch.tensor(np.random.default_rng(seed).uniform(295, 325, n).astype(np.float32), device=DEV).double()
        heat, grad = new(n), new(n, 3, 3)
        for t, j, d, r, ok in _neighbours(pos, reg, 16384):
            w = w_of(reg, r, ok)
            den = r * r * (1 / p.FruidThermalConductivity + p.FruidThermalResistance / r)
            heat[t] = ((temp[j] - temp[t][:, None]) * w / den).sum(1)
            grad[t] = torch.einsum("ija,ijb,ij->iab", vel[j] - vel[t][:, None], d, w / (r * r))
        temp = temp + dt * 2 * p.Dimension / (n0 * rho * p.FruidSpecificHeat) * heat
        temp = temp.clamp(p.MinWallTemperature, p.MaxWallTemperature)
        out["out_temperature"] = temp
        out["out_kin_visc"] = p.ViscosityUpdateParameterA * temp + p.ViscosityUpdateParameterB
        grad = grad * (p.Dimension / n0)
        sym = 0.5 * (grad + grad.transpose(1, 2))
        strain = (torch.diagonal(grad, dim1=1, dim2=2).square().sum(1)
                  + 2 * (sym[:, 0, 1] ** 2 + sym[:, 0, 2] ** 2 + sym[:, 1, 2] ** 2))
        tv = ((p.SmagorinskyConstant * p.FilterWidth) ** 2 * (2 * strain).sqrt()).clamp(max=p.TurbulanViscosityRatio)
        tke = (strain * 2 * p.Cnue * l0 * l0 / p.Cepsilon).clamp(max=p.TurbulanceIntensity)
        visc = visc + tv
        # these two are in sorted order
        order = torch.sort(_hash(sc, pos.float()), stable=True).indices
        out["turb_visc"], out["strain"] = tv[order], tke[order]
    if kind == "pressure_gradient":
        dens = new(n)
        for t, j, d, r, ok in _neighbours(pos, reg, 16384):
            dens[t] = w_of(reg, r, ok).sum(1)
        sonic = 20.0   # RefStep's speed of sound
        pr = torch.where(dens > n0 * p.FreeSurfaceThreshold, sonic ** 2 * rho / n0 * (dens - n0), 0 * dens)
        acc = new(n, 3)
        for t, j, d, r, ok in _neighbours(pos, reg, 16384):
            pc = 0.5 * (pr[j] + pr[t][:, None]) * w_of(reg, r, ok) / (r * r)
            acc[t] = (pc[..., None] * d).sum(1)
        v = vel - dt / rho * (2 * p.Dimension / n0) * acc
        most, a = l0 * p.CourantNumber / dt, v.norm(dim=1, keepdim=True)
        v = torch.where(a > most, most * v / a, v)
        return {"out_pressure": pr, "out_density": dens, "out_pos": pos + (v - vel) * dt, "out_vel": v}
    lap, art, col = new(n, 3), new(n, 3), new(n, 3)
    rc = float(p.r_coeff) * l0
    for t, j, d, r, ok in _neighbours(pos, rel, 8192):
        w = w_of(rel, r, ok)
        lap[t] = torch.einsum("ij,ija->ia", w, vel[j] - vel[t][:, None])
        touch = ok & (r < rc)
        art[t] = torch.einsum("ij,ija->ia", torch.where(touch, p.ArtificialPressure * w / (r * r), 0 * w), d)
        col[t] = torch.einsum("ij,ija->ia", torch.where(touch, (rc - r) / r, 0 * w), d)
    g = torch.tensor([p.GravityConstant.x, p.GravityConstant.y, p.GravityConstant.z], device=DEV).double()
    v = vel + dt * (g + 2.0 * p.Dimension / (p.LambdaValue * n0) * lap * visc[:, None])
    v = v + dt * (art * (-p.Dimension / (n0 * rho)) + 0.01 * col)
    out["out_pos"], out["out_vel"] = pos + dt * v, v
    return out


def _exact_poisson(case, seed):
    sc = _scene(case, seed)
    p = sc.param
    l0, dt, rho = float(p.InitialParticleDistance), float(p.Dt), float(p.Density)
    pos, n = torch.tensor(sc.pos, device=DEV), sc.n
    reg, rel = float(p.GradientInfluenceRadiusCoefficient) * l0, float(p.LaplacianInfluenceRadiusCoefficient) * l0
    pnd, sumw = (torch.zeros(n, dtype=torch.float64, device=DEV) for _ in range(2))
    rows, cols, vals = [], [], []
    for t, j, d, r, ok in _neighbours(pos, rel, 8192):
        w = torch.where(ok, rel / r - 1, torch.zeros_like(r))
        sumw[t] = w.sum(1)
        pnd[t] = torch.where(ok & (r < reg), reg / r - 1, torch.zeros_like(r)).sum(1)
        rows.append(t[:, None].expand_as(j)[ok].int())
        cols.append(j[ok].int())
        vals.append(w[ok])
    coef, kappa = 2.0 * p.Dimension / (sc.lam * sc.n0_lap), 1e-9 * rho / (dt * dt)
    inner = pnd > float(p.FreeSurfaceThreshold) * sc.n0_pnd
    diag = torch.where(inner, coef * sumw + kappa, 0 * sumw)
    rhs = torch.where(inner, 0.05 * rho / (dt * dt) * (pnd - sc.n0_pnd) / sc.n0_pnd, 0 * pnd)
    rows, cols, vals = torch.cat(rows).long(), torch.cat(cols).long(), torch.cat(vals)
    vals = torch.where(inner[rows] & inner[cols], coef * vals, 0 * vals)
    A = torch.sparse_coo_tensor(torch.stack([rows, cols]), vals, (n, n)).coalesce().to_sparse_csr()
    safe = torch.where(inner, diag, torch.ones_like(diag))
    x, r = torch.zeros_like(rhs), rhs.clone()
    z = r / safe
    q, rz, stop = z.clone(), torch.dot(r, z), 1e-13 * float(rhs.norm())
    for _ in range(2000):
        if float(r.norm()) <= stop:
            break
        y = diag * q - (A @ q[:, None])[:, 0]
        a = rz / torch.dot(q, y)
        x, r = x + a * q, r - a * y
        z = r / safe
        new = torch.dot(r, z)
        q, rz = z + new / rz * q, new
    return {"diagonal": diag, "rhs": rhs, "pressure": x}


def _hash(sc, pos):
    """Cell keys of single-precision positions."""
    lo = sc.box.m_BufferedZone.m_MinBound
    lo = torch.tensor([lo.x, lo.y, lo.z], dtype=torch.float32, device=DEV)
    c = ((pos - lo) / torch.tensor(sc.box.m_CellSize, dtype=torch.float32, device=DEV)).trunc().long()
    size = sc.box.m_GridSize
    return (c[:, 0] * size.y + c[:, 1]) * size.z + c[:, 2]


def _exact_topology(case, seed):
    sc = _scene(case, seed)
    pos = torch.tensor(sc.pos.astype(np.float32), device=DEV)
    order = torch.sort(_hash(sc, pos), stable=True).indices
    out = {k: None for k in OUT["topology"]}
    zero = torch.zeros(sc.n, dtype=torch.float64, device=DEV)
    out.update(pos=pos[order].double(), vel=torch.tensor(sc.vel, device=DEV)[order],
               pressure=zero, density=zero, temperature=zero, solid_rate=zero,
               kin_visc=torch.tensor(sc.visc.astype(np.float32), device=DEV).double()[order])
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind in ("mlp_infer", "mlp_grad"):
        x, t = _rows(case, seed)
        ps = [p.to(DEV).double().requires_grad_(kind == "mlp_grad") for p in _weights(seed)]
        h = x.double()
        for k in range(0, 8, 2):
            h = h @ ps[k] + ps[k + 1]
            if k < 6:
                h = torch.nn.functional.silu(h)
        if kind == "mlp_infer":
            return h
        loss = ((h - t.double()).square() * torch.tensor([1.0, 0.25], device=DEV).double()).sum() / x.shape[0]
        loss.backward()
        return {"loss": float(loss), "grad": torch.cat([p.grad.reshape(-1) for p in ps])}
    if kind == "poisson":
        return _exact_poisson(case, seed)
    if kind == "topology":
        return _exact_topology(case, seed)
    if kind in ("viscous", "pressure_gradient", "heat_turbulence"):
        return _exact_layers(case, seed)
    return None   # whole steps, and the reference's own wall distance, have no value in 64 bits of the same meaning
