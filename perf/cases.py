"""What a user of this package has the GPU do, as cases that can be timed and compared.

Whole calls: the large step replayed from its CUDA graph (``Model``), from the smallest mesh
of the tests to the headline mesh, in both precisions, dry and moist, flat and over terrain;
a batched ensemble; and a gradient (the forward and reverse mode of a short run).  Single
stages through the C entry points on a resident model (``Model.call``), as a host model calls
them: the tendencies, the implicit acoustic stage, the diagnostics with the wind
reconstruction, and both scalar transports.

Meshes, level counts, tracers and time steps come from the benchmark's workloads and the
tests; ``draw`` spreads the same ranges (meshes of 162 to 10242 cells, 8 to 64 levels, 1 to 8
tracers).  ``exact`` evaluates the single stages in plain float64 torch; the whole calls
chain hundreds of stage calls and have no such value here.
"""

from __future__ import annotations

import ctypes as C
import functools
import math
from types import SimpleNamespace

import numpy as np
import torch

from mpas_dycore_pytorch_gb300.api import Model
from mpas_dycore_pytorch_gb300.cases import CaseSpec, build_mesh, initial_state
from mpas_dycore_pytorch_gb300.diagnostics import physics_interface_surface_pressure, surface_pressure_functional
from mpas_dycore_pytorch_gb300.dyn_adjoint import DynamicsAdjoint, run_vjp
from mpas_dycore_pytorch_gb300.ensemble import Ensemble
from mpas_dycore_pytorch_gb300.loader import load_arrays

GRAVITY, RGAS, CP, P0 = 9.80616, 287.0, 1004.5, 100000.0
TIME_STEP = {2: 1800.0, 3: 1800.0, 4: 1800.0, 5: 900.0, 6: 720.0}  # seconds, per mesh level
LEN_DISP, SMDIV, EPSSM, COEF3, C_S = 120000.0, 0.1, 0.1, 0.25, 0.125


def _case(name, kind, level, nlev, tracers=1, mono=False, precision="float64", order="native", moist=False,
          terrain=0.0, rk=3, members=1, steps=1):
    return {"name": name, "kind": kind, "level": level, "nlev": nlev, "tracers": tracers, "mono": mono,
            "precision": precision, "order": order, "moist": moist, "terrain": terrain, "rk": rk,
            "members": members, "steps": steps}


def listed():
    return [
        # the smallest forecast of the tests: a step is a chain of tiny kernels
        _case("step-162x12", "step", 2, 12, tracers=2, mono=True),
        # the CPU-runnable workload: explicit transport of one tracer
        _case("step-2562x26", "step", 4, 26),
        # a moist forecast over a hill, odd level count: every slope and moisture path
        _case("step-moist-hill-10242x33", "step", 5, 33, tracers=2, mono=True, moist=True, terrain=1500.0),
        # the headline forecast, float64 and mixed, in the benchmark's mesh order
        _case("step-40962x55", "step", 6, 55, tracers=3, mono=True, order="sfc"),
        _case("step-mixed-40962x55", "step", 6, 55, tracers=3, mono=True, order="sfc", precision="mixed"),
        # an ensemble of uneven meshes in one graph
        _case("ensemble-mixed-8x41", "ensemble", 4, 41, tracers=2, mono=True, precision="mixed", members=8),
        # the first RK stage's tendencies, with every mixing term
        _case("tendencies-10242x41", "tendencies", 5, 41, rk=1),
        # the implicit coefficients and two acoustic substeps with divergence damping
        _case("acoustic-40962x55", "acoustic", 6, 55),
        # diagnostics of a prepared or stepped state and the cell winds
        _case("diagnostics-10242x41", "diagnostics", 5, 41),
        # the limited last transport stage of the headline forecast, and an explicit stage
        # with as many tracers as the package takes, on an odd level count
        _case("monotone-40962x55x3", "monotone", 6, 55, tracers=3),
        _case("transport-2562x37x8", "transport", 4, 37, tracers=8),
        # gradient of the surface-pressure objective through a short dry run
        _case("gradient-2562x26", "gradient", 4, 26, steps=3),
    ]


def draw(rng):
    kind = rng.choice(["step", "step", "step", "ensemble", "tendencies", "acoustic", "diagnostics", "monotone",
                       "transport", "gradient"])
    level = rng.choice([2, 3, 4, 5])
    nlev = int(round(math.exp(rng.uniform(math.log(8), math.log(64)))))
    tracers = rng.randint(1, 8)
    c = _case(None, kind, level, nlev, tracers=tracers, rk=rng.randint(1, 3))
    del c["name"]
    if kind == "step":
        c.update(mono=rng.random() < 0.6, precision=rng.choice(["float64", "float64", "mixed"]),
                 order=rng.choice(["native", "sfc"]), moist=rng.random() < 0.3,
                 terrain=rng.choice([0.0, 0.0, 1500.0]), tracers=rng.randint(1, 4))
    elif kind == "ensemble":
        c.update(level=rng.choice([2, 3, 4]), members=rng.randint(2, 8), tracers=2, mono=True,
                 precision=rng.choice(["float64", "mixed"]))
    elif kind == "gradient":
        c.update(level=rng.choice([2, 3, 4]), steps=rng.randint(1, 4), nlev=min(nlev, 41), tracers=1)
    elif kind in ("tendencies", "acoustic", "diagnostics"):
        c.update(tracers=1)
    return c


# ---------------------------------------------------------------------------- inputs
def _config(case, level):
    return {"config_time_integration_order": 3, "config_len_disp": LEN_DISP, "config_number_of_sub_steps": 2,
            "config_dynamics_split_steps": 3, "config_monotonic": bool(case["mono"]),
            "config_dt": TIME_STEP[level], "config_precision": case["precision"]}


@functools.lru_cache(maxsize=4)
def _grid(level):
    return build_mesh(level)


def _spec(case, level, seed):
    return CaseSpec(level=level, nlev=case["nlev"], seed=seed, n_bumps=8,
                    n_tracers=case["tracers"] - (1 if case["moist"] else 0),
                    u_noise=0.5, w_sine=0.1, qv_surface=0.012 if case["moist"] else 0.0, terrain=case["terrain"])


@functools.lru_cache(maxsize=2)
def _base(level, key):
    """The loaded mesh with one initial state (seed 0): what does not depend on the seed."""
    case = dict(key)
    grid = dict(_grid(level))
    init = initial_state(grid, _spec(case, level, 0))
    for k in ("deriv_two", "defc_a", "defc_b"):
        init[k] = grid.pop(k)
    return load_arrays(init, grid, _config(case, level), as_torch=False)


def _loaded(case, level, seed):
    """The loaded state and mesh of one seed: theta bumps, wind noise."""
    key = tuple(sorted((k, case[k]) for k in ("nlev", "tracers", "moist", "terrain", "mono", "precision")))
    out = dict(_base(level, key))
    init = initial_state(_grid(level), _spec(case, level, seed))
    for k in ("u", "w", "theta", "rho", "scalars", "qv"):
        a = np.asarray(init[k], dtype=np.float64)
        out[k] = np.concatenate([a, np.zeros_like(a[:1])])
    return out


def _gpu(a, dtype=torch.float64):
    return torch.as_tensor(np.asarray(a), dtype=dtype, device="cuda")


def _geometry(st):
    """Mesh arrays on the GPU: 0-based connectivity (missing neighbours read the padding
    row), slot masks, per-slot weights."""
    nc, ne, nv, nl = (int(st[k]) for k in ("nCells", "nEdges", "nVertices", "nVertLevels"))

    def conn(name, rows, n):
        a = np.asarray(st[name]).astype(np.int64)[:rows]
        return _gpu(np.where((a >= 1) & (a <= n), a - 1, n), torch.int64)

    g = SimpleNamespace(nc=nc, ne=ne, nv=nv, nl=nl)
    g.coe, g.voe = conn("cellsOnEdge", ne, nc), conn("verticesOnEdge", ne, nv)
    g.eoc, g.coc, g.voc = conn("edgesOnCell", nc, ne), conn("cellsOnCell", nc, nc), conn("verticesOnCell", nc, nv)
    g.eov, g.eoe, g.adv = conn("edgesOnVertex", nv, ne), conn("edgesOnEdge", ne, ne), conn("advCellsForEdge", ne, nc)
    slots = lambda n, width: torch.arange(width, device="cuda")[None, :] < _gpu(n, torch.int64)[:, None]
    g.on_cell = slots(np.asarray(st["nEdgesOnCell"])[:nc], g.eoc.shape[1])
    g.on_edge = slots(np.asarray(st["nEdgesOnEdge"])[:ne], g.eoe.shape[1])
    g.on_adv = slots(np.asarray(st["nAdvCellsForEdge"])[:ne], g.adv.shape[1])
    for k, n in (("dvEdge", ne), ("dcEdge", ne), ("invDcEdge", ne), ("invDvEdge", ne), ("invAreaCell", nc),
                 ("invAreaTriangle", nv), ("edgesOnCell_sign", nc), ("edgesOnVertex_sign", nv), ("weightsOnEdge", ne),
                 ("adv_coefs", ne), ("adv_coefs_3rd", ne), ("defc_a", nc), ("defc_b", nc), ("fVertex", nv),
                 ("meshScalingDel2", ne), ("meshScalingDel4", ne), ("kiteAreasOnVertex", nv), ("zz", nc),
                 ("zxu", ne), ("dss", nc), ("rho_base", nc), ("theta_base", nc), ("latCell", nc), ("lonCell", nc),
                 ("coeffs_reconstruct", nc), ("areaCell", nc)):
        setattr(g, k, _gpu(st[k])[:n])
    for k in ("rdzw", "rdzu", "fzm", "fzp", "rdnw", "fnm", "fnp"):
        setattr(g, k, _gpu(st[k])[:nl])
    kite = np.asarray(st["kiteForCell"]).astype(np.int64)[:nc]
    g.kite = _gpu(np.maximum(kite - 1, 0), torch.int64)
    return g


def _pad(x, value=0.0):
    return torch.cat([x, torch.full_like(x[:1], value)])


def _sum(weights, mask, index, field):
    """sum_j weights[:, j] field[index[:, j]] over the valid slots."""
    out = None
    for j in range(index.shape[1]):
        t = torch.where(mask[:, j], weights[:, j], 0.0)[:, None] * field[index[:, j]]
        out = t if out is None else out + t
    return out


def _stage_inputs(case, seed):
    """Fields of a dry state in mid-step, from the loaded state alone: the coupled variables,
    their saved values (a little apart, as after an RK stage), the diagnostics."""
    st = _loaded(case, case["level"], seed)
    g = _geometry(st)
    gen = torch.Generator(device="cuda").manual_seed(1000 + int(seed))
    noise = lambda shape, scale: scale * torch.randn(shape, dtype=torch.float64, device="cuda", generator=gen)
    nc, ne, nl = g.nc, g.ne, g.nl
    f = {"u": _gpu(st["u"])[:ne], "theta_m": _gpu(st["theta"])[:nc], "scalars": _gpu(st["scalars"])[:nc]}
    c1, c2 = g.coe[:, 0], g.coe[:, 1]
    w = _gpu(st["w"])[:nc] + noise((nc, nl + 1), 0.02)
    w[:, 0] = 0.0
    w[:, nl] = 0.0
    f["w"] = w
    rz = _gpu(st["rho"])[:nc] / g.zz
    f["rho_zz"] = rz
    f["rho_p"] = rz - g.rho_base
    f["rr_save"] = f["rho_p"] + noise((nc, nl), 1e-6)
    rtb = g.theta_base * g.rho_base
    f["rtheta_base"] = rtb
    f["rtheta_p"] = f["theta_m"] * f["rho_p"] + g.rho_base * (f["theta_m"] - g.theta_base)
    rcv = RGAS / (CP - RGAS)
    f["exner"] = (g.zz * (RGAS / P0) * (f["rtheta_p"] + rtb)) ** rcv
    f["exner_base"] = (g.zz * (RGAS / P0) * rtb) ** rcv
    f["pressure_p"] = g.zz * RGAS * (f["exner"] * f["rtheta_p"] + rtb * (f["exner"] - f["exner_base"]))
    f["ru"] = 0.5 * f["u"] * (rz[c1] + rz[c2])
    rw = torch.zeros_like(w)
    rw[:, 1:nl] = w[:, 1:nl] * (g.fzp[1:] * rz[:, :-1] + g.fzm[1:] * rz[:, 1:]) * \
        (g.fzp[1:] * g.zz[:, :-1] + g.fzm[1:] * g.zz[:, 1:])
    f["rw"] = rw
    f["ru_save"] = f["ru"] + noise((ne, nl), 0.02)
    f["rw_save"] = rw + torch.where(rw != 0.0, noise((nc, nl + 1), 0.002), 0.0)
    f["theta_m_save"] = f["theta_m"] + noise((nc, nl), 0.01)
    f["qtot"] = torch.zeros_like(rz)
    f["cqw"] = torch.ones_like(w)
    f["cqu_e"] = torch.ones_like(f["u"])
    f["tend_u"] = noise((ne, nl), 1e-4)
    f["tend_rho"] = noise((nc, nl), 1e-7)
    f["tend_theta"] = noise((nc, nl), 1e-4)
    f["tend_rw"] = noise((nc, nl + 1), 1e-5)
    f["tend_u_euler"] = noise((ne, nl), 1e-5)
    f["tend_w_euler"] = noise((nc, nl + 1), 1e-6)
    f["tend_theta_euler"] = noise((nc, nl), 1e-6)
    f["kdiff"] = noise((nc, nl), 1.0).abs()
    # the transport's substep-averaged fluxes and the end density they lead to
    f["ruAvg"], f["wwAvg"] = f["ru"], rw
    f["rho_zz_old_split"] = rz + noise((nc, nl), 1e-6)
    s = f["scalars"]
    f["scalars_init"] = s
    f["scalars_a"] = s * (1.0 + noise(s.shape, 1e-3))
    f.update(_exact_diagnostics(g, f["u"], rz, TIME_STEP[case["level"]]))
    return st, g, f


FIELD_PADS = {"rho_zz": 1.0, "rho_zz_old_split": 1.0}


def prepare(case, seed):
    kind, level = case["kind"], case["level"]
    if kind == "step":
        st = _loaded(case, level, seed)
        model = Model(st, _config(case, level), TIME_STEP[level], num_scalars=case["tracers"], order=case["order"])
        model.prepare(st)
        model.step()
        model.capture_graph()
        return {"kind": kind, "model": model}
    if kind == "ensemble":
        members = [_loaded(case, max(2, level - (b % 2)), 100 * seed + b) for b in range(case["members"])]
        ens = Ensemble(members, _config(case, level), 900.0, precision=case["precision"])
        ens.step()
        ens.capture_graph()
        return {"kind": kind, "model": ens.model}
    if kind == "gradient":
        st = _loaded(case, level, seed)
        cfg = dict(_config(case, level), config_dt=900.0)
        model = Model(st, cfg, 900.0, num_scalars=case["tracers"])
        dev = {k: _gpu(st[k]) for k in ("zz", "zgrid", "areaCell")}
        return {"kind": kind, "model": model, "adjoint": DynamicsAdjoint(model), "loaded": st, "mesh": dev,
                "nc": int(st["nCells"]), "steps": case["steps"]}
    st, _, f = _stage_inputs(case, seed)
    model = Model(st, _config(case, level), TIME_STEP[level], num_scalars=case["tracers"])
    model.state.load({k: _pad(v, FIELD_PADS.get(k, 0.0)) for k, v in f.items()})
    return {"kind": kind, "model": model, "rk": case["rk"], "dt": TIME_STEP[level]}


# ---------------------------------------------------------------------------- one pass
def _gradient(s):
    nc, mesh = s["nc"], s["mesh"]

    def cotangents(final):
        leaves = {k: final[k].detach().clone().requires_grad_(True) for k in ("rho_zz", "pressure_p")}
        sp = physics_interface_surface_pressure(
            nCells=nc, rho_zz=leaves["rho_zz"], zz=mesh["zz"], qv=torch.zeros_like(final["rho_zz"]),
            pressure_p=leaves["pressure_p"], pressure_base=final["pressure_base"], zgrid=mesh["zgrid"])
        ref = torch.full_like(sp, 1.0e5)
        loss = surface_pressure_functional(sp, ref, mesh["areaCell"], nc)
        return dict(zip(leaves, torch.autograd.grad(loss, list(leaves.values()))))

    grads, final = run_vjp(s["model"], s["loaded"], s["steps"], cotangents, s["adjoint"])
    return {"grads": grads, "final": {k: v for k, v in final.items() if k not in ("rho_edge", "ur_cell", "vr_cell")}}


def run(state):
    kind, m = state["kind"], state["model"]
    if kind in ("step", "ensemble"):
        m.step()
        return m.state.export()
    if kind == "gradient":
        return _gradient(state)
    f, dt = m.state.f, state["dt"]
    nc, ne, nv = m.dmesh.nCells, m.dmesh.nEdges, m.dmesh.nVertices
    if kind == "tendencies":
        m.call("mpasg_dyn_tend", C.c_int(state["rk"]))
        out = {k: f[k][:ne] for k in ("tend_u", "tend_u_euler")}
        out.update({k: f[k][:nc] for k in ("tend_w", "tend_theta", "tend_rho", "tend_w_euler", "tend_theta_euler",
                                           "h_divergence", "kdiff", "rthdynten")})
        return out
    if kind == "acoustic":
        dts = dt / 3.0 / 2.0
        m.call("mpasg_vert_imp_coefs", C.c_double(dts))
        for small in (1, 2):
            m.call("mpasg_acoustic_step", C.c_int(small), C.c_double(dts))
            m.call("mpasg_divergence_damping", C.c_double(dts))
        out = {k: f[k][:ne] for k in ("ru_p", "ruAvg")}
        out.update({k: f[k][:nc] for k in ("rw_p", "wwAvg", "rho_pp", "rtheta_pp", "rtheta_pp_old", "alpha_tri",
                                           "gamma_tri")})
        return out
    if kind == "diagnostics":
        m.call("mpasg_solve_diagnostics", C.c_int(3))
        m.call("mpasg_reconstruct_2d")
        out = {k: f[k][:ne] for k in ("h_edge", "v", "pv_edge")}
        out.update({k: f[k][:nc] for k in ("divergence", "ke", "uReconstructX", "uReconstructY", "uReconstructZ",
                                           "uReconstructZonal", "uReconstructMeridional")})
        out["vorticity"] = f["vorticity"][:nv]
        return out
    if kind == "monotone":
        m.call("mpasg_advance_scalars_mono", C.c_double(dt))
    else:
        m.call("mpasg_advance_scalars", C.c_int(state["rk"]), C.c_double(dt / 3.0))
    return f["scalars_b"][:nc]


# ---------------------------------------------------------------------------- work
def work(case):
    """Bytes: every array a pass has to read or write, once; flops: the stencils' multiplies
    and adds, a fused pair as two."""
    cells = lambda lv: 10 * 4 ** lv + 2
    L, S = case["nlev"], case["tracers"]
    kind = case["kind"]
    n = cells(case["level"])
    if kind == "ensemble":
        n = sum(cells(max(2, case["level"] - (b % 2))) for b in range(case["members"]))
    cl = float(n * L)
    word = 8.0
    if kind in ("step", "ensemble", "gradient"):
        # one step's inputs and outputs (14 cell, 5 edge (3 a cell), 1 vertex (2 a cell) fields, the scalars)
        fields = 14 + 15 + 2 + S
        flops = 9 * 607.0 + 12 * 130.0 + 9 * 200.0 + 3 * 70.0 * S + 100.0 * S
        passes = 1 if kind != "gradient" else 3 * case["steps"]
        return {"bytes": 2 * fields * word * cl * passes, "flops": flops * cl * passes}
    if kind == "tendencies":
        # reads 5 edge, 1 vertex and 14 cell fields, writes 2 edge and 8 cell fields
        return {"bytes": word * cl * (15 + 2 + 14 + 6 + 8), "flops": 607.0 * cl}
    if kind == "acoustic":
        # reads 3 edge and 14 cell fields, writes 2 edge and 11 cell fields
        return {"bytes": word * cl * (9 + 14 + 6 + 11), "flops": (2 * 130.0 + 60.0) * cl}
    if kind == "diagnostics":
        return {"bytes": word * cl * (3 + 1 + 9 + 2 + 7), "flops": 230.0 * cl}
    # the old and new scalars, the mass fluxes (3 edge, 1 cell a cell) and two densities in; one set of scalars out
    per = 190.0 if kind == "monotone" else 85.0
    return {"bytes": word * cl * (3 * S + 3 + 1 + 2), "flops": per * S * cl}


# ---------------------------------------------------------------------------- 64-bit values
def _flux3(qm2, qm1, q0, qp1, ua, c3):
    return (ua * (7.0 * (q0 + qm1) - (qp1 + qm2)) + c3 * ua.abs() * ((qp1 - qm2) - 3.0 * (q0 - qm1))) / 12.0


def _interfaces(q, vel, fm, fp, c3):
    """Vertical fluxes at the interfaces 0..L of a column field: zero at the ends, second
    order next to them, third order inside (``vel``: the interface velocity, 0..L)."""
    L = q.shape[1]
    wide = (slice(None), slice(None)) + (None,) * (q.dim() - 2)
    out = torch.zeros((q.shape[0], L + 1) + q.shape[2:], dtype=q.dtype, device=q.device)
    lin = lambda k: vel[:, k:k + 1][wide] * (fm[k] * q[:, k:k + 1] + fp[k] * q[:, k - 1:k])
    out[:, 1:2] = lin(1)
    out[:, L - 1:L] = lin(L - 1)
    out[:, 2:L - 1] = _flux3(q[:, :L - 3], q[:, 1:L - 2], q[:, 2:L - 1], q[:, 3:], vel[:, 2:L - 1][wide], c3)
    return out


def _adv(g, uh, q):
    """sum over the advection stencil of an edge, the coefficients by the sign of the flux;
    ``q`` is (cells + 1, levels) or (cells + 1, levels, scalars)."""
    s = torch.where(uh >= 0.0, 1.0, -1.0)
    out = None
    for j in range(g.adv.shape[1]):
        m = g.on_adv[:, j]
        c = torch.where(m, g.adv_coefs[:, j], 0.0)[:, None] + s * torch.where(m, g.adv_coefs_3rd[:, j], 0.0)[:, None]
        x = q[torch.where(m, g.adv[:, j], 0)]
        t = c * x if q.dim() == 2 else c[..., None] * x
        out = t if out is None else out + t
    return out


def _exact_diagnostics(g, u, rho_zz, dt):
    c1, c2, v1, v2 = g.coe[:, 0], g.coe[:, 1], g.voe[:, 0], g.voe[:, 1]
    up = _pad(u)
    o = {"h_edge": 0.5 * (rho_zz[c1] + rho_zz[c2])}
    kee = _pad((g.dcEdge * g.dvEdge)[:, None] * u * u)
    valid = g.eov < g.ne
    dc, dv = _pad(g.dcEdge), _pad(g.dvEdge)
    o["vorticity"] = _sum(g.edgesOnVertex_sign[:, :g.eov.shape[1]] * dc[g.eov], valid, g.eov, up) * g.invAreaTriangle[:, None]
    kev = 0.25 * g.invAreaTriangle[:, None] * _sum(torch.ones_like(g.eov, dtype=torch.float64), valid, g.eov, kee)
    ia = g.invAreaCell[:, None]
    o["divergence"] = _sum(g.edgesOnCell_sign * dv[g.eoc], g.on_cell, g.eoc, up) * ia
    ke = 0.625 * ia * _sum(torch.full_like(g.edgesOnCell_sign, 0.25), g.on_cell, g.eoc, kee)
    kites = torch.where(g.on_cell, _pad(g.kiteAreasOnVertex)[g.voc.clamp(max=g.nv), g.kite], 0.0)
    pvv = _pad(g.fVertex[:, None] + o["vorticity"])
    o["ke"] = ke + ia * _sum(0.375 * kites, g.on_cell, g.voc, _pad(kev))
    pvc = ia * _sum(kites, g.on_cell, g.voc, pvv)
    o["v"] = _sum(g.weightsOnEdge[:, :g.eoe.shape[1]], g.on_edge, g.eoe, up)
    pv1, pv2 = pvv[v1], pvv[v2]
    grad_t = (pv2 - pv1) * g.invDvEdge[:, None]
    grad_n = (pvc[c2] - pvc[c1]) * g.invDcEdge[:, None]
    o["pv_edge"] = 0.5 * (pv1 + pv2) - 0.5 * dt * (o["v"] * grad_t + u * grad_n)
    return o


def _exact_reconstruct(g, u):
    x, y, z = (_sum(g.coeffs_reconstruct[:, :, i], g.on_cell, g.eoc, _pad(u)) for i in range(3))
    cl, sl, co, so = (t[:, None] for t in (g.latCell.cos(), g.latCell.sin(), g.lonCell.cos(), g.lonCell.sin()))
    return {"uReconstructX": x, "uReconstructY": y, "uReconstructZ": z, "uReconstructZonal": -x * so + y * co,
            "uReconstructMeridional": -(x * co + y * so) * sl + z * cl}


def _exact_tendencies(g, f, rk, dt):
    nc, ne, L = g.nc, g.ne, g.nl
    c1, c2 = g.coe[:, 0], g.coe[:, 1]
    ia, dv = g.invAreaCell[:, None], _pad(g.dvEdge)
    sdv = g.edgesOnCell_sign * dv[g.eoc]
    idc, idv = g.invDcEdge[:, None], g.invDvEdge[:, None]
    cell = lambda weights, e: _sum(weights, g.on_cell, g.eoc, _pad(e))
    one = g.edgesOnCell_sign
    u, w, ru, rw, th, ths, rz = (f[k] for k in ("u", "w", "ru", "rw", "theta_m", "theta_m_save", "rho_zz"))
    rho_e = f["h_edge"]
    o = {"h_divergence": ia * cell(sdv, ru), "kdiff": f["kdiff"], "tend_rho": f["tend_rho"]}
    hd = o["h_divergence"]
    if rk == 1:
        o["tend_rho"] = -hd - g.rdzw * (rw[:, 1:] - rw[:, :L])
        dpdz = -GRAVITY * (g.rho_base * f["qtot"] + f["rr_save"] * (1.0 + f["qtot"]))
        dd = cell(g.defc_a[:, :one.shape[1]], u) - cell(g.defc_b[:, :one.shape[1]], f["v"])
        do = cell(g.defc_b[:, :one.shape[1]], u) + cell(g.defc_a[:, :one.shape[1]], f["v"])
        o["kdiff"] = torch.clamp((C_S * LEN_DISP) ** 2 * torch.sqrt(dd * dd + do * do), max=0.01 * LEN_DISP ** 2 / dt)
    wd = _interfaces(u, 0.5 * (rw[c1] + rw[c2]), g.fzm, g.fzp, 1.0)
    up, pvp = _pad(u), _pad(f["pv_edge"])
    woe = g.weightsOnEdge[:, :g.eoe.shape[1]]
    q = 0.5 * (f["pv_edge"] * _sum(woe, g.on_edge, g.eoe, up) + _sum(woe, g.on_edge, g.eoe, up * pvp))
    tu = -g.rdzw * (wd[:, 1:] - wd[:, :L]) + rho_e * (q - (f["ke"][c2] - f["ke"][c1]) * idc) - \
        0.5 * u * (hd[c1] + hd[c2])
    visc4 = 0.05 * LEN_DISP ** 3
    teu = f["tend_u_euler"]
    if rk == 1:
        kd, zz = o["kdiff"], g.zz
        teu = -f["cqu_e"] * ((f["pressure_p"][c2] - f["pressure_p"][c1]) * idc / (0.5 * (zz[c2] + zz[c1])) -
                             0.5 * g.zxu * (dpdz[c1] + dpdz[c2]))
        r_dv = torch.minimum(idv, 4.0 * idc)
        lap = (f["divergence"][c2] - f["divergence"][c1]) * idc - \
            (f["vorticity"][g.voe[:, 1]] - f["vorticity"][g.voe[:, 0]]) * r_dv
        teu = teu + rho_e * 0.5 * (kd[c1] + kd[c2]) * lap * g.meshScalingDel2[:, None]
        lapp = _pad(lap)
        dvort = _sum(g.invAreaTriangle[:, None] * _pad(g.dcEdge)[g.eov] * g.edgesOnVertex_sign[:, :g.eov.shape[1]],
                     g.eov < g.ne, g.eov, lapp)
        ddiv = ia * cell(sdv, lap)
        mix = g.meshScalingDel4[:, None] * visc4
        teu = teu - rho_e * ((ddiv[c2] - ddiv[c1]) * mix * 10.0 * idc -
                             (dvort[g.voe[:, 1]] - dvort[g.voe[:, 0]]) * mix * r_dv)
    o["tend_u_euler"] = teu
    o["tend_u"] = tu + teu
    # w and theta: del2 / del4 mixing at the first stage
    twe, tte = f["tend_w_euler"], f["tend_theta_euler"]
    sdc = sdv * _pad(g.invDcEdge)[g.eoc]
    ms2 = g.meshScalingDel2[:, None]
    if rk == 1:
        he = torch.zeros((ne, L + 1), dtype=torch.float64, device=u.device)
        he[:, 1:L] = 0.5 * (rho_e[:, 1:] + rho_e[:, :-1]) * (w[c2] - w[c1])[:, 1:L]
        k2 = kd[c1] + kd[c2]
        mixed = torch.zeros_like(he)
        mixed[:, 1:L] = he[:, 1:L] * ms2 * 0.25 * (k2[:, 1:] + k2[:, :-1])
        lapw = ia * cell(sdc, he)
        twe = ia * cell(sdc, mixed)
        ht = (th[c2] - th[c1]) * rho_e
        lapt = ia * cell(sdc, ht)
        tte = ia * cell(sdc, ht * 0.5 * k2 * ms2)
        ms4 = g.meshScalingDel4[:, None] * visc4
        d4w = ia * cell(sdc, ms4 * (lapw[c2] - lapw[c1]))
        d4w[:, 0] = 0.0
        d4w[:, L] = 0.0
        twe = twe - d4w
        tte = tte - ia * cell(sdc, ms4 * (lapt[c2] - lapt[c1]))
    # w
    ruw = torch.zeros((ne, L + 1), dtype=torch.float64, device=u.device)
    ruw[:, 1:L] = g.fzm[1:] * ru[:, 1:] + g.fzp[1:] * ru[:, :-1]
    flux = ruw * _adv(g, ruw, _pad(w))
    wd = torch.zeros((nc, L + 1), dtype=torch.float64, device=u.device)  # flux between w levels k - 1 and k
    half = lambda k: 0.5 * (rw[:, k] + rw[:, k - 1])
    for k in (1, L - 1):
        wd[:, k] = half(k) * 0.5 * (w[:, k] + w[:, k - 1])
    wd[:, 2:L - 1] = _flux3(w[:, :L - 3], w[:, 1:L - 2], w[:, 2:L - 1], w[:, 3:L],
                            0.5 * (rw[:, 2:L - 1] + rw[:, 1:L - 2]), 1.0)
    tw = torch.zeros((nc, L + 1), dtype=torch.float64, device=u.device)
    tw[:, 1:L] = (-ia * cell(one, flux))[:, 1:L] - g.rdzu[1:] * (wd[:, 2:] - wd[:, 1:L])
    if rk == 1:
        twe = twe.clone()
        twe[:, 1:L] -= f["cqw"][:, 1:L] * (g.rdzu[1:] * (f["pressure_p"][:, 1:] - f["pressure_p"][:, :-1]) -
                                           (g.fzm[1:] * dpdz[:, 1:] + g.fzp[1:] * dpdz[:, :-1]))
        twe[:, 0] = 0.0
        twe[:, L] = 0.0
    tw[:, 1:L] += twe[:, 1:L]
    o["tend_w"], o["tend_w_euler"] = tw, twe
    # theta
    tt = -ia * cell(one, ru * _adv(g, ru, _pad(th)))
    if rk > 1:
        tt = tt - ia * cell(sdv, (f["ru_save"] - ru) * 0.5 * (ths[c1] + ths[c2]))
    vf = _interfaces(th, rw, g.fzm, g.fzp, COEF3)
    k = slice(1, L - 1)
    lin = lambda q, k: g.fzm[k] * q[:, k] + g.fzp[k] * q[:, slice(k.start - 1, k.stop - 1)]
    vf[:, k] += (f["rw_save"] - rw)[:, k] * lin(ths, k)
    k = slice(L - 1, L)
    vf[:, k] = f["rw_save"][:, k] * lin(th, k)
    tt = tt - g.rdzw * (vf[:, 1:] - vf[:, :L])
    o["rthdynten"] = None  # a difference of nearly equal terms: only its rounding is left
    o["tend_theta_euler"] = tte
    o["tend_theta"] = tt + tte
    return o


def _exact_acoustic(g, f, dts):
    nc, ne, L = g.nc, g.ne, g.nl
    c1, c2 = g.coe[:, 0], g.coe[:, 1]
    rcv = RGAS / (CP - RGAS)
    half, resm = 0.5 * dts * (1.0 + EPSSM), (1.0 - EPSSM) / (1.0 + EPSSM)
    zz, ex, th, ths = g.zz, f["exner"], f["theta_m"], f["theta_m_save"]
    at = lambda q: g.fzm[1:] * q[:, 1:] + g.fzp[1:] * q[:, :-1]
    zeros = lambda n, w: torch.zeros((n, w), dtype=torch.float64, device=zz.device)
    cofrz = half * g.rdzw
    cofwr, cofwz, coftz = zeros(nc, L), zeros(nc, L), zeros(nc, L + 1)
    cofwr[:, 1:] = 0.5 * half * GRAVITY * at(zz)
    cofwz[:, 1:] = half * CP * rcv * at(zz) * g.rdzu[1:] * f["cqw"][:, 1:L] * at(ex)
    coftz[:, 1:L] = half * at(th)
    cofwt = 0.5 * half * rcv * zz * GRAVITY * g.rho_base * ex / ((f["rtheta_base"] + f["rtheta_p"]) * f["exner_base"])
    lo, hi = coftz[:, :L - 1], coftz[:, 2:]
    mid, dn, up = coftz[:, 1:L], g.rdzw[:-1], g.rdzw[1:]
    a = -cofwz[:, 1:] * lo * dn * zz[:, :-1] + cofwr[:, 1:] * cofrz[:-1] - cofwt[:, :-1] * lo * dn
    b = 1.0 + cofwz[:, 1:] * (mid * up * zz[:, 1:] + mid * dn * zz[:, :-1]) - \
        mid * (cofwt[:, 1:] * up - cofwt[:, :-1] * dn) + cofwr[:, 1:] * (cofrz[1:] - cofrz[:-1])
    c = -cofwz[:, 1:] * hi * up * zz[:, 1:] - cofwr[:, 1:] * cofrz[1:] + cofwt[:, 1:] * hi * up
    alpha, gamma = zeros(nc, L), zeros(nc, L)
    for k in range(1, L):
        alpha[:, k] = 1.0 / (b[:, k - 1] - a[:, k - 1] * gamma[:, k - 1])
        gamma[:, k] = c[:, k - 1] * alpha[:, k]
    geo = g.edgesOnCell_sign * _pad(g.dvEdge)[g.eoc] * g.invAreaCell[:, None]
    cell = lambda e: _sum(geo, g.on_cell, g.eoc, _pad(e))
    th_e = 0.5 * (ths[c1] + ths[c2])
    rho, rt, rwp, ww = zeros(nc, L), zeros(nc, L), zeros(nc, L + 1), zeros(nc, L + 1)
    rup, avg = zeros(ne, L), zeros(ne, L)
    for small in (1, 2):
        if small > 1:
            p = (rt[c2] - rt[c1]) * g.invDcEdge[:, None] / (0.5 * (zz[c2] + zz[c1]))
            p = f["cqu_e"] * 0.5 * CP * rcv * (ex[c1] + ex[c2]) * p + 0.5 * g.zxu * GRAVITY * (rho[c1] + rho[c2])
            rup = rup + dts * (f["tend_u"] - p)
            avg = avg + rup
        else:
            rup = dts * f["tend_u"]
            avg = rup
        old = rt
        rs = rho + dts * f["tend_rho"] - dts * cell(rup) - cofrz * resm * (rwp[:, 1:] - rwp[:, :L])
        ts = rt + dts * f["tend_theta"] - dts * cell(rup * th_e) - \
            resm * g.rdzw * (coftz[:, 1:] * rwp[:, 1:] - coftz[:, :L] * rwp[:, :L])
        ww = ww + 0.5 * (1.0 - EPSSM) * rwp
        x = rwp.clone()
        x[:, 1:L] += dts * f["tend_rw"][:, 1:L] - \
            cofwz[:, 1:] * ((zz * ts)[:, 1:] - (zz * ts)[:, :-1] + resm * ((zz * rt)[:, 1:] - (zz * rt)[:, :-1])) - \
            cofwr[:, 1:] * (rs[:, 1:] + rs[:, :-1] + resm * (rho[:, 1:] + rho[:, :-1])) + \
            cofwt[:, 1:] * (ts + resm * rt)[:, 1:] + cofwt[:, :-1] * (ts + resm * rt)[:, :-1]
        for k in range(1, L):
            x[:, k] = (x[:, k] - a[:, k - 1] * x[:, k - 1]) * alpha[:, k]
        for k in range(L - 1, 0, -1):
            x[:, k] = x[:, k] - gamma[:, k] * x[:, k + 1]
        d = (f["rw_save"] - f["rw"])[:, 1:L]
        damp = dts * g.dss[:, 1:]
        x[:, 1:L] = (x[:, 1:L] + d - damp * at(zz) * at(f["rho_zz"]) * f["w"][:, 1:L]) / (1.0 + damp) - d
        ww = ww + 0.5 * (1.0 + EPSSM) * x
        ww[:, 0] = 0.0
        ww[:, L] = 0.0
        rho = rs - cofrz * (x[:, 1:] - x[:, :L])
        rt = ts - g.rdzw * (coftz[:, 1:] * x[:, 1:] - coftz[:, :L] * x[:, :L])
        rwp = x
        rup = rup + 2.0 * SMDIV * LEN_DISP / dts * ((old[c2] - rt[c2]) - (old[c1] - rt[c1])) / (ths[c1] + ths[c2])
    return {"ru_p": rup, "ruAvg": avg, "rw_p": rwp, "wwAvg": ww, "rho_pp": rho, "rtheta_pp": rt, "rtheta_pp_old": old,
            "alpha_tri": alpha, "gamma_tri": gamma}


def _cell_scalars(g, weights, e):
    """sum over a cell's edges of an (edges, levels, scalars) field."""
    out = None
    for j in range(g.eoc.shape[1]):
        ok = g.on_cell[:, j]
        t = torch.where(ok, weights[:, j], 0.0)[:, None, None] * e[torch.where(ok, g.eoc[:, j], 0)]
        out = t if out is None else out + t
    return out


def _exact_transport(g, f, rk, dt):
    so, sn, uh, ww = f["scalars_init"], f["scalars_a"], f["ruAvg"], f["wwAvg"]
    L = g.nl
    h = uh[..., None] * _adv(g, uh, _pad(sn))
    vf = _interfaces(sn, ww, g.fnm, g.fnp, COEF3)
    tend = -g.invAreaCell[:, None, None] * _cell_scalars(g, g.edgesOnCell_sign, h) - \
        g.rdnw[None, :, None] * (vf[:, 1:] - vf[:, :L])
    new = {1: 1.0 / 3.0, 2: 0.5, 3: 1.0}[rk]
    old = f["rho_zz_old_split"]
    rho = (1.0 - new) * old + new * f["rho_zz"]
    return (so * old[..., None] + dt * tend) / rho[..., None]


def _exact_monotone(g, f, dt):
    so, sn, uh, ww, old = f["scalars_init"], f["scalars_a"], f["ruAvg"], f["wwAvg"], f["rho_zz_old_split"]
    L = g.nl
    c1, c2 = g.coe[:, 0], g.coe[:, 1]
    ia, rd, sg = g.invAreaCell[:, None, None], g.rdnw[None, :, None], g.edgesOnCell_sign
    pos, neg = lambda x: x.clamp(min=0.0), lambda x: x.clamp(max=0.0)
    # low-order (upwind) and correction fluxes, positive outward of c1 and upward
    up = torch.where((uh >= 0.0)[..., None], so[c1], so[c2]) * (uh * g.dvEdge[:, None])[..., None] * dt
    corr = dt * uh[..., None] * _adv(g, uh, _pad(sn)) - up
    vup = torch.zeros(so.shape[0], L + 1, so.shape[2], dtype=so.dtype, device=so.device)
    wi = ww[:, 1:L, None]
    vup[:, 1:L] = dt * wi * torch.where(wi >= 0.0, so[:, :-1], so[:, 1:])
    vcorr = dt * _interfaces(sn, ww, g.fnm, g.fnp, COEF3) - vup
    rho = old - dt * (g.invAreaCell[:, None] * _sum(sg * _pad(g.dvEdge)[g.eoc], g.on_cell, g.eoc, _pad(uh)) +
                      g.rdnw * (ww[:, 1:] - ww[:, :L]))
    hi, lo = so.clone(), so.clone()
    hi[:, 1:], lo[:, 1:] = torch.maximum(hi[:, 1:], so[:, :-1]), torch.minimum(lo[:, 1:], so[:, :-1])
    hi[:, :-1], lo[:, :-1] = torch.maximum(hi[:, :-1], so[:, 1:]), torch.minimum(lo[:, :-1], so[:, 1:])
    for j in range(g.coc.shape[1]):
        ok = (g.on_cell[:, j] & (g.coc[:, j] < g.nc))[:, None, None]
        x = so[g.coc[:, j].clamp(max=g.nc - 1)]
        hi, lo = torch.where(ok, torch.maximum(hi, x), hi), torch.where(ok, torch.minimum(lo, x), lo)
    low = so * old[..., None] - rd * (vup[:, 1:] - vup[:, :L]) - ia * _cell_scalars(g, sg, up)
    inflow = -rd * (neg(vcorr[:, 1:]) - pos(vcorr[:, :L]))
    outflow = -rd * (pos(vcorr[:, 1:]) - neg(vcorr[:, :L]))
    for j in range(g.eoc.shape[1]):
        ok = g.on_cell[:, j][:, None, None]
        x = sg[:, j, None, None] * corr[torch.where(g.on_cell[:, j], g.eoc[:, j], 0)]
        outflow = outflow - torch.where(ok, pos(x) * ia, 0.0)
        inflow = inflow - torch.where(ok, neg(x) * ia, 0.0)
    r = rho[..., None]
    fin = ((hi * r - low) / (inflow + 1e-20)).clamp(0.0, 1.0)
    fout = ((lo * r - low) / (outflow - 1e-20)).clamp(0.0, 1.0)
    lim = corr * torch.where(corr >= 0.0, torch.minimum(fout[c1], fin[c2]), torch.minimum(fin[c1], fout[c2]))
    vlim = vcorr.clone()
    wc = vcorr[:, 1:L]
    vlim[:, 1:L] = wc * torch.where(wc >= 0.0, torch.minimum(fout[:, :-1], fin[:, 1:]),
                                    torch.minimum(fout[:, 1:], fin[:, :-1]))
    return pos((low - ia * _cell_scalars(g, sg, lim) - rd * (vlim[:, 1:] - vlim[:, :L])) / r)


def exact(case, seed):
    kind = case["kind"]
    if kind in ("step", "ensemble", "gradient"):
        return None
    _, g, f = _stage_inputs(case, seed)
    dt = TIME_STEP[case["level"]]
    if kind == "tendencies":
        return _exact_tendencies(g, f, case["rk"], dt)
    if kind == "acoustic":
        return _exact_acoustic(g, f, dt / 6.0)
    if kind == "diagnostics":
        o = _exact_diagnostics(g, f["u"], f["rho_zz"], dt)
        o.update(_exact_reconstruct(g, f["u"]))
        return o
    if kind == "monotone":
        return _exact_monotone(g, f, dt)
    return _exact_transport(g, f, case["rk"], dt / 3.0)
