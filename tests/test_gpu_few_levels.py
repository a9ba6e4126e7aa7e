"""Rows of few values, where a block covers so many edges or cells that its tables pass the 48 KB
of shared memory a kernel has without asking: four levels with one tracer and wide stencils
through whole steps (suite's bound), one to three levels through the stage entry points
(stage bound 1e-12; the oracle's vertical fluxes start at two levels)."""

import ctypes as C

import numpy as np
import pytest
import torch

from fixtures import rel_l2
from gpu_helpers import need_gpu, to_np
from test_gpu_stencil_sizes import _case, _compare, _widen

pytestmark = pytest.mark.gpu

TOL = 1e-12
DT = 900.0


@pytest.mark.parametrize("mono", [False, True])
@pytest.mark.parametrize("extra", [1, 4])
def test_one_tracer_four_levels_wide_stencils(extra, mono):
    need_gpu()
    st, cfg = _case(4, 1, mono)
    _compare(_widen(st, extra), cfg)


def _more_cell_slots(st, extra):
    """Room for more edges a cell (unused: every cell keeps its own)."""
    nc, me = int(st["nCells"]), int(st["maxEdges"])
    for k, v in st.items():
        a = np.asarray(v)
        if a.ndim >= 2 and a.shape[0] in (nc, nc + 1) and a.shape[1] == me:
            st[k] = np.concatenate([a, np.zeros((a.shape[0], extra, *a.shape[2:]), a.dtype)], 1)
    st["maxEdges"] = me + extra
    return st


@pytest.mark.parametrize("wide", [False, True])
@pytest.mark.parametrize("nlev,tracers", [(1, 1), (1, 2), (2, 1), (2, 3), (3, 1)])
def test_stage_calls(nlev, tracers, wide):
    need_gpu()
    from mpas_dycore_pytorch_gb300.api import Model
    from oracle import stages
    st, cfg = _case(4, tracers, False)
    if wide:
        st = _more_cell_slots(_widen(st, 4), 2)
    model = Model(st, cfg, DT, num_scalars=tracers)
    model.dmesh.struct.nVertLevels = nlev  # the stages below read no more levels of the mesh
    nc, ne, nv = (int(st[k]) for k in ("nCells", "nEdges", "nVertices"))
    rng = np.random.default_rng(nlev * 10 + tracers)

    def field(name, rows, *shape):
        n = int(np.prod((rows + 1, *shape)))
        return model.state.f[name].flatten()[:n].view(rows + 1, *shape)

    def put(name, a):
        field(name, a.shape[0] - 1, *a.shape[1:]).copy_(torch.as_tensor(a))
        return a

    rows = lambda n, *s: rng.standard_normal((n + 1, *s))
    old, new = (put(k, 0.5 + 0.4 * np.tanh(rows(nc, nlev, tracers))) for k in ("scalars_init", "scalars_a"))
    uh, ww = put("ruAvg", 10.0 * rows(ne, nlev)), 0.01 * rows(nc, nlev + 1)
    ww[:, 0] = ww[:, nlev] = 0.0
    put("wwAvg", ww)
    rho_old = put("rho_zz_old_split", 1.0 + 0.1 * np.tanh(rows(nc, nlev)))
    rho = put("rho_zz", 1.0 + 0.1 * np.tanh(rows(nc, nlev)))
    u, v = put("u", 10.0 * rows(ne, nlev)), put("v", 10.0 * rows(ne, nlev))
    a = {**st, "nVertLevels": nlev, "rk_step": 1, "config_time_integration_order": 3, "advance_density": 1, "dt": DT,
         "coef_3rd_order": 0.25, "scalar_old": old, "scalar_new": new, "scalars_old": old, "scalars_new": new,
         "uhAvg": uh, "wwAvg": ww, "rho_zz_old": rho_old, "rho_zz_new": rho, "scalar_tend_save": 0.0 * old,
         "scalar_tend": 0.0 * old, "horiz_flux_arr": np.zeros((ne + 1, nlev, tracers)), "u": u, "h": rho, "v_in": v,
         "config_apvm_upwinding": 0.5}

    def check(name, got, want, n):
        err = rel_l2(to_np(got)[:n], want[:n])
        assert err <= TOL, (name, err)

    if nlev == 1:  # two levels that exchange nothing, the lower one compared
        two = lambda k: np.repeat(a[k], 2, axis=1)
        b = {**a, "nVertLevels": 2, "wwAvg": np.zeros((nc + 1, 3)), **{k: two(k) for k in (
            "scalar_old", "scalar_new", "scalars_old", "scalars_new", "uhAvg", "rho_zz_old", "rho_zz_new",
            "scalar_tend_save", "scalar_tend", "horiz_flux_arr")}}
    else:
        b = a
    out = lambda: field("scalars_b", nc, nlev, tracers)
    want = stages.advance_scalars(b)["scalar_new"][:, :nlev]
    for entry in ("mpasg_advance_scalars", "mpasg_advance_scalars_static"):
        out().zero_()
        model.call(entry, C.c_int(1), C.c_double(DT))
        check(entry, out(), want, nc)
    if nlev > 1:
        out().zero_()
        model.call("mpasg_advance_scalars_mono", C.c_double(DT))
        check("mono", out(), stages.advance_scalars_mono(b)["scalars_new"], nc)
    for rk in (3, 1):
        want = stages.solve_diagnostics({**a, "rk_step": rk, "v_in": a["v_in"]})
        model.call("mpasg_solve_diagnostics", C.c_int(rk))
        for k, n in (("h_edge", ne), ("divergence", nc), ("vorticity", nv), ("ke", nc), ("pv_edge", ne), ("v", ne)):
            check(k, field(k, n, nlev), want[k], n)
        a["v_in"] = to_np(field("v", ne, nlev)).copy()
