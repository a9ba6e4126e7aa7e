"""Diagnostics of cells whose corner has no kite (kiteForCell 0: a vertex outside the mesh) while
a vertex of the mesh holds NaN: the missing corner adds nothing, whatever other vertices hold.
Against the oracle, same NaN places and 1e-12 relative L2 elsewhere."""

import ctypes as C

import numpy as np
import pytest
import torch

from fixtures import rel_l2
from gpu_helpers import need_gpu, to_np
from test_gpu_stencil_sizes import _case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nlev", [4, 13])
def test_missing_corner(nlev):
    need_gpu()
    from mpas_dycore_pytorch_gb300.api import Model
    from oracle import stages
    st, cfg = _case(nlev, 1, False)
    nc, ne, nv = (int(st[k]) for k in ("nCells", "nEdges", "nVertices"))
    kites = np.asarray(st["kiteForCell"]).copy()
    kites[[40, 90, 150], [0, 3, 4]] = 0
    st["kiteForCell"] = kites
    model = Model(st, cfg, 900.0, num_scalars=1)
    rng = np.random.default_rng(nlev)
    u, rho = 10.0 * rng.standard_normal((ne + 1, nlev)), 1.0 + 0.1 * rng.random((nc + 1, nlev))
    u[np.asarray(st["edgesOnVertex"])[0] - 1] = np.nan
    f = model.state.f
    for k, a in (("u", u), ("rho_zz", rho), ("v", 0.0 * u)):
        f[k].copy_(torch.as_tensor(a))
    model.call("mpasg_solve_diagnostics", C.c_int(1))
    want = stages.solve_diagnostics({**st, "nVertLevels": nlev, "rk_step": 1, "dt": 900.0, "u": u, "h": rho,
                                     "v_in": 0.0 * u, "config_apvm_upwinding": 0.5})
    for k, n in (("divergence", nc), ("vorticity", nv), ("ke", nc), ("pv_edge", ne)):
        g, w = to_np(f[k])[:n], want[k][:n]
        nan = np.isnan(w)
        assert nan.any() and np.array_equal(np.isnan(g), nan), k
        assert rel_l2(g[~nan], w[~nan]) <= 1e-12, k
