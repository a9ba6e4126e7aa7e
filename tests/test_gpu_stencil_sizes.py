"""The float64 step against the oracle where the kernels' blocks, tables and slots can go
wrong: the fewest levels, level counts around the warp size, one to eight tracers (one of
them zero over most of the sphere), stencils wider than a table holds, terrain.  Bound: the
suite's 1e-12 relative L2 after whole steps."""

import numpy as np
import pytest

from fixtures import STEP_TOL, rel_l2
from gpu_helpers import need_gpu, to_np

pytestmark = pytest.mark.gpu

KEYS = ("u", "w", "theta_m", "rho_zz", "scalars", "exner", "pressure_p", "v", "vorticity", "divergence", "ke",
        "pv_edge", "uReconstructZonal", "ruAvg", "wwAvg")


def _case(nlev, tracers, mono, terrain=0.0, moist=False):
    from mpas_dycore_pytorch_gb300.cases import CaseSpec
    from mpas_dycore_pytorch_gb300.loader import load_case
    cfg = {"config_time_integration_order": 3, "config_len_disp": 120000.0, "config_monotonic": mono,
           "config_dt": 900.0}
    spec = CaseSpec(level=2, nlev=nlev, seed=nlev, n_bumps=4, n_tracers=tracers - moist, u_noise=0.5, w_sine=0.1,
                    terrain=terrain, qv_surface=0.012 if moist else 0.0)
    st, _ = load_case(spec, cfg, as_torch=False)
    return dict(st), cfg


def _widen(st, extra):
    """The same stencils with ``extra`` more slots that add nothing (zero weights)."""
    ne = int(st["nEdges"])
    rng = np.random.default_rng(1)

    def wider(conn, weights, count, n):
        a = np.asarray(st[conn])
        idx = np.zeros((a.shape[0], a.shape[1] + extra), a.dtype)
        idx[:, :a.shape[1]] = a
        num = np.asarray(st[count]).copy()
        for e in range(0, ne, 3):  # a third of the edges use the new slots
            k = int(num[e])
            idx[e, k:k + extra] = rng.integers(1, n + 1, extra)
            num[e] = k + extra
        st[conn], st[count] = idx, num
        for w in weights:
            b = np.asarray(st[w])
            st[w] = np.concatenate([b, np.zeros((b.shape[0], extra))], 1)

    wider("edgesOnEdge", ["weightsOnEdge"], "nEdgesOnEdge", ne)
    wider("advCellsForEdge", ["adv_coefs", "adv_coefs_3rd"], "nAdvCellsForEdge", int(st["nCells"]))
    st["maxEdges2"] = st["edgesOnEdge"].shape[1]
    st["nAdvCellsMax"] = st["advCellsForEdge"].shape[1]
    return st


def _compare(st, cfg, steps=2):
    from mpas_dycore_pytorch_gb300.api import Model
    from oracle.step import Stepper
    model = Model(st, cfg, 900.0, num_scalars=st["scalars"].shape[-1])
    model.prepare(st)
    ref = Stepper(st, cfg)
    rs = ref.prepare(st, 900.0)
    for _ in range(steps):
        model.step()
        rs = ref.srk3_step(rs, 900.0)
    got = model.export()
    for k in KEYS:
        err = rel_l2(to_np(got[k])[:-1], rs[k][:-1])
        assert err <= STEP_TOL, (k, err)


@pytest.mark.parametrize("nlev,tracers,mono", [(4, 1, False), (5, 8, True), (7, 3, True), (31, 2, False), (32, 1, True),
                                               (33, 5, False), (64, 3, True)])
def test_level_and_tracer_counts(nlev, tracers, mono):
    need_gpu()
    _compare(*_case(nlev, tracers, mono))


@pytest.mark.parametrize("nlev,moist", [(6, False), (19, True)])
def test_terrain(nlev, moist):
    need_gpu()
    _compare(*_case(nlev, 2, True, terrain=1500.0, moist=moist))


@pytest.mark.parametrize("extra", [1, 4, 6])
def test_wide_stencils(extra):
    need_gpu()
    st, cfg = _case(9, 2, True)
    _compare(_widen(st, extra), cfg)
