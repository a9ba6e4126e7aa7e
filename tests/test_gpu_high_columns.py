"""Columns too high for shared memory: the implicit coefficients (above 1700 levels) and the
acoustic columns (above 1066) through memory instead, against the oracle; the mixed form, which
has no such kernels, refuses its acoustic columns above 193 levels.

Bounds.  Stages: the sweeps of 1800 levels pass their roundings on, a few of 2^-53 a level,
2e-12 in all: 1e-11 relative L2.  A whole step: ten times that."""

import ctypes as C

import numpy as np
import pytest

from fixtures import rel_l2
from gpu_helpers import need_gpu, to_np

pytestmark = pytest.mark.gpu

DT = 120.0


def _case(nlev, precision="float64"):
    from mpas_dycore_pytorch_gb300.api import Model
    from mpas_dycore_pytorch_gb300.cases import CaseSpec
    from mpas_dycore_pytorch_gb300.loader import load_case
    cfg = {"config_time_integration_order": 3, "config_len_disp": 120000.0, "config_monotonic": False,
           "config_dt": DT, "config_precision": precision}
    spec = CaseSpec(level=2, nlev=nlev, seed=1, n_bumps=4, n_tracers=1, w_sine=0.1)
    st, _ = load_case(spec, cfg, as_torch=False)
    model = Model(st, cfg, DT, num_scalars=1)
    model.prepare(st)
    return model, dict(st), cfg


@pytest.mark.parametrize("nlev", [1100, 1800])
def test_columns_through_memory(nlev):
    need_gpu()
    from mpas_dycore_pytorch_gb300.stages import run_stage
    from oracle.step import STAGE_NAMES, Stepper
    model, st, cfg = _case(nlev)
    calls = {k: [] for k in ("vimp", "acoustic")}
    keys = {STAGE_NAMES[k]: k for k in calls}

    def on_stage(name, a, out):
        if name in keys and len(calls[keys[name]]) < 3:
            calls[keys[name]].append((dict(a), out))

    ref = Stepper(st, cfg, on_stage)
    want = ref.srk3_step(ref.prepare(st, DT), DT)
    model.step()
    got = model.export()
    for k in ("u", "w", "theta_m", "rho_zz", "rtheta_p", "ruAvg", "wwAvg", "scalars"):
        err = rel_l2(to_np(got[k])[:-1], want[k][:-1])
        assert err <= 1e-10, (k, err)
    for key, taken in calls.items():
        assert taken
        for a, out in taken:
            res = run_stage(model, key, a)
            for k, g in res.items():
                r = np.asarray(out[k])
                rows = model.dmesh.nCells if r.shape[0] in (model.dmesh.nCells, model.dmesh.nCells + 1) else \
                    model.dmesh.nEdges if r.ndim > 1 else r.shape[0]
                err = rel_l2(to_np(g)[:rows], r[:rows])
                assert err <= 1e-11, (key, k, err)


def test_mixed_form_refuses_high_columns():
    need_gpu()
    from mpas_dycore_pytorch_gb300.errors import MpasConfigError
    for nlev in (193, 194):
        model, _, _ = _case(nlev, "mixed")
        model.call("mpasg_moist_coefficients")
        model.call("mpasg_vert_imp_coefs", C.c_double(DT))
        model.call("mpasg_dyn_tend", C.c_int(1))
        if nlev == 193:
            model.call("mpasg_acoustic_step", C.c_int(1), C.c_double(DT))
            model.step()
            assert model.check_finite() == 0
            continue
        with pytest.raises(MpasConfigError):
            model.call("mpasg_acoustic_step", C.c_int(1), C.c_double(DT))
        with pytest.raises(MpasConfigError):
            model.step()
