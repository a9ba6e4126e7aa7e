"""The acoustic columns in one launch against the same columns in parts, and a captured step,
whose independent kernels run side by side, against the step launched in order: bit for bit."""

import ctypes as C

import pytest
import torch

from gpu_helpers import need_gpu

pytestmark = pytest.mark.gpu

DT = 900.0
ACOUSTIC = ("ru_p", "ruAvg", "rw_p", "wwAvg", "rho_pp", "rtheta_pp", "rtheta_pp_old", "ac_rs", "ac_ts", "ac_x")


def _model(nlev, terrain=0.0, level=2, **options):
    from mpas_dycore_pytorch_gb300.api import Model
    from mpas_dycore_pytorch_gb300.cases import CaseSpec
    from mpas_dycore_pytorch_gb300.loader import load_case
    cfg = {"config_time_integration_order": 3, "config_len_disp": 120000.0, "config_monotonic": True,
           "config_dt": DT, **options}
    spec = CaseSpec(level=level, nlev=nlev, seed=nlev, n_bumps=4, n_tracers=2, u_noise=0.5, w_sine=0.1,
                    terrain=terrain)
    st, _ = load_case(spec, cfg, as_torch=False)
    model = Model(st, cfg, DT, num_scalars=2)
    model.prepare(st)
    return model, st


# levels: the fewest, one over a full pass of a block's threads at the smallest block, the widest
# columns of a block, columns beyond 48 KB of shared memory
@pytest.mark.parametrize("nlev,terrain", [(4, 0.0), (12, 0.0), (13, 1500.0), (33, 0.0), (63, 1500.0), (64, 0.0),
                                          (127, 0.0), (300, 0.0)])
def test_columns_in_one_launch(nlev, terrain):
    need_gpu()
    from mpas_dycore_pytorch_gb300.dyn_adjoint import DynamicsTangent
    model, _ = _model(nlev, terrain)
    tan = DynamicsTangent(model)
    st, dts = model.state, DT / 3.0 / 2.0
    model.step()  # the time-level saves the substeps read
    model.call("mpasg_moist_coefficients")
    model.call("mpasg_vert_imp_coefs", C.c_double(dts))
    model.call("mpasg_dyn_tend", C.c_int(1))
    model.call("mpasg_smlstep_pert")
    for small in (1, 2, 3):
        start = st.arena.clone()
        args = [C.byref(s) for s in (model.dmesh.struct, model.cstruct, st.struct, tan.d.struct)]
        stream = C.c_void_p(torch.cuda.current_stream().cuda_stream)
        tan.d.arena.zero_()
        assert model.lib.mpasg_acoustic_jvp(*args, small, dts, C.c_void_p(tan.work.data_ptr()), stream) == 0
        parts = {k: st.f[k][:-1].clone() for k in ACOUSTIC}
        st.arena.copy_(start)
        model.call("mpasg_acoustic_step", C.c_int(small), C.c_double(dts))
        for k in ACOUSTIC:
            assert torch.equal(st.f[k][:-1], parts[k]), (small, k)
        assert st.f["rw_p"].abs().max() > 0
        model.call("mpasg_divergence_damping", C.c_double(dts))


@pytest.mark.parametrize("options", [{}, {"config_dynamics_split_steps": 1}, {"config_precision": "mixed"},
                                     {"config_precision": "mixed", "config_dynamics_split_steps": 1},
                                     {"config_time_integration_order": 2}])
@pytest.mark.parametrize("terrain", [0.0, 1500.0])
def test_captured_step_with_branches(options, terrain):
    need_gpu()
    eager, st = _model(20, terrain, level=3, **options)
    for _ in range(4):
        eager.step()
    want = eager.export()
    model, _ = _model(20, terrain, level=3, **options)
    model.step()
    model.capture_graph()
    for _ in range(3):
        model.step()
    got = model.export()
    for k, v in want.items():
        assert torch.equal(got[k], v), k


def test_implicit_coefficients_of_high_columns():
    """Blocks whose columns leave no room for the level coefficients in shared memory (2562
    columns of 300 levels) against blocks that hold them (the same columns on 162 cells)."""
    need_gpu()
    big, _ = _model(300, level=4)
    small, _ = _model(300, level=2)
    big.call("mpasg_moist_coefficients")
    nc = small.dmesh.nCells
    columns = ("exner", "exner_base", "rtheta_base", "rtheta_p", "qtot", "theta_m", "cqw")
    for k in columns:
        small.state.f[k][:nc].copy_(big.state.f[k][:nc])
    small.dmesh._keep["rho_base"][:nc].copy_(big.dmesh._keep["rho_base"][:nc])
    assert torch.equal(small.dmesh._keep["zz"][:nc], big.dmesh._keep["zz"][:nc])
    for model in (big, small):
        model.call("mpasg_vert_imp_coefs", C.c_double(DT / 6.0))
    for k in ("cofrz",):
        assert torch.equal(small.state.f[k].flatten()[:300], big.state.f[k].flatten()[:300])
    for k in ("cofwr", "cofwz", "cofwt", "coftz", "a_tri", "b_tri", "c_tri", "alpha_tri", "gamma_tri"):
        assert torch.equal(small.state.f[k][:nc], big.state.f[k][:nc]), k
        assert torch.isfinite(small.state.f[k][:nc]).all(), k
