"""The mixed form's results by value: SHA-256 of two whole steps and of an acoustic stage over
terrain, as the kernels gave them when every stage ran apart (one kernel for the edges, three
for the columns, saves and flux sums in passes of their own).  A last bit of a float32 stencil
grows to the seventh digit of a step, so a kernel of this form that joins or reorders the others
keeps their roundings; no tolerance would show that it does not."""

import ctypes as C
import hashlib

import pytest
import torch

from gpu_helpers import need_gpu

pytestmark = pytest.mark.gpu

DT = 900.0
ACOUSTIC = ("ru_p", "ruAvg", "rw_p", "wwAvg", "rho_pp", "rtheta_pp", "rtheta_pp_old", "ac_rs", "ac_ts", "ac_x")


def _model(terrain, moist, mono=True, order="native", nlev=14, **options):
    from mpas_dycore_pytorch_gb300.api import Model
    from mpas_dycore_pytorch_gb300.cases import CaseSpec
    from mpas_dycore_pytorch_gb300.loader import load_case
    cfg = {"config_time_integration_order": 3, "config_len_disp": 120000.0, "config_monotonic": mono,
           "config_dt": DT, "config_precision": "mixed", **options}
    spec = CaseSpec(level=2, nlev=nlev, seed=3, n_bumps=4, n_tracers=2 - moist, u_noise=0.5, w_sine=0.1,
                    terrain=terrain, qv_surface=0.012 if moist else 0.0)
    st, _ = load_case(spec, cfg, as_torch=False)
    model = Model(st, cfg, DT, num_scalars=2, order=order)
    model.prepare(st)
    return model


def _digest(fields):
    h = hashlib.sha256()
    for k in sorted(fields):
        v = fields[k]
        h.update((v[:-1] if v.dim() > 1 else v).add(0.0).cpu().numpy().tobytes())  # -0 counts as 0
    return h.hexdigest()[:16]


# (terrain, moist, monotone) -> two steps, in either order of the mesh
STEPS = {
    (0.0, False, False): "633c6c5aa2c90def",
    (0.0, False, True): "85a29c9a8d4747a5",
    (0.0, True, False): "3533ca41cf938a8c",
    (0.0, True, True): "5a3229e01290f083",
    (1500.0, False, False): "e39ed5a96d1caf1c",
    (1500.0, False, True): "573df3af401a0e2a",
    (1500.0, True, False): "357e001d378d5ec4",
    (1500.0, True, True): "7808f487c893a190",
}


@pytest.mark.parametrize("case", STEPS, ids=str)
@pytest.mark.parametrize("order", ["native", "sfc"])
def test_steps(case, order):
    need_gpu()
    model = _model(*case, order=order)
    model.step()
    model.step()
    assert model.check_finite() == 0
    assert _digest(model.export()) == STEPS[case]


OPTIONS = {"coupled": {"config_dynamics_split_steps": 1}, "rk2": {"config_time_integration_order": 2},
           "six_substeps": {"config_number_of_sub_steps": 6},
           "mixing": {"config_horiz_mixing": "2d_fixed", "config_h_mom_eddy_visc4": 1.0e10,
                      "config_h_theta_eddy_visc4": 5.0e9, "config_h_theta_eddy_visc2": 2.0e4,
                      "config_v_mom_eddy_visc2": 1.0, "config_v_theta_eddy_visc2": 1.0}}
# (option, terrain) -> two moist steps
OPTION_STEPS = {
    ("coupled", 0.0): "6a94c03e16a504bc",
    ("coupled", 1500.0): "93a574454b711544",
    ("rk2", 0.0): "a32dfb4c85de4154",
    ("rk2", 1500.0): "bb87dd0ea018b052",
    ("six_substeps", 0.0): "89d790ec152145d9",
    ("six_substeps", 1500.0): "d706c74c0e1043c1",
    ("mixing", 0.0): "994c7fa5e1bf76ae",
    ("mixing", 1500.0): "b36f34910f4239b6",
}


@pytest.mark.parametrize("case", OPTION_STEPS, ids=str)
def test_options(case):
    need_gpu()
    model = _model(case[1], True, **OPTIONS[case[0]])
    model.step()
    model.step()
    assert model.check_finite() == 0
    assert _digest(model.export()) == OPTION_STEPS[case]


# (levels, terrain) -> four acoustic substeps, damping between them, after a step
STAGES = {
    (4, 0.0): "ae6358346b3ec64e 3fe64f8eb25a5d16 57b108b5fad07abb "
              "4627e9f3cc85649b e9c427fe5a65e850",
    (4, 1500.0): "60b261cb7f96c9d3 fec76f942557e804 e8a3d0b85d081647 "
                 "cbfec300c195b1ee fa3f60deae465728",
    (14, 0.0): "6b05485ab36ce6dd 3934d28f54b97ed3 14529e8524125033 "
               "d8dab90a2a399375 3b3808ad268ae8aa",
    (14, 1500.0): "d900481472cf5782 db44408c31efa5ba de15910ff359a05c "
                  "bc1c1a51b9686b4b 5c155523499c305e",
    (33, 0.0): "6cb410c2f9e7e352 b2432798b1ac962a 5083492d6e16d392 "
               "4cc58d4ee9be11b1 a05dc349a0d34a70",
    (33, 1500.0): "f5790e76492acc67 afda1e8f73c5e8ba aa836794e32b09fa "
                  "b8eccc706b44c756 812e82b92136d558",
    (64, 0.0): "5fe04a51c86fbd15 cf5f3b0faa2a4969 d10369fae860b54a "
               "abe1fb21cd423308 95f2c19bbfbe0836",
    (64, 1500.0): "257115280090d71e 3d408ef40e99fe31 83c26a934aa5776f "
                  "1b6eb11ef9c54a57 b813fc97a04a7bdb",
}


@pytest.mark.parametrize("case", STAGES, ids=str)
def test_acoustic_stage(case):
    need_gpu()
    nlev, terrain = case
    model = _model(terrain, True, nlev=nlev)
    dts = DT / 6.0
    model.step()
    model.call("mpasg_moist_coefficients")
    model.call("mpasg_vert_imp_coefs", C.c_double(dts))
    model.call("mpasg_dyn_tend", C.c_int(1))
    model.call("mpasg_smlstep_pert")
    digests = []
    for small in (1, 2, 3, 4):
        model.call("mpasg_acoustic_step", C.c_int(small), C.c_double(dts))
        digests.append(_digest({k: model.state.f[k] for k in ACOUSTIC}))
        model.call("mpasg_divergence_damping", C.c_double(dts))
    model.call("mpasg_recover_large_step", C.c_int(3), C.c_int(4), C.c_double(DT / 3.0))
    assert model.check_finite() == 0
    digests.append(_digest(model.export()))
    assert digests == STAGES[case].split()


# a step from rest whose u tendencies lie about the smallest normal float32 (those below it are
# kept as zero, and so the substeps take them)
TINY_STEP = "5f47b54a917551f9"


def test_tendencies_about_the_smallest_normal():
    need_gpu()
    model = _model(0.0, False, config_horiz_mixing="2d_fixed")  # (without mixing: its coefficients are zero)
    f = model.state.f
    for k in ("u", "v", "ru", "w", "rw", "rho_p", "rtheta_p", "divergence", "vorticity", "ke", "pv_edge"):
        f[k].zero_()
    base = (f["rtheta_base"][:-1] / f["theta_m"][:-1])  # rho_zz of the base state for this theta
    f["rho_zz"][:-1].copy_(base)
    n = f["pressure_p"].numel()
    k = torch.arange(n, dtype=torch.float64, device="cuda") % 41
    f["pressure_p"].copy_((2.0 ** (-110.0 + k % 7) * (1.0 + k)).view_as(f["pressure_p"]))
    model.step()
    assert 0.0 < f["ru"].abs().max().item() < 1e-20
    assert _digest(model.export()) == TINY_STEP
