"""Float64 transport of more (row, level, tracer) values than one launch numbers: a build whose
launches take few rows against the library's, bit for bit (each value is formed by the same
expressions whatever launch it falls to), and an explicit stage of 2^32 edge values against
its tracers one by one (the two halves of an edge's values are summed on different pipes: the
stage bound, 1e-12)."""

import ctypes as C
import subprocess

import pytest
import torch

from gpu_helpers import need_gpu
from test_gpu_stencil_sizes import _case

pytestmark = pytest.mark.gpu

DT = 900.0


def _model(nlev, tracers, level=2):
    from mpas_dycore_pytorch_gb300.api import Model
    from mpas_dycore_pytorch_gb300.cases import CaseSpec
    from mpas_dycore_pytorch_gb300.loader import load_case
    if level == 2:
        st, cfg = _case(nlev, tracers, True)
    else:
        cfg = {"config_time_integration_order": 3, "config_len_disp": 120000.0, "config_dt": DT}
        st, _ = load_case(CaseSpec(level=level, nlev=nlev, n_tracers=1), cfg, as_torch=False)
    model = Model(st, cfg, DT, num_scalars=tracers)
    model.prepare(st)
    return model


@pytest.fixture(scope="module", params=[1, 3000])  # one row a launch; a few, the last launch shorter
def few(request, tmp_path_factory):
    """The transport's entry points, built with that many threads a launch."""
    need_gpu()
    from mpas_dycore_pytorch_gb300 import build
    d = tmp_path_factory.mktemp("transport")
    stub, so = d / "count.cu", d / "libtransport.so"
    stub.write_text("void mpasg_count_launch() {}\n")
    flags = build._flags((f"-DMPASG_MAX_THREADS={request.param}",))
    subprocess.run([build.nvcc_path(), *flags, "-shared", "-o", str(so), str(build.CSRC / "kern_transport.cu"),
                    str(stub)], check=True)
    return C.CDLL(str(so))


@pytest.mark.parametrize("nlev,tracers", [(4, 1), (13, 3), (26, 8)])
def test_several_launches(few, nlev, tracers):
    model = _model(nlev, tracers)
    model.step()
    f = model.state.f
    f["scalars_a"].copy_(f["scalars"])
    args = [C.byref(s) for s in (model.dmesh.struct, model.cstruct, model.state.struct)]
    for entry, extra in (("mpasg_advance_scalars", (C.c_int(1), C.c_double(DT))),
                         ("mpasg_advance_scalars_mono", (C.c_double(DT),))):
        got = []
        for lib in (model.lib, few):
            for k in ("scalars_b", "hflux", "flux_up", "flux_tmp", "rows", "scale_in", "scale_out"):
                f[k].zero_()
            stream = C.c_void_p(torch.cuda.current_stream().cuda_stream)
            assert getattr(lib, entry)(*args, *extra, stream) == 0
            torch.cuda.synchronize()
            got.append({k: f[k].clone() for k in ("scalars_b", "hflux")})
        for k in got[0]:
            assert torch.equal(got[0][k], got[1][k]), (entry, k)
        assert got[0]["scalars_b"].abs().max() > 0


def test_more_than_32_bits_of_values():
    """30720 edges of 17500 levels with 8 tracers: 4.3e9 edge values (34 GB), 1.43e9 cell values."""
    need_gpu()
    nlev, tracers = 17500, 8
    torch.cuda.empty_cache()
    if torch.cuda.mem_get_info()[0] < 100e9:
        pytest.skip("needs 100 GB of free device memory")
    model = _model(4, 1, level=5)
    m, f, c = model.dmesh.struct, model.state.struct, model.cstruct
    ne, nc = model.dmesh.nEdges, model.dmesh.nCells
    assert ne * nlev * tracers > 2 ** 32
    g = torch.Generator(device="cuda").manual_seed(1)
    rand = lambda *s: torch.rand(s, generator=g, dtype=torch.float64, device="cuda")
    keep = {"fnm": 0.5 + 0.0 * rand(nlev), "fnp": 0.5 + 0.0 * rand(nlev), "rdnw": 1e-3 * (1.0 + rand(nlev))}
    for k, v in keep.items():
        setattr(m, k, v.data_ptr())
    m.nVertLevels = nlev
    ru, ww = 20.0 * (rand(ne + 1, nlev) - 0.5), 0.02 * (rand(nc + 1, nlev + 1) - 0.5)
    rho_old, rho = 1.0 + 0.1 * rand(nc + 1, nlev), 1.0 + 0.1 * rand(nc + 1, nlev)
    for k, v in (("ruAvg", ru), ("wwAvg", ww), ("rho_zz_old_split", rho_old), ("rho_zz", rho)):
        setattr(f, k, v.data_ptr())

    def stage(init, new):
        n = init.shape[-1]
        out, flux = torch.empty_like(init), torch.empty((ne + 1, nlev, n), dtype=torch.float64, device="cuda")
        for k, v in (("scalars_init", init), ("scalars_a", new), ("scalars_b", out), ("hflux", flux)):
            setattr(f, k, v.data_ptr())
        c.num_scalars = n
        model.call("mpasg_advance_scalars", C.c_int(1), C.c_double(DT))
        torch.cuda.synchronize()
        return out[:nc]

    init, new = rand(nc + 1, nlev, tracers), rand(nc + 1, nlev, tracers)
    got = stage(init, new)
    assert bool(torch.isfinite(got).all())
    for s in range(tracers):
        want = stage(init[..., s:s + 1].contiguous(), new[..., s:s + 1].contiguous())[..., 0]
        assert ((got[..., s] - want).norm() / want.norm()).item() <= 1e-12, s
    del got, want, init, new
    torch.cuda.empty_cache()
