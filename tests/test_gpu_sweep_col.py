"""The sweep with register-held columns (the solver's own form) on the widths,
partial tiles and boundaries that its configurations split on: rows taken
whole, rows cut into tiles, rows with idle lanes, a last row tile of one row,
few planes.

Against other forms: every form of the fused sweep does the same updates in the
same order, so a defect-correction solve gives the same pressure to the bit as
the merged-phase form (FP32) and the pair form (FP32 and FP64), and a CG solve
the same to rounding (assert_same_solve).  Against the oracle's cycle: on levels
that take each configuration, whole and cut."""
import os
import warnings

import numpy as np
import pytest

from sweep_case import assert_same_solve, problem as _problem

pytestmark = pytest.mark.gpu

KEYS = ("PARIS_SWEEP_MERGED", "PARIS_SWEEP_PAIRS", "PARIS_SWEEP_TMA", "PARIS_SWEEP_RS")


def _solve(runtime, capi, desc, cvof, vel, env, mode, pcg):
    old = {k: os.environ.get(k) for k in KEYS}
    os.environ.update({k: env.get(k, "0") for k in KEYS})
    try:
        with runtime.ParisGpu(desc) as gpu:
            gpu.upload(capi.F_CVOF, cvof)
            for f, a in zip((capi.F_U, capi.F_V, capi.F_W), vel):
                gpu.upload(f, a)
            gpu.linfunc(capi.F_RHO)
            gpu.setup_poisson(1e-3)
            gpu.fill_field(capi.F_P, 0.0)
            r = gpu.new_solver(0.0, maxit=3, mode=mode, rel_tol=1e-300, pcg=pcg, beta=1.1)
            return gpu.download(capi.F_P), r
    finally:
        for k, v in old.items():
            if v is None:
                del os.environ[k]
            else:
                os.environ[k] = v


@pytest.mark.parametrize("mode", ["mixed", "fp64"])
@pytest.mark.parametrize("n,bc", [((64, 26, 32), "wall"), ((60, 32, 64), (0, 1, 1, 0, 1, 1)), ((128, 16, 32), "periodic"),
                                  ((104, 28, 16), (1, 0, 1, 1, 0, 1)), ((256, 16, 16), "wall"), ((256, 64, 8), "periodic"),
                                  ((248, 48, 8), (0, 1, 0, 0, 1, 0)), ((512, 16, 8), "periodic"),
                                  ((400, 20, 16), "wall"), ((136, 32, 32), "wall"), ((192, 64, 16), "periodic")])
def test_column_sweep_matches_other_forms(gpu_lib, capi, runtime, orc, workloads, n, bc, mode):
    desc, cvof, vel = _problem(capi, orc, workloads, n, bc, seed=7)
    m = capi.MG_MIXED if mode == "mixed" else capi.MG_FP64
    other = {"PARIS_SWEEP_MERGED": "1"} if mode == "mixed" else {"PARIS_SWEEP_PAIRS": "1"}
    with warnings.catch_warnings():
        warnings.simplefilter("ignore")
        for pcg in (0, 1):
            p_d, r_d = _solve(runtime, capi, desc, cvof, vel, {}, m, pcg)
            p_o, r_o = _solve(runtime, capi, desc, cvof, vel, other, m, pcg)
            assert_same_solve(p_d, r_d, p_o, r_o, pcg, mode == "mixed")


# levels that take the FP32 configurations 0 to 6 and the FP64 ones 0 to 4 as
# whole rows and (all but FP32 5) cut into tiles
WALL, MIXED = "wall", (0, 1, 1, 0, 1, 1)
F32 = [((32, 8, 128), "periodic"), ((128, 8, 32), MIXED), ((68, 8, 100), WALL), ((228, 8, 64), "periodic"),
       ((132, 40, 32), (1, 0, 1, 1, 0, 1)), ((244, 88, 8), WALL), ((228, 8, 128), WALL), ((396, 56, 16), "periodic"),
       ((20, 56, 32), MIXED), ((228, 8, 32), WALL), ((340, 8, 128), "periodic"), ((132, 8, 100), MIXED),
       ((244, 8, 64), WALL), ((260, 20, 16), "periodic"), ((520, 12, 8), MIXED)]
F64 = [((32, 8, 128), "periodic"), ((128, 16, 16), MIXED), ((64, 8, 64), WALL), ((128, 8, 32), "periodic"),
       ((68, 16, 100), (1, 0, 1, 1, 0, 1)), ((144, 8, 100), WALL), ((124, 8, 128), "periodic"), ((372, 8, 64), MIXED),
       ((20, 56, 32), WALL), ((68, 40, 16), "periodic")]


@pytest.mark.parametrize("n,bc,mode", [(*c, "mixed") for c in F32] + [(*c, "fp64") for c in F64])
def test_column_sweep_follows_oracle(gpu_lib, capi, runtime, orc, workloads, n, bc, mode):
    """Two defect-correction cycles: the oracle's residual and its pressure up to
    the free constant.  FP64: the updates and their order are the oracle's, but
    the device contracts a*b+c into one rounding, a few 1e-16 of a value in each
    update, and later updates damp what came before: 1e-14 of the largest pressure
    (4.5e-16 seen).  FP32 cycles sum in another order and divide to two ulps
    (2e-7): 4e-6 (4.8e-7 seen)."""
    desc, cvof, vel = _problem(capi, orc, workloads, n, bc, seed=7)
    rho = orc.linfunc(desc, cvof, desc.rho1, desc.rho2, capi.MEAN_ARITH)
    _, A = orc.setup_poisson(desc, *vel, rho, 1e-3)
    ref, _, hist = orc.fastmg_solve(desc, A, np.zeros(n[::-1]), 1e-300, maxit=2, mixed=mode == "mixed", pcg=False,
                                    omega=1.1)
    with runtime.ParisGpu(desc) as gpu, warnings.catch_warnings():
        warnings.simplefilter("ignore")
        gpu.upload(capi.F_CVOF, cvof)
        gpu.upload(capi.F_RHO, rho)
        for f, a in zip((capi.F_U, capi.F_V, capi.F_W), vel):
            gpu.upload(f, a)
        gpu.setup_poisson(1e-3)
        gpu.fill_field(capi.F_P, 0.0)
        r = gpu.new_solver(0.0, maxit=2, mode=capi.MG_MIXED if mode == "mixed" else capi.MG_FP64, rel_tol=1e-300, pcg=0,
                           beta=1.1)
        p = orc.interior(desc, gpu.download(capi.F_P))
    tol = 4e-6 if mode == "mixed" else 1e-14
    d = (p - p.mean()) - (ref - ref.mean())
    assert np.abs(d).max() <= tol * np.abs(ref).max()
    assert abs(r.rel_res - hist[-1]) <= 10 * tol * hist[-1]
