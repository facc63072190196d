"""The sweep with register-held columns (the solver's own form) on the widths,
partial tiles and boundaries that its configurations split on: rows of 16, 32,
64 and 128 chunks taken whole, rows cut into tiles, rows with idle lanes, a
last row tile of one row, few planes.

Every form of the fused sweep does the same updates in the same order, so a
defect-correction solve gives the same pressure to the bit as the merged-phase
form (FP32) and the pair form (FP32 and FP64), and a CG solve the same to
rounding (assert_same_solve)."""
import os
import warnings

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
