"""Coarsest levels that are no power of two, against the CPU oracle's cycle:
relaxed in one block (up to 5.7 thousand cells FP64, 11.5 FP32; 4.8 and 9.6 with a
seam) and by launches (above), with odd extents over periodic seams, where the first and the last cell
of a row share a colour, and between walls."""
import warnings

import numpy as np
import pytest

from sweep_case import problem as _problem
from test_oracle_fastmg import seam_pairs

pytestmark = pytest.mark.gpu


# coarsest levels 5x3x7, 9x10x11 and 15x9x21 in one block, 18x17x17, 25x17x21 and
# 27x26x13 in one block (FP32, and 18x17x17 between walls) and by launches (FP64),
# 33x25x15 by launches, 45x23x27 (the whole grid) with no level above it
GRIDS = [((20, 12, 28), "periodic"), ((36, 40, 44), (1, 0, 1, 1, 0, 1)), ((60, 36, 84), "wall"),
         ((60, 36, 84), "periodic"), ((36, 34, 34), "periodic"), ((36, 34, 34), "wall"), ((50, 34, 42), "periodic"),
         ((54, 52, 26), (0, 1, 1, 0, 1, 1)), ((50, 34, 42), "wall"), ((66, 50, 30), "periodic"),
         ((45, 23, 27), "periodic")]


@pytest.mark.parametrize("mode", ["fp64", "mixed"])
@pytest.mark.parametrize("n,bc", GRIDS)
def test_cycles_follow_oracle(gpu_lib, capi, runtime, orc, workloads, n, bc, mode):
    """Three defect-correction cycles: the pressure of the oracle's cycles up to
    its free constant, and the same bits when run again.  FP64: the updates and
    their order are the oracle's, but the device contracts a*b+c into one
    rounding, a few 1e-16 of a value in each update, and later updates damp what
    came before: 1e-14 of the largest pressure.  FP32 cycles sum in another order
    and divide to two ulps (2e-7): 4e-6."""
    desc, cvof, vel = _problem(capi, orc, workloads, n, bc, seed=5)
    rho = orc.linfunc(desc, cvof, desc.rho1, desc.rho2, capi.MEAN_ARITH)
    _, A = orc.setup_poisson(desc, *vel, rho, 1e-3)
    ref, _, hist = orc.fastmg_solve(desc, A, np.zeros(n[::-1]), 1e-300, maxit=3, mixed=mode == "mixed", pcg=False,
                                    omega=1.1)
    out = []
    with runtime.ParisGpu(desc) as gpu, warnings.catch_warnings():
        warnings.simplefilter("ignore")
        gpu.upload(capi.F_CVOF, cvof)
        gpu.upload(capi.F_RHO, rho)
        for f, a in zip((capi.F_U, capi.F_V, capi.F_W), vel):
            gpu.upload(f, a)
        gpu.setup_poisson(1e-3)
        for _ in range(2):
            gpu.fill_field(capi.F_P, 0.0)
            r = gpu.new_solver(0.0, maxit=3, mode=capi.MG_FP64 if mode == "fp64" else capi.MG_MIXED, rel_tol=1e-300,
                               pcg=0, beta=1.1)
            out.append(orc.interior(desc, gpu.download(capi.F_P)))
    tol = 1e-14 if mode == "fp64" else 4e-6
    d = (out[0] - out[0].mean()) - (ref - ref.mean())
    assert np.array_equal(out[0], out[1])
    assert np.abs(d).max() <= tol * np.abs(ref).max()
    assert abs(r.rel_res - hist[-1]) <= 10 * tol * hist[-1]


@pytest.mark.parametrize("omega", [1.0, 1.25, 1.5])
def test_pairs_over_an_odd_seam(gpu_lib, capi, runtime, orc, omega):
    """Light cells of one colour facing each other over a seam: the solver follows
    the oracle's CG within one iteration."""
    desc, rho, vel, A = seam_pairs(capi, orc)
    _, it, _ = orc.fastmg_solve(desc, A, np.zeros((9, 9, 9)), 1e-10, maxit=100, mixed=False, pcg=True, omega=omega)
    with runtime.ParisGpu(desc) as gpu:
        gpu.upload(capi.F_RHO, rho)
        for f, a in zip((capi.F_U, capi.F_V, capi.F_W), vel):
            gpu.upload(f, a)
        gpu.setup_poisson(1e-3)
        gpu.fill_field(capi.F_P, 0.0)
        r = gpu.new_solver(0.0, maxit=100, mode=capi.MG_FP64, rel_tol=1e-10, pcg=1, beta=omega)
    assert r.rel_res < 1e-10 and abs(r.it - it) <= 1


def test_handles_in_threads(gpu_lib, capi, runtime, orc, workloads):
    """Handles whose coarse cycles take 219, 137 and 45 KB of shared memory,
    solving in three threads at once, give the bits that each gives alone: what a
    kernel may take is lifted per device and never lowered for another handle."""
    import threading

    cases = [((64, 64, 64), "periodic"), ((32, 16, 40), "wall"), ((20, 12, 28), "periodic")]
    handles = []
    try:
        for n, bc in cases:
            desc, cvof, vel = _problem(capi, orc, workloads, n, bc, seed=9)
            gpu = runtime.ParisGpu(desc)
            handles.append(gpu)
            gpu.upload(capi.F_CVOF, cvof)
            for f, a in zip((capi.F_U, capi.F_V, capi.F_W), vel):
                gpu.upload(f, a)
            gpu.linfunc(capi.F_RHO)
            gpu.setup_poisson(1e-3)
        out = [[] for _ in cases]

        def solve(q):
            gpu = handles[q]
            gpu.fill_field(capi.F_P, 0.0)
            gpu.new_solver(0.0, maxit=60, mode=capi.MG_FP64, rel_tol=1e-9, pcg=1)
            out[q].append(gpu.download(capi.F_P))

        threads = [threading.Thread(target=lambda q=q: [solve(q) for _ in range(3)]) for q in range(3)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        for q in (2, 0, 1):
            solve(q)
    finally:
        for gpu in handles:
            gpu.close()
    for o in out:
        assert len(o) == 4
        for p in o[:3]:
            assert np.array_equal(p, o[3])
