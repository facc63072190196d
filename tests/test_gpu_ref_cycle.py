"""The reference multigrid's cycle as one cooperative kernel, on level chains
that lie wholly in block 0, wholly on the grid (a second level above 4096
cells), and across both; walls, periodic and mixed boundaries, sym_MG and more
than one number of smoothing sweeps: the iterates equal the oracle's to 1e-12
of the largest pressure, as the other tests of this mode ask."""
import warnings

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,bc,sym,nrelax", [((8, 8, 8), "wall", 0, 3), ((16, 16, 16), "periodic", 0, 3),
                                             ((32, 16, 64), "wall", 0, 2), ((8, 256, 128), "wall", 0, 1),
                                             ((64, 8, 256), "periodic", 0, 3), ((64, 64, 64), (1, 0, 1, 1, 0, 1), 0, 3),
                                             ((32, 32, 32), "periodic", 1, 3), ((8, 512, 8), "wall", 1, 2)])
def test_cycle_follows_oracle(gpu_lib, capi, runtime, orc, n, bc, sym, nrelax):
    desc = capi.make_desc(n, bc=bc, rho1=1.0, rho2=100.0)
    rng = np.random.default_rng(4)
    cvof, vel = orc.zeros(desc), [orc.zeros(desc) for _ in range(3)]
    orc.interior(desc, cvof)[...] = rng.random((n[2], n[1], n[0])).round()
    for f in vel:
        orc.interior(desc, f)[...] = rng.standard_normal((n[2], n[1], n[0]))
    for f in (cvof, *vel):
        orc.fill_ghosts(desc, f)
    for d in range(3):
        if bc == "wall" or (bc != "periodic" and bc[d] == 0):   # nothing through the walls
            vel[d].swapaxes(0, 2 - d)[[1, 1 + n[d]]] = 0.0
    desc.sym_mg, desc.nrelax = sym, nrelax
    rho = orc.linfunc(desc, cvof, desc.rho1, desc.rho2, capi.MEAN_ARITH)
    _, A = orc.setup_poisson(desc, *vel, rho, 1e-3)
    ref = orc.zeros(desc)
    orc.new_solver_mg(desc, A, ref, max_error=1e-300, maxit=4, beta=1.2)
    with runtime.ParisGpu(desc) as gpu, warnings.catch_warnings():
        warnings.simplefilter("ignore")
        gpu.upload(capi.F_CVOF, cvof)
        gpu.upload(capi.F_RHO, rho)
        for f, a in zip((capi.F_U, capi.F_V, capi.F_W), vel):
            gpu.upload(f, a)
        gpu.setup_poisson(1e-3)
        gpu.fill_field(capi.F_P, 0.0)
        gpu.new_solver(1e-300, beta=1.2, maxit=4, mode=capi.MG_REFERENCE)
        p = gpu.download(capi.F_P)
    a, b = orc.interior(desc, p), orc.interior(desc, ref)
    assert np.abs(a - b).max() <= 1e-12 * max(1.0, np.abs(b).max())
