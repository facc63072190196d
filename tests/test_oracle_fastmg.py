"""CPU tests of the oracle's restatement of the B200 multigrid (og_fastmg.c):
the smoother's relaxation factor on the levels below the finest."""
import numpy as np
import pytest

from test_gpu_projection import drop_problem

N = 32
TOL = 1e-10


def _system(capi, orc, workloads):
    desc, cvof, rho, vel = drop_problem(capi, orc, workloads, N, bc="periodic", ndrops=4)
    _, A = orc.setup_poisson(desc, *vel, rho, 1e-3)
    return desc, A


def _solve(orc, desc, A, **kw):
    return orc.fastmg_solve(desc, A, np.zeros((N, N, N)), TOL, maxit=60, mixed=False, pcg=True, nu_coarse=4,
                            coarse_from=1, coarse_to=2, **kw)


def test_coarse_factor_equal_to_beta_is_the_same_cycle(capi, orc, workloads):
    """omega_coarse == omega is the cycle without it, bit for bit."""
    desc, A = _system(capi, orc, workloads)
    p0, it0, h0 = _solve(orc, desc, A, omega=1.1)
    p1, it1, h1 = _solve(orc, desc, A, omega=1.1, omega_coarse=1.1)
    assert it0 == it1 and np.array_equal(h0, h1) and np.array_equal(p0, p1)


def test_coarse_factor_changes_the_cycle_not_the_solution(capi, orc, workloads):
    """Another factor below the finest level gives another residual history,
    and the same pressure to the solver's tolerance."""
    desc, A = _system(capi, orc, workloads)
    p0, it0, h0 = _solve(orc, desc, A, omega=1.1)
    p1, it1, h1 = _solve(orc, desc, A, omega=1.1, omega_coarse=1.25)
    assert h1[-1] < TOL and h0[-1] < TOL
    assert not np.array_equal(h0[:min(it0, it1)], h1[:min(it0, it1)])
    d = (p1 - p1.mean()) - (p0 - p0.mean())
    assert np.abs(d).max() <= 1e-8 * np.abs(p0 - p0.mean()).max()


def seam_pairs(capi, orc):
    """9^3 periodic, three pairs of light cells (density 1 in 1e6) that face each
    other over the seam in x: cells of one colour that see little but each other."""
    n = 9
    desc = capi.make_desc((n, n, n), rho1=1.0, rho2=1000.0)
    rho = orc.zeros(desc) + 1e6
    r = orc.interior(desc, rho)
    for j, k in ((2, 3), (6, 5), (4, 7)):
        r[k, j, 0] = r[k, j, n - 1] = 1.0
    orc.fill_ghosts(desc, rho)
    rng = np.random.default_rng(0)
    vel = []
    for _ in range(3):
        f = orc.zeros(desc)
        orc.interior(desc, f)[...] = rng.standard_normal((n, n, n))
        orc.fill_ghosts(desc, f)
        vel.append(f)
    st, A = orc.setup_poisson(desc, *vel, rho, 1e-3)
    assert st == 0
    return desc, rho, vel, A


@pytest.mark.parametrize("omega", [1.0, 1.25, 1.5])
def test_pairs_over_an_odd_seam_do_not_grow(capi, orc, omega):
    """An over-relaxed pass that takes such pairs as they were before it grows
    without bound (1e16 after six cycles at 1.25) unless the diagonal is raised:
    the cycles' residual stays below the right-hand side, and CG converges."""
    desc, _, _, A = seam_pairs(capi, orc)
    z = np.zeros((9, 9, 9))
    _, _, h = orc.fastmg_solve(desc, A, z, 1e-300, maxit=20, mixed=False, pcg=False, omega=omega)
    assert h.max() < 1.0
    _, it, h = orc.fastmg_solve(desc, A, z, 1e-10, maxit=100, mixed=False, pcg=True, omega=omega)
    assert h[-1] < 1e-10 and it <= 40
