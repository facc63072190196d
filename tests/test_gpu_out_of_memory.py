"""A call that finds no device memory for its arrays fails with PARIS_CUDA_ERROR
and leaves nothing half made: the same call with memory available gives what a
handle that never ran short gives, and calls in between work."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N = 128
LEFT = 48 << 20   # less than any of the calls needs, more than its first array


def prepare(capi, runtime, workloads):
    desc = capi.make_desc((N, N, N), rho1=1.0, rho2=100.0, mu1=1e-3, mu2=1e-2, sigma=0.01)
    gpu = runtime.ParisGpu(desc)
    cen, rad = workloads.drop_layout(6, rmin=0.1, rmax=0.15, seed=4, h=1.0 / N)
    gpu.init_spheres(cen, rad, refinement=2)
    rng = np.random.default_rng(5)
    for f in (capi.F_U, capi.F_V, capi.F_W):
        gpu.upload(f, 0.1 * rng.standard_normal(gpu.shape))
    gpu.set_velocity_bc()
    gpu.linfunc(capi.F_RHO)
    gpu.setup_poisson(1e-4)
    return gpu


def solve(mode):
    def call(gpu, capi):
        gpu.fill_field(capi.F_P, 0.0)
        gpu.new_solver(1e-3, maxit=100, mode=getattr(capi, mode), rel_tol=1e-6, pcg=0 if mode == "MG_REFERENCE" else 1)
    return call, ("F_P",)


def heights(gpu, capi):
    gpu.get_all_heights()
    gpu.surface_force()


def momcons(gpu, capi):
    gpu.vof_mom_sweeps(1, 1e-4)


CALLS = {"reference": solve("MG_REFERENCE"), "fp64": solve("MG_FP64"), "mixed": solve("MG_MIXED"),
         "heights": (heights, ("F_HEIGHT", "F_KAPPA", "F_DU")), "momcons": (momcons, ("F_DU", "F_DV", "F_DW"))}


@pytest.mark.parametrize("name", list(CALLS))
def test_call_after_no_memory(gpu_lib, capi, runtime, workloads, name):
    torch = pytest.importorskip("torch")
    call, fields = CALLS[name]
    with prepare(capi, runtime, workloads) as gpu:
        call(gpu, capi)
        want = [gpu.download(getattr(capi, f)) for f in fields]
    with prepare(capi, runtime, workloads) as gpu:
        gpu.sync()
        torch.cuda.empty_cache()
        hold = torch.empty(torch.cuda.mem_get_info()[0] - LEFT, dtype=torch.uint8, device="cuda")
        try:
            for _ in range(2):
                with pytest.raises(runtime.ParisError) as e:
                    call(gpu, capi)
                assert e.value.status == capi.CUDA_ERROR
            gpu.linfunc(capi.F_RHO)   # a call that needs no more memory
        finally:
            del hold
            torch.cuda.empty_cache()
        call(gpu, capi)
        for f, w in zip(fields, want):
            assert np.array_equal(gpu.download(getattr(capi, f)), w), f
