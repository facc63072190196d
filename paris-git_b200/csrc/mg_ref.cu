// mg_ref.cu -- the reference multigrid, step for step, in FP64 on the B200
// (PARIS_MG_REFERENCE): NewSolverMG / MG_iteration / get_MGmatrix_coef /
// fill_coefficients / coarse_from_fine / coarse_fine_interp / get_residual /
// compute_residual (MGsolver.f90:84-405) with RedBlackRelax and apply_BC_MG
// (newsolver.f90:192-247).  Levels are interior-only arrays: the one-layer
// halo of pMG/EMG is resolved in the kernels by periodic wrap, and is zero on
// walls, where ghost_MG_* never writes and the arrays are zeroed.  Every
// colour of a red-black pass only reads the other colour, so one thread per
// cell reproduces the sequential loop exactly.  Built with -fmad=false.
#include "ctx.cuh"

struct LvlDims {
    int n0, n1, n2;
    long N;
};

__device__ inline double powabs(double r, int norm) {
    double a = fabs(r);
    return norm == 2 ? a * a : (norm == 1 ? a : pow(a, (double)norm));
}

// ---- MG_iteration in one kernel ---------------------------------------------
// One cycle is some seventy dependent passes over levels of 64^3 cells and less:
// as launches of their own they took 5.9 us each, whatever their size, 530 us
// per iteration at 64^3 (its residual and host wait included); as one kernel
// 245 us, bound by the latency of a pass (a barrier over the grid and one round
// of loads from L2).  Here the whole cycle is one cooperative kernel, a block
// per SM, with a barrier over the grid after each pass; levels of at most
// kRefOneBlock cells are worked by block 0 alone, with block barriers.  Passes
// that need no barrier between them are one: the first colour from a zero
// iterate also zeroes the other; the residual and its restriction; the
// prolonged correction is read from the coarse iterate where it is used, never
// stored; the sum with the correction and the residual after it.
// All level extents are powers of two (init_MG), so cells come from shifts.
// Values that other blocks write within the kernel are read past L1 (__ldcg).
static constexpr int kRefThreads = 1024;
static constexpr int kRefOneBlock = 512;   // (16^3 over the grid: its colour pass is two cells a thread in one block)
static constexpr int kRefMaxLevels = 16;
static constexpr long kRefSpin = 1L << 24;   // polls of a barrier before it gives up (seconds)

struct RefLvl {
    int b0, b1, b2;   // log2 of the extents
    double *K, *p, *e;
    const double* q;   // beta / K7, formed once per solve
};
struct RefCycle {
    RefLvl l[kRefMaxLevels + 1];   // 1..lmg
    int lmg, nrelax, sym;
    double beta;
};

__device__ inline int ref_cell(const RefLvl& l, int i, int j, int k) { return (((k << l.b1) + j) << l.b0) + i; }

// the six neighbours' values f(i,j,k), 0 beyond a wall: loaded at the wrapped
// index without a branch, so that all of them are in flight together
template <typename F>
__device__ inline void ref_nbrs(const RefLvl& l, const Bnd& B, int i, int j, int k, F f, double x[6]) {
    const int e0 = (1 << l.b0) - 1, e1 = (1 << l.b1) - 1, e2 = (1 << l.b2) - 1;
    x[0] = f((i - 1) & e0, j, k);
    x[1] = f((i + 1) & e0, j, k);
    x[2] = f(i, (j - 1) & e1, k);
    x[3] = f(i, (j + 1) & e1, k);
    x[4] = f(i, j, (k - 1) & e2);
    x[5] = f(i, j, (k + 1) & e2);
    if (!B.per[0]) {
        if (i == 0) x[0] = 0.0;
        if (i == e0) x[1] = 0.0;
    }
    if (!B.per[1]) {
        if (j == 0) x[2] = 0.0;
        if (j == e1) x[3] = 0.0;
    }
    if (!B.per[2]) {
        if (k == 0) x[4] = 0.0;
        if (k == e2) x[5] = 0.0;
    }
}

// RedBlackRelax, one colour: (i+j+k+color) even cells (local indices); zero:
// the iterate is zero and is written whole
__device__ inline void ref_relax(const RefLvl& l, double* x, const Bnd& B, double beta, int color, bool zero, int t0,
                                 int st) {
    const int N = 1 << (l.b0 + l.b1 + l.b2), h = l.b0 - 1;
    const double* K = l.K;
    auto f = [&](int i, int j, int k) { return __ldcg(x + ref_cell(l, i, j, k)); };
    for (int t = t0; t < N / 2; t += st) {
        const int j = (t >> h) & ((1 << l.b1) - 1), k = t >> (h + l.b1);
        const int i = 2 * (t & ((1 << h) - 1)) + ((j + k + color) & 1), m = ref_cell(l, i, j, k);
        const double k7 = __ldcg(K + 7L * N + m);
        if (zero) {
            x[m] = (1.0 - beta) * 0.0 + l.q[m] * (0.0 + k7);
            x[m ^ 1] = 0.0;
            continue;
        }
        double y[6];
        ref_nbrs(l, B, i, j, k, f, y);
        x[m] = (1.0 - beta) * __ldcg(x + m) +
               l.q[m] * (K[m] * y[0] + K[1L * N + m] * y[1] + K[2L * N + m] * y[2] + K[3L * N + m] * y[3] +
                         K[4L * N + m] * y[4] + K[5L * N + m] * y[5] + k7);
    }
}

// get_residual of cell m with the iterate f: K8 <- K8 - K7 x + sum K_n x_n
template <typename F>
__device__ inline double ref_residual(const RefLvl& l, const Bnd& B, int i, int j, int k, int m, F f) {
    const int N = 1 << (l.b0 + l.b1 + l.b2);
    double* K = l.K;
    double y[6];
    ref_nbrs(l, B, i, j, k, f, y);
    const double r = __ldcg(K + 7L * N + m) - K[6L * N + m] * f(i, j, k) + K[m] * y[0] + K[1L * N + m] * y[1] +
                     K[2L * N + m] * y[2] + K[3L * N + m] * y[3] + K[4L * N + m] * y[4] + K[5L * N + m] * y[5];
    K[7L * N + m] = r;
    return r;
}

// The blocks of the grid meet: monotonic arrivals at bar[0].  A block that
// polls too long raises bar[1] and *err, and every block leaves the kernel.
__device__ inline bool ref_grid_sync(unsigned* bar, unsigned& want, int* err) {
    __shared__ int gone;
    want += gridDim.x;
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        atomicAdd(bar, 1u);
        gone = 0;
        long polls = 0;
        unsigned v;
        do {
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(bar) : "memory");
            if (++polls > kRefSpin || *(volatile unsigned*)(bar + 1)) {
                gone = 1;
                atomicExch(bar + 1, 1u);
                *err = 1;
                break;
            }
        } while (v < want);
        __threadfence();
    }
    __syncthreads();
    return gone == 0;
}

// MG_iteration, MGsolver.f90:253-320
__global__ void __launch_bounds__(kRefThreads, 1) k_ref_cycle(const RefCycle C, const Bnd B, unsigned* bar, int* err) {
    unsigned want = 0;
    const int gt = blockIdx.x * kRefThreads + threadIdx.x, gs = gridDim.x * kRefThreads;
    const double beta = C.beta;
    auto size = [](const RefLvl& l) { return 1 << (l.b0 + l.b1 + l.b2); };
    int q = 1;   // levels 1..q are worked by block 0 alone
    while (q < C.lmg && size(C.l[q + 1]) <= kRefOneBlock) q++;
    // the passes of a level on the way down: relaxed from zero, its residual,
    // and the coarse right-hand side; in the order of coarse_from_fine
    // (k1 fastest, then j1, i1)
    auto restrict_ = [&](const RefLvl& l, const RefLvl& c, int t0, int st) {
        const int Nc = size(c);
        auto f = [&](int i, int j, int k) { return __ldcg(l.p + ref_cell(l, i, j, k)); };
        for (int t = t0; t < Nc; t += st) {
            const int i = t & ((1 << c.b0) - 1), j = (t >> c.b0) & ((1 << c.b1) - 1), k = t >> (c.b0 + c.b1);
            double s = 0.0;
#pragma unroll 2
            for (int u = 0; u < 8; u++) {
                const int I = 2 * i + (u >> 2), J = 2 * j + ((u >> 1) & 1), Kk = 2 * k + (u & 1);
                s = s + ref_residual(l, B, I, J, Kk, ref_cell(l, I, J, Kk), f) * 0.125;
            }
            c.K[7L * Nc + t] = s;
        }
    };
    // the correction injected from the level below (sym_MG weights it by the
    // just-zeroed correction): residual with it, and the iterate plus it
    auto correct = [&](const RefLvl& l, const RefLvl& c, int t0, int st) {
        const int N = size(l);
        const double wt = C.sym ? 0.0 : 1.0;
        auto f = [&](int i, int j, int k) { return wt * __ldcg(c.p + ref_cell(c, i >> 1, j >> 1, k >> 1)); };
        for (int m = t0; m < N; m += st) {
            const int i = m & ((1 << l.b0) - 1), j = (m >> l.b0) & ((1 << l.b1) - 1), k = m >> (l.b0 + l.b1);
            ref_residual(l, B, i, j, k, m, f);
            l.p[m] = __ldcg(l.p + m) + f(i, j, k);
        }
    };
    // the iterate plus the relaxed correction e, and the residual with e
    auto finish = [&](const RefLvl& l, int t0, int st) {
        const int N = size(l);
        auto f = [&](int i, int j, int k) { return __ldcg(l.e + ref_cell(l, i, j, k)); };
        for (int m = t0; m < N; m += st) {
            const int i = m & ((1 << l.b0) - 1), j = (m >> l.b0) & ((1 << l.b1) - 1), k = m >> (l.b0 + l.b1);
            l.p[m] = __ldcg(l.p + m) + f(i, j, k);
            ref_residual(l, B, i, j, k, m, f);
        }
    };
#define REF_SYNC()                                    \
    do {                                              \
        if (one) __syncthreads();                     \
        else if (!ref_grid_sync(bar, want, err)) return; \
    } while (0)
    for (int part = 0; part < 3; part++) {
        // down the large levels; the small levels down and up (block 0); up the large levels
        const bool one = part == 1;
        const int t0 = one ? threadIdx.x : gt, st = one ? kRefThreads : gs;
        if (!one || blockIdx.x == 0) {
            const int hi = one ? q : C.lmg, low = one ? 2 : (q + 1 > 2 ? q + 1 : 2);
            if (part < 2)
                for (int L = hi; L >= low; L--) {
                    const RefLvl& l = C.l[L];
                    for (int r = 0; r < 2 * C.nrelax; r++) {
                        ref_relax(l, l.p, B, beta, r & 1, r == 0, t0, st);
                        REF_SYNC();
                    }
                    restrict_(l, C.l[L - 1], t0, st);
                    REF_SYNC();
                }
            if ((one && q >= 2) || (part == 2 && q < 2)) {   // level 2 once more
                for (int color = 0; color < 2; color++) {
                    ref_relax(C.l[2], C.l[2].p, B, beta, color, false, t0, st);
                    REF_SYNC();
                }
            }
            if (part > 0)
                for (int L = one ? 3 : (q + 1 > 3 ? q + 1 : 3); L <= hi; L++) {
                    const RefLvl& l = C.l[L];
                    correct(l, C.l[L - 1], t0, st);
                    REF_SYNC();
                    for (int r = 0; r < 2 * C.nrelax; r++) {
                        ref_relax(l, l.e, B, beta, r & 1, r == 0, t0, st);
                        REF_SYNC();
                    }
                    finish(l, t0, st);
                    REF_SYNC();
                }
        }
        if (one && !ref_grid_sync(bar, want, err)) return;
    }
#undef REF_SYNC
}

// K8 <- K8 - K7 p + sum K_n p_n on the finest level (initial residual) and its
// sum |r|^norm
__global__ void k_ref_initial_residual(const RefLvl l, const Bnd B, int norm, double* part) {
    __shared__ double sh[32];
    double s = 0.0;
    const int N = 1 << (l.b0 + l.b1 + l.b2);
    auto f = [&](int i, int j, int k) { return l.p[ref_cell(l, i, j, k)]; };
    for (int m = blockIdx.x * blockDim.x + threadIdx.x; m < N; m += gridDim.x * blockDim.x) {
        const int i = m & ((1 << l.b0) - 1), j = (m >> l.b0) & ((1 << l.b1) - 1), k = m >> (l.b0 + l.b1);
        s += powabs(ref_residual(l, B, i, j, k, m, f), norm);
    }
    s = block_sum<256>(s, sh);
    if (threadIdx.x == 0) part[blockIdx.x] = s;
}

// compute_residual on the finest level with the caller's A and the ghosted p
__global__ void k_ref_compute_residual(const double* __restrict__ A, const double* __restrict__ p, const Layout L,
                                       int norm, double* part) {
    __shared__ double sh[32];
    double s = 0.0;
    const long N = (long)L.n[0] * L.n[1] * L.n[2];
    ROWS_BEGIN(L.n[0], L.n[1], L.n[2])
        const long m = cidx(L.n[0], L.n[1], i, j, k), n = lidx(L, i, j, k);
        double r = A[7 * N + m] - A[6 * N + m] * p[n] + A[0 * N + m] * p[n - 1] + A[1 * N + m] * p[n + 1] +
                   A[2 * N + m] * p[n - L.pitch] + A[3 * N + m] * p[n + L.pitch] +
                   A[4 * N + m] * p[n - L.plane] + A[5 * N + m] * p[n + L.plane];
        s += powabs(r, norm);
    ROWS_END
    s = block_sum<256>(s, sh);
    if (linear_tid() == 0) part[blockIdx.x] = s;
}

// beta / K7 of a level (RedBlackRelax divides in every pass; the same quotient)
__global__ void k_ref_quotient(const double* __restrict__ K7, double* __restrict__ q, double beta, long N) {
    const long m = blockIdx.x * (long)blockDim.x + threadIdx.x;
    if (m < N) q[m] = beta / K7[m];
}

// fill_coefficients: 0.125*(sum of the 8 children in the Fortran order)
__global__ void k_ref_fill_coef(const double* __restrict__ Kf, const LvlDims f, double* __restrict__ Kc,
                                const LvlDims c) {
    long t = blockIdx.x * (long)blockDim.x + threadIdx.x;
    if (t >= 8 * c.N) return;
    int comp = (int)(t / c.N);
    long m = t % c.N;
    int i = (int)(m % c.n0), j = (int)((m / c.n0) % c.n1), k = (int)(m / ((long)c.n0 * c.n1));
    const double* F = Kf + comp * f.N;
    int I = 2 * i, J = 2 * j, Kk = 2 * k;
    double s = F[cidx(f.n0, f.n1, I, J, Kk)] + F[cidx(f.n0, f.n1, I, J + 1, Kk)] + F[cidx(f.n0, f.n1, I, J, Kk + 1)] +
               F[cidx(f.n0, f.n1, I, J + 1, Kk + 1)] + F[cidx(f.n0, f.n1, I + 1, J, Kk)] +
               F[cidx(f.n0, f.n1, I + 1, J + 1, Kk)] + F[cidx(f.n0, f.n1, I + 1, J, Kk + 1)] +
               F[cidx(f.n0, f.n1, I + 1, J + 1, Kk + 1)];
    Kc[comp * c.N + m] = 0.125 * s;
}

// pMG(LMG) <- p (interior) and p <- p + pMG(LMG)
__global__ void k_ref_field_io(double* __restrict__ pf, double* __restrict__ pm, const Layout L, int add) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x, j = blockIdx.y, k = blockIdx.z;
    if (i >= L.n[0]) return;
    const long m = cidx(L.n[0], L.n[1], i, j, k), n = lidx(L, i, j, k);
    if (add) pf[n] = pf[n] + pm[m];
    else pm[m] = pf[n];
}

static LvlDims dims(const RefLevel& l) { return LvlDims{l.n[0], l.n[1], l.n[2], l.N}; }

static int ref_levels(paris_ctx* c) {
    int nd[3] = {c->d.nx, c->d.ny, c->d.nz};
    int lmg = 1000;
    for (int a = 0; a < 3; a++) {
        if (nd[a] & (nd[a] - 1)) {
            ctx_set_error(c, "multigrid requires 2^n cells per direction (MGsolver.f90:43-46)");
            return PARIS_BAD_ARGS;
        }
        int L = 0;
        while ((1 << (L + 1)) <= nd[a]) L++;
        lmg = L < lmg ? L : lmg;
    }
    if (lmg < 2 || lmg > kRefMaxLevels || c->N > 1L << 30) {
        ctx_set_error(c, "multigrid of %d levels over %ld cells: 2 to %d levels and at most 2^30 cells", lmg, c->N,
                      kRefMaxLevels);
        return PARIS_BAD_ARGS;
    }
    c->ref_lmg = lmg;
    c->ref.resize(lmg + 1);
    for (int L = lmg; L >= 1; L--) {
        RefLevel& l = c->ref[L];
        for (int a = 0; a < 3; a++) l.n[a] = nd[a] >> (lmg - L);
        l.N = (long)l.n[0] * l.n[1] * l.n[2];
        PARIS_CHECK(ctx_malloc(c, &l.K, 8 * l.N * sizeof(double)));
        PARIS_CHECK(ctx_malloc(c, &l.p, l.N * sizeof(double)));
        PARIS_CHECK(ctx_malloc(c, &l.e, l.N * sizeof(double)));
        PARIS_CHECK(ctx_malloc(c, &l.q, l.N * sizeof(double)));
    }
    return PARIS_OK;
}

// all levels or, where memory does not last, none
static int ref_alloc(paris_ctx* c) {
    if (!c->ref.empty()) return PARIS_OK;
    const int st = ref_levels(c);
    if (st != PARIS_OK) {
        for (RefLevel& l : c->ref)
            for (double* p : {l.K, l.p, l.e, l.q}) cudaFree(p);
        c->ref.clear();
    }
    return st;
}

static int log2_of(int n) {
    int b = 0;
    while ((1 << (b + 1)) <= n) b++;
    return b;
}

static RefLvl ref_level(const RefLevel& l) {
    return RefLvl{log2_of(l.n[0]), log2_of(l.n[1]), log2_of(l.n[2]), l.K, l.p, l.e, l.q};
}

// one cycle: a cooperative launch, so that all its blocks are resident
static int mg_iteration(paris_ctx* c, const RefCycle& C) {
    PARIS_CHECK(ctx_malloc(c, &c->ref_bar, 2 * sizeof(unsigned)));
    PARIS_CUDA_TRY(c, cudaMemsetAsync(c->ref_bar, 0, 2 * sizeof(unsigned), c->stream));
    RefCycle a = C;
    void* args[] = {&a, &c->bnd, &c->ref_bar, &c->err_dev};
    const bool prof = prof_enabled(c);
    if (prof) prof_begin(c, "k_ref_cycle", c->N);
    const cudaError_t e = cudaLaunchCooperativeKernel((const void*)k_ref_cycle, dim3(c->nsm), dim3(kRefThreads), args, 0,
                                                      c->stream);
    if (prof) prof_end(c);
    c->launches++;
    PARIS_CUDA_TRY(c, e);
    return PARIS_OK;
}

// NewSolverMG, MGsolver.f90:346-405
int mg_ref_solve(paris_ctx* c, const paris_solve_opts* o, paris_solve_result* res) {
    PARIS_CHECK(ref_alloc(c));
    if (!c->A_valid) PARIS_CHECK(poisson_build_full_A(c));
    int lmg = c->ref_lmg;
    RefLevel& lf = c->ref[lmg];
    PARIS_CUDA_TRY(c, cudaMemcpyAsync(lf.K, c->A, 8 * lf.N * sizeof(double), cudaMemcpyDeviceToDevice, c->stream));
    for (int L = lmg - 1; L >= 1; L--)
        PARIS_LAUNCH(c, k_ref_fill_coef, div_up(8 * c->ref[L].N, 256), 256, 0, c->ref[L + 1].K, dims(c->ref[L + 1]),
                     c->ref[L].K, dims(c->ref[L]));
    for (int L = lmg; L >= 2; L--)
        PARIS_LAUNCH(c, k_ref_quotient, div_up(c->ref[L].N, 256), 256, 0, c->ref[L].K + 6 * c->ref[L].N, c->ref[L].q,
                     o->beta, c->ref[L].N);
    double* p = c->fld[PARIS_FIELD_P];
    PARIS_LAUNCH(c, k_ref_field_io, dim3(div_up(c->d.nx, 128), c->d.ny, c->d.nz), 128, 0, p, lf.p, c->L, 0);
    PARIS_LAUNCH(c, k_ref_initial_residual, red_grid(c, k_ref_initial_residual, 256), 256, 0, ref_level(lf), c->bnd,
                 o->norm, c->red_part);
    double s;
    PARIS_CHECK(ctx_reduce_finish(c, 1, &s));
    double nxyz = (double)c->d.nx * (double)c->d.ny * (double)c->d.nz;
    double tres2 = s / nxyz;
    res->res0 = o->norm == 2 ? sqrt(tres2) : tres2;
    PARIS_CUDA_TRY(c, cudaMemsetAsync(lf.p, 0, lf.N * sizeof(double), c->stream));
    RefCycle C;
    for (int L = 1; L <= lmg; L++) C.l[L] = ref_level(c->ref[L]);
    C.lmg = lmg;
    C.nrelax = c->d.nrelax > 0 ? c->d.nrelax : 3;
    C.sym = c->d.sym_mg;
    C.beta = o->beta;
    int it;
    for (it = 1; it <= o->maxit; it++) {
        PARIS_CHECK(mg_iteration(c, C));
        PARIS_LAUNCH(c, k_ref_field_io, dim3(div_up(c->d.nx, 128), c->d.ny, c->d.nz), 128, 0, p, lf.p, c->L, 1);
        PARIS_CHECK(ctx_ghost_fill(c, p));
        PARIS_LAUNCH(c, k_ref_compute_residual, red_grid(c, k_ref_compute_residual, 256), kRowBlock, 0, c->A, p, c->L, o->norm, c->red_part);
        PARIS_CHECK(ctx_reduce_finish(c, 1, &s));
        if (*c->err_host) {
            *c->err_host = 0;
            ctx_set_error(c, "a barrier of the reference multigrid cycle ran out");
            return PARIS_CUDA_ERROR;
        }
        tres2 = s / nxyz;
        if (o->norm == 2) tres2 = sqrt(tres2);
        if (tres2 != tres2) {
            res->it = it; res->res = tres2;
            ctx_set_error(c, "pressure residual is NaN after %d cycles", it);
            return PARIS_NAN_DETECTED;
        }
        if (tres2 < o->max_error) break;
    }
    res->it = it;
    res->res = tres2;
    return it == o->maxit + 1 ? PARIS_NOT_CONVERGED : PARIS_OK;
}
