// The multigrid's smoothing kernels on the CPU (cuda_on_host.h) against the
// colour passes written out; ThreadSanitizer ends the program at the first race.
// Arguments: "col <float|double> <configuration> n0 n1 n2 px py pz form zc", the
// column sweep, form 0 plain, 1 zero iterate, 2 with the coarse correction;
// "coarse <type> <levels> n0 n1 n2 px py pz threads", the cycle in shared memory;
// "passes <type> 0 n0 n1 n2 px py pz", colour passes by launches.
static double rnd() {
    static uint64_t s = 88172645463325252ull;
    s ^= s << 13; s ^= s >> 7; s ^= s << 17;
    return (double)(s >> 11) / 9007199254740992.0;
}

template <typename T>
struct Problem {
    int n0, n1, n2;
    Bnd B{};
    T *cx, *cy, *cz, *b, *x, *x2, *xc;
    Problem(int a, int c, int d, const int* per) : n0(a), n1(c), n2(d) {
        const long N = (long)n0 * n1 * n2;
        T** all[] = {&cx, &cy, &cz, &b, &x, &x2, &xc};
        for (T** p : all) {
            *p = (T*)aligned_alloc(16, (N * sizeof(T) + 31) / 16 * 16);
            for (long m = 0; m < N; m++) (*p)[m] = (T)(0.5 + rnd());
        }
        for (int q = 0; q < 3; q++) B.per[q] = per[q];
        for (int k = 0; k < n2; k++)   // no flux through a wall
            for (int j = 0; j < n1; j++)
                for (int i = 0; i < n0; i++) {
                    const long m = cidx(n0, n1, i, j, k);
                    if (!per[0] && i == n0 - 1) cx[m] = 0;
                    if (!per[1] && j == n1 - 1) cy[m] = 0;
                    if (!per[2] && k == n2 - 1) cz[m] = 0;
                }
    }
    LV<T> view(T* it, T w) const { return LV<T>{cx, cy, cz, b, it, n0, n1, n2, (long)n0 * n1 * n2, w}; }
};

// a colour pass, cell after cell (i fastest), with the update of the sweep
template <typename T>
static void pass(const LV<T>& v, const Bnd& B, int color, bool sweep) {
    for (int k = 0; k < v.n2; k++)
        for (int j = 0; j < v.n1; j++)
            for (int i = (j + k + color) & 1; i < v.n0; i += 2) {
                if (!sweep) { smooth_cell(v, B, i, j, k); continue; }
                const long m = cidx(v.n0, v.n1, i, j, k);
                T a1, a3, a5, xw, xe, xs, xn, xb, xt, t;
                west_coefs(v, B, i, j, k, m, a1, a3, a5);
                nbrs(v, v.x, B, i, j, k, m, xw, xe, xs, xn, xb, xt);
                if (SwUpd<T>::apply(a1, v.cx[m], a3, v.cy[m], a5, v.cz[m], xw, xe, xs, xn, xb, xt, v.b[m], v.x[m],
                                    v.omega, t))
                    v.x[m] = t;
            }
}

// the same on a level with odd periodic seams: from the values before the pass
template <typename T>
static void pass_seam(const LV<T>& v, const Bnd& B, int color) {
    const std::vector<T> old(v.x, v.x + v.N);
    const bool s[3] = {B.per[0] && v.n0 % 2, B.per[1] && v.n1 % 2, B.per[2] && v.n2 % 2};
    for (int k = 0; k < v.n2; k++)
        for (int j = 0; j < v.n1; j++)
            for (int i = (j + k + color) & 1; i < v.n0; i += 2) {
                const long m = cidx(v.n0, v.n1, i, j, k);
                T a1, a3, a5, xw, xe, xs, xn, xb, xt, e = 0;
                west_coefs(v, B, i, j, k, m, a1, a3, a5);
                const T a2 = v.cx[m], a4 = v.cy[m], a6 = v.cz[m];
                nbrs(v, old.data(), B, i, j, k, m, xw, xe, xs, xn, xb, xt);
                if (s[0]) e += i == 0 ? a1 : (i == v.n0 - 1 ? a2 : (T)0);
                if (s[1]) e += j == 0 ? a3 : (j == v.n1 - 1 ? a4 : (T)0);
                if (s[2]) e += k == 0 ? a5 : (k == v.n2 - 1 ? a6 : (T)0);
                const T d = a1 + a2 + a3 + a4 + a5 + a6;
                const T sum = a1 * xw + a2 * xe + a3 * xs + a4 * xn + a5 * xb + a6 * xt + v.b[m];
                const T up = (T)0.5 * v.omega * (d + e) > d ? (T)0.5 * v.omega * (d + e) - d : (T)0;
                if (d > 0) v.x[m] = relax((sum + up * old[m]) / (d + up), old[m], v.omega);
            }
}

template <typename T>
static int same(const T* a, const T* b, long N, const char* what) {
    for (long m = 0; m < N; m++)
        if (memcmp(a + m, b + m, sizeof(T))) {
            printf("%s: cell %ld is %.17g, should be %.17g\n", what, m, (double)a[m], (double)b[m]);
            return 1;
        }
    return 0;
}

template <class C>
static int run_col(const int* n, const int* per, int form, int zc) {
    using T = typename C::T;
    Problem<T> p(n[0], n[1], n[2], per);
    const long N = (long)n[0] * n[1] * n[2];
    SwColGeo g;
    sweep_col_tiles<C>(n[0], g);
    g.zc = zc;
    int bad = 0;
    for (int first = 0; first < 2; first++) {
        const LV<T> v = p.view(p.x, (T)1.1);
        const dim3 grid((n[0] + g.W - 1) / g.W, (n[1] + C::TY - 1) / C::TY, (n[2] + zc - 1) / zc);
        std::vector<T> ref(N), out(N, (T)-1);
        for (int k = 0; k < n[2]; k++)
            for (int j = 0; j < n[1]; j++)
                for (int i = 0; i < n[0]; i++) {
                    const long m = cidx(n[0], n[1], i, j, k);
                    ref[m] = form == 1 ? (T)0 : p.x[m];
                    if (form == 2) ref[m] += p.xc[cidx(n[0] / 2, n[1] / 2, i / 2, j / 2, k / 2)];
                }
        T* dst = p.x2;
        if (form == 0) launch(grid, C::NT, [&] { k_rb_sweep_col<C, false, false>(v, p.x, dst, nullptr, p.B, first, g, nullptr); });
        if (form == 1) launch(grid, C::NT, [&] { k_rb_sweep_col<C, true, false>(v, nullptr, dst, nullptr, p.B, first, g, nullptr); });
        if (form == 2) launch(grid, C::NT, [&] { k_rb_sweep_col<C, false, true>(v, p.x, dst, p.xc, p.B, first, g, nullptr); });
        const LV<T> r = p.view(ref.data(), (T)1.1);
        pass(r, p.B, first, true);
        pass(r, p.B, 1 - first, true);
        bad += same(dst, ref.data(), N, "sweep");
    }
    return bad;
}

template <typename T>
static int run_coarse(const int* n, const int* per, int nl, unsigned threads) {
    LVSet<T> S{};
    std::vector<Problem<T>*> p;
    size_t cells = 0;
    for (int L = 0; L < nl; L++) {
        p.push_back(new Problem<T>(n[0] >> L, n[1] >> L, n[2] >> L, per));
        S.l[L] = p[L]->view(p[L]->x, (T)1.1);
        cells += 5 * S.l[L].N;
    }
    const LV<T>& last = S.l[nl - 1];
    auto* const kernel = seam_axes(p[0]->B, last.n0, last.n1, last.n2) ? &k_coarse_cycle_smem<T, true> : &k_coarse_cycle_smem<T, false>;
    launch(dim3(1), threads, [&] { kernel(S, 0, nl, p[0]->B, 2, 2, 0, 1, 0, (int)cells); });
    if (nl > 1) return 0;   // (races only)
    std::vector<T> ref(S.l[0].N, (T)0);
    const LV<T> r = p[0]->view(ref.data(), (T)1.1);
    const bool seam = seam_axes(p[0]->B, r.n0, r.n1, r.n2) > 0;
    for (int s = 0; s < 4 * kCoarseSweeps; s++) {
        const int color = s < 2 * kCoarseSweeps ? s & 1 : 1 - (s & 1);
        if (seam) pass_seam(r, p[0]->B, color);
        else pass(r, p[0]->B, color, false);
    }
    return same(p[0]->x, ref.data(), r.N, "coarse cycle");
}

// colour passes over a whole level by launches, four of them
template <typename T>
static int run_passes(const int* n, const int* per) {
    Problem<T> p(n[0], n[1], n[2], per);
    const LV<T> v = p.view(p.x, (T)1.1);
    std::vector<T> ref(p.x, p.x + v.N);
    const LV<T> r = p.view(ref.data(), (T)1.1);
    T* at[2] = {p.x, p.x};
    for (int q = 0; q < 4; q++) {
        const int color = q & 1;
        T* const out = at[color] == p.x ? p.x2 : p.x;
        launch(dim3(1, n[1], n[2]), 32, [&] { k_fast_smooth_seam<T>(v, at[color], at[1 - color], out, p.B, color); });
        at[color] = out;
        pass_seam(r, p.B, color);
    }
    return same(p.x, ref.data(), v.N, "colour passes");
}

int main(int argc, char** argv) {
    auto arg = [&](int q) { return q < argc ? atoi(argv[q]) : 0; };
    const std::string kind = argv[1], type = argv[2];
    const int n[3] = {arg(4), arg(5), arg(6)}, per[3] = {arg(7), arg(8), arg(9)};
    if (kind == "coarse") return type == "float" ? run_coarse<float>(n, per, arg(3), arg(10)) : run_coarse<double>(n, per, arg(3), arg(10));
    if (kind == "passes") return type == "float" ? run_passes<float>(n, per) : run_passes<double>(n, per);
#define COL(t, id, ...) \
    if (kind == "col" && type == #t && arg(3) == id) return run_col<SwColCfg<t, __VA_ARGS__>>(n, per, arg(10), arg(11));
    COLUMN_CONFIGURATIONS
    return 2;
}
