// mg_sweep_col.cuh -- fused red-black Gauss-Seidel sweep of the B200 multigrid
// with the columns of a tile held in registers (included by mg_fast.cu after
// mg_sweep.cuh).
//
// One full sweep (colour F = `first`, then the other colour S) in one pass
// over memory.  The iterate is read from `xin` (ZERO: it is zero) and written to
// `xout`, never in place, so blocks never see each other's new values and the
// sweep computes the two colour passes of k_fast_smooth (in FP64 exactly; in
// FP32 with the update arithmetic of SwUpd<float>).  With CORR, the coarse-grid
// correction `xc` (injection) is added to the iterate as it arrives; with
// bx_part, the sweep also sums b x over the cells it stores (in FP64), one
// partial per block: on the last sweep of a V-cycle on the finest level that is
// r.z, the dot product the CG needs next.  A thread
// owns VEC = 16 / sizeof(T) neighbouring cells of a row (one 16-byte chunk)
// and marches up a chunk of planes.  Step k updates F at plane k and then S at
// plane k-1, which is final and stored:
//   - the iterate of the thread's own cells at planes k-2..k+1 and the
//     coefficients of its S cells at plane k-1 stay in registers; the rows
//     around come from shared memory, the cells left and right as one scalar
//     each;
//   - F of plane k reads S cells from the staged iterate, which is not written
//     again once a step has begun to read it; the new F values go to a ring of
//     their own, U = VEC / 2 of them a chunk, where S of plane k reads them a
//     step later.  No step reads what it writes, so one barrier per plane orders
//     everything (a ring of its own also holds no S cells, which S has in
//     registers: half the bytes per row that S reads);
//   - the cells a thread updates are the same half of its chunk in both
//     colours, by the parity of its row and plane.  Rows are dealt to warps
//     even rows first, so a warp takes one parity and runs its steps in pairs
//     with the parity known at compile time.
// F runs on the tile and one row below and above it (and, where a tile is
// narrower than the grid, one chunk left and right).  Planes of the iterate
// and the coefficients are staged by 16-byte cp.async, D planes ahead.
// Rows and columns outside a wall are zero in every slot from the start and are
// never written; planes outside a wall are not staged and not updated.
//
// What bounds it: on the finest level, instruction issue and HBM together.
// Scalar shared-memory operands and two barriers per pair of planes held the
// earlier form to 138 us per FP32 256^3 sweep (2.9 TB/s of its 24 B/cell); this
// one takes 84 us (4.8 TB/s), 65 from a zero iterate, 104 with the correction, at
// 263 instructions per warp and step of 128 cells (436 with run-time row pitches,
// register copies and a branch on the parity in every step; 87 and 110 us with
// the new F values stored into the staged planes).  On the lower
// levels, resident in L2, the depth of the march: (planes per block + 2) steps.
// Requirements (checked by the host): n0 a multiple of 4, n1 and n2 even, fewer
// than 2^32 cells.
#pragma once

// 16 bytes, asynchronously
__device__ inline void cp_async16_full(uint32_t saddr, const void* g) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(saddr), "l"(g) : "memory");
}

// a configuration: element type, chunks a staged row has room for, tile rows,
// planes staged ahead, blocks per SM the registers are budgeted for
template <typename T_, int PITCH_, int TY_, int D_, int MINB_>
struct SwColCfg {
    using T = T_;
    static constexpr int PITCH = PITCH_, TY = TY_, D = D_, MINB = MINB_;
    static constexpr int VEC = 16 / (int)sizeof(T);
    static constexpr int EV = (TY + 3) / 2, OD = (TY + 2) / 2;               // even and odd rows of 0..TY+1
    static constexpr int NE = (EV * PITCH + 31) / 32 * 32, NT = NE + (OD * PITCH + 31) / 32 * 32;
    static constexpr int XS = D + 2, CS = D + 1;                             // planes in the rings
    static constexpr uint32_t ROW = PITCH * 16, XSLOT = ROW * (TY + 4);
    static constexpr uint32_t NROW = PITCH * 8, NSLOT = NROW * (TY + 4);     // new F cells: rows y0-2..y0+TY+1, of which S uses y0-1..y0+TY
    static constexpr uint32_t O_CY = ROW * (TY + 2), O_CZ = O_CY + ROW * (TY + 3), O_B = O_CZ + ROW * (TY + 2);
    static constexpr uint32_t CSLOT = O_B + ROW * (TY + 2);
    static constexpr size_t SMEM = (size_t)XSLOT * XS + (size_t)CSLOT * CS + 2 * (size_t)NSLOT;
    static_assert(SMEM <= 227 * 1024 && NT <= 1024, "one block fits an SM");
    static_assert(EV >= 3, "the first three rows of threads stage the rows only read");
};

template <typename T, int VEC>
struct alignas(16) SwChunk {
    T v[VEC];
};

// the tiles across a row of n0 cells: as wide as the grid where its chunks fit
// a staged row, else equal tiles with one ring chunk on either side
template <class C>
inline void sweep_col_tiles(int n0, SwColGeo& g) {
    const int V = C::VEC;
    if (n0 / V <= C::PITCH) {
        g.W = n0;
        g.H = 0;
    } else {
        const int t = (n0 + (C::PITCH - 2) * V - 1) / ((C::PITCH - 2) * V);
        g.W = ((n0 + t - 1) / t + V - 1) / V * V;
        g.H = V;
    }
    g.lanes = (g.W + 2 * g.H) / V;
}

template <class C, bool ZERO, bool CORR>
__global__ void __launch_bounds__(C::NT, C::MINB)
    k_rb_sweep_col(const LV<typename C::T> v, const typename C::T* __restrict__ xin, typename C::T* __restrict__ xout,
                   const typename C::T* __restrict__ xc, const Bnd B, int first, const SwColGeo g,
                   double* __restrict__ bx_part) {
    using T = typename C::T;
    constexpr int VEC = C::VEC, U = VEC / 2, TY = C::TY, D = C::D, XS = C::XS, CS = C::CS;
    constexpr uint32_t ROW = C::ROW;
    using Chunk = SwChunk<T, VEC>;
    extern __shared__ __align__(16) unsigned char sw_raw[];
    const int n0 = v.n0, n1 = v.n1, n2 = v.n2;
    const uint32_t plane = (uint32_t)n0 * (uint32_t)n1;
    const int x0 = blockIdx.x * g.W, y0 = blockIdx.y * TY;
    const int z0 = blockIdx.z * g.zc, z1 = min(z0 + g.zc, n2);
    const int tid = threadIdx.x;

    // the thread's row r (0..TY+1 for j = y0-1..y0+TY) and chunk; threads
    // beyond the rows and lanes in use shadow row 0's first chunk and store nothing
    const bool odd = tid >= C::NE;
    const int tq = odd ? tid - C::NE : tid, tr = tq / C::PITCH, tl = tq - tr * C::PITCH;
    const bool on = 2 * tr + (odd ? 1 : 0) < TY + 2 && tl < g.lanes;
    const int q = on ? tr : 0, lane = on ? tl : 0, r = on ? 2 * tr + (odd ? 1 : 0) : 0;
    const int gi0 = x0 - g.H + VEC * lane, j = y0 - 1 + r;
    const int wi = sw_wrap(gi0, n0, B.per[0]), wj = sw_wrap(j, n1, B.per[1]);
    const bool ok = on && wi >= 0 && wj >= 0;   // false outside a wall: zeros are kept there, nothing is updated
    // 32-bit cell indices: a level has fewer than 2^32 cells (checked by the host)
    const uint32_t goff = ok ? (uint32_t)wi + (uint32_t)n0 * (uint32_t)wj : 0u;
    // and a chunk of the rows only read: x at y0-2 (q 0) and y0+TY+1 (q 1), cy at y0-2 (q 2)
    const bool eon = on && !odd && q < 3;
    const int ej = sw_wrap(q == 1 ? y0 + TY + 1 : y0 - 2, n1, B.per[1]);
    const bool eok = eon && wi >= 0 && ej >= 0;
    const uint32_t eoff = eok ? (uint32_t)wi + (uint32_t)n0 * (uint32_t)ej : 0u;
    const bool ex = eok && q < 2, ecy = eok && q == 2;

    const uint32_t o = ROW * r + 16u * lane;                          // the thread's chunk in cx, cz, b and, a row up, x, cy
    const uint32_t oe = ROW * (q == 1 ? TY + 3 : 0) + 16u * lane;     // its chunk of the rows only read
    const uint32_t s_x = (uint32_t)__cvta_generic_to_shared(sw_raw);
    constexpr uint32_t C0 = XS * C::XSLOT;                            // the coefficient ring starts here
    constexpr uint32_t N0 = C0 + CS * C::CSLOT;                       // and the two planes of new F cells here
    constexpr uint32_t NB = U * sizeof(T);
    const uint32_t fo = C::NROW * (r + 1) + NB * lane;               // the thread's F cells in a plane of them
    // the cells left and right of the chunk: across a seam in a whole row, absent (zero) at a wall
    const bool whole = g.H == 0;
    const bool wz = whole && lane == 0 && !B.per[0], ez = whole && lane == g.lanes - 1 && !B.per[0];
    const uint32_t ow = o + (lane > 0 ? -(int)sizeof(T) : (whole ? g.lanes * 16 - (int)sizeof(T) : 0));
    const uint32_t oea = o + (lane < g.lanes - 1 ? 16 : (whole ? 16 - g.lanes * 16 : 16 - (int)sizeof(T)));

    // the F cell left (the last of a chunk's) and right (the first) of the chunk
    const uint32_t fow = fo + (lane > 0 ? -(int)sizeof(T) : (whole ? g.lanes * (int)NB - (int)sizeof(T) : 0));
    const uint32_t foe = fo + (lane < g.lanes - 1 ? (int)NB : (whole ? (int)NB - g.lanes * (int)NB : 0));

    struct alignas(U * sizeof(T)) Half {
        T v[U];
    };
    auto ldh = [](uint32_t a) { return *reinterpret_cast<const Half*>(sw_raw + a); };
    auto ldc = [](uint32_t a) { return *reinterpret_cast<const Chunk*>(sw_raw + a); };   // a: offset from sw_raw
    auto lds = [](uint32_t a) { return *reinterpret_cast<const T*>(sw_raw + a); };
    const bool pz = B.per[2];
    auto inside = [&](int k) { return pz || (k >= 0 && k < n2); };   // plane k exists (or its periodic image)
    auto first_cell = [&](int k) {                                   // of plane k or its image
        return plane * (uint32_t)(k < 0 ? k + n2 : (k >= n2 ? k - n2 : k));
    };
    auto stage_x = [&](int k, uint32_t d) {   // iterate plane k into the slot at byte d of the ring
        if (ZERO || !inside(k)) return;
        const uint32_t p = first_cell(k);
        if (ok) cp_async16_full(s_x + d + o + ROW, xin + (p + goff));
        if (ex) cp_async16_full(s_x + d + oe, xin + (p + eoff));
    };
    auto stage_c = [&](int k, uint32_t d) {   // the coefficients of plane k
        if (!inside(k)) return;
        const uint32_t p = first_cell(k), m = p + goff, s = s_x + d + o;
        if (ok) {
            cp_async16_full(s, v.cx + m);
            cp_async16_full(s + C::O_CY + ROW, v.cy + m);
            cp_async16_full(s + C::O_CZ, v.cz + m);
            cp_async16_full(s + C::O_B, v.b + m);
        }
        if (ecy) cp_async16_full(s_x + d + C::O_CY + 16u * lane, v.cy + (p + eoff));
    };
    auto st0 = [](uint32_t a) { *reinterpret_cast<Chunk*>(sw_raw + a) = Chunk{}; };
    if (on && !ok) {   // outside a wall in x or y
        for (int d = 0; d < XS; d++) st0(d * C::XSLOT + o + ROW);
        for (int d = 0; d < CS; d++) {
            const uint32_t s = C0 + d * C::CSLOT + o;
            st0(s);
            st0(s + C::O_CY + ROW);
            st0(s + C::O_CZ);
            st0(s + C::O_B);
        }
        for (int d = 0; d < 2; d++) *reinterpret_cast<Half*>(sw_raw + N0 + d * C::NSLOT + fo) = Half{};
    }
    if (eon && !eok) {
        for (int d = 0; d < XS; d++)
            if (q < 2) st0(d * C::XSLOT + oe);
        for (int d = 0; d < CS; d++)
            if (q == 2) st0(C0 + d * C::CSLOT + C::O_CY + 16u * lane);
    }

    // the coarse correction (injection): a thread adds it to the chunks it
    // staged, fetched a plane ahead.  Neighbours read iterate plane k+1 from
    // step k+1 on, so step k adds it after its barrier; plane z0-1 gets it
    // before the first one.
    const uint32_t cn0 = (uint32_t)n0 >> 1, cplane = cn0 * ((uint32_t)n1 >> 1);
    const uint32_t coff = ok ? ((uint32_t)wi >> 1) + cn0 * ((uint32_t)wj >> 1) : 0u;
    const uint32_t ecoff = ex ? ((uint32_t)wi >> 1) + cn0 * ((uint32_t)ej >> 1) : 0u;
    Half cown{}, cext{};
    auto fetch = [&](int k) {
        const int gk = k < 0 ? k + n2 : (k >= n2 ? k - n2 : k);
        const uint32_t c = inside(k) ? cplane * ((uint32_t)gk >> 1) : 0u;   // (the value is not added outside a wall)
        if (ok) cown = *reinterpret_cast<const Half*>(xc + (c + coff));
        if (ex) cext = *reinterpret_cast<const Half*>(xc + (c + ecoff));
    };
    auto add_ext = [&](uint32_t d) {
        if (ex) {
            Chunk t = ldc(d + oe);
#pragma unroll
            for (int e = 0; e < VEC; e++) t.v[e] += cext.v[e >> 1];
            *reinterpret_cast<Chunk*>(sw_raw + d + oe) = t;
        }
    };

    // prologue: iterate plane z0-1, then D groups (group k: iterate plane k+1
    // and the coefficients of plane k).  Slot of iterate plane k: (k - z0 + 1)
    // mod XS, of coefficient plane k: (k - z0 + 1) mod CS.
    stage_x(z0 - 1, 0);
#pragma unroll
    for (int d = 0; d < D; d++) {
        if (z0 - 1 + d <= z1) {
            stage_x(z0 + d, (d + 1) * C::XSLOT);
            stage_c(z0 - 1 + d, C0 + d * C::CSLOT);
        }
        cp_async_commit();
    }
    Chunk xa{}, xb{}, x1{}, czm{};   // iterate at planes k-2, k-1, k; cz at k-1
    T a1[U], a2[U], a3[U], a4[U], a5[U], a6[U];   // coefficients of the S cells of plane k-1
    Chunk bb{};                                   // b at plane k-1
#pragma unroll
    for (int u = 0; u < U; u++) a1[u] = a2[u] = a3[u] = a4[u] = a5[u] = a6[u] = (T)0;
    if (ok && inside(z0 - 2)) {
        const uint32_t p = first_cell(z0 - 2) + goff;
        czm = *reinterpret_cast<const Chunk*>(v.cz + p);
        if (!ZERO) xb = *reinterpret_cast<const Chunk*>(xin + p);
        if (CORR) {
            fetch(z0 - 2);
#pragma unroll
            for (int e = 0; e < VEC; e++) xb.v[e] += cown.v[e >> 1];
        }
    }
    const bool out = ok && r >= 1 && r <= TY && j < n1 && gi0 >= x0 && gi0 < x0 + g.W && gi0 < n0;
    uint32_t xo = (uint32_t)gi0 + (uint32_t)n0 * (uint32_t)j + plane * (uint32_t)(z0 - 3);   // the chunk at plane k-1 once advanced (mod 2^32)
    double bx = 0.0;
    const T w = v.omega;
    // byte offsets of the slots of iterate and coefficient planes k-1, k, and of
    // the new F cells of planes k-1, k.  The planes staged at step k, k+1+D and
    // k+D, take the slots of planes k-1, and the F cells of plane k those of
    // plane k-2: last read in step k-1.
    uint32_t xm = (XS - 1) * C::XSLOT, xk = 0;
    uint32_t cm = C0 + (CS - 1) * C::CSLOT, ck = C0;
    uint32_t nm = N0 + C::NSLOT, nk = N0;

    auto step = [&](auto PC, int k) {   // PC: parity of the updated cells of the chunk
        constexpr int P = decltype(PC)::value;
        constexpr int L = VEC - 1;
        const uint32_t xp = xk == (XS - 1) * C::XSLOT ? 0 : xk + C::XSLOT;
        cp_async_wait_newest<D - 1>();
        if (CORR && k == z0 - 1) {
            if (ok && inside(k)) {
                Chunk t = ldc(xk + o + ROW);
#pragma unroll
                for (int e = 0; e < VEC; e++) t.v[e] += cown.v[e >> 1];
                *reinterpret_cast<Chunk*>(sw_raw + xk + o + ROW) = t;
            }
            if (inside(k)) add_ext(xk);
            fetch(z0);
        }
        __syncthreads();
        if (k + D <= z1) {
            stage_x(k + 1 + D, xm);
            stage_c(k + D, cm);
        }
        cp_async_commit();
        xo += plane;
        const uint32_t fx = xk + o, fc = ck + o;
        const bool in = inside(k);
        // F at plane k
        Chunk x2{}, xs{}, xn{};
        T xl = (T)0;
        if (!ZERO) {
            if (k == z0 - 1 && in) x1 = ldc(fx + ROW);
            if (inside(k + 1)) {
                if (!CORR) x2 = ldc(xp + o + ROW);
                if (CORR) {
                    if (ok) {   // (another thread's chunk is still being added to)
                        x2 = ldc(xp + o + ROW);
#pragma unroll
                        for (int e = 0; e < VEC; e++) x2.v[e] += cown.v[e >> 1];
                        *reinterpret_cast<Chunk*>(sw_raw + xp + o + ROW) = x2;
                    }
                    add_ext(xp);
                }
            }
            if (CORR) fetch(k + 2);
            xs = ldc(fx);
            xn = ldc(fx + 2 * ROW);
            xl = lds(xk + ROW + (P == 0 ? ow : oea));
            if (P == 0 ? wz : ez) xl = (T)0;
        }
        const Chunk cx = ldc(fc), cys = ldc(fc + C::O_CY), cy = ldc(fc + C::O_CY + ROW), b = ldc(fc + C::O_B);
        Chunk cz = ldc(fc + C::O_CZ);
        T cw = lds(ck + ow);
        if (wz) cw = (T)0;
        const bool fok = ok && in;
        Chunk nx = x1;
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int e = P + 2 * u;
            T t;
            if (SwUpd<T>::apply(e > 0 ? cx.v[e > 0 ? e - 1 : 0] : cw, cx.v[e], cys.v[e], cy.v[e], czm.v[e], cz.v[e],
                                e > 0 ? x1.v[e > 0 ? e - 1 : 0] : xl, e < L ? x1.v[e < L ? e + 1 : 0] : xl, xs.v[e],
                                xn.v[e], xb.v[e], x2.v[e], b.v[e], x1.v[e], w, t) && fok)
                nx.v[e] = t;
        }
        if (ok) {   // (zero where plane k is outside a wall)
            Half nf;
#pragma unroll
            for (int u = 0; u < U; u++) nf.v[u] = nx.v[P + 2 * u];
            *reinterpret_cast<Half*>(sw_raw + nk + fo) = nf;
        }
        // S at plane k-1, final: stored
        const Half ps = ldh(nm + fo - C::NROW), pn = ldh(nm + fo + C::NROW);
        T pl = lds(nm + (P == 0 ? fow : foe));
        if (P == 0 ? wz : ez) pl = (T)0;
        Chunk ns = xb;
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int e = P + 2 * u;
            T t;
            if (SwUpd<T>::apply(a1[u], a2[u], a3[u], a4[u], a5[u], a6[u], e > 0 ? xb.v[e > 0 ? e - 1 : 0] : pl,
                                e < L ? xb.v[e < L ? e + 1 : 0] : pl, ps.v[u], pn.v[u], xa.v[e], nx.v[e], bb.v[e],
                                xb.v[e], w, t))
                ns.v[e] = t;
        }
        if (out && k > z0) {
            *reinterpret_cast<Chunk*>(xout + xo) = ns;
            if (bx_part) {
#pragma unroll
                for (int e = 0; e < VEC; e++) bx += (double)bb.v[e] * (double)ns.v[e];
            }
        }
        // the other cells of plane k are the S cells of the next step
        if (!in) cz = Chunk{};   // (not staged)
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int e = 1 - P + 2 * u;
            a1[u] = e > 0 ? cx.v[e > 0 ? e - 1 : 0] : cw;
            a2[u] = cx.v[e];
            a3[u] = cys.v[e];
            a4[u] = cy.v[e];
            a5[u] = czm.v[e];
            a6[u] = cz.v[e];
        }
        bb = b;
        czm = cz;
        xa = xb;
        xb = nx;
        x1 = x2;
        xm = xk;
        xk = xp;
        const uint32_t nt = nm;
        nm = nk;
        nk = nt;
        cm = ck;
        ck = ck == C0 + (CS - 1) * C::CSLOT ? C0 : ck + C::CSLOT;
    };

    if (CORR) fetch(z0 - 1);
    // F cells have i + j + k + first even and a chunk starts at an even i; the
    // number of steps, z1 - z0 + 2, is even.  The warps of either parity meet at
    // the same barriers.
    if (((y0 - 1 + (odd ? 1 : 0) + z0 - 1 + first) & 1) == 0)
        for (int k = z0 - 1; k <= z1; k += 2) {
            step(std::integral_constant<int, 0>{}, k);
            step(std::integral_constant<int, 1>{}, k + 1);
        }
    else
        for (int k = z0 - 1; k <= z1; k += 2) {
            step(std::integral_constant<int, 1>{}, k);
            step(std::integral_constant<int, 0>{}, k + 1);
        }
    cp_async_wait_all_groups();
    if (bx_part) {   // b.x of the block: one partial per block, in launch order
        __shared__ double bsh[32];
        bx = block_sum<C::NT>(bx, bsh);
        if (tid == 0) bx_part[blockIdx.x + gridDim.x * (blockIdx.y + gridDim.y * blockIdx.z)] = bx;
    }
}
