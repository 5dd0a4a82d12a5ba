// Whole time steps of the quiet-Sun forms with each z-pencil on chip: FP64
// (options 4, 17 and the velocity form 2) and FP32 option 2; FP32 options 4
// and 17 have fused.cu.
//
// Layout.  A pencil (one horizontal mode of one source) is cut into chunks of
// CH levels, one per thread: TP threads (whole warps, or in FP64 a
// half or a quarter of one: two or four pencils a warp), padded to TP CH levels.  `a`
// sits in shared memory as [field][pencil][chunk], scr in registers, the PML
// planes in shared memory; a CTA holds P pencils.  A pencil's step needs
// nothing of another pencil, so a launch takes up to FUSED_STEPS steps
// (pencil_steps in FP64) before the state goes back to HBM.
//
// What bounds it: FP64 issue.  GB300 issues two FP64 lanes a clock and SM, so
// the kernel is written for few FP64 instructions per level and stage (63 in
// option 4), and everything else (table reads through L1, shared memory,
// shuffles, HBM once in 16 steps) hides behind them:
//   * horizontal components.  The right-hand side sees (xi_x, xi_y) and (v_x,
//     v_y) only through their components along k = (kx, ky); the ones across
//     follow T' = U, U' = -gamma U, whose five stages are one factor per mode.
//     A step forms the along components once, its stages work on four fields
//     instead of six, and the update turns their right-hand sides back;
//   * the compact scheme A f' = C1 d1 + C2 d2 with d1(j) = f(j+1) - f(j-1),
//     d2(j) = f(j+2) - f(j-2) = d1(j+1) + d1(j-1) is solved for y = f' -
//     (C2/alpha) d1, since A y = (C1 - C2/alpha) d1 on every interior row:
//     one difference per level and one neighbour on each side;
//   * stretch, 1/rho0 and the coefficients are folded into the elimination
//     rows (each solve returns the scaled derivative), the boundary closures
//     into five coefficients per row, the same instructions for both ends;
//   * a warp's PML planes are spread over its lanes, one plane per lane.
//
// The solves (dbyd2.f90:198-201, mtridag.f90:94-111) are first-order linear
// recurrences: each thread eliminates its chunk with a zero carry, the chunk
// maps u -> B + M u compose by a scan over the threads below (from above for
// the back substitution), and every level adds its response K or G to the
// carry.  The products M depend on z only and come from a host table.  A scan
// over 16 chunks within the warp (four shuffle steps) and one value of the
// neighbouring warp hold every term above 2^-60 of a chunk value, beneath the
// rounding of FP64; the host checks that bound for the boundary codes in use
// (else the per-stage kernels run).
//
// Shape (pencil_shape): the levels per thread and threads per pencil of the least
// issue cost, on grids with few modes those of the shortest chain; it depends on
// the grid only, so a source's arithmetic does not depend on the batch around it.
// Chunks are stored CHP = CH or CH+1 (odd) values apart, which keeps the 16-byte
// accesses of a warp free of bank conflicts.  Where the per-stage kernels are
// faster (few levels and many modes), capi.cu keeps to them.
//
// Measured per step, against one launch per stage with the pencils in HBM:
// 128x128x150, one source, FP64 2.40 -> 1.36 ms; 256x256x300 FP64 adjoint
// 15.6 -> 10.5 ms; 256x1x300 FP64 (option 17) 1.55 -> 0.072 ms; 128x64x101
// FP64 velocity form 3.07 -> 0.55 ms.
#include <algorithm>
#include <type_traits>

#include "internal.cuh"

namespace {

constexpr int GC = 2;      // ghost chunks of the tile on each side (the z filter reaches 5 levels)

// complex arithmetic with real multipliers; FP32 as paired instructions
__device__ __forceinline__ double2 cfma(double s, double2 v, double2 a) { return make_double2(fma(s, v.x, a.x), fma(s, v.y, a.y)); }
__device__ __forceinline__ float2 cfma(float s, float2 v, float2 a) { return pfma(bc2(s), v, a); }
__device__ __forceinline__ double2 cscale(double s, double2 v) { return make_double2(s * v.x, s * v.y); }
__device__ __forceinline__ float2 cscale(float s, float2 v) { return pmul(bc2(s), v); }
// a + i k v
template <typename T, typename CT>
__device__ __forceinline__ CT ifma(T k, CT v, CT a) {
    CT r;
    r.x = fma(-k, v.y, a.x);
    r.y = fma(k, v.x, a.y);
    return r;
}

// the value d lanes below / above, of the same pencil (seg lanes of the warp hold one)
template <typename CT> __device__ __forceinline__ CT shfl_up_c(CT v, int d, int seg) {
    CT r;
    r.x = __shfl_up_sync(0xffffffffu, v.x, d, seg);
    r.y = __shfl_up_sync(0xffffffffu, v.y, d, seg);
    return r;
}
template <typename CT> __device__ __forceinline__ CT shfl_down_c(CT v, int d, int seg) {
    CT r;
    r.x = __shfl_down_sync(0xffffffffu, v.x, d, seg);
    r.y = __shfl_down_sync(0xffffffffu, v.y, d, seg);
    return r;
}

// Barrier over the TP threads of one pencil (a named barrier; one warp or a part of one needs none).
__device__ __forceinline__ void pencil_sync(int pi, int tp) {
    if (tp <= 32) __syncwarp();
    else asm volatile("bar.sync %0, %1;" ::"r"(pi + 1), "r"(tp) : "memory");
}

struct PencilLayout {      // offsets in complex values, identical on host and device
    int tile, xf, xb, cl, pd, ptile, spt, cells, total, LZ, LX;
};
__host__ __device__ inline PencilLayout pencil_layout(int P, int TP, int CH, int nzpml, int option) {
    PencilLayout L;
    L.LZ = (TP + 2 * GC) * (CH | 1);
    L.LX = TP + 2;
    int o = 0;
    L.tile = o;  o += (option == 4 ? 8 : option == 2 ? 7 : 6) * P * L.LZ;   // the state, and its components along k
    L.xf = o;    o += P * L.LX;          // first and last value of every chunk of the exchanged field
    L.xb = o;    o += P * L.LX;
    L.cl = o;    o += P * 10;            // its five levels at each end
    L.pd = o;    o += P * nzpml;         // exchange of the PML planes
    L.ptile = o; o += 2 * nzpml * P;     // [pencil][2][plane]
    L.spt = o;   o += 2 * nzpml * P;
    L.cells = o; o += 2 * P * ((TP + 31) / 32);         // forward and backward carries between warps
    L.total = o;
    return L;
}

// One solve of a pencil: the scaled d/dz of the exchanged field (own[q] the
// thread's levels, left and right the neighbours' next ones, cl the five
// levels at each end of the pencil, from the end inwards) on the levels
// j0..j0+CH-1.  top: the caller-set value of bc 3.  zt: the thread's column
// of the elimination rows (row stride NZP, level q at q TP), ct: of the carry
// rows (row stride TP), ce: the closure coefficients of this solve.
template <int CH, bool PART, typename T, typename CT>
__device__ __forceinline__ void pencil_solve(const CT (&own)[CH], CT left, CT right, const CT* cl,
                                             const T* __restrict__ zt, const T* __restrict__ ct,
                                             const T* __restrict__ ce, bool has_top, CT top, int NZP, int TP, int nz,
                                             int j0, bool lo, bool hi, int t, CT* cf, CT* cb, int pi, CT (&out)[CH]) {
    auto Z = [&](int row, int q) -> T { return __ldg(&zt[row * NZP + q * TP]); };
    auto C = [&](int row) -> T { return __ldg(&ct[row * TP]); };
    const int lane = t & 31, w = t >> 5, seg = PART ? TP : 32;
    CT d1[CH], u[CH];
    #pragma unroll
    for (int q = 0; q < CH; ++q) {
        d1[q] = (q + 1 < CH ? own[q + 1 < CH ? q + 1 : 0] : right) - (q > 0 ? own[q > 0 ? q - 1 : 0] : left);
        u[q] = cscale(Z(PS_D, q), d1[q]);
    }
    if (lo || hi) {     // rows 0, 1 or nz-2, nz-1 (dbyd2.f90:104-173)
        const CT* b = cl + (lo ? 0 : 5);
        const T* e = ce + (lo ? 0 : PE_COUNT);
        CT near = cscale(__ldg(&e[0]), b[0]), end = cscale(__ldg(&e[5]), b[0]);
        #pragma unroll
        for (int i = 1; i < 5; ++i) {
            near = cfma(__ldg(&e[i]), b[i], near);
            end = cfma(__ldg(&e[5 + i]), b[i], end);
        }
        if (has_top) end = cfma(__ldg(&e[PE_TOP]), top, end);
        const int jn = lo ? 1 : nz - 2, je = lo ? 0 : nz - 1;
        #pragma unroll
        for (int q = 0; q < CH; ++q) {
            if (j0 + q == jn) u[q] = near;
            if (j0 + q == je) u[q] = end;
        }
    }
    // elimination with zero carry-in
    CT run = u[0];
    #pragma unroll
    for (int q = 1; q < CH; ++q) {
        run = cfma(Z(PS_M, q), run, u[q]);
        u[q] = run;
    }
    // carry from the chunks below: exclusive scan over 16 chunks of the warp,
    // then the last value of the warp below
    CT e = shfl_up_c(run, 1, seg);
    if (lane == 0) e = czero<CT>();
    #pragma unroll
    for (int k = 0; k < 4; ++k) e = cfma(C(PC_F + k), shfl_up_c(e, 1 << k, seg), e);   // zero coefficient where it leaves the pencil's lanes
    if (TP > 32 && lane == 31) cf[w] = cfma(C(PC_FL), e, run);
    // back substitution with zero carries
    CT x = u[CH - 1];
    out[CH - 1] = x;
    #pragma unroll
    for (int q = CH - 2; q >= 0; --q) {
        x = cfma(Z(PS_G, q), x, u[q]);
        out[q] = x;
    }
    pencil_sync(pi, TP);         // the exchanged values have been read (the caller rewrites them), the carries are in
    if (w > 0) e = cfma(C(PC_FW), cf[w - 1], e);
    // y(j) = x0(j) + K(j) e + G(j) f, f the carry from the chunks above
    x = cfma(Z(PS_K, 0), e, x);
    CT f = shfl_down_c(x, 1, seg);
    if (lane == seg - 1) f = czero<CT>();
    #pragma unroll
    for (int k = 0; k < 4; ++k) f = cfma(C(PC_B + k), shfl_down_c(f, 1 << k, seg), f);
    if (TP > 32) {
        if (lane == 0) cb[w] = cfma(C(PC_BL), f, x);
        pencil_sync(pi, TP);
        if ((w + 1) * 32 < TP) f = cfma(C(PC_BW), cb[w + 1], f);
    }
    out[0] = cfma(Z(PS_A, 0), d1[0], cfma(Z(PS_GC, 0), f, x));
    #pragma unroll
    for (int q = 1; q < CH; ++q)
        out[q] = cfma(Z(PS_A, q), d1[q], cfma(Z(PS_GC, q), f, cfma(Z(PS_K, q), e, out[q])));
}

// FORM 4, 17 or 2 (the option codes).  Fields of the tile: 4: xi_x, xi_y, xi_z,
// v_x, v_y, v_z, then xi and v along k at the start of the step; 17: xi_x,
// (xi_y), xi_z, v_x, (v_y), v_z; 2: rho, v_x, v_y, v_z, p, (unused), then v
// along k.  The fields in brackets have no right-hand side: they are only
// filtered, and only where a CTA holds a non-zero value of them.
// PART: a pencil takes a part of a warp (seg lanes of it).
template <typename T, int FORM, int CH, bool PART>
__global__ void __launch_bounds__(256, sizeof(T) == 4 ? 2 : 1) pencil_step_kernel(const PencilArgs<T> A) {
    typedef typename CplxOf<T>::type CT;
    constexpr bool D3 = FORM != 17, VEL = FORM == 2;
    constexpr int CHP = CH | 1;
    // tile index of the fields that the stages evolve, in the order of sc
    constexpr int F0 = FORM == 4 ? 6 : 0, F1 = VEL ? 6 : 2, F2 = FORM == 4 ? 7 : 3, F3 = VEL ? 4 : 5;
    constexpr int FZ = VEL ? 2 : 1;                       // sc index of the field the first solve differentiates
    constexpr int FV = VEL ? 2 : 3;                       // sc index of v_z
    extern __shared__ __align__(16) unsigned char smraw[];
    const int W = A.W, P = A.pencils, TP = PART ? A.part : 32 * W, NZP = TP * CH;
    const int nz = A.nz, M = A.M, nzpml = A.nzpml, nb = A.npmlbot, nt = A.npmltop;
    const long long fs = A.fs;
    const PencilLayout Ly = pencil_layout(P, TP, CH, nzpml, FORM);
    const int LZ = Ly.LZ, FT = P * LZ;                    // field stride of the tile
    CT* sm = (CT*)smraw;
    CT* tile = sm + Ly.tile;
    const int pi = threadIdx.x / TP, t = threadIdx.x - pi * TP, j0 = t * CH;
    CT* xf = sm + Ly.xf + pi * Ly.LX + 1;                 // chunks 0..TP-1, a zero at TP
    CT* xb = sm + Ly.xb + pi * Ly.LX + 1;                 // a zero at -1
    CT* cl = sm + Ly.cl + pi * 10;
    CT* pd = sm + Ly.pd + pi * nzpml;
    CT* ptile = sm + Ly.ptile + pi * 2 * nzpml;
    CT* spt = sm + Ly.spt + pi * 2 * nzpml;
    CT* cf = sm + Ly.cells + 2 * pi * W;
    CT* cb = cf + W;
    const int ntile = (M + P - 1) / P;
    const int s = blockIdx.x / ntile;
    const int m0 = (blockIdx.x - s * ntile) * P;
    const int m = m0 + pi;
    const bool mvalid = m < M;
    CT* gA = A.a + (long long)s * 6 * fs;
    CT* gS = A.scr + (long long)s * 6 * fs;
    CT* gP = A.pml + (long long)s * 2 * A.ps;

    // ---- load: the tile transposed ([z][m] in HBM, [pencil][chunk] on chip) by
    // asynchronous copies; ghost and padding levels zero ----
    {
        const int q = threadIdx.x % P, z0 = threadIdx.x / P;
        const bool qv = m0 + q < M;
        CT* dst = tile + q * LZ;
        for (int r = z0; r < LZ; r += TP) {               // r: place in the line, level z (or a ghost, padding or gap)
            const int c = r / CHP - GC, k = r % CHP, z = c * CH + k;
            const bool real = c >= 0 && k < CH && z < nz;
            for (int f = 0; f < 6; ++f) {
                if (qv && real) {
                    const unsigned d = (unsigned)__cvta_generic_to_shared(dst + f * FT + r);
                    const size_t g = __cvta_generic_to_global(gA + f * fs + (long long)z * M + m0 + q);
                    if (sizeof(CT) == 16) asm volatile("cp.async.ca.shared.global [%0], [%1], 16;\n" ::"r"(d), "l"(g) : "memory");
                    else asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(d), "l"(g) : "memory");
                } else {
                    dst[f * FT + r] = czero<CT>();
                }
            }
        }
        for (int r = z0; r < 2 * nzpml; r += TP)
            sm[Ly.ptile + q * 2 * nzpml + r] = qv ? gP[(long long)r * M + m0 + q] : czero<CT>();
        if (t == 0) xb[-1] = xf[TP] = czero<CT>();
    }
    const int tl0 = *A.clk.time - A.clk.t0[s];            // this slot's clock at the first step
    const T kx = mvalid ? A.pt[PT_KX * (long long)M + m] : (T)0;
    const T ky = (mvalid && D3) ? A.pt[PT_KY * (long long)M + m] : (T)0;
    const T ngd = (mvalid && A.damp) ? -A.pt[PT_DAMP * (long long)M + m] : (T)0;
    // the unit vector along k, and the factor of the across components' stages:
    // r = 1, r <- 1 - gamma beta r
    const T kap = D3 ? sqrt(kx * kx + ky * ky) : kx;
    const T ex = (D3 && kap > (T)0) ? kx / kap : (T)1, ey = (D3 && kap > (T)0) ? ky / kap : (T)0;
    T r5 = (T)1;
    if (D3) {
        #pragma unroll
        for (int rk = 1; rk < 5; ++rk) r5 = fma(ngd * A.betas[rk], r5, (T)1);
    }
    asm volatile("cp.async.wait_all;\n" ::: "memory");
    __syncthreads();

    const bool lo = j0 == 0, hi = j0 <= nz - 1 && j0 + CH > nz - 2;
    // PML levels of this chunk: bit q of pmask, plane index pipv + q; and the
    // planes of the levels of this pencil's lanes in the warp: nbw bottom ones from plane pb, ntw top ones from plane pt
    unsigned pmask = 0;
    int pipv = 0;
    if (j0 < nb) {
        pmask = (1u << min(CH, nb - j0)) - 1u;
        pipv = j0;
    } else {
        const int l0 = max(j0, nz - nt), l1 = min(j0 + CH, nz);
        if (l1 > l0) {
            pmask = ((1u << (l1 - l0)) - 1u) << (l0 - j0);
            pipv = nb + (j0 - (nz - nt));
        }
    }
    const int lane = t & 31, seg = PART ? TP : 32, wl = (t - lane) * CH, wh = wl + seg * CH;
    const int nbw = max(0, min(nb, wh) - wl), tl_ = max(nz - nt, wl), ntw = max(0, min(nz, wh) - tl_);
    const int npw = nbw + ntw;
    auto plane = [&](int i) { return i < nbw ? wl + i : nb + tl_ - (nz - nt) + (i - nbw); };

    const T* zt = A.tab + t;                              // level q of row r: zt[r * NZP + q * TP]
    const T* c1 = A.tab + PZ_COUNT * NZP + t;
    const T* c2 = c1 + PC_COUNT * TP;
    const T* ce = A.tab + PZ_COUNT * NZP + 2 * PC_COUNT * TP;      // closures [2 solves][2 ends][PE_COUNT]
    const T* pz = ce + 4 * PE_COUNT;                               // a_z, a_z rho0, b_z of the PML planes
    auto Z = [&](int row, int q) -> T { return __ldg(&zt[row * NZP + q * TP]); };
    CT* tp = tile + pi * LZ + (GC + t) * CHP;             // this thread's levels: field f, level q at tp[f * FT + q]

    // whether the fields without a right-hand side hold anything
    bool extra = false;
    if (!D3 || VEL) {
        #pragma unroll
        for (int q = 0; q < CH; ++q) {
            const CT u = tp[(VEL ? 5 : 1) * FT + q], v = tp[(VEL ? 5 : 4) * FT + q];
            extra = extra || u.x != (T)0 || u.y != (T)0 || v.x != (T)0 || v.y != (T)0;
        }
        extra = __syncthreads_or(extra);
    }

    CT sc[4][CH];
    #pragma unroll
    for (int f = 0; f < 4; ++f)
        #pragma unroll
        for (int q = 0; q < CH; ++q) sc[f][q] = czero<CT>();
    CT F = czero<CT>();
    bool src_t = false;
    // whether level q of the chunk has a zero right-hand side (the first row; in 3-D the last one too)
    auto zero_row = [&](int q) { return j0 + q == 0 || (D3 && j0 + q == nz - 1); };
    // put a field's chunk up for the neighbours and the closures
    auto exchange = [&](const CT (&v)[CH]) {
        xf[t] = v[0];
        xb[t] = v[CH - 1];
        if (j0 < 5 || (j0 < nz && j0 + CH > nz - 5)) {
            #pragma unroll
            for (int q = 0; q < CH; ++q) {
                const int j = j0 + q;
                if (j < 5) cl[j] = v[q];
                if (j >= nz - 5 && j < nz) cl[5 + nz - 1 - j] = v[q];
            }
        }
        pencil_sync(pi, TP);
    };

    // one LDDRK stage; hs: the argument is a + beta*scr (stages 2-5) rather than a
    auto stage = [&](auto hs_c, const T beta) {
        constexpr bool hs = decltype(hs_c)::value;
        auto arg = [&](int f, int i, int q) -> CT {
            const CT v = tp[f * FT + q];
            return hs ? cfma(beta, sc[i][q], v) : v;
        };
        // psi of the PML planes of auxiliary k (psi_vz, psi_p): right-hand side a d + b psi, psi back in pd
        auto pml = [&](int k, const T* az) {
            __syncwarp();
            for (int i = lane; i < npw; i += seg) {
                const int ip = plane(i), o = k * nzpml + ip;
                CT psi = ptile[o];
                if (hs) psi = cfma(beta, spt[o], psi);
                spt[o] = cfma(__ldg(&az[ip]), pd[ip], cscale(__ldg(&pz[2 * nzpml + ip]), psi));
                pd[ip] = psi;
            }
            __syncwarp();
        };
        CT own[CH], d[CH];
        #pragma unroll
        for (int q = 0; q < CH; ++q) own[q] = arg(VEL ? F2 : F1, FZ, q);
        CT top = czero<CT>();
        if (FORM == 17 && hi) {      // caller-set top value of bc 3 (physics2d.f90:960)
            #pragma unroll
            for (int q = 0; q < CH; ++q)
                if (j0 + q == nz - 1) top = cscale(-A.unstr_top, ifma(kap, arg(F0, 0, q), czero<CT>()));
        }
        exchange(own);
        pencil_solve<CH, PART, T, CT>(own, xb[t - 1], xf[t + 1], cl, zt + PZ_S1 * NZP, c1, ce, FORM == 17, top, NZP, TP, nz,
                                j0, lo, hi, t, cf, cb, pi, d);
        if (npw) {                   // psi_vz
            #pragma unroll
            for (int q = 0; q < CH; ++q)
                if (pmask & (1u << q)) pd[pipv + q] = d[q];
            pml(0, pz);
            #pragma unroll
            for (int q = 0; q < CH; ++q)
                if (pmask & (1u << q)) d[q] = d[q] + pd[pipv + q];
        }
        #pragma unroll
        for (int q = 0; q < CH; ++q) {
            if constexpr (VEL) {
                const CT vl = arg(F1, 1, q), rho = arg(F0, 0, q), p = arg(F3, 3, q), vz = own[q];
                const CT div = ifma(kap, vl, d[q]);
                const bool zr = zero_row(q);
                sc[0][q] = cfma(-Z(PZ_GR, q), vz, cscale(-Z(PZ_R0, q), div));
                sc[3][q] = cfma(-Z(PZ_GP, q), vz, cscale(-Z(PZ_C2R, q), div));
                const T ri = zr ? (T)0 : Z(PZ_RI, q), gr = zr ? (T)0 : Z(PZ_E1, q);
                if (zr) sc[0][q] = sc[3][q] = czero<CT>();
                sc[1][q] = ifma(-(ri * kap), p, cscale(ngd, vl));
                sc[2][q] = cfma(-gr, rho, cscale(ngd, vz));
                own[q] = p;
            } else {
                const CT div = ifma(kap, arg(F0, 0, q), d[q]);
                const CT xz = own[q];
                const CT p = cfma(-Z(PZ_GP, q), xz, cscale(-Z(PZ_C2R, q), div));
                const CT b = cfma(Z(PZ_E2, q), xz, cscale(Z(PZ_E1, q), div));      // -g rho'/rho0
                own[q] = p;
                const T ri = Z(PZ_RI, q);
                const CT v = arg(F2, 2, q), vz = arg(F3, 3, q);
                sc[2][q] = ifma(-(ri * kap), p, D3 ? cscale(ngd, v) : czero<CT>());
                sc[0][q] = v;
                sc[3][q] = D3 ? cfma(ngd, vz, b) : b;
                sc[1][q] = vz;
            }
        }
        exchange(own);
        // d: stretch / rho0 times d/dz of p'
        pencil_solve<CH, PART, T, CT>(own, xb[t - 1], xf[t + 1], cl, zt + PZ_S2 * NZP, c2, ce + 2 * PE_COUNT, false,
                                czero<CT>(), NZP, TP, nz, j0, lo, hi, t, cf, cb, pi, d);
        #pragma unroll
        for (int q = 0; q < CH; ++q)
            if (!(VEL && zero_row(q))) sc[FV][q] = sc[FV][q] - d[q];
        if (npw) {                   // psi_p
            #pragma unroll
            for (int q = 0; q < CH; ++q)
                if (pmask & (1u << q)) pd[pipv + q] = d[q];
            pml(1, pz + nzpml);
            #pragma unroll
            for (int q = 0; q < CH; ++q)
                if ((pmask & (1u << q)) && !(VEL && zero_row(q))) sc[FV][q] = cfma(-Z(PZ_RI, q), pd[pipv + q], sc[FV][q]);
        }
        if (src_t) {
            #pragma unroll
            for (int q = 0; q < CH; ++q) {
                if (VEL) {
                    if (abs(j0 + q - A.ksrc) <= 4 && !zero_row(q) && j0 + q < nz)
                        sc[FV][q] = cfma(Z(PZ_SRC, q), F, sc[FV][q]);
                } else if (j0 + q == A.ksrc) {
                    sc[FV][q] = sc[FV][q] + F;
                }
            }
        }
        if constexpr (!VEL) {
            if (lo || hi) {
                #pragma unroll
                for (int q = 0; q < CH; ++q)
                    if (zero_row(q)) sc[0][q] = sc[1][q] = sc[2][q] = sc[3][q] = czero<CT>();
            }
        }
    };

    #pragma unroll 1
    for (int step = 0; step < A.nsteps; ++step) {
        const int tl = tl0 + step;
        // forcing of this step, on the slot's clock
        const int reach = VEL ? 4 : 0;
        src_t = A.src_mode != 0 && slot_src_on(A.clk, tl) && mvalid && A.ksrc + reach >= j0 && A.ksrc - reach < j0 + CH;
        if (src_t) {
            if (A.src_mode == 1) {
                const T w = (tl < A.nseries) ? (T)A.series[(long long)s * A.nseries + tl] : (T)0;
                F = cscale(w, A.planes[(long long)s * A.plane_ss + m]);
            } else {                 // this step's plane, interpolated by source_plane_kernel
                F = A.src_plane[((long long)step * A.nsrc + s) * M + m];
            }
            if (!VEL) F = cscale(A.src_scale, F);
        }
        // the components along k
        if (D3) {
            #pragma unroll
            for (int q = 0; q < CH; ++q) {
                const CT* p = tp + q;
                if constexpr (VEL) {
                    tp[6 * FT + q] = cfma(ex, p[FT], cscale(ey, p[2 * FT]));
                } else {
                    tp[6 * FT + q] = cfma(ex, p[0], cscale(ey, p[FT]));
                    tp[7 * FT + q] = cfma(ex, p[3 * FT], cscale(ey, p[4 * FT]));
                }
            }
        }
        stage(std::integral_constant<bool, false>(), (T)0);
        #pragma unroll 1
        for (int rk = 1; rk < 5; ++rk) {
            const T beta = rk == 1 ? A.betas[1] : rk == 2 ? A.betas[2] : rk == 3 ? A.betas[3] : A.betas[4];
            stage(std::integral_constant<bool, true>(), beta);
        }
        // ---- update a += dt*scr (step.f90:114-116), and the right-hand side of
        // the call's last step for the outputs that read it.  The across
        // components' right-hand sides are r5 U and -gamma r5 U, U = v across k ----
        const bool put_scr = A.write_scr && step == A.nsteps - 1 && mvalid;
        #pragma unroll
        for (int q = 0; q < CH; ++q) {
            CT* p = tp + q;
            CT* g = gS + (long long)(j0 + q) * M + m;
            const bool put = put_scr && j0 + q < nz;
            if constexpr (FORM == 4) {
                const CT vx = p[3 * FT], vy = p[4 * FT];
                const CT c = cscale(zero_row(q) ? (T)0 : r5, cfma(ex, vy, cscale(-ey, vx)));
                if (put) {
                    g[0] = cfma(ex, sc[0][q], cscale(-ey, c));
                    g[fs] = cfma(ey, sc[0][q], cscale(ex, c));
                    g[2 * fs] = sc[1][q];
                    g[3 * fs] = cfma(ex, sc[2][q], cscale(-ey * ngd, c));
                    g[4 * fs] = cfma(ey, sc[2][q], cscale(ex * ngd, c));
                    g[5 * fs] = sc[3][q];
                }
                p[0] = cfma(A.dt * ex, sc[0][q], cfma(-A.dt * ey, c, p[0]));
                p[FT] = cfma(A.dt * ey, sc[0][q], cfma(A.dt * ex, c, p[FT]));
                p[2 * FT] = cfma(A.dt, sc[1][q], p[2 * FT]);
                p[3 * FT] = cfma(A.dt * ex, sc[2][q], cfma(-A.dt * ey * ngd, c, vx));
                p[4 * FT] = cfma(A.dt * ey, sc[2][q], cfma(A.dt * ex * ngd, c, vy));
                p[5 * FT] = cfma(A.dt, sc[3][q], p[5 * FT]);
            } else if constexpr (VEL) {
                const CT vx = p[FT], vy = p[2 * FT];
                const CT c = cscale(ngd * r5, cfma(ex, vy, cscale(-ey, vx)));
                if (put) {
                    g[0] = sc[0][q];
                    g[fs] = cfma(ex, sc[1][q], cscale(-ey, c));
                    g[2 * fs] = cfma(ey, sc[1][q], cscale(ex, c));
                    g[3 * fs] = sc[2][q];
                    g[4 * fs] = sc[3][q];
                }
                p[0] = cfma(A.dt, sc[0][q], p[0]);
                p[FT] = cfma(A.dt * ex, sc[1][q], cfma(-A.dt * ey, c, vx));
                p[2 * FT] = cfma(A.dt * ey, sc[1][q], cfma(A.dt * ex, c, vy));
                p[3 * FT] = cfma(A.dt, sc[2][q], p[3 * FT]);
                p[4 * FT] = cfma(A.dt, sc[3][q], p[4 * FT]);
            } else {
                if (put) {
                    g[0] = sc[0][q];
                    g[2 * fs] = sc[1][q];
                    g[3 * fs] = sc[2][q];
                    g[5 * fs] = sc[3][q];
                    g[fs] = g[4 * fs] = czero<CT>();
                }
                p[0] = cfma(A.dt, sc[0][q], p[0]);
                p[2 * FT] = cfma(A.dt, sc[1][q], p[2 * FT]);
                p[3 * FT] = cfma(A.dt, sc[2][q], p[3 * FT]);
                p[5 * FT] = cfma(A.dt, sc[3][q], p[5 * FT]);
            }
        }
        // pml += dt*scrpml (step.f90:116)
        for (int i = lane; i < 2 * npw; i += seg) {
            const int o = (i < npw ? 0 : nzpml) + plane(i < npw ? i : i - npw);
            ptile[o] = cfma(A.dt, spt[o], ptile[o]);
        }
        pencil_sync(pi, TP);
        // ---- z filter and horizontal filter (FILTER_VARS_3D / _2D): field f into
        // registers, written back once every thread has read its neighbours ----
        const bool hfil = slot_hfilter(A.clk, tl);
        const T hf = (hfil && mvalid) ? A.pt[PT_HF * (long long)M + m] : (T)1;
        const T h1 = (T)(0.5 * 0.41015625), h2 = (T)(0.5 * -0.234375), h3 = (T)(0.5 * 0.087890625);
        const T h4 = (T)(0.5 * -0.01953125), h5 = (T)(0.5 * 0.001953125), h0 = (T)0.75390625, half = (T)0.5;
        const bool ends = j0 < 5 || j0 + CH > nz - 5;
        #pragma unroll 1
        for (int f = 0; f < 6; ++f) {
            if (!extra && (VEL ? f == 5 : (!D3 && (f == 1 || f == 4)))) continue;
            // level q of the chunk, q from -5 to CH + 4: chunk offset floor(q / CH)
            const CT* B = tp + f * FT;
            auto V = [&](int q) -> CT {
                const int c = (q + 2 * CH) / CH - 2;
                return B[c * CHP + (q - c * CH)];
            };
            CT out[CH];
            #pragma unroll
            for (int q = 0; q < CH; ++q) {
                CT acc = cscale(h0, V(q));
                acc = cfma(h1, V(q - 1) + V(q + 1), acc);
                acc = cfma(h2, V(q - 2) + V(q + 2), acc);
                acc = cfma(h3, V(q - 3) + V(q + 3), acc);
                acc = cfma(h4, V(q - 4) + V(q + 4), acc);
                out[q] = cfma(h5, V(q - 5) + V(q + 5), acc);
            }
            if (ends) {
                #pragma unroll
                for (int q = 0; q < CH; ++q) {
                    const int j = j0 + q;
                    if (j == 0 || j == nz - 1) out[q] = V(q);
                    else if (j >= nz) out[q] = czero<CT>();          // padding stays zero
                    else if (j >= nz - 5 || (D3 && j <= 4)) out[q] = cscale(half, V(q + 1) + V(q - 1));
                    else if (j <= 4) out[q] = V(q);
                }
            }
            if (hfil && (D3 ? f < 5 : true)) {
                #pragma unroll
                for (int q = 0; q < CH; ++q) out[q] = cscale(hf, out[q]);
            }
            pencil_sync(pi, TP);
            #pragma unroll
            for (int q = 0; q < CH; ++q) tp[f * FT + q] = out[q];
        }
        // ---- surface record: v_z on the observation plane (driver.f90:455-476) ----
        if (A.rec && mvalid && tl >= 0 && tl % A.rec_steps == 0 && A.rec_k >= j0 && A.rec_k < j0 + CH) {
            const int r = tl / A.rec_steps;
            if (r < A.rec_max) A.rec[((long long)s * A.rec_max + r) * M + m] = tp[(VEL ? 3 : 5) * FT + A.rec_k - j0];
        }
    }
    __syncthreads();
    {
        const int q = threadIdx.x % P, z0 = threadIdx.x / P;
        if (m0 + q < M) {
            const CT* src = tile + q * LZ + GC * CHP;
            for (int z = z0; z < nz; z += TP) {
                const int r = (z / CH) * CHP + z % CH;
                for (int f = 0; f < 6; ++f)
                    if (!VEL || f < 5 || extra) gA[f * fs + (long long)z * M + m0 + q] = src[f * FT + r];
            }
            for (int r = z0; r < 2 * nzpml; r += TP)
                gP[(long long)r * M + m0 + q] = sm[Ly.ptile + q * 2 * nzpml + r];
        }
    }
}

// FP32 is built for the velocity form alone, parts of a warp for FP64 with up to
// five levels a thread (pencil_shape)
template <typename T, int CH, bool PART>
const void* kernel_form(int option) {
    if constexpr (sizeof(T) == 8) {
        if (option == 17) return (const void*)pencil_step_kernel<T, 17, CH, PART>;
        if (option == 4) return (const void*)pencil_step_kernel<T, 4, CH, PART>;
    }
    return (const void*)pencil_step_kernel<T, 2, CH, PART>;
}
template <typename T, int CH>
const void* kernel_ch(int option, int tp) {
    if constexpr (sizeof(T) == 8 && CH <= 5) {
        if (tp < 32) return kernel_form<T, CH, true>(option);
    }
    return kernel_form<T, CH, false>(option);
}
template <typename T>
const void* kernel_of(int option, const PencilShape& sh) {
    switch (sh.ch) {
        case 3: return kernel_ch<T, 3>(option, sh.tp);
        case 4: return kernel_ch<T, 4>(option, sh.tp);
        case 6: return kernel_ch<T, 6>(option, sh.tp);
        case 7: return kernel_ch<T, 7>(option, sh.tp);
        default: return kernel_ch<T, 5>(option, sh.tp);
    }
}

size_t pencil_bytes(const PencilShape& sh, int option, int P, int nzpml, int complex_bytes) {
    return (size_t)pencil_layout(P, sh.tp, sh.ch, nzpml, option).total * complex_bytes;
}

}  // namespace

// Cost of a pencil's step of a shape: warps times the FP64 instructions of a thread
// (per chunk 40 a stage for the scans and 60 for closures and PML, per level 55 a
// stage and 144 for update and filter).  A step takes 4.05 us a unit to within 4 %
// on every shape of option 4 at 512x256.
double pencil_cost(const PencilShape& sh) { return sh.tp / 32.0 * (5 * 100.0 + sh.ch * (5 * 55.0 + 144.0)); }

// Levels per thread and threads per pencil of a grid: the least cost.  FP64
// issue pays for a lane without levels as for a full one, so boxes of up to 40
// levels take a quarter and of up to 80 half of a warp (512x256, option 4, ms a step
// with a whole warp and so: 24 levels 6.94 and 1.84, 48 levels 6.94 and 3.51, 80
// levels 6.94 and 5.21); with 6 or 7 levels a thread such pencils leave an SM four
// or five warps, too few (96 levels on half a warp 7.02, on a whole one 6.94).
// FP32 (option 2) is not bound by FP64 and keeps whole warps.  On grids with few
// modes (an SM holds no more than four pencils of one source) a step is the length
// of its serial chains: 3 levels per thread, as many lanes as that takes
// (256x1x300, one source: 3 levels on four warps 69 us, 4 on three 80, 5 on two
// 93; eight sources, which fill the GPU, 376, 389 and 329: the shape depends on
// the grid alone, so that a source's arithmetic does not depend on the batch
// around it).
PencilShape pencil_shape(int nz, int modes, bool f64, int nsm) {
    PencilShape best = {5, 32 * ((nz + 159) / 160)};
    double cost = 0.0;
    const bool few = modes <= 4 * nsm;
    for (int ch = 3; ch <= 7; ++ch) {
        const bool part = f64 && ch <= 5 && nz <= 16 * ch;
        const PencilShape sh = {ch, part ? (nz <= 8 * ch ? 8 : 16) : 32 * ((nz + 32 * ch - 1) / (32 * ch))};
        if (sh.tp > 256 || (few && ch > 3 && (nz + 95) / 96 <= 8)) continue;
        const double c = pencil_cost(sh);
        if (cost == 0.0 || c < cost) { cost = c; best = sh; }
    }
    return best;
}

// Pencils per CTA: 128 threads (two CTAs an SM overlap one's copies with the
// other's arithmetic), fewer when the launch would leave SMs without two CTAs;
// whole warps.  Part-warp pencils take the size of which an SM holds most warps
// (8 at the kernel's 255 registers), the larger of two that give as many, and two
// warps a CTA at least: CTAs of one warp are a sixth slower (512x256x48, half a
// warp a pencil: 8 or 4 pencils a CTA 3.51 ms a step, 2 pencils 4.13).
// 0: not even one warp fits the shared memory a CTA may use.
int pencil_count(const PencilShape& sh, int option, int nzpml, int complex_bytes, long long pencils, int nsm) {
    const int least = pencil_least(sh);
    auto bytes = [&](int p) { return pencil_bytes(sh, option, p, nzpml, complex_bytes); };
    if (sh.tp > 256 || bytes(least) > 227 * 1024) return 0;
    int P = std::max(least, 128 / sh.tp);
    if (sh.tp < 32) {
        int held = 0;
        for (int p = 128 / sh.tp; p >= 2 * least; p /= 2) {
            const int warps = std::min(8, (int)(228 * 1024 / (bytes(p) + 1024)) * (p / least));
            if (warps > held) { held = warps; P = p; }
        }
    }
    while (P > least && (bytes(P) > 113 * 1024 || (pencils + P - 1) / P < 2LL * nsm)) P /= 2;
    return P;
}

template <typename T>
int pencil_prepare(const PencilShape& sh, int option) {
    return allow_shared_memory(kernel_of<T>(option, sh));
}

template <typename T>
void launch_pencil(const PencilArgs<T>& A, int ch, cudaStream_t s) {
    const PencilShape sh = {ch, A.part ? A.part : 32 * A.W};
    const size_t smem = pencil_bytes(sh, A.option, A.pencils, A.nzpml, 2 * sizeof(T));
    const long long ctas = (long long)((A.M + A.pencils - 1) / A.pencils) * A.nsrc;
    void* args[] = {(void*)&A};
    cudaLaunchKernel(kernel_of<T>(A.option, sh), dim3((unsigned)ctas), dim3(A.pencils * sh.tp), args, smem, s);
}

template int pencil_prepare<double>(const PencilShape&, int);
template int pencil_prepare<float>(const PencilShape&, int);
template void launch_pencil<double>(const PencilArgs<double>&, int, cudaStream_t);
template void launch_pencil<float>(const PencilArgs<float>&, int, cudaStream_t);
