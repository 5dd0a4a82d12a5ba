// Time step of the magnetic forms: MP_MHD_PML_3D_DISPL (option 10,
// displacement.f90:663-849), MP_MHD_PML_2D_DISPL (option 18,
// physics2d.f90:724-943) and the velocity form MP_MHD_PML_3D (option 8,
// pml.f90:80-208) on a physical-space state.
//
// A stage of option 10 (of option 18 without the y parts):
//   x, y    d/dx of xi_x, flux3, flux2; d/dy of xi_y, flux3, flux1; and
//           DAMP_VELOCITY (damping.f90:125-159) of v through the transforms
//   z       d/dz of xi_z, flux1, flux2
//   point1  div, p', rho' and the induced field b
//   x, y, z d/dx and d/dy of p' and b; d/dz of p', b_x, b_y
//   point2  everything else: curl b, the Lorentz forces, gravity, sponge,
//           damping, source, zero rows; it writes the next stage's temporaries
//           and fluxes (a + beta scr at its own points), or scr after the last
//           stage
// Every launch covers all the fields of its group and all sources.  Steps
// replay from graphs: the horizontal filter reads each source's clock on the
// device, so a captured step is valid at any time.
//
// What bounds it: on a large grid in FP32 memory (a stage passes 120 fields
// through it, 137 before the stages were joined; the point-wise kernels run at
// the copy rate, transforms and z solves at 0.55 to 0.8 of it); in FP64 the
// FP64 pipe, two thirds of it in the transforms; on a small grid the launches
// and their serial chains.
//
// The z derivatives pass through memory.  Solving them inside point1 / point2
// (a CTA holding 16 or 32 whole pencils) saves 15 field passes a stage but
// reads 27 fields in 64- or 128-byte pieces, 300 planes apart: measured 1364 us
// a stage against 940 us at 256x256x300 FP32, and slower on every smaller grid
// and in FP64 too.
//
// Measured per step: option 10, 256x256x300 FP32 10.8 -> 8.9 ms, 128x128x150
// FP64 18.0 -> 12.8 ms; option 18, 256x1x300 FP64 5.6 -> 0.42 ms.
#include <algorithm>
#include <cstring>
#include <type_traits>

#include "mhd.cuh"
#include "zsolve.cuh"

namespace {

template <typename T> struct StepArgs {
    long long N, NP, FS;      // points per field, per plane; field stride of the state slots
    int nz, nb, nt, nzpml, both;       // both: PML at both ends (options 8, 18), else the bottom only
    const T* bg; T* work;
    const T* pab; const T* pml; T* spml;
    const T* a; T* scr;
    T beta, beta_next;        // this stage's argument a + beta scr, and the next one's
    int hs, last;             // hs: not the first stage; last: the fifth
    const T* g; const T* sponge; const T* zt;
    int damp, adjoint;
    SlotClock clk;
    int src_mode, ksrc;
    const T* src; long long src_ss;      // this step's plane (mode 2) or the series' plane (mode 1)
    const double* series; int nseries;
    const int* plane; const T* dw;
};

// PML accounting (pml.f90:213-231 form): rhs = a_z deriv + b_z psi, deriv +=
// psi, with psi = pmlvars + beta*scrpml, on plane k, pixel q of source s
template <typename T>
__device__ __forceinline__ T pml_at(const StepArgs<T>& A, int k, long long q, int s, int aux, T deriv) {
    int ip = -1;                                  // pmlindex of the plane
    if (k < A.nb) ip = k;
    else if (A.both && k >= A.nz - A.nt) ip = A.nb + (k - (A.nz - A.nt));
    if (ip < 0) return deriv;
    const long long np = (long long)A.nzpml * A.NP, ipq = (long long)ip * A.NP + q;
    const long long o = ((long long)s * PV_COUNT + aux) * np + ipq;
    T psi = A.pml[o];
    if (A.hs) psi = psi + A.beta * A.spml[o];
    A.spml[o] = A.pab[ipq] * deriv + A.pab[np + ipq] * psi;
    return deriv + psi;
}

// forcing of this step at pixel q of source s (its clock tl)
template <typename T>
__device__ __forceinline__ T forcing(const StepArgs<T>& A, int s, int tl, long long q) {
    const T p = A.src[(long long)s * A.src_ss + q];
    if (A.src_mode != 1) return p;                // interpolated by source_plane_kernel
    return ((tl < A.nseries) ? (T)A.series[(long long)s * A.nseries + tl] : (T)0) * p;
}

// the first stage's temporaries T = a (step.f90:52-71) and the fluxes of
// xi x B0 (displacement.f90:672-674)
template <typename T, int FORM>
__global__ void temp_kernel(const StepArgs<T> A) {
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= A.N) return;
    const int s = blockIdx.y;
    constexpr int NF = FORM == 8 ? 8 : 6, WC = FORM == 8 ? (int)V8_COUNT : (int)MW_COUNT, F1 = FORM == 8 ? V8_F1 : MW_F1;
    const T* as = A.a + (long long)s * NF * A.FS;
    T* w = A.work + (long long)s * WC * A.N;
    T v[NF];
    #pragma unroll
    for (int f = 0; f < NF; ++f) {
        v[f] = as[f * A.FS + t];
        w[f * A.N + t] = v[f];
    }
    constexpr int U = FORM == 8 ? 1 : 0;          // the vector crossed with B0
    const T box = A.bg[MB_BOX * A.N + t], boz = A.bg[MB_BOZ * A.N + t];
    w[(F1 + 1) * A.N + t] = -(v[U] * boz - v[U + 2] * box);
    if (FORM != 18) {
        const T boy = A.bg[MB_BOY * A.N + t];
        w[F1 * A.N + t] = -(v[U + 2] * boy - v[U + 1] * boz);
        w[(F1 + 2) * A.N + t] = -(v[U + 1] * box - v[U] * boy);
    }
}

// After the z derivatives of xi_z and of the fluxes: div, p', rho'
// (displacement.f90:694-697) after the psi_vz accounting, and b
// (displacement.f90:729-757) after psi_ibx, psi_iby, on plane k, pixel q of source
// s; w, bg at the point
template <typename T, int FORM>
__device__ __forceinline__ void point1(const StepArgs<T>& A, T* w, const T* __restrict__ bg, int s, int k, long long q,
                                       T dz, T dzf1, T dzf2) {
    constexpr bool D3 = FORM == 10;
    auto W = [&](int f) -> T { return w[f * A.N]; };
    auto B = [&](int f) -> T { return __ldg(&bg[f * A.N]); };
    // every load first
    const T xx = W(MW_T0), xz = W(MW_T2), dx = W(MW_DX);
    const T c2r = B(MB_C2RHO0), r0 = B(MB_RHO0), gpx = B(MB_GP0X), gpz = B(MB_GP0Z), grx = B(MB_GR0X), grz = B(MB_GR0Z);
    T xy = (T)0, dy = (T)0, gpy = (T)0, gry = (T)0, bx = (T)0, by = (T)0, bz = (T)0, dyf1 = (T)0;
    if (D3) {
        xy = W(MW_T1); dy = W(MW_DY); gpy = B(MB_GP0Y); gry = B(MB_GR0Y);
        bx = W(MW_BX); by = W(MW_BY); bz = W(MW_BZ); dyf1 = W(MW_DYF1);
    }
    dz = pml_at<T>(A, k, q, s, PV_VZ, dz);
    dzf2 = pml_at<T>(A, k, q, s, PV_IBX, dzf2);
    const T div = D3 ? dx + dy + dz : dx + dz;
    T p = -c2r * div - xz * gpz - xx * gpx, r = -r0 * div - xz * grz - xx * grx;
    if constexpr (D3) {
        dzf1 = pml_at<T>(A, k, q, s, PV_IBY, dzf1);
        p = p - xy * gpy;
        r = r - xy * gry;
        w[MW_BX * A.N] = bx - dzf2;
        w[MW_BY * A.N] = -by + dzf1;
        w[MW_BZ * A.N] = bz - dyf1;
    } else {
        w[MW_BX * A.N] = -dzf2;
    }
    w[MW_P * A.N] = p;
    w[MW_R * A.N] = r;
}

// After the z derivatives of p', b_x, b_y, the rest of the stage: psi_p, psi_dzbx,
// psi_dzby, curl b, the two Lorentz terms (CROSS, derivatives.f90:471-480), the
// sponge on the top 36 planes (option 10), gravity, RHSxi = v, damping, the
// source on each pixel's source plane ks while the slot's clock is within the
// forcing gate, and the zero rows (displacement.f90:759-848, physics2d.f90:780-938);
// as and ss at the point
template <typename T, int FORM>
__device__ __forceinline__ void point2(const StepArgs<T>& A, T* w, const T* __restrict__ bg, const T* as, T* ss, int s,
                                       int k, long long q, int ks, T gpz, T dzbx, T dzby) {
    constexpr bool D3 = FORM == 10;
    const bool last = A.last != 0, damp = A.damp != 0;
    auto W = [&](int f) -> T { return w[f * A.N]; };
    auto B = [&](int f) -> T { return __ldg(&bg[f * A.N]); };
    // every load first
    const T gpx = W(MW_GPX), dxbz = W(MW_DXBZ), bx = W(MW_BX), bz = W(MW_BZ), r = W(MW_R);
    const T box = B(MB_BOX), boz = B(MB_BOZ), ri = B(MB_RHOINV), cboy = B(MB_CBOY);
    T vx = W(MW_T3), vy = (T)0, vz = W(MW_T5);
    T dmx = (T)0, dmy = (T)0, dmz = (T)0, gpy = (T)0, by = (T)0, dybz = (T)0, dxby = (T)0, dybx = (T)0;
    T boy = (T)0, cbox = (T)0, cboz = (T)0, a0 = (T)0, a1 = (T)0, a2 = (T)0, a3 = (T)0, a4 = (T)0, a5 = (T)0;
    if (damp) { dmx = W(MW_DMX); dmz = W(MW_DMZ); if (D3) dmy = W(MW_DMY); }
    if (D3) {
        gpy = W(MW_GPY); by = W(MW_BY); dybz = W(MW_DYBZ); dxby = W(MW_DXBY); dybx = W(MW_DYBX); vy = W(MW_T4);
        boy = B(MB_BOY); cbox = B(MB_CBOX); cboz = B(MB_CBOZ);
    }
    if (!last) {
        a0 = as[0]; a2 = as[2 * A.FS]; a3 = as[3 * A.FS]; a5 = as[5 * A.FS];
        if (D3) { a1 = as[A.FS]; a4 = as[4 * A.FS]; }
    }
    gpz = pml_at<T>(A, k, q, s, PV_P, gpz);
    dzbx = pml_at<T>(A, k, q, s, PV_DZBX, dzbx);
    const T cby = -dxbz + dzbx;
    T rvx, rvy = (T)0, rvz;
    if constexpr (D3) {
        dzby = pml_at<T>(A, k, q, s, PV_DZBY, dzby);
        const T cbx = dybz - dzby, cbz = dxby - dybx;
        rvx = ri * (-gpx + (cby * boz - cbz * boy)) + ri * (cboy * bz - cboz * by);
        rvy = ri * (-gpy + (box * cbz - cbx * boz)) + ri * (bx * cboz - cbox * bz);
        rvz = ri * (-gpz + (cbx * boy - cby * box)) + ri * (cbox * by - cboy * bx);
        if (k >= A.nz - 36) {
            const T sp = __ldg(&A.sponge[k]);
            rvx = rvx - sp * vx;
            rvy = rvy - sp * vy;
            rvz = rvz - sp * vz;
        }
    } else {
        rvx = fma(ri, -gpx + cby * boz, ri * (cboy * bz));      // one rounding order (rows2d_f32.cu)
        rvz = ri * (-gpz + (-cby * box)) + ri * (-cboy * bx);
    }
    rvz = rvz - ri * r * __ldg(&A.g[k]);
    rvx = rvx - dmx;
    rvy = rvy - dmy;
    rvz = rvz - dmz;
    if (k == ks) {
        const int tl = *A.clk.time - A.clk.t0[s];
        if (tl >= 0 && tl <= A.clk.gate) {
            const T F = forcing<T>(A, s, tl, q), r0 = B(MB_RHO0), dw = A.dw[q];
            rvz = rvz + ((!D3 && A.adjoint) ? F * dw / r0 : F / r0 * dw);
        }
    }
    if (k == 0 || (D3 && k == A.nz - 1)) vx = vy = vz = rvx = rvy = rvz = (T)0;
    if (last) {
        ss[0] = vx;
        ss[A.FS] = vy;
        ss[2 * A.FS] = vz;
        ss[3 * A.FS] = rvx;
        ss[4 * A.FS] = rvy;
        ss[5 * A.FS] = rvz;
    } else {
        const T bn = A.beta_next;
        a0 = a0 + bn * vx;
        a2 = a2 + bn * vz;
        w[MW_T0 * A.N] = a0;
        w[MW_T2 * A.N] = a2;
        w[MW_T3 * A.N] = a3 + bn * rvx;
        w[MW_T5 * A.N] = a5 + bn * rvz;
        w[MW_F2 * A.N] = -(a0 * boz - a2 * box);
        if (D3) {
            a1 = a1 + bn * vy;
            w[MW_T1 * A.N] = a1;
            w[MW_T4 * A.N] = a4 + bn * rvy;
            w[MW_F1 * A.N] = -(a2 * boy - a1 * boz);
            w[MW_F3 * A.N] = -(a1 * box - a0 * boy);
        }
    }
}

template <typename T, int FORM, int WHICH>
__global__ void __launch_bounds__(256) point_kernel(const StepArgs<T> A) {
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= A.N) return;
    const int s = blockIdx.y, k = (int)(t / A.NP);
    const long long q = t - (long long)k * A.NP;
    T* w = A.work + (long long)s * MW_COUNT * A.N + t;
    const T z0 = w[MW_Z0 * A.N], z1 = FORM == 10 || WHICH == 2 ? w[MW_Z1 * A.N] : (T)0;
    const T z2 = FORM == 10 || WHICH == 1 ? w[MW_Z2 * A.N] : (T)0;
    if (WHICH == 1) point1<T, FORM>(A, w, A.bg + t, s, k, q, z0, z1, z2);
    else point2<T, FORM>(A, w, A.bg + t, A.a + (long long)s * 6 * A.FS + t, A.scr + (long long)s * 6 * A.FS + t, s, k, q,
                         A.src_mode != 0 ? A.plane[q] : -1, z0, z1, z2);
}

// option 8, everything after the derivatives, point-wise: PML_BOUNDARY_ACCOUNTING_3D
// at both ends (pml.f90:213-285), the induction RHS, div, curl b, continuity,
// pressure, the two Lorentz terms (CROSS, derivatives.f90:471-480), gravity,
// the source forcing * source_dep(k) for |k - e_rad| <= 4 (pml.f90:175-181),
// the zero top and bottom rows of all eight fields, then DAMP_VELOCITY; writes
// the next stage's temporaries and fluxes, or scr after the last stage
template <typename T>
__global__ void rhs8_kernel(const StepArgs<T> A) {
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= A.N) return;
    const int s = blockIdx.y;
    const int k = (int)(t / A.NP);
    const long long q = t - (long long)k * A.NP;
    T* w = A.work + (long long)s * V8_COUNT * A.N;
    auto W = [&](int f) -> T { return w[(long long)f * A.N + t]; };
    auto B = [&](int f) -> T { return A.bg[(long long)f * A.N + t]; };
    const T gpz = pml_at<T>(A, k, q, s, PV_P, W(V8_GPZ));
    const T dvzdz = pml_at<T>(A, k, q, s, PV_VZ, W(V8_DVZDZ));
    const T dzf2 = pml_at<T>(A, k, q, s, PV_IBX, W(V8_DZF2));
    const T dzf1 = pml_at<T>(A, k, q, s, PV_IBY, W(V8_DZF1));
    const T dzbx = pml_at<T>(A, k, q, s, PV_DZBX, W(V8_DZBX));
    const T dzby = pml_at<T>(A, k, q, s, PV_DZBY, W(V8_DZBY));
    const T rbx = W(V8_DYF3) - dzf2;
    const T rby = -W(V8_DXF3) + dzf1;
    const T rbz = W(V8_DXF2) - W(V8_DYF1);
    const T div = W(V8_DVXDX) + W(V8_DVYDY) + dvzdz;
    const T cbx = W(V8_DYBZ) - dzby;
    const T cby = -W(V8_DXBZ) + dzbx;
    const T cbz = W(V8_DXBY) - W(V8_DYBX);
    const T rho = W(V8_T0), vx = W(V8_T1), vy = W(V8_T2), vz = W(V8_T3);
    const T bx = W(V8_T5), by = W(V8_T6), bz = W(V8_T7);
    const T rcont = -B(MB_GR0X) * vx - B(MB_GR0Y) * vy - B(MB_GR0Z) * vz - B(MB_RHO0) * div;
    const T rp = -B(MB_C2RHO0) * div - vx * B(MB_GP0X) - vy * B(MB_GP0Y) - vz * B(MB_GP0Z);
    const T box = B(MB_BOX), boy = B(MB_BOY), boz = B(MB_BOZ), ri = B(MB_RHOINV);
    T f1 = cby * boz - cbz * boy, f2 = cbz * box - cbx * boz, f3 = cbx * boy - cby * box;
    T rvx = -ri * (W(V8_GPX) - f1);
    T rvy = -ri * (W(V8_GPY) - f2);
    T rvz = -ri * (gpz - f3);
    const T cbox = B(MB_CBOX), cboy = B(MB_CBOY), cboz = B(MB_CBOZ);
    f1 = cboy * bz - cboz * by; f2 = cboz * bx - cbox * bz; f3 = cbox * by - cboy * bx;
    rvx = rvx + ri * f1;
    rvy = rvy + ri * f2;
    rvz = rvz + ri * f3;
    rvz = rvz - ri * rho * A.g[k];
    if (A.src_mode != 0 && abs(k - A.ksrc) <= 4) {
        const int tl = *A.clk.time - A.clk.t0[s];
        if (slot_src_on(A.clk, tl)) rvz = rvz + forcing<T>(A, s, tl, q) * A.zt[ZT_SRCDEP * A.nz + k];
    }
    T out[8] = {rcont, rvx, rvy, rvz, rp, rbx, rby, rbz};
    if (k == 0 || k == A.nz - 1) {
        #pragma unroll
        for (int f = 0; f < 8; ++f) out[f] = (T)0;
    }
    if (A.damp) {
        out[1] = out[1] - W(V8_DMX);
        out[2] = out[2] - W(V8_DMY);
        out[3] = out[3] - W(V8_DMZ);
    }
    if (A.last) {
        T* ss = A.scr + (long long)s * 8 * A.FS;
        #pragma unroll
        for (int f = 0; f < 8; ++f) ss[f * A.FS + t] = out[f];
        return;
    }
    const T* as = A.a + (long long)s * 8 * A.FS;
    #pragma unroll
    for (int f = 0; f < 8; ++f) {
        out[f] = as[f * A.FS + t] + A.beta_next * out[f];
        w[(V8_T0 + f) * A.N + t] = out[f];
    }
    w[V8_F1 * A.N + t] = -(out[3] * boy - out[2] * boz);
    w[V8_F2 * A.N + t] = -(out[1] * boz - out[3] * box);
    w[V8_F3 * A.N + t] = -(out[2] * box - out[1] * boy);
}

__device__ __forceinline__ double vfma(double s, double v, double a) { return fma(s, v, a); }
__device__ __forceinline__ float2 vfma(float s, float2 v, float2 a) { return pfma(bc2(s), v, a); }
__device__ __forceinline__ float vfma(float s, float v, float a) { return fma(s, v, a); }
__device__ __forceinline__ double vmul(double s, double v) { return s * v; }
__device__ __forceinline__ float vmul(float s, float v) { return s * v; }
__device__ __forceinline__ float2 vmul(float s, float2 v) { return pmul(bc2(s), v); }
__device__ __forceinline__ double vsub(double a, double b) { return a - b; }
__device__ __forceinline__ float2 vsub(float2 a, float2 b) { return psub(a, b); }

constexpr int Z_THREADS = 512;
// d/dz of the fields of a list (grid.y) of every source (grid.z), each pencil on
// chunks of ZCS levels, one per thread; in FP32 a thread takes two neighbouring
// pencils (paired instructions, npix is even).  A CTA holds LP values side by
// side times nw chunks.  A thread reads its chunk and one level on each side
// from HBM, eliminates and back-substitutes it with zero carries, and the
// chunks meet twice through shared memory: the carry from below is the sum over
// the ZKB nearest chunks of their values times the products of the chunk
// multipliers between them, and the same from above.  What is left out is below
// 2^-60 of a chunk value for every nz and boundary code (|multiplier| about 0.38
// a level, 50 levels).  The field is read once and written once; seven operations
// a level.
//
// Bound by memory latency in FP32, by the FP64 pipe in FP64.  One field of
// 256x256x300 FP32 54 -> 40 us (3.9 TB/s) against the solve it replaces, which
// staged its planes in shared memory; one of 128x128x150 FP64 101 -> 41 us
// against a thread per pencil.
template <typename T, typename V>
__global__ void __launch_bounds__(Z_THREADS, sizeof(T) == 4 ? 2 : 1) zderiv_kernel(
    const LineList<T, T> L, const ZCodes codes, const T* __restrict__ ztab, int nz, long long npix, int LP,
    const T* topsrc, T topscale) {
    extern __shared__ __align__(16) unsigned char smraw[];
    V* cf = (V*)smraw;
    V* cb = cf + blockDim.x;
    const long long nv = npix / (long long)(sizeof(V) / sizeof(T));
    const int nw = z_chunks(nz), nzp = nw * ZCS, cell = threadIdx.x, w = threadIdx.x / LP, j0 = w * ZCS;
    const long long m0 = (long long)blockIdx.x * LP + (threadIdx.x & (LP - 1));
    const bool on = m0 < nv;
    const long long m = on ? m0 : nv - 1;              // lanes past the last pencil repeat it and store nothing
    const T* c = ztab + (size_t)codes.bc[blockIdx.y] * z_code_size(nz);
    const V* in = (const V*)(L.in[blockIdx.y] + blockIdx.z * L.in_ss) + m;
    auto R = [&](int row, int q) -> T { return __ldg(&c[row * nzp + j0 + q]); };
    auto ld = [&](int j) -> V { return in[(long long)j * nv]; };
    V a[ZCS + 2], u[ZCS];
    #pragma unroll
    for (int i = 0; i < ZCS + 2; ++i) {
        const int j = j0 - 1 + i;
        a[i] = (j >= 0 && j < nz) ? ld(j) : vzero<V>();
    }
    #pragma unroll
    for (int q = 0; q < ZCS; ++q) u[q] = vmul(R(PS_D, q), vsub(a[q + 2], a[q]));
    const bool lo = w == 0, hi = j0 + ZCS > nz - 2;
    if (lo || hi) {       // rows 0, 1 or nz-2, nz-1 (dbyd2.f90:104-173)
        const T* e = c + PS_COUNT * nzp + 2 * nw * (ZKB - 1) + (lo ? 0 : PE_COUNT);
        V top = vzero<V>();
        if (hi && topsrc) top = vmul(topscale, ((const V*)(topsrc + blockIdx.z * L.in_ss))[(long long)(nz - 1) * nv + m]);
        V near = vzero<V>(), end = vmul(__ldg(&e[PE_TOP]), top);
        #pragma unroll
        for (int i = 0; i < 5; ++i) {
            const V b = lo ? a[1 + i] : ld(nz - 1 - i);
            near = vfma(__ldg(&e[i]), b, near);
            end = vfma(__ldg(&e[5 + i]), b, end);
        }
        const int jn = lo ? 1 : nz - 2, je = lo ? 0 : nz - 1;
        #pragma unroll
        for (int q = 0; q < ZCS; ++q) {
            if (j0 + q == jn) u[q] = near;
            if (j0 + q == je) u[q] = end;
        }
    }
    V run = u[0];
    #pragma unroll
    for (int q = 1; q < ZCS; ++q) {
        run = vfma(R(PS_M, q), run, u[q]);
        u[q] = run;
    }
    cf[cell] = run;
    // back substitution, with the part outside y added
    V x = run;
    u[ZCS - 1] = vfma(R(PS_A, ZCS - 1), vsub(a[ZCS + 1], a[ZCS - 1]), x);
    #pragma unroll
    for (int q = ZCS - 2; q >= 0; --q) {
        x = vfma(R(PS_G, q), x, u[q]);
        u[q] = vfma(R(PS_A, q), vsub(a[q + 2], a[q]), x);
    }
    __syncthreads();
    const T* pf = c + PS_COUNT * nzp + w * (ZKB - 1);
    const T* pb = pf + nw * (ZKB - 1);
    V e = w > 0 ? cf[cell - LP] : vzero<V>();
    #pragma unroll
    for (int i = 2; i <= ZKB; ++i)
        if (w >= i) e = vfma(__ldg(&pf[i - 2]), cf[cell - i * LP], e);
    cb[cell] = vfma(R(PS_K, 0), e, x);
    __syncthreads();
    V f = w + 1 < nw ? cb[cell + LP] : vzero<V>();
    #pragma unroll
    for (int i = 2; i <= ZKB; ++i)
        if (w + i < nw) f = vfma(__ldg(&pb[i - 2]), cb[cell + i * LP], f);
    if (!on) return;
    V* out = (V*)(L.out[blockIdx.y] + blockIdx.z * L.out_ss) + m;
    #pragma unroll
    for (int q = 0; q < ZCS; ++q)
        if (j0 + q < nz) out[(long long)(j0 + q) * nv] = vfma(R(PS_GC, q), f, vfma(R(PS_K, q), e, u[q]));
}

// values (pencils or pairs) per CTA: 16, at most Z_THREADS threads; fewer where
// the grid would not give every SM two CTAs
int z_pencils(int nz, long long nvalues, int nbatch, int nsm) {
    int lp = 16;
    while (lp > 2 && (lp * z_chunks(nz) > Z_THREADS || nvalues / lp * nbatch < 2LL * nsm)) lp /= 2;
    return lp;
}

// a += dt*scr (step.f90:114) and the z filter of FILTER_VARS_3D / _2D on whole
// pencils: a CTA's columns of a + dt*scr meet in shared memory, so the field is
// read once and written once.  Bound by memory latency: 256x256x300 FP32, six
// fields, 446 us with one column per thread, 359 with two (floor 202 us)
template <typename T, typename V>
__global__ void __launch_bounds__(Z_THREADS, 2) update_kernel(T* __restrict__ a_, const T* __restrict__ scr_, long long FS,
                                                              long long npix, int nz, int nf, int LP, T dt, int mode) {
    extern __shared__ __align__(16) unsigned char smraw[];
    V* col = (V*)smraw;                           // [nz][LP]
    constexpr int VW = sizeof(V) / sizeof(T);
    const int lp = threadIdx.x & (LP - 1), j0 = threadIdx.x / LP * ZCS;
    const long long nv = npix / VW, m = (long long)blockIdx.x * LP + lp, o = ((long long)blockIdx.z * nf + blockIdx.y) * FS;
    V* a = (V*)(a_ + o) + m;
    const V* scr = (const V*)(scr_ + o) + m;
    const bool on = m < nv;
    #pragma unroll
    for (int q = 0; q < ZCS; ++q) {
        const int j = j0 + q;
        if (j < nz && on) col[j * LP + lp] = vfma(dt, scr[(long long)j * nv], a[(long long)j * nv]);
    }
    __syncthreads();
    if (!on) return;
    const T h1 = (T)(0.5 * 0.41015625), h2 = (T)(0.5 * -0.234375), h3 = (T)(0.5 * 0.087890625);
    const T h4 = (T)(0.5 * -0.01953125), h5 = (T)(0.5 * 0.001953125), c0 = (T)0.75390625, hf = (T)0.5;
    #pragma unroll
    for (int q = 0; q < ZCS; ++q) {
        const int j = j0 + q;
        if (j >= nz) break;
        auto W = [&](int i) -> V { return col[(j + i) * LP + lp]; };
        V v;
        if (j == 0 || j == nz - 1) v = W(0);
        else if (j >= nz - 5) v = vmul(hf, W(1) + W(-1));
        else if (j <= 4) v = mode == 0 ? vmul(hf, W(1) + W(-1)) : W(0);
        else if constexpr (VW == 2) {      // the field's value last: rounds once at its size (as fused.cu)
            v = vfma(h1, W(-1) + W(1), vmul(c0 - (T)1, W(0)));
            v = vfma(h3, W(-3) + W(3), vfma(h2, W(-2) + W(2), v));
            v = W(0) + vfma(h5, W(-5) + W(5), vfma(h4, W(-4) + W(4), v));
        } else {
            v = c0 * W(0) + h1 * (W(-1) + W(1)) + h2 * (W(-2) + W(2)) + h3 * (W(-3) + W(3)) + h4 * (W(-4) + W(4)) +
                h5 * (W(-5) + W(5));
        }
        a[(long long)j * nv] = v;
    }
}

// pmlvars += dt*scrpml (step.f90:116)
template <typename T>
__global__ void pml_update_kernel(T* pml, const T* spml, T dt, long long n) {
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t < n) pml[t] = pml[t] + dt * spml[t];
}

// v_z (field fz of nf per slot) of each slot on its observation plane into
// the record buffer (dense planes) when the slot's clock is on the output cadence
template <typename T>
__global__ void record_kernel(const T* __restrict__ a, T* __restrict__ rec, const int* __restrict__ t0,
                              const int* __restrict__ time, int steps, int rec_max, long long FS, long long NP,
                              long long rec_ss, const int* __restrict__ plane, int nf, int fz) {
    const long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const int s = blockIdx.y;
    if (q >= NP) return;
    const int tl = *time - t0[s];
    if (tl < 0 || tl % steps != 0) return;
    const int r = tl / steps;
    if (r >= rec_max) return;
    rec[(long long)s * rec_ss + (long long)r * NP + q] = a[((long long)s * nf + fz) * FS + (long long)plane[q] * NP + q];
}

// ---- a step -------------------------------------------------------------------------

bool lines_cover(const sparc_ctx* c) { return line_ok(c->P.nx) && (c->P.ny == 1 || line_ok(c->P.ny)); }

// fields of source slots through the spectrum and a real multiplier (pt row:
// PT_DAMP or PT_HF), in place or not; gate: only the sources on a filter step
template <typename T>
int filter_fields(sparc_ctx* c, const LineList<T, T>& L, int nsrc, int row, const LineGate& gate) {
    typedef typename CplxOf<T>::type CT;
    MhdState& m = *c->mhd;
    const int nx = c->P.nx, ny = c->P.ny, nz = c->nz;
    const long long nrows = (long long)ny * nz;
    if constexpr (sizeof(T) == 4) {
        if (ny == 1) {
            for (int i0 = 0; i0 < L.n; i0 += 3) {         // m.spec holds three fields of a source
                LineList<float, float2> f;
                LineList<float2, float> h;
                f.n = h.n = std::min(3, L.n - i0);
                for (int i = 0; i < f.n; ++i) {
                    float2* sp = (float2*)m.spec + (size_t)i * c->fs;
                    f.in[i] = L.in[i0 + i]; f.out[i] = sp;
                    h.in[i] = sp; h.out[i] = L.out[i0 + i];
                }
                f.in_ss = L.in_ss; h.out_ss = L.out_ss;
                f.out_ss = h.in_ss = 3 * c->fs;
                rows2d_r2c(f, nsrc, nx, nrows, (float)(1.0 / (double)nx), (const float*)c->pt + (size_t)row * c->M, c->tw_x,
                           gate, c->stream);
                rows2d_c2r(h, nsrc, nx, nrows, (int)nrows, 0LL, c->tw_x, gate, c->stream);
                c->launches += 2;
            }
            return SPARC_OK;
        }
    }
    if (ny == 1) {      // one pass: the packed rows' filter, scaled by 1 / nx
        line_rows<T>(L, nsrc, nx, nrows, line_mul<T>((const T*)m.fx + (row == PT_HF ? nx : 0), true), c->tw_x, gate,
                     c->stream);
        c->launches++;
        return SPARC_OK;
    }
    LineList<T, CT> f;
    LineList<CT, CT> g;
    LineList<CT, T> h;
    f.n = g.n = h.n = L.n;
    for (int i = 0; i < L.n; ++i) {
        CT* sp = (CT*)m.spec + (size_t)i * c->fs;
        f.in[i] = L.in[i]; f.out[i] = sp;
        g.in[i] = g.out[i] = sp;
        h.in[i] = sp; h.out[i] = L.out[i];
    }
    f.in_ss = L.in_ss; h.out_ss = L.out_ss;
    f.out_ss = g.in_ss = g.out_ss = h.in_ss = 3 * c->fs;
    line_r2c<T>(f, nsrc, nx, nrows, (T)(1.0 / ((double)nx * ny)), c->tw_x, gate, c->stream);
    line_cols_filter<T>(g, nsrc, nx / 2 + 1, ny, nz, (const T*)c->pt + (size_t)row * c->M, c->tw_y, gate, c->stream);
    line_c2r<T>(h, nsrc, nx, ny, nrows, nz, 0LL, c->tw_x, gate, c->stream);
    c->launches += 3;
    return SPARC_OK;
}

template <typename T>
LineList<T, T> list_of(T* work, long long N, int wcount, std::initializer_list<std::pair<int, int>> io) {
    LineList<T, T> L;
    L.n = 0;
    L.in_ss = L.out_ss = (long long)wcount * N;
    for (const auto& p : io) {
        L.in[L.n] = work + (size_t)p.first * N;
        L.out[L.n++] = work + (size_t)p.second * N;
    }
    return L;
}

// DAMP_VELOCITY's terms of the listed velocity temporaries
template <typename T>
int damp_terms(sparc_ctx* c, const LineList<T, T>& L, int nsrc) {
    typedef typename CplxOf<T>::type CT;
    if (lines_cover(c)) return filter_fields<T>(c, L, nsrc, PT_DAMP, {});
    for (int s = 0; s < nsrc; ++s)
        for (int i = 0; i < L.n; ++i)
            c->launches += fft_filter_phys<T>(L.in[i] + s * L.in_ss, L.out[i] + s * L.out_ss, (CT*)c->mhd->spec,
                                              (CT*)c->tmp, c->P.nx, c->P.ny, c->nz, c->tw_x, c->tw_y, c->stream,
                                              (const T*)c->pt + (size_t)PT_DAMP * c->M);
    return SPARC_OK;
}

template <typename T, int FORM>
int stage(sparc_ctx* c, const StepArgs<T>& A, int S) {
    constexpr int WC = FORM == 8 ? (int)V8_COUNT : (int)MW_COUNT;
    const long long N = c->N;
    auto list = [&](std::initializer_list<std::pair<int, int>> io) { return list_of<T>(A.work, N, WC, io); };
    const dim3 pg(nb256(N), S);
    int rc;
    if (A.hs == 0) {
        temp_kernel<T, FORM><<<pg, 256, 0, c->stream>>>(A);
        c->launches++;
    }
    if constexpr (FORM == 8) {
        // the six ddxyz calls (pml.f90:106-116), all with bc 1
        if ((rc = mhd_ddx<T>(c, list({{V8_T1, V8_DVXDX}, {V8_F3, V8_DXF3}, {V8_T4, V8_GPX}, {V8_F2, V8_DXF2},
                                      {V8_T6, V8_DXBY}, {V8_T7, V8_DXBZ}}), S)) ||
            (rc = mhd_ddy<T>(c, list({{V8_T2, V8_DVYDY}, {V8_T4, V8_GPY}, {V8_F3, V8_DYF3}, {V8_T7, V8_DYBZ},
                                      {V8_T5, V8_DYBX}, {V8_F1, V8_DYF1}}), S)) ||
            (rc = mhd_ddz<T>(c, list({{V8_T3, V8_DVZDZ}, {V8_F1, V8_DZF1}, {V8_F2, V8_DZF2}, {V8_T5, V8_DZBX},
                                      {V8_T4, V8_GPZ}, {V8_T6, V8_DZBY}}), {{1, 1, 1, 1, 1, 1}}, S)))
            return rc;
        if (A.damp && (rc = damp_terms<T>(c, list({{V8_T1, V8_DMX}, {V8_T2, V8_DMY}, {V8_T3, V8_DMZ}}), S))) return rc;
        rhs8_kernel<T><<<pg, 256, 0, c->stream>>>(A);
        c->launches++;
    } else if constexpr (FORM == 18) {
        // d(xi_x)/dx and d(flux2)/dx, with the damping of v_x, v_z in the same launch where the line transforms cover it
        auto x1 = list({{MW_T0, MW_DX}, {MW_F2, MW_BZ}, {MW_T3, MW_DMX}, {MW_T5, MW_DMZ}});
        if (sizeof(T) == 8 && A.damp && lines_cover(c)) {
            LineMul<T> mul = line_mul<T>((const T*)c->mhd->rx);
            mul.mul[2] = mul.mul[3] = (const T*)c->mhd->fx;
            mul.real = 4 | 8;
            line_rows<T>(x1, S, c->P.nx, c->nz, mul, c->tw_x, {}, c->stream);
            c->launches++;
        } else {
            x1.n = 2;
            if ((rc = mhd_ddx<T>(c, x1, S))) return rc;
            if (A.damp && (rc = damp_terms<T>(c, list({{MW_T3, MW_DMX}, {MW_T5, MW_DMZ}}), S))) return rc;
        }
        // d(xi_z)/dz with bc 3, the top value -dxixdx(nz) * unstretch(nz) (physics2d.f90:731-733)
        const T unstr = (T)c->zt_host[(size_t)ZT_UNSTRETCH * c->nz + c->nz - 1];
        if ((rc = mhd_ddz<T>(c, list({{MW_T2, MW_Z0}, {MW_F2, MW_Z2}}), {{3, 0}}, S, A.work + (size_t)MW_DX * N, -unstr)))
            return rc;
        point_kernel<T, 18, 1><<<pg, 256, 0, c->stream>>>(A);
        if ((rc = mhd_ddx<T>(c, list({{MW_P, MW_GPX}, {MW_BZ, MW_DXBZ}}), S)) ||
            (rc = mhd_ddz<T>(c, list({{MW_P, MW_Z0}, {MW_BX, MW_Z1}}), {{2, 0}}, S)))
            return rc;
        point_kernel<T, 18, 2><<<pg, 256, 0, c->stream>>>(A);
        c->launches += 2;
    } else {
        // ddxyz(xi_x, xi_y, xi_z, bc 1), and the induction: ddxyz(flux3, by, flux3, bx, flux2, .),
        // ddxyz(flux2, bz, flux1, ., flux1, .)
        if ((rc = mhd_ddx<T>(c, list({{MW_T0, MW_DX}, {MW_F3, MW_BY}, {MW_F2, MW_BZ}}), S)) ||
            (rc = mhd_ddy<T>(c, list({{MW_T1, MW_DY}, {MW_F3, MW_BX}, {MW_F1, MW_DYF1}}), S)))
            return rc;
        if (A.damp && (rc = damp_terms<T>(c, list({{MW_T3, MW_DMX}, {MW_T4, MW_DMY}, {MW_T5, MW_DMZ}}), S))) return rc;
        if ((rc = mhd_ddz<T>(c, list({{MW_T2, MW_Z0}, {MW_F1, MW_Z1}, {MW_F2, MW_Z2}}), {{1, 1, 1}}, S))) return rc;
        point_kernel<T, 10, 1><<<pg, 256, 0, c->stream>>>(A);
        // grad p' and curl b: ddxyz(by, curlbz, bz, curlbx, bx, .), ddxyz(bz, curlby, bx, ., by, .)
        if ((rc = mhd_ddx<T>(c, list({{MW_P, MW_GPX}, {MW_BY, MW_DXBY}, {MW_BZ, MW_DXBZ}}), S)) ||
            (rc = mhd_ddy<T>(c, list({{MW_P, MW_GPY}, {MW_BZ, MW_DYBZ}, {MW_BX, MW_DYBX}}), S)) ||
            (rc = mhd_ddz<T>(c, list({{MW_P, MW_Z0}, {MW_BX, MW_Z1}, {MW_BY, MW_Z2}}), {{0, 1, 1}}, S)))
            return rc;
        point_kernel<T, 10, 2><<<pg, 256, 0, c->stream>>>(A);
        c->launches += 2;
    }
    CKL();
    return SPARC_OK;
}

template <typename T>
int enqueue_t(sparc_ctx* c, int nsteps) {
    typedef typename CplxOf<T>::type CT;
    MhdState& m = *c->mhd;
    const int S = c->active_n, opt = c->P.option, nz = c->nz;
    const bool two_d = opt == 18;
    StepArgs<T> A;
    memset(&A, 0, sizeof(A));
    A.N = c->N; A.NP = c->NP; A.FS = 2 * c->fs; A.nz = nz;
    A.nb = c->P.npmlbot; A.nt = c->P.npmltop; A.nzpml = std::max(c->nzpml, 1);
    A.both = opt != 10;
    A.bg = (const T*)m.bg; A.work = (T*)m.work; A.pab = (const T*)m.pab;
    A.pml = (const T*)m.pml; A.spml = (T*)m.spml;
    A.a = (const T*)c->a; A.scr = (T*)c->scr;
    A.g = (const T*)m.g; A.sponge = (const T*)m.sponge; A.zt = (const T*)c->zt;
    A.damp = c->P.damp_waves ? 1 : 0;
    A.adjoint = c->P.compute_adjoint ? 1 : 0;
    A.clk.t0 = c->d_t0; A.clk.time = c->d_time; A.clk.freq = c->freq_filtering; A.clk.two_d = two_d ? 1 : 0;
    A.clk.gate = c->forcing_length * c->cadforcing_step; A.clk.num_steps = c->num_steps;
    A.clk.ts = R4(c->P.timestep); A.clk.cad = R4(c->P.cadforcing);
    A.src_mode = c->src_mode;
    A.ksrc = (c->P.src_k > 0 ? c->P.src_k : c->e_rad) - 1;
    A.src = c->src_mode == 2 ? (const T*)m.src : (const T*)c->planes;
    A.src_ss = c->src_mode == 2 ? c->NP : (long long)c->src_L * c->NP;
    A.series = c->series; A.nseries = c->nseries;
    A.plane = m.plane; A.dw = (const T*)m.dw;
    // update: two neighbouring columns per thread in FP32, but not in 2-D, whose FP32
    // sums keep their order (rows2d_f32.cu)
    const int vw = sizeof(T) == 4 && !two_d ? 2 : 1;
    const long long unv = c->NP / vw;
    const int LP = z_pencils(nz, unv, c->nf * S, c->nsm), nth = LP * z_chunks(nz);
    const dim3 ug((unsigned)((unv + LP - 1) / LP), c->nf, S);
    const size_t usm = (size_t)nz * LP * vw * sizeof(T);
    LineGate gate;
    gate.on = 1;
    gate.clk = A.clk;
    for (int it = 0; it < nsteps; ++it) {
        if (c->src_mode == 2) {      // this step's planes; two neighbouring pixels as one complex value
            launch_source_plane<T>((CT*)m.src, (const CT*)c->planes, (long long)c->src_L * c->NP / 2, c->src_L, A.clk,
                                   (int)(c->NP / 2), 1, S, c->stream);
            c->launches++;
        }
        for (int rk = 0; rk < 5; ++rk) {
            A.beta = (T)c->betas[rk];
            A.beta_next = rk < 4 ? (T)c->betas[rk + 1] : (T)0;
            A.hs = rk > 0;
            A.last = rk == 4;
            const int rc = two_d ? stage<T, 18>(c, A, S) : (opt == 8 ? stage<T, 8>(c, A, S) : stage<T, 10>(c, A, S));
            if (rc) return rc;
        }
        if constexpr (sizeof(T) == 4) {
            if (!two_d)
                update_kernel<T, float2><<<ug, nth, usm, c->stream>>>((T*)c->a, (const T*)c->scr, A.FS, c->NP, nz, c->nf, LP,
                                                                      (T)c->deltat, 0);
        }
        if (vw == 1)
            update_kernel<T, T><<<ug, nth, usm, c->stream>>>((T*)c->a, (const T*)c->scr, A.FS, c->NP, nz, c->nf, LP,
                                                             (T)c->deltat, two_d ? 1 : 0);
        const long long npv = (long long)S * PV_COUNT * A.nzpml * c->NP;
        pml_update_kernel<T><<<nb256(npv), 256, 0, c->stream>>>((T*)m.pml, (const T*)m.spml, (T)c->deltat, npv);
        c->launches += 2;
        CKL();
        // horizontal filter every freq_filtering steps of each slot's clock:
        // 3-D on fields 1..5 when mod(time, 30) = 0 (physics.f90:791-830),
        // 2-D on all six when mod(time+1, 30) = 0 (physics2d.f90:566-584)
        const int nhf = two_d ? 6 : 5;
        if (lines_cover(c)) {
            for (int f0 = 0; f0 < nhf; f0 += two_d ? 6 : 3) {
                LineList<T, T> L;
                L.n = std::min(two_d ? 6 : 3, nhf - f0);
                L.in_ss = L.out_ss = (long long)c->nf * A.FS;
                for (int i = 0; i < L.n; ++i) L.in[i] = L.out[i] = (T*)c->a + (size_t)(f0 + i) * A.FS;
                const int rc = filter_fields<T>(c, L, S, PT_HF, gate);
                if (rc) return rc;
            }
        } else {
            for (int s = 0; s < S; ++s) {
                const int tl = c->time + it - c->t0[s];
                if (tl < 0 || (two_d ? (tl + 1) : tl) % c->freq_filtering != 0) continue;
                for (int f = 0; f < nhf; ++f) {
                    T* fp = (T*)c->a + ((size_t)s * c->nf + f) * A.FS;
                    c->launches += fft_filter_phys<T>(fp, fp, (CT*)m.spec, (CT*)c->tmp, c->P.nx, c->P.ny, nz, c->tw_x,
                                                      c->tw_y, c->stream, (const T*)c->pt + (size_t)PT_HF * c->M);
                }
            }
        }
        if (c->rec_on) {
            record_kernel<T><<<dim3(nb256(c->NP), S), 256, 0, c->stream>>>(
                (const T*)c->a, (T*)c->rec, c->d_t0, c->d_time, c->steps, c->rec_max, A.FS, c->NP,
                (long long)c->rec_max * 2 * c->M, m.plane_obs, c->nf, opt == 8 ? 3 : 5);
            c->launches++;
        }
        launch_tick(c->d_time, 1, c->stream);
        c->launches++;
        CKL();
    }
    return SPARC_OK;
}

}  // namespace

template <typename T>
int mhd_ddz(sparc_ctx* c, const LineList<T, T>& L, const ZCodes& codes, int nsrc, const T* topsrc, T topscale) {
    if constexpr (sizeof(T) == 4) {
        if (c->mhd->rows2d_z) {
            Compact<float> cc;
            cc.C1 = (float)c->cc64.C1; cc.C2 = (float)c->cc64.C2;
            for (int i = 0; i < 5; ++i) cc.Cb[i] = (float)c->cc64.Cb[i];
            for (int i = 0; i < 4; ++i) cc.Cf[i] = (float)c->cc64.Cf[i];
            cc.alpha2 = (float)c->cc64.alpha2; cc.beta1 = (float)c->cc64.beta1; cc.cnst = (float)c->cc64.cnst;
            rows2d_ddz(L, codes, nsrc, (const float*)c->zt, cc, c->NP, c->nz, topsrc, topscale, c->stream);
            c->launches++;
            CKL();
            return SPARC_OK;
        }
    }
    typedef typename std::conditional<sizeof(T) == 4, float2, T>::type V;
    const long long nv = c->NP / (long long)(sizeof(V) / sizeof(T));
    const int LP = z_pencils(c->nz, nv, L.n * nsrc, c->nsm), nth = LP * z_chunks(c->nz);
    zderiv_kernel<T, V><<<dim3((unsigned)((nv + LP - 1) / LP), L.n, nsrc), nth, 2 * nth * sizeof(V), c->stream>>>(
        L, codes, mhd_ztab<T>(c), c->nz, c->NP, LP, topsrc, topscale);
    c->launches++;
    CKL();
    return SPARC_OK;
}
template int mhd_ddz<double>(sparc_ctx*, const LineList<double, double>&, const ZCodes&, int, const double*, double);
template int mhd_ddz<float>(sparc_ctx*, const LineList<float, float>&, const ZCodes&, int, const float*, float);

int mhd_enqueue(sparc_ctx* c, int nsteps) { return c->f32 ? enqueue_t<float>(c, nsteps) : enqueue_t<double>(c, nsteps); }

bool mhd_graphs(const sparc_ctx* c) { return lines_cover(c); }

int mhd_ready(sparc_ctx* c) {
    if (c->mhd && c->mhd->have_bg) return SPARC_OK;
    return fail(c, SPARC_ESTATE, c->P.option == 18 ? "option 18 needs sparc_gpu_set_mhd2d_background"
                                                    : "options 8 and 10 need sparc_gpu_set_mhd_background");
}
