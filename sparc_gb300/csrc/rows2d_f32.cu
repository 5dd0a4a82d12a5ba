// Row transforms and z derivatives of the FP32 2-D forms (options 17 and 18,
// ny = 1).  After a source has acted, their FP32 results carry 1e-5 to 5e-5 of
// rounding (v_z in the top rows, where p' and the buoyancy cancel), so any other
// order of the sums moves the results by as much.  These kernels therefore keep
// one order of sums, whatever the line transforms and the z solver of the other
// forms do: a row of 64 or 256 points as two passes of radix-2 register DFTs
// (8 x 8, 16 x 16), any other as shared-memory Stockham radix-2, and the z solve
// on eight chunks whose carries are composed one after the other.
//
// All fields and sources of a list in one launch (grid.y, grid.z).  A 2-D grid
// holds a few hundred rows of 512 points at most: every kernel is bound by the
// latency of its launch and its passes.  Measured per step of option 18, 256x1x300:
// 0.75 ms (one source) and 1.66 ms (four) with a launch per field and source, 0.23
// and 0.26 ms here, 0.11 and 0.17 ms through the line transforms.
#include <algorithm>

#include "mhd.cuh"

namespace {

// in-register DFT of length R (decimation in frequency): on return v[brev(k)]
// holds X[k]; w[j] = W_R^j for j < R/2
template <int R>
__device__ __forceinline__ void reg_dft(float2 (&v)[R], const float2 (&w)[R / 2]) {
    #pragma unroll
    for (int len = R; len >= 2; len >>= 1) {
        const int half = len >> 1, step = R / len;
        #pragma unroll
        for (int b = 0; b < R; b += len) {
            #pragma unroll
            for (int k = 0; k < half; ++k) {
                const float2 a = v[b + k], c = v[b + k + half];
                v[b + k] = bsum(a, c);
                const float2 d = bdif(a, c);
                v[b + k + half] = (k == 0) ? d : cmul(d, w[k * step]);
            }
        }
    }
}

template <int R>
__host__ __device__ constexpr int brev(int k) {
    int r = 0;
    for (int b = 1, m = R >> 1; b < R; b <<= 1, m >>= 1)
        if (k & b) r |= m;
    return r;
}

template <int R>
__device__ __forceinline__ void twiddles(float2 (&w)[R / 2], const double* __restrict__ tw, float sign) {
    #pragma unroll
    for (int j = 0; j < R / 2; ++j) w[j] = tw_n<float, float2>(tw, j * R, R * R, sign);
}

// whether a gated launch leaves this source alone (the same for the whole CTA)
__device__ __forceinline__ bool gated_off(const LineGate& g) {
    return g.on && !slot_hfilter(g.clk, *g.clk.time - g.clk.t0[blockIdx.z]);
}

// A CTA's rows, two to a complex line: R = 8, 16: R*R points, R threads a line,
// 256 / R lines; R = 0: any size, one line.  z(i): point i of the packed line;
// out(i, value); the line's FFT of the given sign.
template <int R> struct Lines {
    float2* z;           // this thread's line (R: R rows of R + 1)
    int r, n;            // thread of the line; points
    long long r0;        // first of the two rows
    __device__ Lines(unsigned char* sm, int nx) {
        r = threadIdx.x % R;
        n = R * R;
        const int pp = threadIdx.x / R;
        z = (float2*)sm + pp * R * (R + 1);
        r0 = 2LL * ((long long)blockIdx.x * (256 / R) + pp);
    }
    // n = R n1 + n2 in registers -> k = r + R k2 in registers, v[brev(k2)]
    __device__ __forceinline__ void fft(float2 (&v)[R], const float2 (&w)[R / 2], float sign, const double* __restrict__ tw) {
        reg_dft<R>(v, w);
        #pragma unroll
        for (int k1 = 0; k1 < R; ++k1) {
            float2 y = v[brev<R>(k1)];
            if (k1 > 0 && r > 0) y = cmul(y, tw_n<float, float2>(tw, r * k1, R * R, sign));
            z[k1 * (R + 1) + r] = y;
        }
        __syncthreads();
        #pragma unroll
        for (int n2 = 0; n2 < R; ++n2) v[n2] = z[r * (R + 1) + n2];
        reg_dft<R>(v, w);
    }
};

template <int R>
__global__ void __launch_bounds__(256) rows_deriv_kernel(const LineList<float, float> L, int nx, long long nrows,
                                                         const float* __restrict__ mul, const double* __restrict__ tw) {
    extern __shared__ __align__(16) unsigned char smraw[];
    const float* in = L.in[blockIdx.y] + blockIdx.z * L.in_ss;
    float* out = L.out[blockIdx.y] + blockIdx.z * L.out_ss;
    if constexpr (R > 0) {
        Lines<R> l(smraw, nx);
        const int r = l.r, n = l.n;
        const long long r0 = l.r0, r1 = r0 + 1;
        const bool has0 = r0 < nrows, has1 = r1 < nrows;
        float2 wf[R / 2], wi[R / 2], v[R], u[R];
        twiddles<R>(wf, tw, -1.f);
        twiddles<R>(wi, tw, 1.f);
        #pragma unroll
        for (int n1 = 0; n1 < R; ++n1) {
            v[n1].x = has0 ? in[r0 * n + R * n1 + r] : 0.f;
            v[n1].y = has1 ? in[r1 * n + R * n1 + r] : 0.f;
        }
        l.fft(v, wf, -1.f, tw);
        __syncthreads();                                   // the tile is rewritten below
        #pragma unroll
        for (int k2 = 0; k2 < R; ++k2) {
            const float2 X = v[brev<R>(k2)];
            const float m = __ldg(&mul[r + R * k2]);
            u[k2].x = -m * X.y;
            u[k2].y = m * X.x;
        }
        l.fft(u, wi, 1.f, tw);                             // mirrored: ends where it began
        #pragma unroll
        for (int n1 = 0; n1 < R; ++n1) {
            const float2 y = u[brev<R>(n1)];
            if (has0) out[r0 * n + R * n1 + r] = y.x;
            if (has1) out[r1 * n + R * n1 + r] = y.y;
        }
    } else {
        float2* b0 = (float2*)smraw;
        float2* b1 = b0 + nx;
        const long long r0 = 2LL * blockIdx.x, r1 = r0 + 1;
        const bool has1 = r1 < nrows;
        for (int i = threadIdx.x; i < nx; i += blockDim.x) b0[i] = make_float2(in[r0 * nx + i], has1 ? in[r1 * nx + i] : 0.f);
        __syncthreads();
        float2* Z = smem_fft<float, float2>(b0, b1, nx, 1, -1.f, tw);
        for (int k = threadIdx.x; k < nx; k += blockDim.x) Z[k] = make_float2(-mul[k] * Z[k].y, mul[k] * Z[k].x);
        __syncthreads();
        float2* Y = smem_fft<float, float2>(Z, Z == b0 ? b1 : b0, nx, 1, 1.f, tw);
        for (int i = threadIdx.x; i < nx; i += blockDim.x) {
            out[r0 * nx + i] = Y[i].x;
            if (has1) out[r1 * nx + i] = Y[i].y;
        }
    }
}

// rows of nx reals -> rows of H = nx/2+1 complex, split by Hermitian symmetry,
// scaled, then times mul[k] if given
template <int R>
__global__ void __launch_bounds__(256) rows_r2c_kernel(const LineList<float, float2> L, int nx, long long nrows, float scale,
                                                       const float* __restrict__ mul, const double* __restrict__ tw,
                                                       const LineGate gate) {
    extern __shared__ __align__(16) unsigned char smraw[];
    if (gated_off(gate)) return;
    const float* in = L.in[blockIdx.y] + blockIdx.z * L.in_ss;
    float2* out = L.out[blockIdx.y] + blockIdx.z * L.out_ss;
    const int H = nx / 2 + 1;
    const float hs = 0.5f * scale;
    const float2* Z;
    long long r0;
    int k0, kstep;
    if constexpr (R > 0) {
        Lines<R> l(smraw, nx);
        const int r = l.r;
        r0 = l.r0;
        float2 w[R / 2], v[R];
        twiddles<R>(w, tw, -1.f);
        #pragma unroll
        for (int n1 = 0; n1 < R; ++n1) {
            v[n1].x = r0 < nrows ? in[r0 * nx + R * n1 + r] : 0.f;
            v[n1].y = r0 + 1 < nrows ? in[(r0 + 1) * nx + R * n1 + r] : 0.f;
        }
        l.fft(v, w, -1.f, tw);
        __syncthreads();                                   // the tile now takes the spectrum
        #pragma unroll
        for (int k2 = 0; k2 < R; ++k2) l.z[r + R * k2] = v[brev<R>(k2)];
        __syncthreads();
        Z = l.z;
        k0 = r;
        kstep = R;
    } else {
        float2* b0 = (float2*)smraw;
        r0 = 2LL * blockIdx.x;
        for (int i = threadIdx.x; i < nx; i += blockDim.x)
            b0[i] = make_float2(in[r0 * nx + i], r0 + 1 < nrows ? in[(r0 + 1) * nx + i] : 0.f);
        __syncthreads();
        Z = smem_fft<float, float2>(b0, b0 + nx, nx, 1, -1.f, tw);
        k0 = threadIdx.x;
        kstep = blockDim.x;
    }
    for (int k = k0; k < H; k += kstep) {
        const float2 zk = Z[k], zn = Z[(nx - k) & (nx - 1)];
        float2 x1 = make_float2((zk.x + zn.x) * hs, (zk.y - zn.y) * hs);
        float2 x2 = make_float2((zk.y + zn.y) * hs, -(zk.x - zn.x) * hs);
        if (mul) {
            x1 = mul[k] * x1;
            x2 = mul[k] * x2;
        }
        if (r0 < nrows) out[r0 * H + k] = x1;
        if (r0 + 1 < nrows) out[(r0 + 1) * H + k] = x2;
    }
}

// rows of H complex -> rows of nx reals, inverse, unscaled (DC and Nyquist
// imaginary parts dropped as FFTW c2r does); row r at (r / ppg) gstride + (r % ppg) H
template <int R>
__global__ void __launch_bounds__(256) rows_c2r_kernel(const LineList<float2, float> L, int nx, long long nrows, int ppg,
                                                       long long gstride, const double* __restrict__ tw, const LineGate gate) {
    extern __shared__ __align__(16) unsigned char smraw[];
    if (gated_off(gate)) return;
    const float2* in = L.in[blockIdx.y] + blockIdx.z * L.in_ss;
    float* out = L.out[blockIdx.y] + blockIdx.z * L.out_ss;
    const int H = nx / 2 + 1, half = nx / 2;
    const float2 zero = make_float2(0.f, 0.f);
    if constexpr (R > 0) {
        Lines<R> l(smraw, nx);
        const int r = l.r;
        const long long r0 = l.r0, r1 = r0 + 1;
        const bool has0 = r0 < nrows, has1 = r1 < nrows;
        const long long o0 = has0 ? grp_off(r0, ppg, gstride, H) : 0, o1 = has1 ? grp_off(r1, ppg, gstride, H) : 0;
        float2 w[R / 2], v[R];
        twiddles<R>(w, tw, 1.f);
        #pragma unroll
        for (int n1 = 0; n1 < R; ++n1) {
            const int idx = R * n1 + r;
            const bool mirror = idx > half;
            const int k = mirror ? R * R - idx : idx;
            const float2 x1 = has0 ? in[o0 + k] : zero, x2 = has1 ? in[o1 + k] : zero;
            if (k == 0 || k == half) v[n1] = make_float2(x1.x, x2.x);
            else if (!mirror) v[n1] = make_float2(x1.x - x2.y, x1.y + x2.x);
            else v[n1] = make_float2(x1.x + x2.y, -x1.y + x2.x);
        }
        l.fft(v, w, 1.f, tw);
        #pragma unroll
        for (int k2 = 0; k2 < R; ++k2) {
            const float2 zz = v[brev<R>(k2)];
            if (has0) out[r0 * nx + r + R * k2] = zz.x;
            if (has1) out[r1 * nx + r + R * k2] = zz.y;
        }
    } else {
        float2* b0 = (float2*)smraw;
        const long long r0 = 2LL * blockIdx.x, r1 = r0 + 1;
        const bool has1 = r1 < nrows;
        const long long o0 = grp_off(r0, ppg, gstride, H), o1 = has1 ? grp_off(r1, ppg, gstride, H) : 0;
        for (int k = threadIdx.x; k <= half; k += blockDim.x) {
            const float2 x1 = in[o0 + k], x2 = has1 ? in[o1 + k] : zero;
            if (k == 0 || k == half) {
                b0[k] = make_float2(x1.x, x2.x);
            } else {
                b0[k] = make_float2(x1.x - x2.y, x1.y + x2.x);
                b0[nx - k] = make_float2(x1.x + x2.y, -x1.y + x2.x);
            }
        }
        __syncthreads();
        const float2* Z = smem_fft<float, float2>(b0, b0 + nx, nx, 1, 1.f, tw);
        for (int i = threadIdx.x; i < nx; i += blockDim.x) {
            out[r0 * nx + i] = Z[i].x;
            if (has1) out[r1 * nx + i] = Z[i].y;
        }
    }
}

int radix(int n) { return n == 256 ? 16 : n == 64 ? 8 : 0; }

// launch shape: line pairs per CTA, threads, shared memory
struct Shape { unsigned x, thr; size_t sm; };
Shape shape(int nx, long long nrows) {
    const int R = radix(nx);
    const long long pairs = (nrows + 1) / 2;
    if (R) return {(unsigned)((pairs + 256 / R - 1) / (256 / R)), 256, (size_t)256 * (R + 1) * sizeof(float2)};
    return {(unsigned)pairs, (unsigned)std::min(std::max(nx / 2, 32), 256), 2 * (size_t)nx * sizeof(float2)};
}

// ---- d/dz --------------------------------------------------------------------------

constexpr int NCH = 8;      // chunks of a pencil, one warp each
// bytes of the five coefficient tables, rounded up so the float2 buffers after them are 8-byte aligned
__host__ __device__ inline size_t tables_bytes(int nz) { return (((size_t)5 * nz + 1) * 4 + 15) & ~(size_t)15; }
size_t chunk_bytes(int nz) {
    const int cs = (nz + NCH - 1) / NCH;
    return tables_bytes(nz) + (size_t)NCH * 32 * (8 + 4) + (size_t)NCH * (cs + 4) * 32 * 8;
}

// DBYD2's right-hand side of row j (0-based) for boundary code bc (the rows of
// compact_forward): interior 6th-order stencil, 5th-order rows 1 and nz-2,
// the bc-dependent closures of rows 0 and nz-1 (caller-set 0 / top for bc 2 / 3)
template <typename Ld>
__device__ __forceinline__ float rhs_of(int j, int nz, int bc, Ld B, float top, const Compact<float>& c) {
    if (j == 1 || j == 0) {
        const float R1 = c.Cb[0] * B(0) + c.Cb[1] * B(1) + c.Cb[2] * B(2) + c.Cb[3] * B(3) + c.Cb[4] * B(4);
        if (j == 1) return R1;
        if (bc == 0 || bc == 2) return 0.f;
        const float R0 = c.Cf[0] * B(0) + c.Cf[1] * B(1) + c.Cf[2] * B(2) + c.Cf[3] * B(3);
        return (c.alpha2 * R0 - c.beta1 * R1) * c.cnst;
    }
    const float Rn2 = -(c.Cb[0] * B(nz - 1) + c.Cb[1] * B(nz - 2) + c.Cb[2] * B(nz - 3) + c.Cb[3] * B(nz - 4) +
                        c.Cb[4] * B(nz - 5));
    if (j == nz - 2) return Rn2;
    if (bc == 0) return 0.f;
    if (bc == 3) return top;
    const float Rn1 = -(c.Cf[0] * B(nz - 1) + c.Cf[1] * B(nz - 2) + c.Cf[2] * B(nz - 3) + c.Cf[3] * B(nz - 4));
    return (c.alpha2 * Rn1 - c.beta1 * Rn2) * c.cnst;
}

// d/dz of dense fields (DBYD2 * stretch) by chunks: 64 pencils per CTA (two
// neighbours per lane, as paired FP32), NCH warps, warp w owning planes
// [w*cs, w*cs + cs).  Forward elimination y_j = (R_j - low_j y_{j-1}) ibd_j is
// affine in y_{j-1}: each warp eliminates its chunk from zero (y'), keeping the
// product of the multipliers -low_j ibd_j, and after one barrier adds the
// carry-in composed from the chunks below.  The back substitution x_j = y_j -
// gam_{j+1} x_{j+1} runs the same way from the top.  Each warp stages its chunk
// and two halo planes either side in its own rows of shared memory (row i =
// plane s-2+i); the input is read once and the result written once.
__global__ void __launch_bounds__(32 * NCH) ddz_kernel(const LineList<float, float> L, const ZCodes codes,
                                                       const float* __restrict__ zt, Compact<float> cc, long long npix,
                                                       int nz, const float* __restrict__ topsrc, float topscale) {
    extern __shared__ __align__(16) unsigned char smraw[];
    const int bc = codes.bc[blockIdx.y];
    const float* in = L.in[blockIdx.y] + blockIdx.z * L.in_ss;
    float* out = L.out[blockIdx.y] + blockIdx.z * L.out_ss;
    const int cs = (nz + NCH - 1) / NCH, rows = cs + 4;
    float* tmf = (float*)smraw;              // [nz] -low_j ibd_j
    float* tib = tmf + nz;                   // [nz] ibd_j
    float* tlo = tib + nz;                   // [nz] low_j
    float* tga = tlo + nz;                   // [nz+1] gam_j (gam_nz = 0)
    float* tst = tga + nz + 1;               // [nz] stretch_j
    float2* Cy = (float2*)(smraw + tables_bytes(nz));   // [NCH][32] chunk-end values
    float* Cp = (float*)(Cy + NCH * 32);     // [NCH][32] chunk multiplier products
    float2* Yall = (float2*)(Cp + NCH * 32); // [NCH][rows][32]
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    {
        const float* low = zt + (ZT_TH + 3 * bc) * nz;
        const float* ibd = zt + (ZT_TH + 3 * bc + 1) * nz;
        const float* gam = zt + (ZT_TH + 3 * bc + 2) * nz;
        for (int j = threadIdx.x; j <= nz; j += blockDim.x) {
            if (j < nz) {
                const float l = j > 0 ? low[j] : 0.f, ib = ibd[j];
                tlo[j] = l;
                tib[j] = ib;
                tmf[j] = -l * ib;
                tst[j] = zt[ZT_STRETCH * nz + j];
            }
            tga[j] = (j > 0 && j < nz) ? gam[j] : 0.f;
        }
    }
    float2* Y = Yall + (long long)w * rows * 32 + lane;   // Y[i * 32] = plane s - 2 + i
    const long long m = (long long)blockIdx.x * 64 + 2 * lane;
    const bool on = m < npix;                             // npix even: both pencils or neither
    const float* b = in + (on ? m : 0);
    float* o = out + m;
    const int s = w * cs, e = min(nz, s + cs) - 1;        // empty chunk when s > e
    auto B = [&](int j) -> float2 { return *(const float2*)(b + (long long)j * npix); };
    float2 top = make_float2(0.f, 0.f);
    if (bc == 3 && on) {
        const float2 tv = *(const float2*)(topsrc + blockIdx.z * L.in_ss + (long long)(nz - 1) * npix + m);
        top = pmul(bc2(topscale), tv);
    }
    if (s <= e) {
        for (int i = 0; i < e - s + 5; ++i) {
            const int j = s - 2 + i;
            if (j >= 0 && j < nz) {
                const unsigned dst = (unsigned)__cvta_generic_to_shared(Y + i * 32);
                const float* src = b + (long long)j * npix;
                asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(dst), "l"(src) : "memory");
            } else {
                Y[i * 32] = make_float2(0.f, 0.f);
            }
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
        asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    }
    __syncthreads();
    // the closures, from the staged planes (before the forward pass overwrites
    // them) or, outside this chunk's staged range, from global memory
    auto Bs = [&](int j) -> float2 { return (j >= s - 2 && j <= e + 2) ? Y[(j - s + 2) * 32] : B(j); };
    auto rhs_row = [&](int j) -> float2 {
        return make_float2(rhs_of(j, nz, bc, [&](int k) { return Bs(k).x; }, top.x, cc),
                           rhs_of(j, nz, bc, [&](int k) { return Bs(k).y; }, top.y, cc));
    };
    const float2 Z2 = make_float2(0.f, 0.f);
    float2 Rlo0 = Z2, Rlo1 = Z2, Rhi2 = Z2, Rhi1 = Z2;
    if (s <= e && s <= 1) { Rlo0 = rhs_row(0); Rlo1 = rhs_row(1); }
    if (s <= e && e >= nz - 2) { Rhi2 = rhs_row(nz - 2); Rhi1 = rhs_row(nz - 1); }
    const float2 C1p = bc2(cc.C1), C2p = bc2(cc.C2);
    float2 y = Z2;
    float pr = 1.f;
    if (s <= e) {
        float2 wm2 = Y[0], wm1 = Y[32], w0 = Y[64], w1 = Y[96], w2 = Y[128];
        for (int j = s, i = 2; j <= e; ++j, ++i) {
            float2 R;
            if (j >= 2 && j <= nz - 3) R = pfma(C2p, psub(w2, wm2), pmul(C1p, psub(w1, wm1)));
            else R = j == 0 ? Rlo0 : (j == 1 ? Rlo1 : (j == nz - 2 ? Rhi2 : Rhi1));
            y = pmul(bc2(tib[j]), pfma(bc2(-tlo[j]), y, R));
            pr = pr * tmf[j];
            wm2 = wm1; wm1 = w0; w0 = w1; w1 = w2;
            if (j < e) w2 = Y[(i + 3) * 32];
            Y[i * 32] = y;
        }
    }
    Cy[w * 32 + lane] = y;
    Cp[w * 32 + lane] = pr;
    __syncthreads();
    float2 cin = Z2;
    for (int q = 0; q < w; ++q) cin = pfma(bc2(Cp[q * 32 + lane]), cin, Cy[q * 32 + lane]);
    float2 x = Z2;
    pr = 1.f;
    if (s <= e) {
        if (w > 0) {
            float pj = 1.f;
            for (int j = s, i = 2; j <= e; ++j, ++i) {
                pj = pj * tmf[j];
                Y[i * 32] = pfma(bc2(pj), cin, Y[i * 32]);
            }
        }
        for (int j = e, i = e - s + 2; j >= s; --j, --i) {
            const float g = tga[j + 1];
            x = pfma(bc2(-g), x, Y[i * 32]);
            pr = pr * (-g);
            Y[i * 32] = x;
        }
    }
    __syncthreads();                         // all chunk-end values of the forward pass are read
    Cy[w * 32 + lane] = x;                   // x' at the chunk's first plane
    Cp[w * 32 + lane] = pr;
    __syncthreads();
    float2 xin = Z2;
    for (int q = NCH - 1; q > w; --q) xin = pfma(bc2(Cp[q * 32 + lane]), xin, Cy[q * 32 + lane]);
    if (s <= e && on) {
        float pj = 1.f;
        for (int j = e, i = e - s + 2; j >= s; --j, --i) {
            pj = pj * (-tga[j + 1]);
            *(float2*)(o + (long long)j * npix) = pmul(bc2(tst[j]), pfma(bc2(pj), xin, Y[i * 32]));
        }
    }
}

}  // namespace

void rows2d_deriv(const LineList<float, float>& L, int nsrc, int nx, long long nrows, const float* mul, const double* tw,
                  cudaStream_t s) {
    const Shape h = shape(nx, nrows);
    const dim3 g(h.x, L.n, nsrc);
    if (radix(nx) == 16) rows_deriv_kernel<16><<<g, h.thr, h.sm, s>>>(L, nx, nrows, mul, tw);
    else if (radix(nx) == 8) rows_deriv_kernel<8><<<g, h.thr, h.sm, s>>>(L, nx, nrows, mul, tw);
    else rows_deriv_kernel<0><<<g, h.thr, h.sm, s>>>(L, nx, nrows, mul, tw);
}

void rows2d_r2c(const LineList<float, float2>& L, int nsrc, int nx, long long nrows, float scale, const float* mul,
                const double* tw, const LineGate& gate, cudaStream_t s) {
    const Shape h = shape(nx, nrows);
    const dim3 g(h.x, L.n, nsrc);
    if (radix(nx) == 16) rows_r2c_kernel<16><<<g, h.thr, h.sm, s>>>(L, nx, nrows, scale, mul, tw, gate);
    else if (radix(nx) == 8) rows_r2c_kernel<8><<<g, h.thr, h.sm, s>>>(L, nx, nrows, scale, mul, tw, gate);
    else rows_r2c_kernel<0><<<g, h.thr, h.sm, s>>>(L, nx, nrows, scale, mul, tw, gate);
}

void rows2d_c2r(const LineList<float2, float>& L, int nsrc, int nx, long long nrows, int ppg, long long gstride,
                const double* tw, const LineGate& gate, cudaStream_t s) {
    const Shape h = shape(nx, nrows);
    const dim3 g(h.x, L.n, nsrc);
    if (radix(nx) == 16) rows_c2r_kernel<16><<<g, h.thr, h.sm, s>>>(L, nx, nrows, ppg, gstride, tw, gate);
    else if (radix(nx) == 8) rows_c2r_kernel<8><<<g, h.thr, h.sm, s>>>(L, nx, nrows, ppg, gstride, tw, gate);
    else rows_c2r_kernel<0><<<g, h.thr, h.sm, s>>>(L, nx, nrows, ppg, gstride, tw, gate);
}

// pencils that fit the kernel's shared memory (about 700 levels; taller ones go through mhd_ddz's own solver)
bool rows2d_ddz_ok(int nz) {
    return chunk_bytes(nz) <= 200 * 1024 && allow_shared_memory((const void*)ddz_kernel);
}

void rows2d_ddz(const LineList<float, float>& L, const ZCodes& codes, int nsrc, const float* zt, const Compact<float>& cc,
                long long npix, int nz, const float* topsrc, float topscale, cudaStream_t s) {
    ddz_kernel<<<dim3((unsigned)((npix + 63) / 64), L.n, nsrc), 32 * NCH, chunk_bytes(nz), s>>>(L, codes, zt, cc, npix, nz,
                                                                                               topsrc, topscale);
}
