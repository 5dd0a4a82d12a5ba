// Kernels of lines.cuh for one element type; lines_f32.cu and lines_f64.cu
// instantiate them (two translation units, compiled in parallel).
#include <algorithm>

#include "lines.cuh"

namespace {

// ---- register DFTs -------------------------------------------------------------

// cos(2 pi j / 32), j = 0..8
__device__ constexpr double COS32[9] = {1.0, 0.98078528040323044913, 0.92387953251128675613, 0.83146961230254523708,
                                        0.70710678118654752440, 0.55557023301960222474, 0.38268343236508977173,
                                        0.19509032201612826785, 0.0};
__host__ __device__ constexpr double cos32(int j) {
    j &= 31;
    return j <= 8 ? COS32[j] : j <= 16 ? -COS32[16 - j] : j <= 24 ? -COS32[j - 16] : COS32[32 - j];
}

// v times exp(-+ 2 pi i J / 32) (the upper sign forward), J a constant
template <int J, bool INV, typename T, typename CT>
__device__ __forceinline__ CT rot(CT v) {
    constexpr int j = (INV ? -J : J) & 31;            // v * (cos - i sin) of 2 pi j / 32
    CT r;
    if constexpr (j == 0) return v;
    else if constexpr (j == 8) { r.x = v.y; r.y = -v.x; return r; }
    else if constexpr (j == 16) { r.x = -v.x; r.y = -v.y; return r; }
    else if constexpr (j == 24) { r.x = -v.y; r.y = v.x; return r; }
    else {
        constexpr T c = (T)cos32(j), s = (T)cos32(j - 8);     // sin(a) = cos(a - pi/2)
        if constexpr (j == 4 || j == 28) {                     // (1 -+ i) / sqrt 2
            const CT w = v;
            if constexpr (j == 4) { r.x = c * (w.x + w.y); r.y = c * (w.y - w.x); }
            else { r.x = c * (w.x - w.y); r.y = c * (w.y + w.x); }
        } else {
            r.x = fma(c, v.x, s * v.y);
            r.y = fma(c, v.y, -s * v.x);
        }
        return r;
    }
}

template <bool INV, typename CT>
__device__ __forceinline__ void dft4(CT& a, CT& b, CT& c, CT& d) {
    const CT s0 = bsum(a, c), d0 = bdif(a, c), s1 = bsum(b, d), d1 = bdif(b, d);
    CT e;                                              // -+ i d1
    if (INV) { e.x = -d1.y; e.y = d1.x; } else { e.x = d1.y; e.y = -d1.x; }
    a = bsum(s0, s1);
    c = bdif(s0, s1);
    b = bsum(d0, e);
    d = bdif(d0, e);
}

// in place, natural order
template <typename T, typename CT, bool INV> __device__ __forceinline__ void dft(CT (&v)[4]) { dft4<INV>(v[0], v[1], v[2], v[3]); }
template <typename T, typename CT, bool INV> __device__ __forceinline__ void dft(CT (&v)[8]) {
    dft4<INV>(v[0], v[2], v[4], v[6]);
    dft4<INV>(v[1], v[3], v[5], v[7]);
    const CT o1 = rot<4, INV, T>(v[3]), o2 = rot<8, INV, T>(v[5]), o3 = rot<12, INV, T>(v[7]);
    const CT e0 = v[0], e1 = v[2], e2 = v[4], e3 = v[6], o0 = v[1];
    v[0] = bsum(e0, o0); v[4] = bdif(e0, o0);
    v[1] = bsum(e1, o1); v[5] = bdif(e1, o1);
    v[2] = bsum(e2, o2); v[6] = bdif(e2, o2);
    v[3] = bsum(e3, o3); v[7] = bdif(e3, o3);
}
template <typename T, typename CT, bool INV> __device__ __forceinline__ void dft(CT (&v)[16]) {
    // n = 4 n1 + n2, k = k1 + 4 k2
    #pragma unroll
    for (int n2 = 0; n2 < 4; ++n2) dft4<INV>(v[n2], v[4 + n2], v[8 + n2], v[12 + n2]);     // v[4 k1 + n2]
    v[5] = rot<2, INV, T>(v[5]);   v[6] = rot<4, INV, T>(v[6]);    v[7] = rot<6, INV, T>(v[7]);
    v[9] = rot<4, INV, T>(v[9]);   v[10] = rot<8, INV, T>(v[10]);  v[11] = rot<12, INV, T>(v[11]);
    v[13] = rot<6, INV, T>(v[13]); v[14] = rot<12, INV, T>(v[14]); v[15] = rot<18, INV, T>(v[15]);
    #pragma unroll
    for (int k1 = 0; k1 < 4; ++k1) dft4<INV>(v[4 * k1], v[4 * k1 + 1], v[4 * k1 + 2], v[4 * k1 + 3]);   // v[4 k1 + k2]
    #pragma unroll
    for (int a = 0; a < 4; ++a)
        #pragma unroll
        for (int b = a + 1; b < 4; ++b) {
            const CT x = v[4 * a + b];
            v[4 * a + b] = v[4 * b + a];
            v[4 * b + a] = x;
        }
}
template <int N2, typename T, typename CT, bool INV> __device__ __forceinline__ void rot32(CT (&a)[8]) {
    a[1] = rot<N2, INV, T>(a[1]);     a[2] = rot<2 * N2, INV, T>(a[2]); a[3] = rot<3 * N2, INV, T>(a[3]);
    a[4] = rot<4 * N2, INV, T>(a[4]); a[5] = rot<5 * N2, INV, T>(a[5]); a[6] = rot<6 * N2, INV, T>(a[6]);
    a[7] = rot<7 * N2, INV, T>(a[7]);
}
template <typename T, typename CT, bool INV> __device__ __forceinline__ void dft(CT (&v)[32]) {
    // n = 4 n1 + n2 (n1 < 8), k = k1 + 8 k2
    CT a[4][8];
    #pragma unroll
    for (int n2 = 0; n2 < 4; ++n2) {
        #pragma unroll
        for (int n1 = 0; n1 < 8; ++n1) a[n2][n1] = v[4 * n1 + n2];
        dft<T, CT, INV>(a[n2]);
    }
    rot32<1, T, CT, INV>(a[1]);
    rot32<2, T, CT, INV>(a[2]);
    rot32<3, T, CT, INV>(a[3]);
    #pragma unroll
    for (int k1 = 0; k1 < 8; ++k1) {
        dft4<INV>(a[0][k1], a[1][k1], a[2][k1], a[3][k1]);
        #pragma unroll
        for (int k2 = 0; k2 < 4; ++k2) v[k1 + 8 * k2] = a[k2][k1];
    }
}

// ---- a line on TL threads --------------------------------------------------------

template <int N> struct Plan {
    static constexpr int R1 = N >= 512 ? 32 : N >= 128 ? 16 : N >= 32 ? 8 : 4, R2 = N / R1, TL = R2, G = R1 / R2;
};

// times W_N^(-+ q), q < N
template <bool INV, int N, typename T, typename CT>
__device__ __forceinline__ CT twid(CT v, int q, const double* __restrict__ tw) {
    return cmul(v, tw_n<T, CT>(tw, q, N, INV ? (T)1 : (T)-1));
}

// v[n1] = x[R2 n1 + t]  ->  v[g R2 + k2] = X[(t + R2 g) + R1 k2]; zs(k1, n2) the
// line's exchange cells.  One barrier inside; the caller puts one before the
// cells are written again.
template <bool INV, int N, typename T, typename CT, typename ZS>
__device__ __forceinline__ void line_pass(CT (&v)[Plan<N>::R1], int t, ZS zs, const double* __restrict__ tw) {
    typedef Plan<N> P;
    dft<T, CT, INV>(v);
    #pragma unroll
    for (int k1 = 0; k1 < P::R1; ++k1) zs(k1, t) = k1 > 0 ? twid<INV, N, T>(v[k1], t * k1, tw) : v[k1];
    __syncthreads();
    #pragma unroll
    for (int g = 0; g < P::G; ++g) {
        CT w[P::R2];
        #pragma unroll
        for (int n2 = 0; n2 < P::R2; ++n2) w[n2] = zs(t + P::R2 * g, n2);
        dft<T, CT, INV>(w);
        #pragma unroll
        for (int k2 = 0; k2 < P::R2; ++k2) v[g * P::R2 + k2] = w[k2];
    }
}
// the mirrored form: v[g R2 + k2] = X[(t + R2 g) + R1 k2]  ->  v[n1] = x[R2 n1 + t]
template <bool INV, int N, typename T, typename CT, typename ZS>
__device__ __forceinline__ void line_mirror(CT (&v)[Plan<N>::R1], int t, ZS zs, const double* __restrict__ tw) {
    typedef Plan<N> P;
    #pragma unroll
    for (int g = 0; g < P::G; ++g) {
        CT w[P::R2];
        #pragma unroll
        for (int k2 = 0; k2 < P::R2; ++k2) w[k2] = v[g * P::R2 + k2];
        dft<T, CT, INV>(w);
        const int k1 = t + P::R2 * g;
        #pragma unroll
        for (int n2 = 0; n2 < P::R2; ++n2) zs(k1, n2) = n2 > 0 ? twid<INV, N, T>(w[n2], n2 * k1, tw) : w[n2];
    }
    __syncthreads();
    #pragma unroll
    for (int k1 = 0; k1 < P::R1; ++k1) v[k1] = zs(k1, t);
    dft<T, CT, INV>(v);
}

// whether a gated launch leaves this source alone (the same for the whole CTA)
__device__ __forceinline__ bool gated_off(const LineGate& g) {
    return g.on && !slot_hfilter(g.clk, *g.clk.time - g.clk.t0[blockIdx.z]);
}

// ---- kernels ---------------------------------------------------------------------

// forward, i mul (or mul), inverse of rows of N reals, two rows packed as the
// real and imaginary part of a line: both multipliers act on the parts separately
// KIND 0: all fields derivatives; 1: all filters; 2: some of each
template <typename T, int N, int KIND>
__global__ void __launch_bounds__(256) rows_kernel(const LineList<T, T> L, long long nrows, const LineMul<T> M,
                                                   const double* __restrict__ tw, const LineGate gate) {
    typedef typename CplxOf<T>::type CT;
    typedef Plan<N> P;
    extern __shared__ __align__(16) unsigned char smraw[];
    if (gated_off(gate)) return;
    const int t = threadIdx.x % P::TL, pp = threadIdx.x / P::TL;
    CT* Z = (CT*)smraw + pp * P::R1 * (P::R2 + 1);
    auto zs = [&](int k1, int n2) -> CT& { return Z[k1 * (P::R2 + 1) + n2]; };
    const T* in = L.in[blockIdx.y] + blockIdx.z * L.in_ss;
    T* out = L.out[blockIdx.y] + blockIdx.z * L.out_ss;
    const T* __restrict__ mul = M.mul[blockIdx.y];
    const bool real = KIND == 2 ? (M.real >> blockIdx.y) & 1 : KIND == 1;
    const long long r0 = 2LL * ((long long)blockIdx.x * (blockDim.x / P::TL) + pp), r1 = r0 + 1;
    const bool has0 = r0 < nrows, has1 = r1 < nrows;
    CT v[P::R1];
    #pragma unroll
    for (int n1 = 0; n1 < P::R1; ++n1) {
        v[n1].x = has0 ? in[r0 * N + P::R2 * n1 + t] : (T)0;
        v[n1].y = has1 ? in[r1 * N + P::R2 * n1 + t] : (T)0;
    }
    line_pass<false, N, T>(v, t, zs, tw);
    __syncthreads();
    #pragma unroll
    for (int g = 0; g < P::G; ++g)
        #pragma unroll
        for (int k2 = 0; k2 < P::R2; ++k2) {
            const T m = __ldg(&mul[t + P::R2 * g + P::R1 * k2]);
            const CT X = v[g * P::R2 + k2];
            v[g * P::R2 + k2].x = m * (real ? X.x : -X.y);
            v[g * P::R2 + k2].y = m * (real ? X.y : X.x);
        }
    line_mirror<true, N, T>(v, t, zs, tw);
    #pragma unroll
    for (int n1 = 0; n1 < P::R1; ++n1) {
        if (has0) out[r0 * N + P::R2 * n1 + t] = v[n1].x;
        if (has1) out[r1 * N + P::R2 * n1 + t] = v[n1].y;
    }
}

// d/dy of dense (N, nx) planes: NC pairs of adjacent columns per CTA, a pair
// read and written as one complex value
template <typename T, int N, int NC>
__global__ void __launch_bounds__(256) cols_deriv_kernel(const LineList<T, T> L, int nx, const T* __restrict__ mul,
                                                         const double* __restrict__ tw) {
    typedef typename CplxOf<T>::type CT;
    typedef Plan<N> P;
    extern __shared__ __align__(16) unsigned char smraw[];
    CT* Z = (CT*)smraw;
    const int npair = nx / 2, ntile = (npair + NC - 1) / NC;
    const long long plane = blockIdx.x / ntile;
    const int c = threadIdx.x % NC, t = threadIdx.x / NC;
    const int cp = (blockIdx.x % ntile) * NC + c;
    const bool cv = cp < npair;
    auto zs = [&](int k1, int n2) -> CT& { return Z[(k1 * P::R2 + n2) * NC + c]; };
    const CT* src = (const CT*)(L.in[blockIdx.y] + blockIdx.z * L.in_ss + plane * (long long)N * nx) + cp;
    CT* dst = (CT*)(L.out[blockIdx.y] + blockIdx.z * L.out_ss + plane * (long long)N * nx) + cp;
    CT v[P::R1];
    #pragma unroll
    for (int n1 = 0; n1 < P::R1; ++n1) v[n1] = cv ? src[(long long)(P::R2 * n1 + t) * npair] : czero<CT>();
    line_pass<false, N, T>(v, t, zs, tw);
    __syncthreads();
    #pragma unroll
    for (int g = 0; g < P::G; ++g)
        #pragma unroll
        for (int k2 = 0; k2 < P::R2; ++k2) v[g * P::R2 + k2] = imul(__ldg(&mul[t + P::R2 * g + P::R1 * k2]), v[g * P::R2 + k2]);
    line_mirror<true, N, T>(v, t, zs, tw);
    if (cv) {
        #pragma unroll
        for (int n1 = 0; n1 < P::R1; ++n1) dst[(long long)(P::R2 * n1 + t) * npair] = v[n1];
    }
}

// two real rows packed as one complex line, split by Hermitian symmetry
template <typename T, int N>
__global__ void __launch_bounds__(256) r2c_kernel(const LineList<T, typename CplxOf<T>::type> L, long long nrows,
                                                  T scale, const double* __restrict__ tw, const LineGate gate) {
    typedef typename CplxOf<T>::type CT;
    typedef Plan<N> P;
    constexpr int H = N / 2 + 1;
    extern __shared__ __align__(16) unsigned char smraw[];
    if (gated_off(gate)) return;
    const int t = threadIdx.x % P::TL, pp = threadIdx.x / P::TL;
    CT* Z = (CT*)smraw + pp * P::R1 * (P::R2 + 1);
    auto zs = [&](int k1, int n2) -> CT& { return Z[k1 * (P::R2 + 1) + n2]; };
    const T* in = L.in[blockIdx.y] + blockIdx.z * L.in_ss;
    CT* out = L.out[blockIdx.y] + blockIdx.z * L.out_ss;
    const long long r0 = 2LL * ((long long)blockIdx.x * (blockDim.x / P::TL) + pp), r1 = r0 + 1;
    const bool has0 = r0 < nrows, has1 = r1 < nrows;
    CT v[P::R1];
    #pragma unroll
    for (int n1 = 0; n1 < P::R1; ++n1) {
        v[n1].x = has0 ? in[r0 * N + P::R2 * n1 + t] : (T)0;
        v[n1].y = has1 ? in[r1 * N + P::R2 * n1 + t] : (T)0;
    }
    line_pass<false, N, T>(v, t, zs, tw);
    __syncthreads();                                     // the cells now take the spectrum, in natural order
    #pragma unroll
    for (int g = 0; g < P::G; ++g)
        #pragma unroll
        for (int k2 = 0; k2 < P::R2; ++k2) Z[t + P::R2 * g + P::R1 * k2] = v[g * P::R2 + k2];
    __syncthreads();
    const T hs = (T)0.5 * scale;
    for (int k = t; k < H; k += P::TL) {
        const CT zk = Z[k], zn = Z[(N - k) & (N - 1)];
        CT x1, x2;
        x1.x = (zk.x + zn.x) * hs;
        x1.y = (zk.y - zn.y) * hs;
        x2.x = (zk.y + zn.y) * hs;
        x2.y = -(zk.x - zn.x) * hs;
        if (has0) out[r0 * H + k] = x1;
        if (has1) out[r1 * H + k] = x2;
    }
}

// two half-spectrum rows packed, inverse (FFTW c2r semantics: the imaginary
// parts of DC and Nyquist are dropped)
template <typename T, int N>
__global__ void __launch_bounds__(256) c2r_kernel(const LineList<typename CplxOf<T>::type, T> L, long long nrows,
                                                  int ny, int ppg, long long gstride, const double* __restrict__ tw,
                                                  const LineGate gate) {
    typedef typename CplxOf<T>::type CT;
    typedef Plan<N> P;
    constexpr int H = N / 2 + 1, half = N / 2;
    extern __shared__ __align__(16) unsigned char smraw[];
    if (gated_off(gate)) return;
    const int t = threadIdx.x % P::TL, pp = threadIdx.x / P::TL;
    CT* Z = (CT*)smraw + pp * P::R1 * (P::R2 + 1);
    auto zs = [&](int k1, int n2) -> CT& { return Z[k1 * (P::R2 + 1) + n2]; };
    const CT* in = L.in[blockIdx.y] + blockIdx.z * L.in_ss;
    T* out = L.out[blockIdx.y] + blockIdx.z * L.out_ss;
    const long long r0 = 2LL * ((long long)blockIdx.x * (blockDim.x / P::TL) + pp), r1 = r0 + 1;
    const bool has0 = r0 < nrows, has1 = r1 < nrows;
    const long long pe = (long long)ny * H;
    const long long o0 = has0 ? grp_off(r0 / ny, ppg, gstride, pe) + (r0 % ny) * H : 0;
    const long long o1 = has1 ? grp_off(r1 / ny, ppg, gstride, pe) + (r1 % ny) * H : 0;
    CT v[P::R1];
    #pragma unroll
    for (int n1 = 0; n1 < P::R1; ++n1) {
        const int idx = P::R2 * n1 + t;
        const bool mirror = idx > half;
        const int k = mirror ? N - idx : idx;
        const CT x1 = has0 ? in[o0 + k] : czero<CT>();
        const CT x2 = has1 ? in[o1 + k] : czero<CT>();
        CT z;
        if (k == 0 || k == half) { z.x = x1.x; z.y = x2.x; }
        else if (!mirror) { z.x = x1.x - x2.y; z.y = x1.y + x2.x; }
        else { z.x = x1.x + x2.y; z.y = -x1.y + x2.x; }
        v[n1] = z;
    }
    line_pass<true, N, T>(v, t, zs, tw);
    #pragma unroll
    for (int g = 0; g < P::G; ++g)
        #pragma unroll
        for (int k2 = 0; k2 < P::R2; ++k2) {
            const int i = t + P::R2 * g + P::R1 * k2;
            if (has0) out[r0 * N + i] = v[g * P::R2 + k2].x;
            if (has1) out[r1 * N + i] = v[g * P::R2 + k2].y;
        }
}

// complex columns along y, NC per CTA
template <typename T, int N, bool INV, int NC>
__global__ void __launch_bounds__(256) cols_kernel(const typename CplxOf<T>::type* __restrict__ in,
                                                   typename CplxOf<T>::type* __restrict__ out, int H, int ppg,
                                                   long long gstride, const T* __restrict__ mul,
                                                   const double* __restrict__ tw) {
    typedef typename CplxOf<T>::type CT;
    typedef Plan<N> P;
    extern __shared__ __align__(16) unsigned char smraw[];
    CT* Z = (CT*)smraw;
    const int ntile = (H + NC - 1) / NC;
    const long long plane = blockIdx.x / ntile;
    const int c = threadIdx.x % NC, t = threadIdx.x / NC;
    const int kx = (blockIdx.x % ntile) * NC + c;
    const bool cv = kx < H;
    auto zs = [&](int k1, int n2) -> CT& { return Z[(k1 * P::R2 + n2) * NC + c]; };
    const CT* src = in + grp_off(plane, ppg, gstride, (long long)N * H) + kx;
    CT* dst = out + plane * (long long)N * H + kx;
    CT v[P::R1];
    #pragma unroll
    for (int n1 = 0; n1 < P::R1; ++n1) v[n1] = cv ? src[(long long)(P::R2 * n1 + t) * H] : czero<CT>();
    line_pass<INV, N, T>(v, t, zs, tw);
    if (cv) {
        #pragma unroll
        for (int g = 0; g < P::G; ++g)
            #pragma unroll
            for (int k2 = 0; k2 < P::R2; ++k2) {
                const long long y = t + P::R2 * g + P::R1 * k2;
                CT val = v[g * P::R2 + k2];
                if (mul) val = __ldg(&mul[y * H + kx]) * val;
                dst[y * H] = val;
            }
    }
}

template <typename T, int N, int NC>
__global__ void __launch_bounds__(256) cols_filter_kernel(
    const LineList<typename CplxOf<T>::type, typename CplxOf<T>::type> L, int H, const T* __restrict__ mul,
    const double* __restrict__ tw, const LineGate gate) {
    typedef typename CplxOf<T>::type CT;
    typedef Plan<N> P;
    extern __shared__ __align__(16) unsigned char smraw[];
    if (gated_off(gate)) return;
    CT* Z = (CT*)smraw;
    const int ntile = (H + NC - 1) / NC;
    const long long plane = blockIdx.x / ntile;
    const int c = threadIdx.x % NC, t = threadIdx.x / NC;
    const int kx = (blockIdx.x % ntile) * NC + c;
    const bool cv = kx < H;
    auto zs = [&](int k1, int n2) -> CT& { return Z[(k1 * P::R2 + n2) * NC + c]; };
    const CT* src = L.in[blockIdx.y] + blockIdx.z * L.in_ss + plane * (long long)N * H + kx;
    CT* dst = L.out[blockIdx.y] + blockIdx.z * L.out_ss + plane * (long long)N * H + kx;
    CT v[P::R1];
    #pragma unroll
    for (int n1 = 0; n1 < P::R1; ++n1) v[n1] = cv ? src[(long long)(P::R2 * n1 + t) * H] : czero<CT>();
    line_pass<false, N, T>(v, t, zs, tw);
    __syncthreads();
    #pragma unroll
    for (int g = 0; g < P::G; ++g)
        #pragma unroll
        for (int k2 = 0; k2 < P::R2; ++k2) {
            const long long y = t + P::R2 * g + P::R1 * k2;
            v[g * P::R2 + k2] = cv ? __ldg(&mul[y * H + kx]) * v[g * P::R2 + k2] : czero<CT>();
        }
    line_mirror<true, N, T>(v, t, zs, tw);
    if (cv) {
        #pragma unroll
        for (int n1 = 0; n1 < P::R1; ++n1) dst[(long long)(P::R2 * n1 + t) * H] = v[n1];
    }
}

// ---- launches ----------------------------------------------------------------------

template <typename F> void by_size(int n, F f) {
    switch (n) {
        case 16: f(std::integral_constant<int, 16>()); break;
        case 32: f(std::integral_constant<int, 32>()); break;
        case 64: f(std::integral_constant<int, 64>()); break;
        case 128: f(std::integral_constant<int, 128>()); break;
        case 256: f(std::integral_constant<int, 256>()); break;
        case 512: f(std::integral_constant<int, 512>()); break;
        case 1024: f(std::integral_constant<int, 1024>()); break;
    }
}
template <typename K> void smem_of(K k, size_t bytes) {
    if (bytes > 48 * 1024) cudaFuncSetAttribute((const void*)k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
}

// SMs of the device
int sm_count() {
    static const int n = [] {
        int dev = 0, v = 0;
        if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) v = 0;
        cudaGetLastError();
        return v > 0 ? v : 152;
    }();
    return n;
}
// A launch over row pairs: CTAs, threads and exchange bytes.  Two warps (their
// barriers cost least: 256x256x300 FP32 d/dx 33 -> 30 us, FP64 the same as
// larger CTAs); one while the launch would leave an SM with less than four CTAs
// -- a few lines of FP64 keep an SM's pipe busy for tens of microseconds, so
// they have to be spread (300 rows of 256: 60 -> 29 us)
template <int N, typename CT> struct RowLaunch {
    int b;
    unsigned ctas;
    size_t smem;
    RowLaunch(long long nrows, int batch) {
        const long long pairs = (nrows + 1) / 2;
        b = pairs * batch / (64 / Plan<N>::TL) < 4LL * sm_count() ? 32 : 64;
        const int per = b / Plan<N>::TL;
        ctas = (unsigned)((pairs + per - 1) / per);
        smem = (size_t)per * Plan<N>::R1 * (Plan<N>::R2 + 1) * sizeof(CT);
    }
};
// Columns (or pairs) per CTA: rows of 128 bytes, two warps at least.  Wider
// CTAs waste columns of the nx/2+1 of a half spectrum (FP64, 65 columns: 32 a
// CTA 154 us, 8 a CTA 126 us); on the nx/2 pairs of a plane there is no such
// waste and 256 threads are the faster ones (FP64 128: 104 against 100 us)
template <int N, typename CT> constexpr int narrow() {
    const int least = sizeof(CT) == 16 || Plan<N>::TL == 32 ? 8 : 16;
    return least > 64 / Plan<N>::TL ? least : 64 / Plan<N>::TL;
}
template <int N> constexpr int wide() { return 256 / Plan<N>::TL; }

}  // namespace

template <typename T>
void line_rows(const LineList<T, T>& L, int nsrc, int nx, long long nrows, const LineMul<T>& mul, const double* tw,
               const LineGate& gate, cudaStream_t s) {
    typedef typename CplxOf<T>::type CT;
    by_size(nx, [&](auto n) {
        constexpr int N = decltype(n)::value;
        const int all = (1 << L.n) - 1, kind = (mul.real & all) == 0 ? 0 : (mul.real & all) == all ? 1 : 2;
        auto k = kind == 0 ? rows_kernel<T, N, 0> : kind == 1 ? rows_kernel<T, N, 1> : rows_kernel<T, N, 2>;
        const RowLaunch<N, CT> g(nrows, L.n * nsrc);
        smem_of(k, g.smem);
        k<<<dim3(g.ctas, L.n, nsrc), g.b, g.smem, s>>>(L, nrows, mul, tw, gate);
    });
}
template <typename T>
void line_cols_deriv(const LineList<T, T>& L, int nsrc, int nx, int ny, long long nplanes, const T* mul,
                     const double* tw, cudaStream_t s) {
    typedef typename CplxOf<T>::type CT;
    by_size(ny, [&](auto n) {
        constexpr int N = decltype(n)::value;
        auto launch = [&](auto k, int NC) {
            const long long tiles = (nx / 2 + NC - 1) / NC;
            smem_of(k, (size_t)NC * N * sizeof(CT));
            k<<<dim3((unsigned)(nplanes * tiles), L.n, nsrc), NC * Plan<N>::TL, (size_t)NC * N * sizeof(CT), s>>>(L, nx, mul, tw);
        };
        if (nplanes * (nx / 2) / wide<N>() * L.n * nsrc >= 4LL * sm_count()) launch(cols_deriv_kernel<T, N, wide<N>()>, wide<N>());
        else launch(cols_deriv_kernel<T, N, narrow<N, CT>()>, narrow<N, CT>());
    });
}
template <typename T>
void line_r2c(const LineList<T, typename CplxOf<T>::type>& L, int nsrc, int nx, long long nrows, T scale,
              const double* tw, const LineGate& gate, cudaStream_t s) {
    typedef typename CplxOf<T>::type CT;
    by_size(nx, [&](auto n) {
        constexpr int N = decltype(n)::value;
        const RowLaunch<N, CT> g(nrows, L.n * nsrc);
        smem_of(r2c_kernel<T, N>, g.smem);
        r2c_kernel<T, N><<<dim3(g.ctas, L.n, nsrc), g.b, g.smem, s>>>(L, nrows, scale, tw, gate);
    });
}
template <typename T>
void line_c2r(const LineList<typename CplxOf<T>::type, T>& L, int nsrc, int nx, int ny, long long nrows, int ppg,
              long long gstride, const double* tw, const LineGate& gate, cudaStream_t s) {
    typedef typename CplxOf<T>::type CT;
    by_size(nx, [&](auto n) {
        constexpr int N = decltype(n)::value;
        const RowLaunch<N, CT> g(nrows, L.n * nsrc);
        smem_of(c2r_kernel<T, N>, g.smem);
        c2r_kernel<T, N><<<dim3(g.ctas, L.n, nsrc), g.b, g.smem, s>>>(L, nrows, ny, ppg, gstride, tw, gate);
    });
}
template <typename T>
void line_cols(const typename CplxOf<T>::type* in, typename CplxOf<T>::type* out, int H, int ny, long long nplanes,
               int ppg, long long gstride, int sign, const T* mul, const double* tw, cudaStream_t s) {
    typedef typename CplxOf<T>::type CT;
    by_size(ny, [&](auto n) {
        constexpr int N = decltype(n)::value;
        constexpr int NC = narrow<N, CT>();
        auto k = sign > 0 ? cols_kernel<T, N, true, NC> : cols_kernel<T, N, false, NC>;
        const size_t smem = (size_t)NC * N * sizeof(CT);
        smem_of(k, smem);
        const long long tiles = (H + NC - 1) / NC;
        k<<<(unsigned)(nplanes * tiles), NC * Plan<N>::TL, smem, s>>>(in, out, H, ppg, gstride, mul, tw);
    });
}
template <typename T>
void line_cols_filter(const LineList<typename CplxOf<T>::type, typename CplxOf<T>::type>& L, int nsrc, int H, int ny,
                      long long nplanes, const T* mul, const double* tw, const LineGate& gate, cudaStream_t s) {
    typedef typename CplxOf<T>::type CT;
    by_size(ny, [&](auto n) {
        constexpr int N = decltype(n)::value;
        constexpr int NC = narrow<N, CT>();
        const size_t smem = (size_t)NC * N * sizeof(CT);
        smem_of(cols_filter_kernel<T, N, NC>, smem);
        const long long tiles = (H + NC - 1) / NC;
        cols_filter_kernel<T, N, NC><<<dim3((unsigned)(nplanes * tiles), L.n, nsrc), NC * Plan<N>::TL, smem, s>>>(L, H, mul, tw, gate);
    });
}

#define INST_LINES(T, CT)                                                                                             \
    template void line_rows<T>(const LineList<T, T>&, int, int, long long, const LineMul<T>&, const double*,          \
                               const LineGate&, cudaStream_t);                                                        \
    template void line_cols_deriv<T>(const LineList<T, T>&, int, int, int, long long, const T*, const double*,        \
                                     cudaStream_t);                                                                   \
    template void line_r2c<T>(const LineList<T, CT>&, int, int, long long, T, const double*, const LineGate&,         \
                              cudaStream_t);                                                                          \
    template void line_c2r<T>(const LineList<CT, T>&, int, int, int, long long, int, long long, const double*,        \
                              const LineGate&, cudaStream_t);                                                         \
    template void line_cols<T>(const CT*, CT*, int, int, long long, int, long long, int, const T*, const double*,     \
                               cudaStream_t);                                                                         \
    template void line_cols_filter<T>(const LineList<CT, CT>&, int, int, int, long long, const T*, const double*,     \
                                      const LineGate&, cudaStream_t);
