// Transforms of whole lines (rows along x, columns along y) of n = 16..1024
// points in registers, shared by the spectral derivatives, the horizontal
// filters and the physical <-> spectral transforms.
//
// n = R1 R2 (R1 >= R2): TL = R2 threads hold a line, R1 points each.  Pass 1
// (thread n2): an R1-point DFT in registers over n1 of x[R2 n1 + n2], times
// the twiddle W_n^(n2 k1); one exchange through shared memory; pass 2: R1/R2
// DFTs of R2 points over n2, for k1 = t + R2 g, give X[k1 + R1 k2].  The
// mirrored form starts from that layout and ends in the first one, so a
// derivative or a filter (forward, multiply, inverse) needs no reordering.
// The register DFTs are radix-4 steps with their rotations as constants.
//
// FP64 issue bounds the FP64 kernels (79 % of the pipe), memory latency and L1
// the FP32 ones.  Measured at 128x128x150 FP64, one field, against shared-memory
// radix-2: d/dx 138 -> 104 us, d/dy 143 -> 104 us, forward rows 84 -> 65 us,
// inverse rows 73 -> 60 us, filter columns 212 -> 157 us.
#pragma once
#include "internal.cuh"

// fields of one batched launch (grid.y the field, grid.z the source): field
// i of source s is in[i] + s in_ss -> out[i] + s out_ss (element strides)
constexpr int LINE_FIELDS = 8;
template <typename A, typename B> struct LineList {
    const A* in[LINE_FIELDS];
    B* out[LINE_FIELDS];
    int n;
    long long in_ss, out_ss;
};
// Launches that only act on the steps of the horizontal filter: a source whose
// clock is not on one is left alone
struct LineGate {
    int on;
    SlotClock clk;
};

static inline bool line_ok(int n) { return n >= 16 && n <= 1024 && (n & (n - 1)) == 0; }

// Per field of a list of rows: the factors mul[nx] of the spectrum, times i
// (a derivative) or real (a filter)
template <typename T> struct LineMul {
    const T* mul[LINE_FIELDS];
    int real;           // bit i: field i's factors are real
};
template <typename T> LineMul<T> line_mul(const T* mul, bool real = false) {
    LineMul<T> m;
    for (const T*& p : m.mul) p = mul;
    m.real = real ? -1 : 0;
    return m;
}

// d/dx or a filter of rows of nx reals, nrows rows per field
template <typename T>
void line_rows(const LineList<T, T>& L, int nsrc, int nx, long long nrows, const LineMul<T>& mul, const double* tw,
               const LineGate& gate, cudaStream_t s);
// d/dy of dense (ny, nx) planes
template <typename T>
void line_cols_deriv(const LineList<T, T>& L, int nsrc, int nx, int ny, long long nplanes, const T* mul,
                     const double* tw, cudaStream_t s);
// rows of nx reals -> rows of nx/2+1 complex, scaled
template <typename T>
void line_r2c(const LineList<T, typename CplxOf<T>::type>& L, int nsrc, int nx, long long nrows, T scale,
              const double* tw, const LineGate& gate, cudaStream_t s);
// rows of nx/2+1 complex -> rows of nx reals, inverse, unscaled.  Input planes of ny rows may come in
// groups: plane p at (p / ppg) gstride + (p % ppg) ny (nx/2+1)
template <typename T>
void line_c2r(const LineList<typename CplxOf<T>::type, T>& L, int nsrc, int nx, int ny, long long nrows, int ppg,
              long long gstride, const double* tw, const LineGate& gate, cudaStream_t s);
// complex columns along y of [plane][y][kx] data (H columns), sign -1 or +1, times mul[ky][kx] if given
template <typename T>
void line_cols(const typename CplxOf<T>::type* in, typename CplxOf<T>::type* out, int H, int ny, long long nplanes,
               int ppg, long long gstride, int sign, const T* mul, const double* tw, cudaStream_t s);
// forward columns, the real multiplier mul[ky][kx], inverse columns, in place
template <typename T>
void line_cols_filter(const LineList<typename CplxOf<T>::type, typename CplxOf<T>::type>& L, int nsrc, int H, int ny,
                      long long nplanes, const T* mul, const double* tw, const LineGate& gate, cudaStream_t s);

// The FP32 2-D forms' row transforms (rows2d_f32.cu), any nx: d/dx; rows of nx
// reals -> rows of nx/2+1 complex, scaled, times mul[k] if given; its inverse, row
// r at (r / ppg) gstride + (r % ppg) (nx/2+1)
void rows2d_deriv(const LineList<float, float>& L, int nsrc, int nx, long long nrows, const float* mul, const double* tw,
                  cudaStream_t s);
void rows2d_r2c(const LineList<float, float2>& L, int nsrc, int nx, long long nrows, float scale, const float* mul,
                const double* tw, const LineGate& gate, cudaStream_t s);
void rows2d_c2r(const LineList<float2, float>& L, int nsrc, int nx, long long nrows, int ppg, long long gstride,
                const double* tw, const LineGate& gate, cudaStream_t s);

// offset of input plane p when planes come in groups of ppg, group g starting
// at g * gstride (complex elements); pe = elements per plane
__device__ __forceinline__ long long grp_off(long long p, int ppg, long long gstride, long long pe) {
    const long long g = p / ppg;
    return g * gstride + (p - g * ppg) * pe;
}
