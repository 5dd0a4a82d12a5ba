// Horizontal transforms between physical planes a(nx,ny) and the normalised
// r2c half-spectrum state (the FFTW plans of initialize.f90:323-337 and
// damping.f90:46-58 are the reference's counterpart; cuFFT is not used): the
// register transforms of lines.cuh for 16 to 1024 points, shared-memory
// Stockham radix-2 FFTs for 4 and 8; FP32 rows of a 2-D grid go through
// rows2d_f32.cu.
//
//   phys -> spec : rows_r2c   (two real rows packed as one complex FFT along x,
//                              split by Hermitian symmetry, scaled 1/(nx*ny))
//                  cols_fft   (complex FFT along y on tiles of kx columns)
//   spec -> phys : cols_fft (inverse), rows_c2r (two rows per complex inverse
//                  FFT; DC/Nyquist imaginary parts dropped as FFTW c2r does)
//
// Also: point-wise spectral multipliers and the sensitivity-kernel
// accumulation of kernels.f90:273-311 on physical fields.
#include "internal.cuh"
#include "lines.cuh"

// phys (nrows rows of nx reals) -> out (nrows rows of H = nx/2+1 complex), scaled by `scale`
template <typename T>
__global__ void rows_r2c_kernel(const T* __restrict__ phys, typename CplxOf<T>::type* __restrict__ out,
                                int nx, long long nrows, T scale, const double* __restrict__ tw) {
    typedef typename CplxOf<T>::type CT;
    extern __shared__ __align__(16) unsigned char smraw[];
    CT* b0 = (CT*)smraw;
    CT* b1 = b0 + nx;
    const long long r0 = 2LL * blockIdx.x, r1 = r0 + 1;
    const bool has1 = r1 < nrows;
    for (int i = threadIdx.x; i < nx; i += blockDim.x) {
        CT v;
        v.x = phys[r0 * nx + i];
        v.y = has1 ? phys[r1 * nx + i] : (T)0;
        b0[i] = v;
    }
    __syncthreads();
    CT* Z = smem_fft<T, CT>(b0, b1, nx, 1, (T)-1, tw);
    const int H = nx / 2 + 1;
    const T hs = (T)0.5 * scale;
    for (int k = threadIdx.x; k < H; k += blockDim.x) {
        CT zk = Z[k], zn = Z[(nx - k) & (nx - 1)];
        CT x1, x2;
        x1.x = (zk.x + zn.x) * hs;
        x1.y = (zk.y - zn.y) * hs;
        x2.x = (zk.y + zn.y) * hs;
        x2.y = -(zk.x - zn.x) * hs;
        out[r0 * H + k] = x1;
        if (has1) out[r1 * H + k] = x2;
    }
}

// in (nrows rows of H complex) -> phys (nrows rows of nx reals), inverse, unscaled
template <typename T>
__global__ void rows_c2r_kernel(const typename CplxOf<T>::type* __restrict__ in, T* __restrict__ phys,
                                int nx, long long nrows, const double* __restrict__ tw, int ny, int ppg,
                                long long gstride) {
    typedef typename CplxOf<T>::type CT;
    extern __shared__ __align__(16) unsigned char smraw[];
    CT* b0 = (CT*)smraw;
    CT* b1 = b0 + nx;
    const long long r0 = 2LL * blockIdx.x, r1 = r0 + 1;
    const bool has1 = r1 < nrows;
    const int H = nx / 2 + 1, half = nx / 2;
    const long long pe = (long long)ny * H;
    const long long o0 = grp_off(r0 / ny, ppg, gstride, pe) + (r0 % ny) * H;
    const long long o1 = has1 ? grp_off(r1 / ny, ppg, gstride, pe) + (r1 % ny) * H : 0;
    for (int k = threadIdx.x; k <= half; k += blockDim.x) {
        CT x1 = in[o0 + k];
        CT x2 = has1 ? in[o1 + k] : czero<CT>();
        if (k == 0 || k == half) {
            CT z; z.x = x1.x; z.y = x2.x;
            b0[k] = z;
        } else {
            CT z;
            z.x = x1.x - x2.y; z.y = x1.y + x2.x;
            b0[k] = z;
            z.x = x1.x + x2.y; z.y = -x1.y + x2.x;
            b0[nx - k] = z;
        }
    }
    __syncthreads();
    CT* Z = smem_fft<T, CT>(b0, b1, nx, 1, (T)1, tw);
    for (int i = threadIdx.x; i < nx; i += blockDim.x) {
        CT z = Z[i];
        phys[r0 * nx + i] = z.x;
        if (has1) phys[r1 * nx + i] = z.y;
    }
}

// complex FFT along y on tiles of W kx-columns: data [plane][y][kx], H columns
template <typename T>
__global__ void cols_fft_kernel(const typename CplxOf<T>::type* __restrict__ in,
                                typename CplxOf<T>::type* __restrict__ out, int ny, int H, int W, T sign,
                                const double* __restrict__ tw, int ppg, long long gstride) {
    typedef typename CplxOf<T>::type CT;
    extern __shared__ __align__(16) unsigned char smraw[];
    CT* b0 = (CT*)smraw;
    CT* b1 = b0 + (long long)W * ny;
    const int ntile = (H + W - 1) / W;
    const long long plane = blockIdx.x / ntile;
    const int kx0 = (blockIdx.x % ntile) * W;
    const int w = min(W, H - kx0);
    const long long base = plane * (long long)ny * H;
    const long long ibase = grp_off(plane, ppg, gstride, (long long)ny * H);
    for (int t = threadIdx.x; t < W * ny; t += blockDim.x) {
        int y = t / W, c = t - y * W;
        b0[c * ny + y] = (c < w) ? in[ibase + (long long)y * H + kx0 + c] : czero<CT>();
    }
    __syncthreads();
    CT* Z = smem_fft<T, CT>(b0, b1, ny, W, sign, tw);
    for (int t = threadIdx.x; t < W * ny; t += blockDim.x) {
        int y = t / W, c = t - y * W;
        if (c < w) out[base + (long long)y * H + kx0 + c] = Z[c * ny + y];
    }
}

static int col_tile(int) { return 16; }    // sizes below the line transforms (4, 8)

// spec[plane][m] *= mul[m] (a real pencil multiplier, m < M)
template <typename T>
__global__ void spec_mul_kernel(typename CplxOf<T>::type* spec, const T* __restrict__ mul, int M, long long n) {
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t < n) spec[t] = mul[t % M] * spec[t];
}

// phys -> normalised half-spectrum; with mul, each spectral plane is also
// multiplied by the real pencil multiplier mul[m] (in the column pass when
// there is one)
// rows of nx reals -> rows of H complex (the forward row pass of fft_phys_to_spec)
template <typename T>
static void rows_forward(const T* phys, typename CplxOf<T>::type* dst, int nx, int ny, long long nrows, T scale,
                         const double* tw_x, cudaStream_t s) {
    typedef typename CplxOf<T>::type CT;
    if constexpr (sizeof(T) == 4) {
        if (ny == 1) return rows2d_r2c({{phys}, {dst}, 1, 0, 0}, 1, nx, nrows, scale, nullptr, tw_x, {}, s);
    }
    if (line_ok(nx)) {
        line_r2c<T>({{phys}, {dst}, 1, 0, 0}, 1, nx, nrows, scale, tw_x, {}, s);
        return;
    }
    size_t sm = 2 * (size_t)nx * sizeof(CT);
    rows_r2c_kernel<T><<<(unsigned)((nrows + 1) / 2), 32, sm, s>>>(phys, dst, nx, nrows, scale, tw_x);
}

template <typename T>
void fft_phys_to_spec(const T* phys, typename CplxOf<T>::type* spec, typename CplxOf<T>::type* tmp,
                      int nx, int ny, int nplanes, const double* tw_x, const double* tw_y, cudaStream_t s,
                      const T* mul) {
    typedef typename CplxOf<T>::type CT;
    const int H = nx / 2 + 1;
    const long long nrows = (long long)ny * nplanes;
    CT* dst = (ny == 1) ? spec : tmp;
    const T scale = (T)(1.0 / ((double)nx * ny));
    rows_forward<T>(phys, dst, nx, ny, nrows, scale, tw_x, s);
    if (ny > 1 && line_ok(ny)) {
        line_cols<T>(tmp, spec, H, ny, nplanes, nplanes, 0LL, -1, mul, tw_y, s);
        return;
    }
    if (ny > 1) {
        int W = col_tile(ny);
        size_t sm2 = 2 * (size_t)W * ny * sizeof(CT);
        int ntile = (H + W - 1) / W;
        cols_fft_kernel<T><<<(unsigned)(ntile * (long long)nplanes), 256, sm2, s>>>(tmp, spec, ny, H, W, (T)-1, tw_y,
                                                                                   nplanes, 0LL);
    }
    if (mul) {
        const long long n = (long long)nplanes * ny * H;
        spec_mul_kernel<T><<<(unsigned)((n + 255) / 256), 256, 0, s>>>(spec, mul, ny * H, n);
    }
}

// rows of H complex -> rows of nx reals (the inverse row pass of fft_spec_to_phys_g)
template <typename T>
static void rows_inverse(const typename CplxOf<T>::type* src, T* phys, int nx, int ny, long long nrows,
                         int rppg, long long rgs, const double* tw_x, cudaStream_t s) {
    typedef typename CplxOf<T>::type CT;
    if constexpr (sizeof(T) == 4) {
        if (ny == 1) return rows2d_c2r({{src}, {phys}, 1, 0, 0}, 1, nx, nrows, rppg, rgs, tw_x, {}, s);
    }
    if (line_ok(nx)) {
        line_c2r<T>({{src}, {phys}, 1, 0, 0}, 1, nx, ny, nrows, rppg, rgs, tw_x, {}, s);
        return;
    }
    size_t sm = 2 * (size_t)nx * sizeof(CT);
    rows_c2r_kernel<T><<<(unsigned)((nrows + 1) / 2), 32, sm, s>>>(src, phys, nx, nrows, tw_x, ny, rppg, rgs);
}

template <typename T>
void fft_spec_to_phys_g(const typename CplxOf<T>::type* spec, int ppg, long long gstride, T* phys,
                        typename CplxOf<T>::type* tmp, int nx, int ny, int nplanes, const double* tw_x,
                        const double* tw_y, cudaStream_t s) {
    typedef typename CplxOf<T>::type CT;
    const int H = nx / 2 + 1;
    const long long nrows = (long long)ny * nplanes;
    const CT* src = spec;
    int rppg = ppg;
    long long rgs = gstride;
    if (ny > 1) {
        if (line_ok(ny)) {
            line_cols<T>(spec, tmp, H, ny, nplanes, ppg, gstride, 1, nullptr, tw_y, s);
        } else {
            int W = col_tile(ny);
            size_t sm2 = 2 * (size_t)W * ny * sizeof(CT);
            int ntile = (H + W - 1) / W;
            cols_fft_kernel<T><<<(unsigned)(ntile * (long long)nplanes), 256, sm2, s>>>(spec, tmp, ny, H, W, (T)1, tw_y,
                                                                                       ppg, gstride);
        }
        src = tmp;
        rppg = nplanes;      // tmp is contiguous
        rgs = 0;
    }
    rows_inverse<T>(src, phys, nx, ny, nrows, rppg, rgs, tw_x, s);
}

// phys -> out through the half spectrum times the real pencil multiplier
// mul[ky][kx] (damping, horizontal filter).  The column passes run as one
// kernel in place on tmp (3 launches) where the line transforms cover ny;
// otherwise as fft_phys_to_spec + fft_spec_to_phys through spec (3 to 5).
// Returns the number of launches.
template <typename T>
int fft_filter_phys(const T* phys, T* out, typename CplxOf<T>::type* spec, typename CplxOf<T>::type* tmp, int nx,
                    int ny, int nplanes, const double* tw_x, const double* tw_y, cudaStream_t s, const T* mul) {
    if (!(ny > 1 && line_ok(ny))) {
        fft_phys_to_spec<T>(phys, spec, tmp, nx, ny, nplanes, tw_x, tw_y, s, mul);
        fft_spec_to_phys<T>(spec, out, tmp, nx, ny, nplanes, tw_x, tw_y, s);
        return ny > 1 ? 5 : 3;
    }
    const long long nrows = (long long)ny * nplanes;
    rows_forward<T>(phys, tmp, nx, ny, nrows, (T)(1.0 / ((double)nx * ny)), tw_x, s);
    line_cols_filter<T>({{tmp}, {tmp}, 1, 0, 0}, 1, nx / 2 + 1, ny, nplanes, mul, tw_y, {}, s);
    rows_inverse<T>(tmp, out, nx, ny, nrows, nplanes, 0LL, tw_x, s);
    return 3;
}

template <typename T>
void fft_spec_to_phys(const typename CplxOf<T>::type* spec, T* phys, typename CplxOf<T>::type* tmp,
                      int nx, int ny, int nplanes, const double* tw_x, const double* tw_y, cudaStream_t s) {
    fft_spec_to_phys_g<T>(spec, nplanes, 0LL, phys, tmp, nx, ny, nplanes, tw_x, tw_y, s);
}

// out = out + i kx fx + i ky fy   (fy may be null)
template <typename T>
__global__ void spec_combine_kernel(typename CplxOf<T>::type* out, const typename CplxOf<T>::type* fx,
                                    const typename CplxOf<T>::type* fy, const T* __restrict__ pt, int M,
                                    long long n, long long out_ss, long long in_ss) {
    long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n) return;
    out += blockIdx.y * out_ss;
    fx += blockIdx.y * in_ss;
    if (fy) fy += blockIdx.y * in_ss;
    int m = (int)(t % M);
    typename CplxOf<T>::type d = imul(pt[PT_KX * (long long)M + m], fx[t]);
    if (fy) d = d + imul(pt[PT_KY * (long long)M + m], fy[t]);
    out[t] = d + out[t];
}

// out(z) = in(z) * zt[row][z]
template <typename T>
__global__ void spec_scale_z_kernel(typename CplxOf<T>::type* out, const typename CplxOf<T>::type* in,
                                    const T* __restrict__ zt, int row, int M, int nz, long long out_ss,
                                    long long in_ss) {
    long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (long long)M * nz) return;
    out += blockIdx.y * out_ss;
    in += blockIdx.y * in_ss;
    int z = (int)(t / M);
    out[t] = in[t] * zt[row * nz + z];
}

// which: 0 -> i kx * in, 1 -> i ky * in, 2 -> damping rate * in, 3 -> horizontal filter * in
template <typename T>
__global__ void spec_dxdy_kernel(typename CplxOf<T>::type* out, const typename CplxOf<T>::type* in,
                                 const T* __restrict__ pt, int which, int M, long long n, long long out_ss,
                                 long long in_ss) {
    long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n) return;
    out += blockIdx.y * out_ss;
    in += blockIdx.y * in_ss;
    int m = (int)(t % M);
    if (which == 0) out[t] = imul(pt[PT_KX * (long long)M + m], in[t]);
    else if (which == 1) out[t] = imul(pt[PT_KY * (long long)M + m], in[t]);
    else if (which == 2) out[t] = pt[PT_DAMP * (long long)M + m] * in[t];
    else out[t] = pt[PT_HF * (long long)M + m] * in[t];
}

// Sensitivity-kernel accumulation, kernels.f90:276-311, for nsrc sources at
// once.  fwd planes (field stride fwd_fs, source stride N): 0 div(f_xi), 1-3
// f_acc (x,y,z), 4-6 f_xi (x,y,z); adj planes (stride adj_fs): 0 div(a_v), 1-3
// a_v, 4-6 grad(g a_vz).  acc [src][3][N]: kernelc2, kernelrho, hessian, FP64.
// The time integral is FP64; the per-snapshot products are formed in T (the
// fields' own precision).
template <typename T>
__global__ void kernel_accum_kernel(double* __restrict__ acc, const T* __restrict__ fwd, long long fwd_fs,
                                    const T* __restrict__ adj, long long adj_fs, const double* __restrict__ zt64,
                                    long long NP, int nz, int use_y, int nsrc, const double* __restrict__ c2f) {
    long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const long long N = NP * nz;
    if (t >= N * nsrc) return;
    const long long g = t / N, i = t - g * N;
    const int z = (int)(i / NP);
    double* A = acc + g * 3 * N;
    const T zero = (T)0;
    const T f1 = fwd[t], fax = fwd[fwd_fs + t], fay = use_y ? fwd[2 * fwd_fs + t] : zero, faz = fwd[3 * fwd_fs + t];
    const T fxx = fwd[4 * fwd_fs + t], fxy = use_y ? fwd[5 * fwd_fs + t] : zero, fxz = fwd[6 * fwd_fs + t];
    const T a1 = adj[t], avx = adj[adj_fs + t], avy = use_y ? adj[2 * adj_fs + t] : zero, avz = adj[3 * adj_fs + t];
    const T d31 = adj[4 * adj_fs + t], d32 = use_y ? adj[5 * adj_fs + t] : zero, d33 = adj[6 * adj_fs + t];
    if constexpr (sizeof(T) == 8) {
        const double c2 = c2f ? c2f[i] : zt64[ZT_C2 * nz + z], gr = zt64[ZT_GRAW * nz + z];
        A[2 * N + i] = A[2 * N + i] + faz * faz + fax * fax + fay * fay;
        const double t1 = f1 * a1;
        A[i] = A[i] + t1;
        double kr = A[N + i] + t1 * c2 + faz * avz + fax * avx + fay * avy;
        kr = kr - gr * fxz * a1 + (fxx * d31 + fxy * d32 + fxz * d33);
        A[N + i] = kr;
    } else {
        const T c2 = (T)(c2f ? c2f[i] : zt64[ZT_C2 * nz + z]), gr = (T)zt64[ZT_GRAW * nz + z];
        const T h = faz * faz + fax * fax + fay * fay;
        const T t1 = f1 * a1;
        const T kr = t1 * c2 + faz * avz + fax * avx + fay * avy - gr * fxz * a1 + (fxx * d31 + fxy * d32 + fxz * d33);
        A[2 * N + i] += (double)h;
        A[i] += (double)t1;
        A[N + i] += (double)kr;
    }
}

// Final scaling kernels.f90:523-539, optionally summed over nsum slots
__global__ void kernel_finish_kernel(double* __restrict__ out, const double* __restrict__ acc,
                                     const double* __restrict__ zt64, long long NP, int nz, double scale_c,
                                     double scale_r, int nsum, long long acc_ss, const double* __restrict__ r0f,
                                     const double* __restrict__ c2f) {
    long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const long long N = NP * nz;
    if (t >= N) return;
    const int z = (int)(t / NP);
    const double r0 = r0f ? r0f[t] : zt64[ZT_RHO0 * nz + z], c2 = c2f ? c2f[t] : zt64[ZT_C2 * nz + z];
    double kc = 0, kr = 0, h = 0;
    for (int s = 0; s < nsum; ++s) {
        const double* A = acc + s * acc_ss;
        kc += -A[t] * r0 * c2 * scale_c;
        kr += -r0 * A[N + t] * scale_r;
        h += A[2 * N + t];
    }
    out[t] = kc;
    out[N + t] = kr;
    out[2 * N + t] = h;
}

template <typename T>
__global__ void copy_convert_kernel(T* dst, const double* src, long long n) {
    long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t < n) dst[t] = (T)src[t];
}
template <typename T>
__global__ void copy_back_kernel(double* dst, const T* src, long long n) {
    long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t < n) dst[t] = (double)src[t];
}

template <typename T>
__global__ void finite_kernel(const T* p, long long n, int* flag) {
    long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    long long stride = (long long)gridDim.x * blockDim.x;
    for (; t < n; t += stride)
        if (!isfinite(p[t])) { *flag = 1; return; }
}

static unsigned nblk(long long n, int b = 256) { return (unsigned)((n + b - 1) / b); }

template <typename T>
void launch_spec_combine(typename CplxOf<T>::type* out, const typename CplxOf<T>::type* fx,
                         const typename CplxOf<T>::type* fy, const T* pt, int M, int nz, int nsrc, long long out_ss,
                         long long in_ss, cudaStream_t s) {
    long long n = (long long)M * nz;
    spec_combine_kernel<T><<<dim3(nblk(n), nsrc), 256, 0, s>>>(out, fx, fy, pt, M, n, out_ss, in_ss);
}
template <typename T>
void launch_spec_scale_z(typename CplxOf<T>::type* out, const typename CplxOf<T>::type* in, const T* zt, int row,
                         int M, int nz, int nsrc, long long out_ss, long long in_ss, cudaStream_t s) {
    spec_scale_z_kernel<T><<<dim3(nblk((long long)M * nz), nsrc), 256, 0, s>>>(out, in, zt, row, M, nz, out_ss, in_ss);
}
template <typename T>
void launch_spec_dxdy(typename CplxOf<T>::type* out, const typename CplxOf<T>::type* in, const T* pt, int which,
                      int M, int nz, int nsrc, long long out_ss, long long in_ss, cudaStream_t s) {
    long long n = (long long)M * nz;
    spec_dxdy_kernel<T><<<dim3(nblk(n), nsrc), 256, 0, s>>>(out, in, pt, which, M, n, out_ss, in_ss);
}
template <typename T>
void launch_kernel_accum(double* acc, const T* fwd, long long fwd_fs, const T* adj, long long adj_fs,
                         const double* zt64, long long NP, int nz, int use_y, int nsrc, cudaStream_t s,
                         const double* c2f) {
    kernel_accum_kernel<T><<<nblk(NP * nz * nsrc), 256, 0, s>>>(acc, fwd, fwd_fs, adj, adj_fs, zt64, NP, nz, use_y,
                                                                nsrc, c2f);
}
void launch_kernel_finish(double* out, const double* acc, const double* zt64, long long NP, int nz, double scale_c,
                          double scale_r, int nsum, long long acc_ss, cudaStream_t s, const double* r0f,
                          const double* c2f) {
    kernel_finish_kernel<<<nblk(NP * nz), 256, 0, s>>>(out, acc, zt64, NP, nz, scale_c, scale_r, nsum, acc_ss, r0f,
                                                       c2f);
}
template <typename T> void launch_copy_convert(T* dst, const double* src, long long n, cudaStream_t s) {
    copy_convert_kernel<T><<<nblk(n), 256, 0, s>>>(dst, src, n);
}
template <typename T> void launch_copy_back(double* dst, const T* src, long long n, cudaStream_t s) {
    copy_back_kernel<T><<<nblk(n), 256, 0, s>>>(dst, src, n);
}
int launch_check_finite_f64(const double* p, long long n, int* flag, cudaStream_t s) {
    finite_kernel<double><<<1024, 256, 0, s>>>(p, n, flag);
    return 0;
}
int launch_check_finite_f32(const float* p, long long n, int* flag, cudaStream_t s) {
    finite_kernel<float><<<1024, 256, 0, s>>>(p, n, flag);
    return 0;
}

#define INST(T)                                                                                                   \
    template int fft_filter_phys<T>(const T*, T*, CplxOf<T>::type*, CplxOf<T>::type*, int, int, int, const double*, \
                                    const double*, cudaStream_t, const T*);                                       \
    template void fft_phys_to_spec<T>(const T*, CplxOf<T>::type*, CplxOf<T>::type*, int, int, int, const double*, \
                                      const double*, cudaStream_t, const T*);                                     \
    template void fft_spec_to_phys<T>(const CplxOf<T>::type*, T*, CplxOf<T>::type*, int, int, int, const double*, \
                                      const double*, cudaStream_t);                                               \
    template void fft_spec_to_phys_g<T>(const CplxOf<T>::type*, int, long long, T*, CplxOf<T>::type*, int, int, \
                                        int, const double*, const double*, cudaStream_t);                         \
    template void launch_spec_combine<T>(CplxOf<T>::type*, const CplxOf<T>::type*, const CplxOf<T>::type*,       \
                                         const T*, int, int, int, long long, long long, cudaStream_t);            \
    template void launch_spec_scale_z<T>(CplxOf<T>::type*, const CplxOf<T>::type*, const T*, int, int, int, int, \
                                         long long, long long, cudaStream_t);                                     \
    template void launch_spec_dxdy<T>(CplxOf<T>::type*, const CplxOf<T>::type*, const T*, int, int, int, int,    \
                                      long long, long long, cudaStream_t);                                        \
    template void launch_kernel_accum<T>(double*, const T*, long long, const T*, long long, const double*,       \
                                         long long, int, int, int, cudaStream_t, const double*);                  \
    template void launch_copy_convert<T>(T*, const double*, long long, cudaStream_t);                             \
    template void launch_copy_back<T>(double*, const T*, long long, cudaStream_t);
INST(double)
INST(float)
