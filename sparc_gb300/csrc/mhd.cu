// The magnetic forms (options 10, 18 and 8): set-up of a background that varies
// in x and y, the derivative launches, and the sensitivity kernels of the 2-D
// form.  The time step is mhd_step.cu.
//
// The background breaks the per-mode structure of the quiet-Sun path, so the
// state lives in physical space: each [source][field] slot of the context holds
// one dense (nz, ny, nx) real field, and a stage takes its 21 derivatives
// explicitly:
//   d/dx  two real rows packed as one complex row, FFT (lines.cuh), times
//         i k normx 2 pi stretchx (the reference's eyekx * stretchx, Nyquist
//         dropped as its c2r does), inverse FFT  (derivatives.f90:28-58);
//   d/dy  two adjacent x-columns packed as one complex column, the same
//         along y (derivatives.f90:62-170); the derivative has a real kernel,
//         so it acts on the packed real and imaginary parts separately;
//   d/dz  DBYD2 on real pencils (zderiv_kernel, mhd_step.cu).
// DAMP_VELOCITY and the horizontal filter go through the normalised 2-D
// transforms and the same pencil multipliers as the quiet path.  The PML has
// six auxiliaries (psi_vz, psi_p, psi_dzbx, psi_dzby, psi_induction_bx,
// psi_induction_by; initialize.f90:487-490,560-566), in option 10 at the bottom
// only; its top has the sponge over the last 36 planes.
#include <cmath>
#include <cstring>
#include <vector>
#include <algorithm>

#include "mhd.cuh"

namespace {

template <typename T>
__device__ __forceinline__ typename CplxOf<T>::type imul_c(T k, typename CplxOf<T>::type z) {
    typename CplxOf<T>::type r;
    r.x = -k * z.y;
    r.y = k * z.x;
    return r;
}

// d/dx of nrows rows of nx reals (rows r = plane*ny + y, dense), two rows per CTA;
// every field (grid.y) and source (grid.z) of a list in one launch, since a grid
// this small is bound by its launches (option 10, 8x8x41, two sources, a step
// with a launch each 1.43 ms in FP32 and 1.87 in FP64, so 0.87 and 1.19)
template <typename T>
__global__ void rowderiv_kernel(const LineList<T, T> L, int nx, long long nrows, const T* __restrict__ rx,
                                const double* __restrict__ tw) {
    typedef typename CplxOf<T>::type CT;
    extern __shared__ __align__(16) unsigned char smraw[];
    const T* in = L.in[blockIdx.y] + blockIdx.z * L.in_ss;
    T* out = L.out[blockIdx.y] + blockIdx.z * L.out_ss;
    CT* b0 = (CT*)smraw;
    CT* b1 = b0 + nx;
    const long long r0 = 2LL * blockIdx.x, r1 = r0 + 1;
    const bool has1 = r1 < nrows;
    for (int i = threadIdx.x; i < nx; i += blockDim.x) {
        CT v;
        v.x = in[r0 * nx + i];
        v.y = has1 ? in[r1 * nx + i] : (T)0;
        b0[i] = v;
    }
    __syncthreads();
    CT* Z = smem_fft<T, CT>(b0, b1, nx, 1, (T)-1, tw);
    for (int k = threadIdx.x; k < nx; k += blockDim.x) Z[k] = imul_c<T>(rx[k], Z[k]);
    __syncthreads();
    CT* Y = smem_fft<T, CT>(Z, Z == b0 ? b1 : b0, nx, 1, (T)1, tw);
    for (int i = threadIdx.x; i < nx; i += blockDim.x) {
        out[r0 * nx + i] = Y[i].x;
        if (has1) out[r1 * nx + i] = Y[i].y;
    }
}

// d/dy of nplanes dense (ny, nx) planes: W complex columns (2W real x) per CTA;
// fields and sources as rowderiv_kernel
template <typename T>
__global__ void colderiv_kernel(const LineList<T, T> L, int nx, int ny, int W, const T* __restrict__ ry,
                                const double* __restrict__ tw) {
    typedef typename CplxOf<T>::type CT;
    extern __shared__ __align__(16) unsigned char smraw[];
    const T* in = L.in[blockIdx.y] + blockIdx.z * L.in_ss;
    T* out = L.out[blockIdx.y] + blockIdx.z * L.out_ss;
    CT* b0 = (CT*)smraw;
    CT* b1 = b0 + (long long)W * ny;
    const int ntile = (nx / 2) / W;
    const long long plane = blockIdx.x / ntile;
    const int c0 = (blockIdx.x % ntile) * W;
    const long long base = plane * (long long)ny * nx;
    for (int t = threadIdx.x; t < W * ny; t += blockDim.x) {
        const int y = t / W, c = t - y * W;
        const long long o = base + (long long)y * nx + 2 * (c0 + c);
        CT v;
        v.x = in[o];
        v.y = in[o + 1];
        b0[c * ny + y] = v;
    }
    __syncthreads();
    CT* Z = smem_fft<T, CT>(b0, b1, ny, W, (T)-1, tw);
    for (int t = threadIdx.x; t < W * ny; t += blockDim.x) {
        const int k = t % ny;
        Z[t] = imul_c<T>(ry[k], Z[t]);
    }
    __syncthreads();
    CT* Y = smem_fft<T, CT>(Z, Z == b0 ? b1 : b0, ny, W, (T)1, tw);
    for (int t = threadIdx.x; t < W * ny; t += blockDim.x) {
        const int y = t / W, c = t - y * W;
        const long long o = base + (long long)y * nx + 2 * (c0 + c);
        const CT v = Y[c * ny + y];
        out[o] = v.x;
        out[o + 1] = v.y;
    }
}

// FILTER_VAR_Z (kernels.f90:845-881) of nfield dense fields in place, one
// thread per pencil: rows 2..nz-1 written (the same stencil as FILTER_VARS_3D)
template <typename T>
__global__ void zfilter_phys_kernel(T* __restrict__ f, long long npix, int nz, long long fstride) {
    const long long m = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (m >= npix) return;
    T* p = f + blockIdx.y * fstride + m;
    zfilter_stream<T, T>(
        nz, 0, [&](int j) { return p[(long long)j * npix]; }, [&](int j, T v) { p[(long long)j * npix] = v; });
}

// a += b
template <typename T>
__global__ void add_kernel(T* __restrict__ a, const T* __restrict__ b, long long n) {
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t < n) a[t] = a[t] + b[t];
}

// out = in * prof[plane]
template <typename T>
__global__ void zscale_kernel(T* __restrict__ out, const T* __restrict__ in, const T* __restrict__ prof,
                              long long npix, long long n) {
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t < n) out[t] = in[t] * prof[t / npix];
}

// ---- set-up kernels (FP64) -------------------------------------------------

// READ_IN_FIELD (all_modules.f90:491-505) and the reduction of the field
// (physics.f90:116-129); taper[k] is the REAL*4 factor ((k-nz)/10.)**4 of the
// top eleven planes (1 elsewhere), cq the quiet sound speed
__global__ void mhd_read_kernel(double* rho0, double* c2, double* p0, double* bx, double* by, double* bz,
                                const double* cq, const double* taper, long long NP, int nz, double dimrho,
                                double dimc, double dimb) {
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= NP * nz) return;
    const int k = (int)(t / NP);
    const double r = rho0[t] / dimrho;
    const double cs = c2[t] / dimc;
    rho0[t] = r;
    c2[t] = pow(cs, 2.0);
    p0[t] = p0[t] / (dimrho * pow(dimc, 2.0));
    double x = bx[t] / dimb, y = by[t] / dimb, z = bz[t] / dimb;
    double red = (pow(z, 2.0) + pow(x, 2.0) + pow(y, 2.0)) / (r * pow(cq[k], 2.0));
    red = 8.0 / (8.0 + red);
    red = red * taper[k];
    const double s = pow(red, 0.5);
    bx[t] = x * s; by[t] = y * s; bz[t] = z * s;
}

// a = -a / d (element-wise)
__global__ void neg_div_kernel(double* a, double d, long long n) {
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t < n) a[t] = -a[t] / d;
}

// a = s1 * b + s2 * c (element-wise)
__global__ void axpby_kernel(double* a, const double* b, double s1, const double* c, double s2, long long n) {
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t < n) a[t] = s1 * b[t] + (c ? s2 * c[t] : 0.0);
}

// PML decay of gradp0_z / gradrho0_z and the bottom a_z, b_z (physics.f90:255-297)
__global__ void mhd_pml_kernel(double* gp0z, double* gr0z, double* az, double* bzp, const double* c2,
                               const double* rho0, const double* bx, const double* by, const double* bz,
                               const double* z, const double* alph, long long NP, int nz, int nb, int nt) {
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= NP * nz) return;
    const int k = (int)(t / NP);        // 0-based plane
    const long long q = t - (long long)k * NP;
    const bool bot = k < nb, top = k >= nz - nt;
    if (!bot && !top) return;
    auto tempin = [&](int kk) {
        const long long i = q + NP * kk;
        return pow(c2[i] + (pow(bx[i], 2.0) + pow(by[i], 2.0) + pow(bz[i], 2.0)) / rho0[i], 0.5);
    };
    double dampz, fdec;
    if (bot) {
        const double r = (z[nb - 1] - z[k]) / (z[nb - 1] - z[0]);
        dampz = 2.0 * 3.0 * 3.0 * tempin(0) / (z[nb - 1] - z[0]) * (r * r);
        fdec = alph[k] / (dampz + alph[k]);
        gp0z[t] *= fdec; gr0z[t] *= fdec;
        az[t] = -dampz;
        bzp[t] = -alph[k] - dampz;
    }
    if (top) {
        const double r = (z[nz - nt] - z[k]) / (z[nz - 1] - z[nz - nt]);
        dampz = 3.0 * 3.0 * tempin(nz - 1) / (z[nz - 1] - z[nz - nt]) * (r * r);
        fdec = alph[k] / (dampz + alph[k]);
        gp0z[t] *= fdec; gr0z[t] *= fdec;
        // pmlindex order: the top planes follow the nb bottom ones (read by
        // option 8; option 10 accounts for the bottom only)
        const long long ip = nb + (k - (nz - nt));
        az[ip * NP + q] = -dampz;
        bzp[ip * NP + q] = -alph[k] - dampz;
    }
}

__global__ void rhoinv_kernel(double* rhoinv, double* c2rho0, const double* rho0, const double* c2, long long n) {
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n) return;
    rhoinv[t] = 1.0 / rho0[t];
    c2rho0[t] = c2[t] * rho0[t];
}

template <typename T>
__global__ void to_t_kernel(T* dst, const double* src, long long n) {
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t < n) dst[t] = (T)src[t];
}

template <typename T>
int ddx_launch(sparc_ctx* c, const T* in, T* out) { return mhd_ddx<T>(c, {{in}, {out}, 1, 0, 0}, 1); }
template <typename T>
int ddy_launch(sparc_ctx* c, const T* in, T* out) { return mhd_ddy<T>(c, {{in}, {out}, 1, 0, 0}, 1); }
template <typename T>
int ddz_launch(sparc_ctx* c, const T* in, T* out, int bc) { return mhd_ddz<T>(c, {{in}, {out}, 1, 0, 0}, {{bc}}, 1); }

}  // namespace

template <typename T> int mhd_ddx(sparc_ctx* c, const LineList<T, T>& L, int nsrc) {
    const int nx = c->P.nx;
    const long long nrows = (long long)c->nz * c->P.ny;
    if constexpr (sizeof(T) == 4) {
        if (c->P.option == 18) {
            rows2d_deriv(L, nsrc, nx, nrows, (const float*)c->mhd->rx, c->tw_x, c->stream);
            c->launches++;
            CKL();
            return SPARC_OK;
        }
    }
    if (line_ok(nx)) {
        line_rows<T>(L, nsrc, nx, nrows, line_mul<T>((const T*)c->mhd->rx), c->tw_x, {}, c->stream);
        c->launches++;
    } else {
        const size_t sm = 2 * (size_t)nx * sizeof(typename CplxOf<T>::type);
        rowderiv_kernel<T><<<dim3((unsigned)((nrows + 1) / 2), L.n, nsrc), 32, sm, c->stream>>>(
            L, nx, nrows, (const T*)c->mhd->rx, c->tw_x);
        c->launches++;
    }
    CKL();
    return SPARC_OK;
}

template <typename T> int mhd_ddy(sparc_ctx* c, const LineList<T, T>& L, int nsrc) {
    const int nx = c->P.nx, ny = c->P.ny;
    if (line_ok(ny)) {
        line_cols_deriv<T>(L, nsrc, nx, ny, c->nz, (const T*)c->mhd->ry, c->tw_y, c->stream);
        c->launches++;
    } else {
        const int W = std::max(1, std::min(nx / 2, 1024 / ny));
        const size_t sm = 2 * (size_t)W * ny * sizeof(typename CplxOf<T>::type);
        colderiv_kernel<T><<<dim3((unsigned)((long long)c->nz * ((nx / 2) / W)), L.n, nsrc), 256, sm, c->stream>>>(
            L, nx, ny, W, (const T*)c->mhd->ry, c->tw_y);
        c->launches++;
    }
    CKL();
    return SPARC_OK;
}
template int mhd_ddx<double>(sparc_ctx*, const LineList<double, double>&, int);
template int mhd_ddx<float>(sparc_ctx*, const LineList<float, float>&, int);
template int mhd_ddy<double>(sparc_ctx*, const LineList<double, double>&, int);
template int mhd_ddy<float>(sparc_ctx*, const LineList<float, float>&, int);

int mhd_create(sparc_ctx* c) {
    c->mhd = new MhdState();
    MhdState& m = *c->mhd;
    const size_t es = esz(c);
    int rc;
    m.rows2d_z = c->f32 && c->P.option == 18 && rows2d_ddz_ok(c->nz);
    if ((rc = dalloc(c, &m.bg, (size_t)MB_COUNT * c->N * es))) return rc;
    CK(cudaMemsetAsync(m.bg, 0, (size_t)MB_COUNT * c->N * es, c->stream));   // 2-D leaves the y rows at 0
    if ((rc = dalloc(c, &m.pab, (size_t)2 * std::max(c->nzpml, 1) * c->NP * es))) return rc;
    if ((rc = dalloc(c, &m.g, (size_t)c->nz * es))) return rc;
    if ((rc = dalloc(c, &m.sponge, (size_t)c->nz * es))) return rc;
    if ((rc = dalloc(c, (void**)&m.plane, (size_t)c->NP * sizeof(int)))) return rc;
    if ((rc = dalloc(c, (void**)&m.plane_obs, (size_t)c->NP * sizeof(int)))) return rc;
    if ((rc = dalloc(c, &m.dw, (size_t)c->NP * es))) return rc;
    if ((rc = dalloc(c, &m.rx, (size_t)c->P.nx * es))) return rc;
    if ((rc = dalloc(c, &m.ry, (size_t)std::max(c->P.ny, 2) * es))) return rc;
    const int nwork = c->P.option == 8 ? (int)V8_COUNT : (int)MW_COUNT;
    if ((rc = dalloc(c, &m.work, (size_t)c->S * nwork * c->N * es))) return rc;
    const size_t pv = (size_t)c->S * PV_COUNT * std::max(c->nzpml, 1) * c->NP * es;
    if ((rc = dalloc(c, &m.pml, pv))) return rc;
    if ((rc = dalloc(c, &m.spml, pv))) return rc;
    CK(cudaMemsetAsync(m.pml, 0, pv, c->stream));
    CK(cudaMemsetAsync(m.spml, 0, pv, c->stream));   // 2-D never writes psi_dzby, psi_induction_by
    if ((rc = dalloc(c, &m.spec, (size_t)3 * c->S * c->fs * csz(c)))) return rc;
    if ((rc = dalloc(c, &m.fx, (size_t)2 * c->P.nx * es))) return rc;
    if ((rc = dalloc(c, &m.src, (size_t)c->S * c->NP * es))) return rc;
    return SPARC_OK;
}

// the pencil multipliers of set_background as factors of a packed row's nx
// complex points, over nx (the 2-D forms' damping and horizontal filter)
int mhd_set_tables(sparc_ctx* c) {
    const int nx = c->P.nx;
    std::vector<double> f(2 * (size_t)nx);
    for (int k = 0; k < nx; ++k) {
        const int h = std::min(k, nx - k);
        f[k] = c->pt_host[PT_DAMP * (size_t)c->M + h] / nx;
        f[nx + k] = c->pt_host[PT_HF * (size_t)c->M + h] / nx;
    }
    const std::vector<float> g(f.begin(), f.end());
    const int rc = c->f32 ? upload(c, c->mhd->fx, g.data(), g.size() * 4) : upload(c, c->mhd->fx, f.data(), f.size() * 8);
    if (rc) return rc;
    CK(cudaStreamSynchronize(c->stream));
    return SPARC_OK;
}

void mhd_destroy(sparc_ctx* c) {
    delete c->mhd;
    c->mhd = nullptr;
}

void* mhd_pml(sparc_ctx* c) { return c->mhd ? c->mhd->pml : nullptr; }
void* mhd_spml(sparc_ctx* c) { return c->mhd ? c->mhd->spml : nullptr; }
const int* mhd_planes(sparc_ctx* c) { return c->mhd ? c->mhd->plane : nullptr; }

// The magnetic parts of mp_Initialize_RHS (physics.f90:62-161, 204-208,
// 255-303, 356-363) in the reference's order; inputs are the 3-D cgs arrays
// READ_IN_FIELD reads, (nz, ny, nx) C order.
int mhd_set_background(sparc_ctx* c, const double* rho, const double* cs, const double* p, const double* bx,
                       const double* by, const double* bz) {
    MhdState& m = *c->mhd;
    const int nz = c->nz, nb = c->P.npmlbot, nt = c->P.npmltop;
    const long long N = c->N, NP = c->NP;
    const std::vector<double>& z = c->zq;
    // FP64 work: 6 inputs, curl (3), horizontal gradients (4), z gradients (2), rhoinv, c2rho0, scratch
    enum { W_RHO, W_C2, W_P, W_BX, W_BY, W_BZ, W_CBX, W_CBY, W_CBZ, W_GP0X, W_GP0Y, W_GR0X, W_GR0Y, W_GP0Z, W_GR0Z,
           W_RI, W_C2R, W_TMP, W_AZ, W_BZP, W_N };
    double* w64 = nullptr;
    int rc = dalloc(c, (void**)&w64, (size_t)W_N * N * 8);
    if (rc) return rc;
    auto W = [&](int i) { return w64 + (size_t)i * N; };
    const double* in[6] = {rho, cs, p, bx, by, bz};
    for (int i = 0; i < 6; ++i)
        if ((rc = upload(c, W(i), in[i], (size_t)N * 8))) return rc;
    // erad_2d / orad_2d (physics.f90:62-87): searched before READ_IN_FIELD,
    // on the density of solar_data (the quiet column) -- the same plane for
    // every pixel; loop bounds clamped to the box
    auto search = [&](int kc) {
        double temp = 1.0;
        int best = kc;
        for (int k = std::max(1, kc - 50); k <= std::min(nz, kc + 10); ++k)
            if (std::fabs(c->rhoq[kc - 1] - c->rhoq[k - 1]) <= temp) {
                temp = std::fabs(c->rhoq[kc - 1] - c->rhoq[k - 1]);
                best = k;
            }
        return best;
    };
    const int erad = search(c->e_rad), orad = search(c->o_rad);
    const int k2 = c->P.compute_adjoint ? orad : erad;
    const int ks = c->P.src_k > 0 ? c->P.src_k : k2;
    std::vector<int> plane(NP, ks - 1), plane_obs(NP, orad - 1);
    const double dw2 = 2.0 / (z[k2] - z[k2 - 2]);
    // spongez (physics.f90:104-108)
    std::vector<double> spz(nz), taper(nz, 1.0), alph(nz), gk(nz);
    for (int k = 0; k < nz; ++k)
        spz[k] = 200.0 / (1.0 + std::exp((R4(1.002) - z[k]) / R4(0.0001))) +
                 300.0 / (1.0 + std::exp((z[k] - (z[0] + R4(0.005))) / R4(0.0005)));
    // ((k-nz)/10.0)**4. in REAL*4 for k = nz-10..nz (physics.f90:123-125)
    for (int k1 = std::max(1, nz - 10); k1 <= nz; ++k1) {
        const float tt = (float)(k1 - nz) / 10.0f;
        taper[k1 - 1] = (double)std::pow(tt, 4.0f);
    }
    // alphaz of the PML planes (physics.f90:269-285)
    for (int k = 1; k <= nz; ++k) {
        double a0 = c->pi * R4(0.005) * c->diml / c->dimc;
        if (k < nb + 1) a0 = c->pi * R4(0.005) * c->diml / c->dimc * (z[k - 1] - z[0]) / (z[nb - 1] - z[0]);
        if (k > nz - nt) a0 = c->pi * R4(0.005) * c->diml / c->dimc * (z[nz - 1] - z[k - 1]) / (z[nz - 1] - z[nz - nt]);
        alph[k - 1] = a0;
    }
    // gravity with the decay of the (1,1) column (physics.f90:287,299), on the host
    {
        const double dimb = std::sqrt(4.0 * c->pi * c->dimc * c->dimc * c->dimrho);
        auto tempin00 = [&](int k) {
            const long long i = (long long)k * NP;
            const double r = rho[i] / c->dimrho, css = cs[i] / c->dimc;
            const double x = bx[i] / dimb, y = by[i] / dimb, zz = bz[i] / dimb;
            double red = (std::pow(zz, 2.0) + std::pow(x, 2.0) + std::pow(y, 2.0)) / (r * std::pow(c->cq[k], 2.0));
            red = 8.0 / (8.0 + red) * taper[k];
            const double sc = std::pow(red, 0.5);
            return std::pow(std::pow(css, 2.0) + (std::pow(x * sc, 2.0) + std::pow(y * sc, 2.0) +
                                                   std::pow(zz * sc, 2.0)) / r, 0.5);
        };
        for (int k = 1; k <= nz; ++k) {
            double fdec = 1.0;
            if (k < nb + 1) {
                const double r = (z[nb - 1] - z[k - 1]) / (z[nb - 1] - z[0]);
                const double dampz = 2.0 * 3.0 * 3.0 * tempin00(0) / (z[nb - 1] - z[0]) * (r * r);
                fdec = alph[k - 1] / (dampz + alph[k - 1]);
            }
            if (k > nz - nt) {
                const double r = (z[nz - nt] - z[k - 1]) / (z[nz - 1] - z[nz - nt]);
                const double dampz = 3.0 * 3.0 * tempin00(nz - 1) / (z[nz - 1] - z[nz - nt]) * (r * r);
                fdec = alph[k - 1] / (dampz + alph[k - 1]);
            }
            gk[k - 1] = c->zt_host[(size_t)ZT_GRAW * nz + k - 1] * fdec;
        }
    }
    double *d_cq = nullptr, *d_taper = nullptr, *d_z = nullptr, *d_alph = nullptr;
    if ((rc = dalloc(c, (void**)&d_cq, nz * 8)) || (rc = dalloc(c, (void**)&d_taper, nz * 8)) ||
        (rc = dalloc(c, (void**)&d_z, nz * 8)) || (rc = dalloc(c, (void**)&d_alph, nz * 8)))
        return rc;
    if ((rc = upload(c, d_cq, c->cq.data(), nz * 8)) || (rc = upload(c, d_taper, taper.data(), nz * 8)) ||
        (rc = upload(c, d_z, z.data(), nz * 8)) || (rc = upload(c, d_alph, alph.data(), nz * 8)))
        return rc;
    const double dimb = std::sqrt(4.0 * c->pi * c->dimc * c->dimc * c->dimrho);
    mhd_read_kernel<<<nb256(N), 256, 0, c->stream>>>(W(W_RHO), W(W_C2), W(W_P), W(W_BX), W(W_BY), W(W_BZ), d_cq,
                                                     d_taper, NP, nz, c->dimrho, c->dimc, dimb);
    CKL();
    // FP64 derivative multipliers for the set-up, then the curl of B0 as the
    // reference forms it (physics.f90:131-159: the d/dz parts are discarded)
    // and the horizontal background gradients (physics.f90:356-363)
    {
        std::vector<double> rx(c->P.nx), ry(std::max(c->P.ny, 2), 0.0);
        for (int k = 0; k < c->P.nx; ++k) {
            const int kk = k < c->P.nx / 2 ? k : (k == c->P.nx / 2 ? 0 : k - c->P.nx);
            rx[k] = (double)kk * c->normx * 2.0 * c->pi * c->stretchx;
        }
        for (int k = 0; k < c->P.ny; ++k) {
            const int kk = k < c->P.ny / 2 ? k : (k == c->P.ny / 2 ? 0 : k - c->P.ny);
            ry[k] = (double)kk * c->normy * 2.0 * c->pi * c->stretchy;
        }
        double *rx64 = nullptr, *ry64 = nullptr;
        if ((rc = dalloc(c, (void**)&rx64, rx.size() * 8)) || (rc = dalloc(c, (void**)&ry64, ry.size() * 8))) return rc;
        if ((rc = upload(c, rx64, rx.data(), rx.size() * 8)) || (rc = upload(c, ry64, ry.data(), ry.size() * 8))) return rc;
        void* rx0 = m.rx; void* ry0 = m.ry;
        m.rx = rx64; m.ry = ry64;                 // FP64 multipliers while setting up
        if ((rc = ddx_launch<double>(c, W(W_BY), W(W_CBZ))) || (rc = ddy_launch<double>(c, W(W_BX), W(W_TMP))))
            return rc;
        axpby_kernel<<<nb256(N), 256, 0, c->stream>>>(W(W_CBZ), W(W_CBZ), 1.0, W(W_TMP), -1.0, N);
        if ((rc = ddy_launch<double>(c, W(W_BZ), W(W_CBX))) || (rc = ddx_launch<double>(c, W(W_BZ), W(W_TMP))))
            return rc;
        axpby_kernel<<<nb256(N), 256, 0, c->stream>>>(W(W_CBY), W(W_TMP), -1.0, nullptr, 0.0, N);
        if ((rc = ddx_launch<double>(c, W(W_RHO), W(W_GR0X))) || (rc = ddy_launch<double>(c, W(W_RHO), W(W_GR0Y))) ||
            (rc = ddx_launch<double>(c, W(W_P), W(W_GP0X))) || (rc = ddy_launch<double>(c, W(W_P), W(W_GP0Y))))
            return rc;
        // d/dz of the background in FP64 (physics.f90:207-208)
        if ((rc = ddz_launch<double>(c, W(W_RHO), W(W_GR0Z), 1)) ||
            (rc = ddz_launch<double>(c, W(W_P), W(W_GP0Z), 1)))
            return rc;
        CKL();
        // multipliers of the element type for the steps
        std::vector<double> rxs = rx, rys = ry;
        m.rx = rx0; m.ry = ry0;
        if (c->f32) {
            std::vector<float> fx(rx.begin(), rx.end()), fy(ry.begin(), ry.end());
            if ((rc = upload(c, m.rx, fx.data(), fx.size() * 4)) || (rc = upload(c, m.ry, fy.data(), fy.size() * 4)))
                return rc;
        } else {
            if ((rc = upload(c, m.rx, rx.data(), rx.size() * 8)) || (rc = upload(c, m.ry, ry.data(), ry.size() * 8)))
                return rc;
        }
    }
    rhoinv_kernel<<<nb256(N), 256, 0, c->stream>>>(W(W_RI), W(W_C2R), W(W_RHO), W(W_C2), N);
    CKL();
    mhd_pml_kernel<<<nb256(N), 256, 0, c->stream>>>(W(W_GP0Z), W(W_GR0Z), W(W_AZ), W(W_BZP), W(W_C2), W(W_RHO),
                                                    W(W_BX), W(W_BY), W(W_BZ), d_z, d_alph, NP, nz, nb, nt);
    CKL();
    // to the element type: background fields, bottom PML coefficients, tables
    const int src_of[MB_COUNT] = {W_BX, W_BY, W_BZ, W_CBX, W_CBY, W_CBZ, W_GP0X, W_GP0Y, W_GP0Z, W_GR0X,
                                  W_GR0Y, W_GR0Z, W_C2R, W_RHO, W_RI};
    // a_z, b_z of all nzpml PML planes in pmlindex order (option 10 reads the bottom nb)
    const long long nbp = (long long)std::max(c->nzpml, 1) * NP, npz = nbp;
    for (int i = 0; i < MB_COUNT; ++i) {
        if (c->f32) to_t_kernel<float><<<nb256(N), 256, 0, c->stream>>>((float*)m.bg + (size_t)i * N, W(src_of[i]), N);
        else to_t_kernel<double><<<nb256(N), 256, 0, c->stream>>>((double*)m.bg + (size_t)i * N, W(src_of[i]), N);
    }
    if (c->f32) {
        to_t_kernel<float><<<nb256(nbp), 256, 0, c->stream>>>((float*)m.pab, W(W_AZ), nbp);
        to_t_kernel<float><<<nb256(nbp), 256, 0, c->stream>>>((float*)m.pab + npz, W(W_BZP), nbp);
    } else {
        to_t_kernel<double><<<nb256(nbp), 256, 0, c->stream>>>((double*)m.pab, W(W_AZ), nbp);
        to_t_kernel<double><<<nb256(nbp), 256, 0, c->stream>>>((double*)m.pab + npz, W(W_BZP), nbp);
    }
    CKL();
    std::vector<double> dwv(NP, dw2);
    if (c->f32) {
        std::vector<float> g32(gk.begin(), gk.end()), s32(spz.begin(), spz.end()), d32(dwv.begin(), dwv.end());
        if ((rc = upload(c, m.g, g32.data(), nz * 4)) || (rc = upload(c, m.sponge, s32.data(), nz * 4)) ||
            (rc = upload(c, m.dw, d32.data(), NP * 4)))
            return rc;
    } else {
        if ((rc = upload(c, m.g, gk.data(), nz * 8)) || (rc = upload(c, m.sponge, spz.data(), nz * 8)) ||
            (rc = upload(c, m.dw, dwv.data(), NP * 8)))
            return rc;
    }
    if ((rc = upload(c, m.plane, plane.data(), NP * sizeof(int)))) return rc;
    if ((rc = upload(c, m.plane_obs, plane_obs.data(), NP * sizeof(int)))) return rc;
    CK(cudaStreamSynchronize(c->stream));
    // release the FP64 set-up buffers
    for (void* pp : {(void*)w64, (void*)d_cq, (void*)d_taper, (void*)d_z, (void*)d_alph}) {
        auto it = std::find(c->allocs.begin(), c->allocs.end(), pp);
        if (it != c->allocs.end()) c->allocs.erase(it);
        cudaFree(pp);
    }
    c->dev_bytes -= (long long)W_N * N * 8 + 4LL * nz * 8;
    m.have_bg = true;
    return SPARC_OK;
}

// ---- option 18 (2-D, ny = 1) ---------------------------------------------------

namespace {

// DBYD1 (dbyd1.f) with ibc = 0 along x for n2 rows of n1: the DBYD2 compact
// scheme with its coefficients in default REAL (the file declares no
// kinds), zero end rows, solved by TRIDAG (tridag.f: Thomas with divisions)
void host_dbyd1_ibc0(std::vector<double>& a, const double* b, int n1, long n2) {
    const float d1i = (float)(n1 - 1);
    const double C1 = (double)(d1i * 7.0f / 9.0f), C2 = (double)(d1i / 36.0f);
    const double B1 = (double)(-43.0f / 96.0f * d1i), B2 = (double)(-5.0f / 6.0f * d1i);
    const double B3 = (double)(9.0f / 8.0f * d1i), B4 = (double)(1.0f / 6.0f * d1i), B5 = (double)(-1.0f / 96.0f * d1i);
    std::vector<double> uppr(n1 + 1, 0.0), lowr(n1 + 1, 0.0), diag(n1 + 1, 1.0), gam(n1 + 1), ud(n1 + 1), r(n1 + 1);
    for (int J = 3; J <= n1 - 2; ++J) uppr[J] = (double)(1.0f / 3.0f);
    uppr[2] = (double)(3.0f / 4.0f);
    uppr[n1 - 1] = (double)(1.0f / 8.0f);
    for (int I = 1; I <= n1; ++I) lowr[I] = uppr[n1 - I + 1];
    lowr[n1] = 0.0;
    a.assign((size_t)n1 * n2, 0.0);
    for (long i = 0; i < n2; ++i) {
        const double* B = b + i * n1 - 1;
        for (int J = 3; J <= n1 - 2; ++J) r[J] = C1 * (B[J + 1] - B[J - 1]) + C2 * (B[J + 2] - B[J - 2]);
        r[2] = B1 * B[1] + B2 * B[2] + B3 * B[3] + B4 * B[4] + B5 * B[5];
        r[n1 - 1] = -(B1 * B[n1] + B2 * B[n1 - 1] + B3 * B[n1 - 2] + B4 * B[n1 - 3] + B5 * B[n1 - 4]);
        r[1] = 0.0;
        r[n1] = 0.0;
        double bet = diag[1];
        ud[1] = r[1] / bet;
        for (int J = 2; J <= n1; ++J) {
            gam[J] = uppr[J - 1] / bet;
            bet = diag[J] - lowr[J] * gam[J];
            ud[J] = (r[J] - lowr[J] * ud[J - 1]) / bet;
        }
        for (int J = n1 - 1; J >= 1; --J) ud[J] = ud[J] - gam[J + 1] * ud[J + 1];
        for (int J = 1; J <= n1; ++J) a[(size_t)i * n1 + J - 1] = ud[J];
    }
}

// physics2d.f90:154-172: non-dimensional background, B = (B_x, B_z) / dimb
__global__ void mhd2d_read_kernel(double* p0, double* rho0, double* c2, double* bx, double* bz, long long n,
                                  double dimrho, double dimc, double dimb) {
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n) return;
    bx[t] = bx[t] / dimb;
    bz[t] = bz[t] / dimb;
    p0[t] = p0[t] / (dimrho * pow(dimc, 2.0));
    rho0[t] = rho0[t] / dimrho;
    c2[t] = pow(c2[t] / dimc, 2.0);
}

// PML of physics2d.f90:262-297 with the magnetic wave speed: tempin at
// plane 1 (bottom) and nz-5 (top), factor 3*3 at both ends; a_z, b_z stored
// in pmlindex order; g(k) decayed with the (1,1) column
__global__ void mhd2d_pml_kernel(double* gp0z, double* gr0z, double* az, double* bzp, double* gk, const double* graw,
                                 const double* c2, const double* rho0, const double* bx, const double* bz,
                                 const double* z, const double* alph, long long NP, int nz, int nb, int nt) {
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= NP * nz) return;
    const int k = (int)(t / NP);
    const long long q = t - (long long)k * NP;
    const bool bot = k < nb, top = k >= nz - nt;
    auto tempin = [&](int kk) {
        const long long i = q + NP * kk;
        return pow(c2[i] + (pow(bx[i], 2.0) + pow(bz[i], 2.0)) / rho0[i], 0.5);
    };
    double fdec = 1.0, dampz = 0.0;
    if (bot) {
        const double r = (z[nb - 1] - z[k]) / (z[nb - 1] - z[0]);
        dampz = 3.0 * 3.0 * tempin(0) / (z[nb - 1] - z[0]) * (r * r);
        fdec = alph[k] / (dampz + alph[k]);
        gp0z[t] *= fdec; gr0z[t] *= fdec;
        az[(long long)k * NP + q] = -dampz;
        bzp[(long long)k * NP + q] = -alph[k] - dampz;
    }
    if (top) {
        const double r = (z[nz - nt] - z[k]) / (z[nz - 1] - z[nz - nt]);
        dampz = 3.0 * 3.0 * tempin(nz - 6) / (z[nz - 1] - z[nz - nt]) * (r * r);
        fdec = alph[k] / (dampz + alph[k]);
        gp0z[t] *= fdec; gr0z[t] *= fdec;
        const long long ip = nb + (k - (nz - nt));
        az[ip * NP + q] = -dampz;
        bzp[ip * NP + q] = -alph[k] - dampz;
    }
    if (q == 0) gk[k] = (bot || top) ? graw[k] * fdec : graw[k];
}

}  // namespace

int mhd2d_set_background(sparc_ctx* c, const double* p, const double* rho, const double* cs, const double* psi) {
    MhdState& m = *c->mhd;
    const int nz = c->nz, nb = c->P.npmlbot, nt = c->P.npmltop, nx = c->P.nx;
    const long long N = c->N, NP = c->NP;
    const std::vector<double>& z = c->zq;
    enum { W_P, W_RHO, W_C2, W_PSI, W_BX, W_BZ, W_CBY, W_TMP, W_RI, W_C2R, W_GR0Z, W_GP0Z, W_GR0X, W_GP0X, W_AZ,
           W_BZP, W_KBX, W_KCY, W_N };
    double* w64 = nullptr;
    int rc = dalloc(c, (void**)&w64, (size_t)W_N * N * 8);
    if (rc) return rc;
    auto W = [&](int i) { return w64 + (size_t)i * N; };
    if ((rc = upload(c, W(W_P), p, N * 8)) || (rc = upload(c, W(W_RHO), rho, N * 8)) ||
        (rc = upload(c, W(W_C2), cs, N * 8)) || (rc = upload(c, W(W_PSI), psi, N * 8)))
        return rc;
    // B_x = -d psi/dz (ddz, bc 1); B_z = DBYD1(psi) * stretchx (physics2d.f90:140-146)
    if ((rc = ddz_launch<double>(c, W(W_PSI), W(W_BX), 1))) return rc;
    axpby_kernel<<<nb256(N), 256, 0, c->stream>>>(W(W_BX), W(W_BX), -1.0, nullptr, 0.0, N);
    std::vector<double> bzh;
    host_dbyd1_ibc0(bzh, psi, nx, (long)nz);
    for (double& v : bzh) v = v * c->stretchx;
    if ((rc = upload(c, W(W_BZ), bzh.data(), N * 8))) return rc;
    const double dimb = std::sqrt(4.0 * c->pi * c->dimc * c->dimc * c->dimrho);
    mhd2d_read_kernel<<<nb256(N), 256, 0, c->stream>>>(W(W_P), W(W_RHO), W(W_C2), W(W_BX), W(W_BZ), N, c->dimrho,
                                                       c->dimc, dimb);
    CKL();
    // curl_y B0 = dBx/dz - dBz/dx (physics2d.f90:180-183), then the gradients
    std::vector<double> rx(nx);
    for (int k = 0; k < nx; ++k) {
        const int kk = k < nx / 2 ? k : (k == nx / 2 ? 0 : k - nx);
        rx[k] = (double)kk * c->normx * 2.0 * c->pi * c->stretchx;
    }
    double* rx64 = nullptr;
    if ((rc = dalloc(c, (void**)&rx64, nx * 8)) || (rc = upload(c, rx64, rx.data(), nx * 8))) return rc;
    void* rx0 = m.rx;
    m.rx = rx64;
    if ((rc = ddz_launch<double>(c, W(W_BX), W(W_CBY), 1)) ||
        (rc = ddx_launch<double>(c, W(W_BZ), W(W_TMP))))
        return rc;
    axpby_kernel<<<nb256(N), 256, 0, c->stream>>>(W(W_CBY), W(W_CBY), 1.0, W(W_TMP), -1.0, N);
    rhoinv_kernel<<<nb256(N), 256, 0, c->stream>>>(W(W_RI), W(W_C2R), W(W_RHO), W(W_C2), N);
    if ((rc = ddz_launch<double>(c, W(W_RHO), W(W_GR0Z), 1)) ||
        (rc = ddz_launch<double>(c, W(W_P), W(W_GP0Z), 1)))
        return rc;
    // PML and gravity
    std::vector<double> alph(nz);
    for (int k = 1; k <= nz; ++k) {
        double a0 = c->pi * R4(0.005) * c->diml / c->dimc;
        if (k < nb + 1) a0 = c->pi * R4(0.005) * c->diml / c->dimc * (z[k - 1] - z[0]) / (z[nb - 1] - z[0]);
        if (k > nz - nt) a0 = c->pi * R4(0.005) * c->diml / c->dimc * (z[nz - 1] - z[k - 1]) / (z[nz - 1] - z[nz - nt]);
        alph[k - 1] = a0;
    }
    double *d_z = nullptr, *d_alph = nullptr, *d_g = nullptr;
    if ((rc = dalloc(c, (void**)&d_z, nz * 8)) || (rc = dalloc(c, (void**)&d_alph, nz * 8)) ||
        (rc = dalloc(c, (void**)&d_g, nz * 8)))
        return rc;
    if ((rc = upload(c, d_z, z.data(), nz * 8)) || (rc = upload(c, d_alph, alph.data(), nz * 8))) return rc;
    mhd2d_pml_kernel<<<nb256(N), 256, 0, c->stream>>>(W(W_GP0Z), W(W_GR0Z), W(W_AZ), W(W_BZP), d_g,
                                                      c->zt64 + (size_t)ZT_GRAW * nz, W(W_C2), W(W_RHO), W(W_BX),
                                                      W(W_BZ), d_z, d_alph, NP, nz, nb, nt);
    CKL();
    // horizontal gradients (physics2d.f90:318-321)
    if ((rc = ddx_launch<double>(c, W(W_RHO), W(W_GR0X))) || (rc = ddx_launch<double>(c, W(W_P), W(W_GP0X))))
        return rc;
    // B0 of kernel mode (kernels.f90:99-133): box = -ddzkern(psi, 0) / dimb
    // (bc 0 and FILTER_VAR_Z, unlike the solve's ddz bc 1), boz as the
    // solve's, curl_y B0 = ddzkern(box, 0) - d boz/dx (CURL_KERN with bcz = 0)
    if ((rc = ddz_launch<double>(c, W(W_PSI), W(W_KBX), 0))) return rc;
    zfilter_phys_kernel<double><<<dim3(nb256(NP), 1), 256, 0, c->stream>>>(W(W_KBX), NP, nz, 0);
    neg_div_kernel<<<nb256(N), 256, 0, c->stream>>>(W(W_KBX), dimb, N);
    if ((rc = ddz_launch<double>(c, W(W_KBX), W(W_KCY), 0))) return rc;
    zfilter_phys_kernel<double><<<dim3(nb256(NP), 1), 256, 0, c->stream>>>(W(W_KCY), NP, nz, 0);
    if ((rc = ddx_launch<double>(c, W(W_BZ), W(W_TMP)))) return rc;
    axpby_kernel<<<nb256(N), 256, 0, c->stream>>>(W(W_KCY), W(W_KCY), 1.0, W(W_TMP), -1.0, N);
    CKL();
    if (!m.kc2) {
        if ((rc = dalloc(c, (void**)&m.kc2, N * 8)) || (rc = dalloc(c, (void**)&m.krho, N * 8)) ||
            (rc = dalloc(c, &m.kbox, N * esz(c))) || (rc = dalloc(c, &m.kcby, N * esz(c))))
            return rc;
    }
    CK(cudaMemcpyAsync(m.kc2, W(W_C2), N * 8, cudaMemcpyDeviceToDevice, c->stream));
    CK(cudaMemcpyAsync(m.krho, W(W_RHO), N * 8, cudaMemcpyDeviceToDevice, c->stream));
    if (c->f32) {
        to_t_kernel<float><<<nb256(N), 256, 0, c->stream>>>((float*)m.kbox, W(W_KBX), N);
        to_t_kernel<float><<<nb256(N), 256, 0, c->stream>>>((float*)m.kcby, W(W_KCY), N);
    } else {
        to_t_kernel<double><<<nb256(N), 256, 0, c->stream>>>((double*)m.kbox, W(W_KBX), N);
        to_t_kernel<double><<<nb256(N), 256, 0, c->stream>>>((double*)m.kcby, W(W_KCY), N);
    }
    m.rx64 = rx64;                           // kept for the kernel scaling in FP64
    m.rx = rx0;
    {
        std::vector<double> rxs(rx);
        if (c->f32) {
            std::vector<float> fx(rxs.begin(), rxs.end());
            if ((rc = upload(c, m.rx, fx.data(), nx * 4))) return rc;
        } else if ((rc = upload(c, m.rx, rxs.data(), nx * 8))) {
            return rc;
        }
    }
    // to the element type (the y components and the other curl components stay 0)
    const int dst_of[] = {MB_BOX, MB_BOZ, MB_CBOY, MB_GP0X, MB_GP0Z, MB_GR0X, MB_GR0Z, MB_C2RHO0, MB_RHO0, MB_RHOINV};
    const int src_of[] = {W_BX, W_BZ, W_CBY, W_GP0X, W_GP0Z, W_GR0X, W_GR0Z, W_C2R, W_RHO, W_RI};
    const long long npz = (long long)std::max(c->nzpml, 1) * NP;
    for (int i = 0; i < 10; ++i) {
        if (c->f32) to_t_kernel<float><<<nb256(N), 256, 0, c->stream>>>((float*)m.bg + (size_t)dst_of[i] * N, W(src_of[i]), N);
        else to_t_kernel<double><<<nb256(N), 256, 0, c->stream>>>((double*)m.bg + (size_t)dst_of[i] * N, W(src_of[i]), N);
    }
    if (c->f32) {
        to_t_kernel<float><<<nb256(npz), 256, 0, c->stream>>>((float*)m.pab, W(W_AZ), npz);
        to_t_kernel<float><<<nb256(npz), 256, 0, c->stream>>>((float*)m.pab + npz, W(W_BZP), npz);
        to_t_kernel<float><<<nb256(nz), 256, 0, c->stream>>>((float*)m.g, d_g, nz);
    } else {
        to_t_kernel<double><<<nb256(npz), 256, 0, c->stream>>>((double*)m.pab, W(W_AZ), npz);
        to_t_kernel<double><<<nb256(npz), 256, 0, c->stream>>>((double*)m.pab + npz, W(W_BZP), npz);
        to_t_kernel<double><<<nb256(nz), 256, 0, c->stream>>>((double*)m.g, d_g, nz);
    }
    CKL();
    // source planes: erad_2d = e_rad, orad_2d = o_rad (physics2d.f90:334-341)
    const int k2 = c->P.compute_adjoint ? c->o_rad : c->e_rad;
    const int ks = c->P.src_k > 0 ? c->P.src_k : k2;
    std::vector<int> plane(NP, ks - 1), plane_obs(NP, c->o_rad - 1);
    std::vector<double> dwv(NP, 2.0 / (z[k2] - z[k2 - 2]));
    if (c->f32) {
        std::vector<float> d32(dwv.begin(), dwv.end());
        if ((rc = upload(c, m.dw, d32.data(), NP * 4))) return rc;
    } else if ((rc = upload(c, m.dw, dwv.data(), NP * 8))) {
        return rc;
    }
    if ((rc = upload(c, m.plane, plane.data(), NP * sizeof(int))) ||
        (rc = upload(c, m.plane_obs, plane_obs.data(), NP * sizeof(int))))
        return rc;
    CK(cudaStreamSynchronize(c->stream));
    for (void* pp : {(void*)w64, (void*)d_z, (void*)d_alph, (void*)d_g}) {
        auto it = std::find(c->allocs.begin(), c->allocs.end(), pp);
        if (it != c->allocs.end()) c->allocs.erase(it);
        cudaFree(pp);
    }
    c->dev_bytes -= (long long)W_N * N * 8 + 3LL * nz * 8;
    m.have_bg = true;
    return SPARC_OK;
}

// ---- sensitivity kernels of the 2-D MHD form (option 18) ---------------------

namespace {

// ddzkern: DBYD2 * stretch, then FILTER_VAR_Z (kernels.f90:609-621)
template <typename T>
int ddzk_launch(sparc_ctx* c, const T* in, T* out, int bc) {
    int rc = ddz_launch<T>(c, in, out, bc);
    if (rc) return rc;
    zfilter_phys_kernel<T><<<dim3(nb256(c->NP), 1), 256, 0, c->stream>>>(out, c->NP, c->nz, 0);
    c->launches++;
    CKL();
    return SPARC_OK;
}

// the seven physical fields of a kernel snapshot of sources s0..s0+G-1 (the
// layout of the quiet path's store): forward div(xi) (COMPUTE_DIV), acc =
// scr(v) (3), xi (3); adjoint div(v), v (3), grad(v_z grav) (3)
template <typename T>
int mhd2d_derive_t(sparc_ctx* c, int s0, int G, bool adjoint, T* out, long long ofs) {
    MhdState& m = *c->mhd;
    const long long N = c->N, fs2 = 2 * c->fs;
    const T* zt = (const T*)c->zt;
    T* sc = (T*)m.work + (size_t)MW_P * N;      // scratch: work fields of slot 0
    T* sc2 = (T*)m.work + (size_t)MW_R * N;
    int rc;
    for (int g = 0; g < G; ++g) {
        const int s = s0 + g;
        auto A = [&](int f) { return (T*)c->a + ((size_t)s * c->nf + f) * fs2; };
        auto S = [&](int f) { return (T*)c->scr + ((size_t)s * c->nf + f) * fs2; };
        auto O = [&](int f) { return out + (size_t)f * ofs + (size_t)g * N; };
        const int fx = adjoint ? 3 : 0;
        if ((rc = ddx_launch<T>(c, A(fx), O(0))) || (rc = ddzk_launch<T>(c, A(fx + 2), sc, 1))) return rc;
        add_kernel<T><<<nb256(N), 256, 0, c->stream>>>(O(0), sc, N);
        for (int q = 0; q < 3; ++q) {
            CK(cudaMemcpyAsync(O(1 + q), adjoint ? A(3 + q) : S(3 + q), N * sizeof(T), cudaMemcpyDeviceToDevice,
                               c->stream));
            if (!adjoint) CK(cudaMemcpyAsync(O(4 + q), A(q), N * sizeof(T), cudaMemcpyDeviceToDevice, c->stream));
        }
        if (adjoint) {
            // grad(v_z grav) (kernels.f90:299-304)
            zscale_kernel<T><<<nb256(N), 256, 0, c->stream>>>(sc2, A(5), zt + (size_t)ZT_GRAW * c->nz, c->NP, N);
            if ((rc = ddx_launch<T>(c, sc2, O(4))) || (rc = ddzk_launch<T>(c, sc2, O(6), 1))) return rc;
            CK(cudaMemsetAsync(O(5), 0, N * sizeof(T), c->stream));
        }
        c->launches += adjoint ? 3 : 1;
        CKL();
    }
    return SPARC_OK;
}

// the y-only products of the MAGNETIC_KERNELS block in 2-D (B0 = (Bx, 0, Bz),
// curl B0 = (0, cby, 0), d/dy = 0): ty = (xi x B0)_y, uy = (v x B0)_y,
// (wx, wz) = v x curl B0, vy = (B0 x xi div v)_y
template <typename T>
__global__ void kb_products_kernel(const T* __restrict__ fxx, const T* __restrict__ fxz, const T* __restrict__ avx,
                                   const T* __restrict__ avz, const T* __restrict__ dA, const T* __restrict__ box,
                                   const T* __restrict__ boz, const T* __restrict__ cby, T* __restrict__ ty,
                                   T* __restrict__ uy, T* __restrict__ wx, T* __restrict__ wz, T* __restrict__ vy,
                                   long long n) {
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n) return;
    ty[t] = box[t] * fxz[t] - fxx[t] * boz[t];
    uy[t] = box[t] * avz[t] - avx[t] * boz[t];
    wx[t] = -(avz[t] * cby[t]);
    wz[t] = avx[t] * cby[t];
    const T tx = fxx[t] * dA[t], tz = fxz[t] * dA[t];
    vy[t] = tx * boz[t] - box[t] * tz;
}

// fb = curl(0, ty, 0) = (-ddzk ty, 0, d ty/dx); ab likewise from uy; t3y = (fb x v)_y
template <typename T>
__global__ void kb_curls_kernel(T* __restrict__ fbx, const T* __restrict__ fbz, T* __restrict__ abx,
                                const T* __restrict__ avx, const T* __restrict__ avz, T* __restrict__ t3y,
                                long long n) {
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n) return;
    const T bx = -fbx[t];
    fbx[t] = bx;
    abx[t] = -abx[t];
    t3y[t] = avx[t] * fbz[t] - bx * avz[t];
}

// kernelb += the six terms in the reference's order (kernels.f90:337-453)
template <typename T>
__global__ void kb_accum_kernel(double* __restrict__ kbx, double* __restrict__ kbz, const T* __restrict__ fxx,
                                const T* __restrict__ fxz, const T* __restrict__ avx, const T* __restrict__ avz,
                                const T* __restrict__ dA, const T* __restrict__ cby, const T* __restrict__ r1,
                                const T* __restrict__ r2, const T* __restrict__ u1, const T* __restrict__ u2,
                                const T* __restrict__ s1, const T* __restrict__ s2, const T* __restrict__ p1,
                                const T* __restrict__ p2, const T* __restrict__ q1, const T* __restrict__ q2,
                                long long n) {
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n) return;
    const T t2y = r1[t] - r2[t];                    // curl(curl(xi x B0))_y
    const T t4y = s1[t] - s2[t];                    // curl(curl(v x B0))_y
    const T sy = p1[t] - p2[t];                     // curl(v x curl B0)_y
    double x = kbx[t], z = kbz[t];
    x = x + (double)(-(avz[t] * t2y)); z = z + (double)(avx[t] * t2y);
    x = x + (double)(-u1[t]);          z = z + (double)u2[t];
    x = x + (double)(-(fxz[t] * t4y)); z = z + (double)(fxx[t] * t4y);
    x = x + (double)(sy * fxz[t]);     z = z + (double)(-(sy * fxx[t]));
    x = x + (double)(-(fxz[t] * cby[t]) * dA[t]);
    z = z + (double)((fxx[t] * cby[t]) * dA[t]);
    x = x + (double)(-q1[t]);          z = z + (double)q2[t];
    kbx[t] = x;
    kbz[t] = z;
}

template <typename T>
int mhd2d_kernel_b_t(sparc_ctx* c, const T* fst, long long sfs, const T* adj, long long afs, int s0, int G) {
    MhdState& m = *c->mhd;
    const long long N = c->N;
    const T* zt = (const T*)c->zt;
    T* w = (T*)m.work;                               // work fields of slot 0 as scratch
    auto Wf = [&](int i) { return w + (size_t)i * N; };
    T *ty = Wf(0), *uy = Wf(1), *wx = Wf(2), *wz = Wf(3), *vy = Wf(4), *fbx = Wf(5), *fbz = Wf(6), *abx = Wf(7);
    T *abz = Wf(8), *p1 = Wf(9), *p2 = Wf(10), *q1 = Wf(11), *q2 = Wf(12), *t3y = Wf(13), *r1 = Wf(14);
    T *r2 = Wf(15), *s1 = Wf(16), *s2 = Wf(17), *u1 = Wf(18), *u2 = Wf(19);
    const unsigned nb = nb256(N);
    int rc;
    for (int g = 0; g < G; ++g) {
        const T* fxx = fst + 4 * sfs + (size_t)g * N;
        const T* fxz = fst + 6 * sfs + (size_t)g * N;
        const T* dA = adj + (size_t)g * N;
        const T* avx = adj + afs + (size_t)g * N;
        const T* avz = adj + 3 * afs + (size_t)g * N;
        double* kb = m.kbacc + (size_t)(s0 + g) * 2 * N;
        kb_products_kernel<T><<<nb, 256, 0, c->stream>>>(fxx, fxz, avx, avz, dA, (const T*)m.kbox,
                                                         (const T*)m.bg + (size_t)MB_BOZ * N, (const T*)m.kcby, ty, uy,
                                                         wx, wz, vy, N);
        if ((rc = ddzk_launch<T>(c, ty, fbx, 0)) || (rc = ddx_launch<T>(c, ty, fbz)) ||
            (rc = ddzk_launch<T>(c, uy, abx, 0)) || (rc = ddx_launch<T>(c, uy, abz)) ||
            (rc = ddzk_launch<T>(c, wx, p1, 0)) || (rc = ddx_launch<T>(c, wz, p2)) ||
            (rc = ddzk_launch<T>(c, vy, q1, 0)) || (rc = ddx_launch<T>(c, vy, q2)))
            return rc;
        kb_curls_kernel<T><<<nb, 256, 0, c->stream>>>(fbx, fbz, abx, avx, avz, t3y, N);
        if ((rc = ddzk_launch<T>(c, fbx, r1, 0)) || (rc = ddx_launch<T>(c, fbz, r2)) ||
            (rc = ddzk_launch<T>(c, abx, s1, 0)) || (rc = ddx_launch<T>(c, abz, s2)) ||
            (rc = ddzk_launch<T>(c, t3y, u1, 0)) || (rc = ddx_launch<T>(c, t3y, u2)))
            return rc;
        kb_accum_kernel<T><<<nb, 256, 0, c->stream>>>(kb, kb + N, fxx, fxz, avx, avz, dA, (const T*)m.kcby, r1, r2,
                                                      u1, u2, s1, s2, p1, p2, q1, q2, N);
        c->launches += 3;
        CKL();
    }
    return SPARC_OK;
}

// kernel_b * scale for x and z, and the vector-potential kernel as the y
// component of CURL_KERN of (kernel_bx, 0, kernel_bz), in FP64
__global__ void kb_finish_kernel(double* __restrict__ out, const double* __restrict__ acc, double scale, int nsum,
                                 long long acc_ss, long long n) {
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n) return;
    double x = 0, z = 0;
    for (int s = 0; s < nsum; ++s) {
        x += acc[s * acc_ss + t];
        z += acc[s * acc_ss + n + t];
    }
    out[t] = x * scale;
    out[n + t] = z * scale;
}

}  // namespace

int mhd2d_derive(sparc_ctx* c, int s0, int G, bool adjoint, void* out, long long ofs) {
    if (!c->mhd || c->P.option != 18) return fail(c, SPARC_EINVAL, "kernel snapshots of the MHD forms need option 18");
    return c->f32 ? mhd2d_derive_t<float>(c, s0, G, adjoint, (float*)out, ofs)
                  : mhd2d_derive_t<double>(c, s0, G, adjoint, (double*)out, ofs);
}

int mhd2d_kernel_b_reset(sparc_ctx* c) {
    MhdState& m = *c->mhd;
    if (!m.kbacc) {
        int rc = dalloc(c, (void**)&m.kbacc, (size_t)c->S * 2 * c->N * 8);
        if (rc) return rc;
    }
    CK(cudaMemsetAsync(m.kbacc, 0, (size_t)c->S * 2 * c->N * 8, c->stream));
    return SPARC_OK;
}

int mhd2d_kernel_b_accumulate(sparc_ctx* c, const void* fst, long long sfs, const void* adj, long long afs, int s0,
                              int G) {
    MhdState& m = *c->mhd;
    if (!m.kbacc) { int rc = mhd2d_kernel_b_reset(c); if (rc) return rc; }
    return c->f32 ? mhd2d_kernel_b_t<float>(c, (const float*)fst, sfs, (const float*)adj, afs, s0, G)
                  : mhd2d_kernel_b_t<double>(c, (const double*)fst, sfs, (const double*)adj, afs, s0, G);
}

int mhd2d_kernels_b(sparc_ctx* c, int src, int sum_slots, double* kbx, double* kbz, double* kpsi) {
    MhdState& m = *c->mhd;
    if (!m.kbacc) return fail(c, SPARC_ESTATE, "no B-field kernel accumulation yet");
    const long long N = c->N;
    // kernels.f90:498-514 (2-D: dimen = (diml 1e-8 xlength 1e-8 dimb)^-1)
    const double dimb = std::sqrt(4.0 * c->pi * c->dimc * c->dimc * c->dimrho);
    const double dimen = 1.0 / (c->diml * (double)1.0e-8f * R4(c->P.xlength) * (double)1.0e-8f * dimb);
    const double scale = (double)c->steps * R4(c->P.timestep) * dimen;
    double* out = nullptr;
    int rc = dalloc(c, (void**)&out, (size_t)4 * N * 8);
    if (rc) return rc;
    const double* acc = m.kbacc + (sum_slots ? 0 : (size_t)src * 2 * N);
    kb_finish_kernel<<<nb256(N), 256, 0, c->stream>>>(out, acc, scale, sum_slots ? c->S : 1, 2 * N, N);
    c->launches++;
    // psi kernel: ddzkern(kernel_bx, 0) - d kernel_bz/dx (FP64 multipliers)
    void* rx0 = m.rx;
    m.rx = m.rx64;
    rc = ddz_launch<double>(c, out, out + 2 * N, 0);
    if (!rc) {
        zfilter_phys_kernel<double><<<dim3(nb256(c->NP), 1), 256, 0, c->stream>>>(out + 2 * N, c->NP, c->nz, 0);
        rc = ddx_launch<double>(c, out + N, out + 3 * N);
    }
    m.rx = rx0;
    if (!rc) {
        axpby_kernel<<<nb256(N), 256, 0, c->stream>>>(out + 2 * N, out + 2 * N, 1.0, out + 3 * N, -1.0, N);
        c->launches += 2;
        if (kbx) CK(cudaMemcpyAsync(kbx, out, N * 8, cudaMemcpyDeviceToHost, c->stream));
        if (kbz) CK(cudaMemcpyAsync(kbz, out + N, N * 8, cudaMemcpyDeviceToHost, c->stream));
        if (kpsi) CK(cudaMemcpyAsync(kpsi, out + 2 * N, N * 8, cudaMemcpyDeviceToHost, c->stream));
        CK(cudaStreamSynchronize(c->stream));
    }
    cudaFree(out);
    c->allocs.erase(std::remove(c->allocs.begin(), c->allocs.end(), (void*)out), c->allocs.end());
    c->dev_bytes -= (long long)4 * N * 8;
    return rc;
}

const double* mhd_kernel_c2(const sparc_ctx* c) { return (c->mhd && c->P.option == 18) ? c->mhd->kc2 : nullptr; }
const double* mhd_kernel_rho0(const sparc_ctx* c) { return (c->mhd && c->P.option == 18) ? c->mhd->krho : nullptr; }
