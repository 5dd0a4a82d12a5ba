// Private to the magnetic forms (mhd.cu: set-up and sensitivity kernels;
// mhd_step.cu: the time step).
#pragma once
#include "ctx.cuh"
#include "lines.cuh"

// background fields (T, N values each)
enum { MB_BOX, MB_BOY, MB_BOZ, MB_CBOX, MB_CBOY, MB_CBOZ, MB_GP0X, MB_GP0Y, MB_GP0Z, MB_GR0X, MB_GR0Y, MB_GR0Z,
       MB_C2RHO0, MB_RHO0, MB_RHOINV, MB_COUNT };
// stage scratch per source (T, N values each) of options 10 and 18: the
// temporaries, the fluxes, p', rho', b (each first holds the d/dx or d/dy part
// of its component), the x, y and z derivatives and the damping terms
enum { MW_T0, MW_T1, MW_T2, MW_T3, MW_T4, MW_T5, MW_F1, MW_F2, MW_F3, MW_P, MW_R, MW_BX, MW_BY, MW_BZ, MW_DX, MW_DY,
       MW_DYF1, MW_GPX, MW_GPY, MW_DXBY, MW_DXBZ, MW_DYBZ, MW_DYBX, MW_DMX, MW_DMY, MW_DMZ, MW_Z0, MW_Z1, MW_Z2,
       MW_COUNT };
// PML auxiliaries (scrpml / pmlvars index, initialize.f90:487-490,560-566)
enum { PV_VZ, PV_P, PV_DZBX, PV_DZBY, PV_IBX, PV_IBY, PV_COUNT };
// work fields of a stage of the MHD velocity form (option 8): the eight
// temporaries, the fluxes of v x B0, the eighteen derivatives of the six
// ddxyz calls of pml.f90:106-116 (named for the derivative they hold) and
// the three damping terms
enum { V8_T0, V8_T1, V8_T2, V8_T3, V8_T4, V8_T5, V8_T6, V8_T7, V8_F1, V8_F2, V8_F3,
       V8_DVXDX, V8_DVYDY, V8_DVZDZ, V8_DXF3, V8_GPY, V8_DZF1, V8_GPX, V8_DYF3, V8_DZF2, V8_DXF2, V8_DYBZ,
       V8_DZBX, V8_DXBY, V8_DYBX, V8_GPZ, V8_DXBZ, V8_DYF1, V8_DZBY, V8_DMX, V8_DMY, V8_DMZ, V8_COUNT };

struct MhdState {
    void* bg = nullptr;        // [MB_COUNT][N] T
    void* pab = nullptr;       // [2][nzpml*NP] T: a_z, b_z of the PML planes (pmlindex order)
    void* g = nullptr;         // [nz] T: gravity with the PML decay of the (1,1) column
    void* sponge = nullptr;    // [nz] T: spongez (PERIODIC: spongexyz(:,:,k) = spongez(k))
    int* plane = nullptr;      // [NP] 0-based source plane of each pixel
    int* plane_obs = nullptr;  // [NP] 0-based observation plane of each pixel (surface records)
    void* dw = nullptr;        // [NP] T: delta_width_2d
    void* rx = nullptr;        // [nx] T: d/dx multipliers of the packed complex FFT
    void* ry = nullptr;        // [ny] T
    void* fx = nullptr;        // [2][nx] T: damping and horizontal filter of a packed row, over nx (ny = 1)
    void* work = nullptr;      // [S][MW_COUNT][N] T ([S][V8_COUNT][N] in option 8)
    void* pml = nullptr;       // [S][6][nzpml*NP] T (pmlvars)
    void* spml = nullptr;      // [S][6][nzpml*NP] T (scrpml)
    void* spec = nullptr;      // [S][3] spectral fields (nz*M complex T): damping / filter transforms
    void* src = nullptr;       // [S][NP] T: a LAGRANGE_INTERP source interpolated to the step
    bool have_bg = false;
    bool rows2d_z = false;     // FP32 option 18: d/dz through rows2d_ddz
    // sensitivity kernels of the 2-D form (kernels.f90:99-133, 337-453)
    void* kbox = nullptr;      // [N] T: B_x of kernel mode, -ddzkern(psi, 0) / dimb
    void* kcby = nullptr;      // [N] T: (curl B0)_y of kernel mode (CURL_KERN)
    double* kc2 = nullptr;     // [N] c^2 (non-dimensional) for the kernel products and scaling
    double* krho = nullptr;    // [N] rho0 (non-dimensional)
    double* rx64 = nullptr;    // [nx] FP64 d/dx multipliers (kernel scaling in FP64)
    double* kbacc = nullptr;   // [S][2][N] B-field kernel sums (x, z)
};

inline unsigned nb256(long long n) { return (unsigned)((n + 255) / 256); }
// the z-solve table of the element type
template <typename T> const T* mhd_ztab(const sparc_ctx* c);
template <> inline const double* mhd_ztab<double>(const sparc_ctx* c) { return c->ztab64; }
template <> inline const float* mhd_ztab<float>(const sparc_ctx* c) { return (const float*)c->ztab; }

// d/dx, d/dy of the fields of a list, nsrc sources (mhd.cu)
template <typename T> int mhd_ddx(sparc_ctx* c, const LineList<T, T>& L, int nsrc);
template <typename T> int mhd_ddy(sparc_ctx* c, const LineList<T, T>& L, int nsrc);
// d/dz of the fields of a list, field i with boundary code bc[i]; caller-set
// values: 0 at the bottom (bc 2), topscale times the top plane of the field
// topsrc (source stride as the list's input) at the top (bc 3) (mhd_step.cu)
struct ZCodes { int bc[LINE_FIELDS]; };
template <typename T>
int mhd_ddz(sparc_ctx* c, const LineList<T, T>& L, const ZCodes& codes, int nsrc, const T* topsrc = nullptr,
            T topscale = (T)0);
// d/dz of the FP32 2-D form (rows2d_f32.cu); rows2d_ddz_ok: nz fits its shared memory
bool rows2d_ddz_ok(int nz);
void rows2d_ddz(const LineList<float, float>& L, const ZCodes& codes, int nsrc, const float* zt, const Compact<float>& cc,
                long long npix, int nz, const float* topsrc, float topscale, cudaStream_t s);
// nsteps steps on the context's stream; the context's time is the caller's to advance
int mhd_enqueue(sparc_ctx* c, int nsteps);
