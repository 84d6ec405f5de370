// modal.cu -- the cylindrical field solve truncated to azimuthal modes m = 0, 1.
//
// The reference's theta-gridded field update (cyl_em_update.F90 and
// cyl_em_update_lehe.F90, restated in cyl.cu) is linear and invariant under
// shifts of the theta index on its ny periodic cells: every theta difference
// couples F(j) with F(j +- 1), the axis conditions couple F(j) with the
// partner F(j + ny/2) (cyl_em_update.F90:143-227), and the Bz axis update
// sums over all j (:231-246).  So it acts on each discrete Fourier mode of
// theta separately.  This form keeps m = 0 and m = 1 only: a component is
//
//     F(i, t, k) = a(i, k) + b(i, k) cos(phi t) + c(i, k) sin(phi t),
//     t = j - 3 (theta index), phi = 2 pi / ny,
//
// stored as three planes (a, b, c) of an (mx, 3, mz) array, and every update
// of cyl.cu is applied to the planes with the theta shifts written as
// rotations of (b, c):
//     F(t + 1) -> (a,  b cos(phi) + c sin(phi),  c cos(phi) - b sin(phi))
//     F(t - 1) -> (a,  b cos(phi) - c sin(phi),  c cos(phi) + b sin(phi))
//     F(t + ny/2) -> (a, -b, -c).
// On fields whose theta content is m <= 1 the result equals the
// theta-gridded update to round-off.  The particles keep the reference's
// theta-gridded mover: the theta-gridded E and B it gathers from are
// synthesised from the modes by every field update, and the current it
// deposits (after the fold) is projected onto the modes before AddCurrent.
// The projection of a charge-conserving current is charge-conserving mode by
// mode (the continuity equation is theta-shift invariant), so the truncated
// run keeps the theta-gridded scheme's Gauss law for m = 0, 1.
#include <cmath>

#include "common.cuh"
#include "field_math.cuh"
#include "kernels.cuh"

namespace pic {

struct ModalP {
    double cphi, sphi;    // cos / sin of 2 pi / ny
    double dtheta, ax_perm_area, rmin;
    int ny;
};

// Three planes of one component at (i, k); T = double or float (the FP32 form).
template <typename T>
struct M3 {
    T a, b, c;
};

template <typename T>
__device__ __forceinline__ M3<T> operator+(M3<T> x, M3<T> y) { return {x.a + y.a, x.b + y.b, x.c + y.c}; }
template <typename T>
__device__ __forceinline__ M3<T> operator-(M3<T> x, M3<T> y) { return {x.a - y.a, x.b - y.b, x.c - y.c}; }
template <typename T>
__device__ __forceinline__ M3<T> operator*(T s, M3<T> x) { return {s * x.a, s * x.b, s * x.c}; }
template <typename T>
__device__ __forceinline__ M3<T> operator/(M3<T> x, T s) { return {x.a / s, x.b / s, x.c / s}; }

// modal grid: the theta dimension holds the planes a, b, c (j = 1, 2, 3)
template <typename T>
__device__ __forceinline__ M3<T> ld3(const GridP &gm, const T *F, int i, int k)
{
    const long long c0 = cidx(gm, i, 1, k);
    return {F[c0], F[c0 + gm.sy], F[c0 + 2 * gm.sy]};
}
template <typename T>
__device__ __forceinline__ void st3(const GridP &gm, T *F, int i, int k, M3<T> v)
{
    const long long c0 = cidx(gm, i, 1, k);
    F[c0] = v.a;
    F[c0 + gm.sy] = v.b;
    F[c0 + 2 * gm.sy] = v.c;
}
// F(t + 1), F(t - 1), F(t + ny/2)
template <typename T>
__device__ __forceinline__ M3<T> tp(const ModalP &m, M3<T> v)
{
    const T cp = (T)m.cphi, sp = (T)m.sphi;
    return {v.a, v.b * cp + v.c * sp, v.c * cp - v.b * sp};
}
template <typename T>
__device__ __forceinline__ M3<T> tm(const ModalP &m, M3<T> v)
{
    const T cp = (T)m.cphi, sp = (T)m.sphi;
    return {v.a, v.b * cp - v.c * sp, v.c * cp + v.b * sp};
}
template <typename T>
__device__ __forceinline__ M3<T> partner(M3<T> v) { return {v.a, -v.b, -v.c}; }

// Lehe directional differences (cyl_em_update_lehe.F90:255-289) on modes.
template <typename T>
__device__ __forceinline__ M3<T> mgx(const GridP &gm, const T *F, int i, int k)
{
    const double *L = gm.lehe;
    M3<T> r = (T)L[0] * (ld3(gm, F, i + 1, k) - ld3(gm, F, i, k));
    r = r + (T)L[4] * (ld3(gm, F, i + 1, k + 1) - ld3(gm, F, i, k + 1));
    r = r + (T)L[4] * (ld3(gm, F, i + 1, k - 1) - ld3(gm, F, i, k - 1));
    return r;
}
template <typename T>
__device__ __forceinline__ M3<T> mgx1(const GridP &gm, const T *F, int i, int k, T rp, T rr)
{
    const double *L = gm.lehe;
    M3<T> r = (T)L[0] * (rp * ld3(gm, F, i + 1, k) - rr * ld3(gm, F, i, k));
    r = r + (T)L[4] * (rp * ld3(gm, F, i + 1, k + 1) - rr * ld3(gm, F, i, k + 1));
    r = r + (T)L[4] * (rp * ld3(gm, F, i + 1, k - 1) - rr * ld3(gm, F, i, k - 1));
    return r;
}
template <typename T>
__device__ __forceinline__ M3<T> mgy(const GridP &gm, const ModalP &m, const T *F, int i, int k)
{
    const double *L = gm.lehe;
    const M3<T> f0 = ld3(gm, F, i, k), fp = ld3(gm, F, i, k + 1), fm = ld3(gm, F, i, k - 1);
    M3<T> r = (T)L[1] * (tp(m, f0) - f0);
    r = r + (T)L[6] * (tp(m, fp) - fp);
    r = r + (T)L[6] * (tp(m, fm) - fm);
    return r;
}
template <typename T>
__device__ __forceinline__ M3<T> mgz(const GridP &gm, const ModalP &m, const T *F, int i, int k)
{
    const double *L = gm.lehe;
    const M3<T> dz0 = ld3(gm, F, i, k + 1) - ld3(gm, F, i, k);
    M3<T> r = (T)L[2] * dz0;
    r = r + (T)L[7] * (ld3(gm, F, i + 1, k + 1) - ld3(gm, F, i + 1, k));
    r = r + (T)L[7] * (ld3(gm, F, i - 1, k + 1) - ld3(gm, F, i - 1, k));
    r = r + (T)L[8] * tp(m, dz0);
    r = r + (T)L[8] * tm(m, dz0);
    r = r + (T)L[11] * (ld3(gm, F, i, k + 2) - ld3(gm, F, i, k - 1));
    return r;
}

// cos and sin of the ny theta angles, in the block's shared memory (dynamic,
// 2 ny doubles): the synthesis of a column needs all of them, and sincospi in
// FP64 costs more than the rest of the update.
__device__ __forceinline__ void theta_table(const ModalP &m, double *cs, double *sn)
{
    for (int t = threadIdx.x + blockDim.x * threadIdx.y; t < m.ny; t += blockDim.x * blockDim.y)
        sincospi(2.0 * (double)t / (double)m.ny, &sn[t], &cs[t]);
    __syncthreads();
}

// v into the planes Fm and its synthesis into the theta-gridded F at (i, k),
// with the z images of both and the theta ghosts.
template <typename T>
__device__ __forceinline__ void emit(const GridP &g, const GridP &gm, const double *cs, const double *sn, T *Fm, T *F,
                                     int i, int k, M3<T> v)
{
    const int kk = image_of(k, g.mz);
    st3(gm, Fm, i, k, v);
    if (kk) st3(gm, Fm, i, kk, v);
    for (int j = 3; j <= g.my - 3; j++) {
        const T f = v.a + v.b * (T)cs[j - 3] + v.c * (T)sn[j - 3];
        const int jj = image_of(j, g.my);
        F[cidx(g, i, j, k)] = f;
        if (jj) F[cidx(g, i, jj, k)] = f;
        if (kk) F[cidx(g, i, j, kk)] = f;
        if (jj && kk) F[cidx(g, i, jj, kk)] = f;
    }
}

// The B and E phases: one thread per interior (r, z) and component updates
// the planes of its cell, applies the axis conditions (the thread next to the axis, whose
// new values they are made of) and writes the planes, their theta-gridded
// synthesis and all images; the columns an update leaves alone are emitted as
// they are.  With launches for the update, the axis, the halo, the synthesis,
// the fold and the projection each, a step had 43 of them (nr 128, nz 1024,
// FP32: 379 us of a 877 us step; now 3 and 90 us).

// B half step (cyl_em_update.F90:66-83; Lehe :62-118): i 4..mx-1; then
// UpdateBzAxis (:231-246: the circulation of Ey(4, :, k) is ny times its m = 0
// plane, and Bz on the axis has no m = 1 part) and UpdateBFldAxis (:187-227).
template <typename T, int FDTD>
__global__ void __launch_bounds__(128) k_modal_bhalf(GridP g, GridP gm, ModalP m, const T *__restrict__ Ex,
                                                     const T *__restrict__ Ey, const T *__restrict__ Ez, T *Bx, T *By,
                                                     T *Bz, T *Fx, T *Fy, T *Fz)
{
    extern __shared__ double tab[];
    const double *cs = tab, *sn = tab + m.ny;
    theta_table(m, tab, tab + m.ny);
    const int i = 1 + blockIdx.x * blockDim.x + threadIdx.x, k = 3 + blockIdx.y * blockDim.y + threadIdx.y;
    if (i > gm.mx || k > gm.mz - 3 || i == 3) return;   // column 3 belongs to the thread of column 4
    const int comp = blockIdx.z;
    T *B = comp == 0 ? Bx : comp == 1 ? By : Bz, *F = comp == 0 ? Fx : comp == 1 ? Fy : Fz;
    M3<T> v = ld3(gm, B, i, k);
    if (i >= 4 && i <= gm.mx - 1) {
        const T h = (T)gm.h, dtheta = (T)m.dtheta;
        const T r = ((T)i - (T)3.0) + (T)m.rmin;
        const T rp_half = r + (T)0.5, rp = r + (T)1.0;
        if (FDTD == PIC_FDTD_YEE) {
            if (comp == 0) {
                const M3<T> ez = ld3(gm, Ez, i, k), ey = ld3(gm, Ey, i, k);
                v = v - (h * (tp(m, ez) - ez)) / (r * dtheta) + h * (ld3(gm, Ey, i, k + 1) - ey);
            } else if (comp == 1) {
                const M3<T> ez = ld3(gm, Ez, i, k), ex = ld3(gm, Ex, i, k);
                v = v - h * (ld3(gm, Ex, i, k + 1) - ex) + h * (ld3(gm, Ez, i + 1, k) - ez);
            } else {
                const M3<T> ex = ld3(gm, Ex, i, k), ey = ld3(gm, Ey, i, k);
                v = v - (h * ((rp * ld3(gm, Ey, i + 1, k) - r * ey) - (tp(m, ex) - ex) / dtheta)) / rp_half;
            }
        } else {
            if (comp == 0) v = v - (h * mgy(gm, m, Ez, i, k)) / (r * dtheta) + h * mgz(gm, m, Ey, i, k);
            else if (comp == 1) v = v - h * mgz(gm, m, Ex, i, k) + h * mgx(gm, Ez, i, k);
            else v = v - (h * (mgx1(gm, Ey, i, k, rp, r) - mgy(gm, m, Ex, i, k) / dtheta)) / rp_half;
        }
    }
    if (i == 4) {
        if (comp == 0) {
            emit<T>(g, gm, cs, sn, B, F, 3, k, {-v.a, v.b, v.c});
        } else if (comp == 1) {
            emit(g, gm, cs, sn, B, F, 3, k, (T)0.5 * (v - partner(v)));
            emit<T>(g, gm, cs, sn, B, F, 2, k, {-v.a, v.b, v.c});
        } else {
            const T s = -(T)(gm.h * m.ax_perm_area) * ((T)m.ny * ld3(gm, Ey, 4, k).a);
            emit<T>(g, gm, cs, sn, B, F, 3, k, {ld3(gm, B, 3, k).a + s, (T)0, (T)0});
            emit(g, gm, cs, sn, B, F, 2, k, partner(v));
        }
    }
    if (i == 2 && comp != 0) return;   // By and Bz of column 2: above
    emit(g, gm, cs, sn, B, F, i, k, v);
}

// Modes of the theta-gridded J at (i, k): a = mean, b = 2/ny sum J cos, c =
// 2/ny sum J sin over the ny interior theta cells (summed in FP64); FOLD: of
// J with its periodic images added (z first, then theta).
template <typename T, bool FOLD>
__device__ __forceinline__ M3<T> project(const GridP &g, const ModalP &m, const double *cs, const double *sn, const T *J,
                                         int i, int k)
{
    const int kk = FOLD ? image_of(k, g.mz) : 0;
    double a = 0.0, b = 0.0, c = 0.0;
    for (int t = 0; t < m.ny; t++) {
        const int j = 3 + t;
        T f = J[cidx(g, i, j, k)];
        if (FOLD) {
            const int jj = image_of(j, g.my);
            if (kk) f = f + J[cidx(g, i, j, kk)];
            if (jj) {
                T w = J[cidx(g, i, jj, k)];
                if (kk) w = w + J[cidx(g, i, jj, kk)];
                f = f + w;
            }
        }
        const double v = (double)f;
        a += v;
        b += v * cs[t];
        c += v * sn[t];
    }
    const double inv = 1.0 / (double)m.ny;
    return {(T)(a * inv), (T)(2.0 * b * inv), (T)(2.0 * c * inv)};
}

// UpdateEfield (cyl_em_update.F90:24-41, MODE 0), AddCurrent of a folded J
// (:128-137, MODE 2), or both with the fold and the zeroing of J (MODE 1, the
// step) on modes: i 4..mx-3; then UpdateEFldAxis (:143-185).
template <typename T, int MODE>
__global__ void __launch_bounds__(128) k_modal_e(GridP g, GridP gm, ModalP m, T *Ex, T *Ey, T *Ez,
                                                 const T *__restrict__ Bx, const T *__restrict__ By,
                                                 const T *__restrict__ Bz, T *Jx, T *Jy, T *Jz, T *Fx, T *Fy, T *Fz)
{
    extern __shared__ double tab[];
    const double *cs = tab, *sn = tab + m.ny;
    theta_table(m, tab, tab + m.ny);
    const int i = 1 + blockIdx.x * blockDim.x + threadIdx.x, k = 3 + blockIdx.y * blockDim.y + threadIdx.y;
    if (i > gm.mx || k > gm.mz - 3) return;
    const int comp = blockIdx.z;
    T *E = comp == 0 ? Ex : comp == 1 ? Ey : Ez, *F = comp == 0 ? Fx : comp == 1 ? Fy : Fz;
    T *J = comp == 0 ? Jx : comp == 1 ? Jy : Jz;
    M3<T> v = ld3(gm, E, i, k);
    if (i >= 4 && i <= gm.mx - 3) {
        const T dtheta = (T)m.dtheta;
        const T r = ((T)i - (T)3.0) + (T)m.rmin;
        const T rp_half = r + (T)0.5, rm_half = r - (T)0.5;
        if (MODE != 2) {
            const T fc = (T)gm.fc;
            if (comp == 0) {
                const M3<T> bz = ld3(gm, Bz, i, k), by = ld3(gm, By, i, k);
                v = v + (fc * (bz - tm(m, bz))) / (rp_half * dtheta) - fc * (by - ld3(gm, By, i, k - 1));
            } else if (comp == 1) {
                const M3<T> bz = ld3(gm, Bz, i, k), bx = ld3(gm, Bx, i, k);
                v = v + fc * (bx - ld3(gm, Bx, i, k - 1)) - fc * (bz - ld3(gm, Bz, i - 1, k));
            } else {
                const M3<T> by = ld3(gm, By, i, k), bx = ld3(gm, Bx, i, k);
                v = v + (fc * (rp_half * by - rm_half * ld3(gm, By, i - 1, k))) / r - (fc * (bx - tm(m, bx))) / (r * dtheta);
            }
        }
        if (MODE != 0) {
            const M3<T> cur = project<T, MODE == 1>(g, m, cs, sn, J, i, k);
            if (comp == 0) v = v - cur / (rp_half * dtheta);
            else if (comp == 1) v = v - cur;
            else v = v - cur / (r * dtheta);
        }
    }
    if (MODE == 1) {   // ResetCurrent
        const int kk = image_of(k, g.mz);
        for (int j = 1; j <= g.my; j++) {
            J[cidx(g, i, j, k)] = (T)0;
            if (kk) J[cidx(g, i, j, kk)] = (T)0;
        }
    }
    if (i == 3) return;   // column 3 belongs to the thread of column 4
    if (i == 4) {
        if (comp == 0) {
            emit(g, gm, cs, sn, E, F, 3, k, (T)0.5 * (v - partner(v)));
            emit<T>(g, gm, cs, sn, E, F, 2, k, {-v.a, v.b, v.c});
        } else if (comp == 1) {
            emit<T>(g, gm, cs, sn, E, F, 3, k, {-v.a, v.b, v.c});
        } else {
            emit(g, gm, cs, sn, E, F, 3, k, partner(v));
        }
    }
    if (i == 2 && comp == 0) return;   // Ex of column 2: above
    emit(g, gm, cs, sn, E, F, i, k, v);
}

// Theta-gridded F(i, j, k) for every ghosted j from the modes at (i, k)
// (loaded fields).
template <typename T>
__global__ void k_modal_synth(GridP g, GridP gm, ModalP m, const T *__restrict__ Fm, T *F)
{
    extern __shared__ double tab[];
    theta_table(m, tab, tab + m.ny);
    const int i = 1 + blockIdx.x * blockDim.x + threadIdx.x, k = 1 + blockIdx.y * blockDim.y + threadIdx.y;
    if (i > g.mx || k > g.mz) return;
    const M3<T> v = ld3(gm, Fm, i, k);
    for (int j = 1; j <= g.my; j++) {
        int t = (j - 3) % m.ny;
        if (t < 0) t += m.ny;
        F[cidx(g, i, j, k)] = v.a + v.b * (T)tab[t] + v.c * (T)tab[m.ny + t];
    }
}

// The modes of a theta-gridded component (loaded fields).
template <typename T>
__global__ void k_modal_project(GridP g, GridP gm, ModalP m, const T *__restrict__ F, T *Fm)
{
    extern __shared__ double tab[];
    theta_table(m, tab, tab + m.ny);
    const int i = 1 + blockIdx.x * blockDim.x + threadIdx.x, k = 1 + blockIdx.y * blockDim.y + threadIdx.y;
    if (i > g.mx || k > g.mz) return;
    st3<T>(gm, Fm, i, k, project<T, false>(g, m, tab, tab + m.ny, F, i, k));
}

GridP modal_grid(const GridP &g)
{
    GridP gm = g;
    gm.my = 3;
    gm.sy = g.mx;
    gm.sz = (long long)g.mx * 3;
    gm.ncell = gm.sz * g.mz;
    return gm;
}

static ModalP modal_params(const GridP &g)
{
    ModalP m;
    const double pi = 3.14159265358979323846264;
    m.ny = g.ny;
    m.dtheta = 2.0 * pi / g.ny;
    m.cphi = std::cos(m.dtheta);
    m.sphi = std::sin(m.dtheta);
    m.ax_perm_area = 4.0 / g.ny;
    m.rmin = -0.5;
    return m;
}

static void modal_shape(const GridP &g, dim3 &grid, dim3 &block, size_t &smem)
{
    block = dim3(32, 4);
    grid = dim3((g.mx + 31) / 32, (g.nz + 3) / 4, 3);
    smem = 2 * sizeof(double) * (size_t)g.ny;
}
template <typename K>
static void allow_smem(K k, size_t smem)   // beyond 3072 theta cells
{
    if (smem > 48 * 1024) cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
}

template <typename T>
void launch_modal_bhalf(const GridP &g, T *const B[3], T *const Em[3], T *const Bm[3], cudaStream_t s)
{
    const GridP gm = modal_grid(g);
    const ModalP m = modal_params(g);
    dim3 grid, block;
    size_t sm;
    modal_shape(g, grid, block, sm);
    auto k = g.fdtd == PIC_FDTD_LEHE ? k_modal_bhalf<T, PIC_FDTD_LEHE> : k_modal_bhalf<T, PIC_FDTD_YEE>;
    allow_smem(k, sm);
    k<<<grid, block, sm, s>>>(g, gm, m, Em[0], Em[1], Em[2], Bm[0], Bm[1], Bm[2], B[0], B[1], B[2]);
    count_launches(1);
}

template <typename T>
void launch_modal_efield(const GridP &g, int mode, T *const E[3], T *const J[3], T *const Em[3], T *const Bm[3],
                         cudaStream_t s)
{
    const GridP gm = modal_grid(g);
    const ModalP m = modal_params(g);
    dim3 grid, block;
    size_t sm;
    modal_shape(g, grid, block, sm);
    auto k = mode == 0 ? k_modal_e<T, 0> : mode == 1 ? k_modal_e<T, 1> : k_modal_e<T, 2>;
    allow_smem(k, sm);
    k<<<grid, block, sm, s>>>(g, gm, m, Em[0], Em[1], Em[2], Bm[0], Bm[1], Bm[2], J[0], J[1], J[2], E[0], E[1], E[2]);
    count_launches(1);
}

template <typename T>
void launch_modal_synth(const GridP &g, T *const Fm[3], T *const F[3], cudaStream_t s)
{
    const GridP gm = modal_grid(g);
    const ModalP m = modal_params(g);
    const dim3 block(32, 4), grid((g.mx + 31) / 32, (g.mz + 3) / 4);
    const size_t sm = 2 * sizeof(double) * (size_t)g.ny;
    allow_smem(k_modal_synth<T>, sm);
    for (int c = 0; c < 3; c++) k_modal_synth<T><<<grid, block, sm, s>>>(g, gm, m, Fm[c], F[c]);
    count_launches(3);
}

template <typename T>
void launch_modal_project(const GridP &g, T *const F[3], T *const Fm[3], cudaStream_t s)
{
    const GridP gm = modal_grid(g);
    const ModalP m = modal_params(g);
    const dim3 block(32, 4), grid((g.mx + 31) / 32, (g.mz + 3) / 4);
    const size_t sm = 2 * sizeof(double) * (size_t)g.ny;
    allow_smem(k_modal_project<T>, sm);
    for (int c = 0; c < 3; c++) k_modal_project<T><<<grid, block, sm, s>>>(g, gm, m, F[c], Fm[c]);
    count_launches(3);
}

template void launch_modal_bhalf<double>(const GridP &, double *const[3], double *const[3], double *const[3],
                                         cudaStream_t);
template void launch_modal_bhalf<float>(const GridP &, float *const[3], float *const[3], float *const[3], cudaStream_t);
template void launch_modal_efield<double>(const GridP &, int, double *const[3], double *const[3], double *const[3],
                                          double *const[3], cudaStream_t);
template void launch_modal_efield<float>(const GridP &, int, float *const[3], float *const[3], float *const[3],
                                         float *const[3], cudaStream_t);
template void launch_modal_synth<double>(const GridP &, double *const[3], double *const[3], cudaStream_t);
template void launch_modal_synth<float>(const GridP &, float *const[3], float *const[3], cudaStream_t);
template void launch_modal_project<double>(const GridP &, double *const[3], double *const[3], cudaStream_t);
template void launch_modal_project<float>(const GridP &, float *const[3], float *const[3], cudaStream_t);

}  // namespace pic
