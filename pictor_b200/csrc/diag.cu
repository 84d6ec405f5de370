// diag.cu -- FP64 diagnostics on the device.
//
// Reference: src/io/savedata_routines.F90:265-348 (CalcEnergy, CalcPrtlEnergy,
// CalcFldEnergy, CalcDivE).  Field energy is a deterministic two-level
// reduction (per-block partial sums in a scratch array, then one block adds
// them in block order); the Gauss residual deposits the CIC charge density of
// q*qi at nodes, folded periodically, and reports max |divE - rho| with divE
// the backward-difference node divergence of CalcDivE.
#include "common.cuh"
#include "kernels.cuh"

namespace pic {

constexpr int kDiagThreads = 256;

int field_energy_blocks(const GridP &g)
{
    const long long nint = (long long)g.nx * g.ny * (g.dims == 3 ? g.nz : 1);
    long long b = (nint + kDiagThreads * 2 - 1) / (kDiagThreads * 2);
    if (b > kSMs * 8) b = kSMs * 8;
    return (int)(b < 1 ? 1 : b);
}

// The interior cells for the warps of the grid, f(offset of the cell, i), with
// no flat index divided per cell: a warp takes pieces of up to kRowPiece cells
// of a row, or, of rows of at most half its lanes, as many rows as fit into
// them.  (A warp per row took 23.5 ms for 2 rows of 2^21 cells, 0.05 ms as a
// square grid, and left lanes idle in short rows.)
constexpr int kRowPiece = 256;
template <typename F>
__device__ __forceinline__ void for_interior_cells(const GridP &g, F f)
{
    const int lane = threadIdx.x & 31, nw = gridDim.x * (kDiagThreads / 32);
    const int gw = blockIdx.x * (kDiagThreads / 32) + (threadIdx.x >> 5), rows = g.ny * (g.dims == 3 ? g.nz : 1);
    auto row_offset = [&](int r) {
        const int kk = g.dims == 3 ? r / g.ny : 0;
        return cidx(g, 0, 3 + (r - kk * g.ny), g.dims == 3 ? 3 + kk : 1);
    };
    if (g.nx > 16) {
        const int cuts = (g.nx - 1) / kRowPiece + 1;
        for (int it = gw; it < rows * cuts; it += nw) {
            const int r = cuts == 1 ? it : it / cuts, i0 = 3 + (it - r * cuts) * kRowPiece;
            const int i1 = min(i0 + kRowPiece, 3 + g.nx);
            const long long c0 = row_offset(r);
            for (int i = i0 + lane; i < i1; i += 32) f(c0 + i, i);
        }
    } else {
        const int lw = 32 - __clz(g.nx - 1);   // 2^lw lanes hold a row
        const int i = 3 + (lane & ((1 << lw) - 1));
        for (int r = (gw << (5 - lw)) + (lane >> lw); r < rows; r += nw << (5 - lw))
            if (i < 3 + g.nx) f(row_offset(r) + i, i);
    }
}

__device__ __forceinline__ double block_sum(double v, double *red)
{
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    double t = 0;
    if (threadIdx.x == 0)
        for (int w = 0; w < kDiagThreads / 32; w++) t += red[w];
    return t;
}

template <typename T>
__global__ void __launch_bounds__(kDiagThreads) k_field_energy_partial(GridP g, const T *__restrict__ Ex, const T *__restrict__ Ey,
                                                                       const T *__restrict__ Ez, const T *__restrict__ Bx,
                                                                       const T *__restrict__ By, const T *__restrict__ Bz,
                                                                       double *partials)
{
    __shared__ double red[kDiagThreads / 32];
    double eb = 0, ee = 0;
    const double dtheta = 2.0 * 3.14159265358979323846264 / g.ny;
    for_interior_cells(g, [&](long long c, int i) {
        const double bx = Bx[c], by = By[c], bz = Bz[c], ex = Ex[c], ey = Ey[c], ez = Ez[c];
        if (g.geom == PIC_GEOM_CYLINDRICAL) {
            // CalcFldEnergy_cyl (cyl_savedata_routines.F90:8-31): r weights, axis cell excluded
            if (i < 4) return;
            const double r = ((double)i - 3.0) + -0.5, rp = r + 0.5;
            eb += ((r * (bx * bx) + rp * (by * by)) + rp * (bz * bz)) * dtheta;
            ee += ((rp * (ex * ex) + r * (ey * ey)) + r * (ez * ez)) * dtheta;
        } else {
            eb += (bx * bx + by * by) + bz * bz;
            ee += (ex * ex + ey * ey) + ez * ez;
        }
    });
    const double sb = block_sum(eb, red);
    const double se = block_sum(ee, red);
    if (threadIdx.x == 0) {
        partials[2 * blockIdx.x] = sb;
        partials[2 * blockIdx.x + 1] = se;
    }
}

// The partial pairs added in a fixed order: thread t its own stride, then the
// threads' sums in a tree (one thread walking 1184 pairs took 33 us).
__global__ void __launch_bounds__(kDiagThreads) k_sum_partials(const double *__restrict__ partials, int nblocks, double *out2)
{
    __shared__ double red[kDiagThreads / 32];
    double sb = 0, se = 0;
    for (int b = threadIdx.x; b < nblocks; b += kDiagThreads) {
        sb += partials[2 * b];
        se += partials[2 * b + 1];
    }
    const double tb = block_sum(sb, red);
    const double te = block_sum(se, red);
    if (threadIdx.x == 0) {
        out2[0] = tb;
        out2[1] = te;
    }
}

void launch_field_energy(const GridP &g, const void *const E[3], const void *const B[3], bool fp32, double *partials,
                         int nblocks, double *out2, cudaStream_t s)
{
    if (fp32)
        k_field_energy_partial<float><<<nblocks, kDiagThreads, 0, s>>>(
            g, (const float *)E[0], (const float *)E[1], (const float *)E[2], (const float *)B[0], (const float *)B[1],
            (const float *)B[2], partials);
    else
        k_field_energy_partial<double><<<nblocks, kDiagThreads, 0, s>>>(
            g, (const double *)E[0], (const double *)E[1], (const double *)E[2], (const double *)B[0],
            (const double *)B[1], (const double *)B[2], partials);
    k_sum_partials<<<1, kDiagThreads, 0, s>>>(partials, nblocks, out2);
    count_launches(1);
    count_launches(1);
}

// ---------------------------------------------------------------------------
// Kinetic energy per species (CalcPrtlEnergy, savedata_routines.F90:283-308),
// with the particle weight wtp = |q| (charge = weight * FlvrCharge).
// ---------------------------------------------------------------------------
__device__ __forceinline__ double species_energy(const GridP &g, double masse, int flv, double q, double u, double v,
                                                 double w)
{
    const double c = g.c;
    const double gm = sqrt(((1.0 + u * u) + v * v) + w * w);
    const double wt = fabs(q);
    if (q > 0) return (((gm - 1.0) * wt) * (q * g.qi / g.qm[flv])) * c * c;
    if (q < 0) return ((gm - 1.0) * wt) * ((masse * c) * c);
    return 0.0;
}

// Sums per flavour: flavours 1 and 2 in registers (an array indexed by the
// flavour lives in local memory), the others, which few runs have, in shared
// memory; one atomic per block and flavour.
struct FlavourSum {
    double a1 = 0, a2 = 0;
    __device__ __forceinline__ void add(double *sh, int flv, double e)
    {
        a1 += flv == 1 ? e : 0.0;
        a2 += flv == 2 ? e : 0.0;
        if (flv > 2) atomicAdd(sh + flv, e);
    }
    __device__ void store(double *sh, double *out)
    {
        double v[2] = {a1, a2};
        for (int f = 0; f < 2; f++) {
            for (int o = 16; o > 0; o >>= 1) v[f] += __shfl_down_sync(0xffffffffu, v[f], o);
            if ((threadIdx.x & 31) == 0 && v[f] != 0.0) atomicAdd(sh + 1 + f, v[f]);
        }
        __syncthreads();
        const int f = 1 + threadIdx.x;
        if (f <= PIC_MAX_FLVR && sh[f] != 0.0) atomicAdd(out + f - 1, sh[f]);
    }
};

__global__ void __launch_bounds__(kDiagThreads) k_pe_f64(GridP g, PartF64 p, const Counters *__restrict__ cnt, double masse,
                                                         double *out)
{
    __shared__ double sh[PIC_MAX_FLVR + 1];
    if (threadIdx.x <= PIC_MAX_FLVR) sh[threadIdx.x] = 0;
    __syncthreads();
    FlavourSum acc;
    const long long n = cnt->used;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const int flv = p.flv[i];
        if (flv <= 0 || flv > PIC_MAX_FLVR) continue;
        acc.add(sh, flv, species_energy(g, masse, flv, p.q[i], p.u[i], p.v[i], p.w[i]));
    }
    acc.store(sh, out);
}

__global__ void __launch_bounds__(kDiagThreads) k_pe_f32(GridP g, PartF32 p, const Counters *__restrict__ cnt, double masse,
                                                         double *out)
{
    __shared__ double sh[PIC_MAX_FLVR + 1];
    if (threadIdx.x <= PIC_MAX_FLVR) sh[threadIdx.x] = 0;
    __syncthreads();
    FlavourSum acc;
    const long long n = cnt->used;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const int flv = (int)(p.key[i] >> kFlvShift);
        if (flv == 0) continue;
        acc.add(sh, flv, species_energy(g, masse, flv, (double)p.w[i], (double)p.ux[i], (double)p.uy[i], (double)p.uz[i]));
    }
    acc.store(sh, out);
}

void launch_particle_energy_f64(const GridP &g, const PartF64 &p, const Counters *cnt, double masse, double *out,
                                cudaStream_t s)
{
    k_pe_f64<<<kSMs * 8, kDiagThreads, 0, s>>>(g, p, cnt, masse, out);
    count_launches(1);
}

void launch_particle_energy_f32(const GridP &g, const PartF32 &p, const Counters *cnt, double masse, double *out,
                                cudaStream_t s)
{
    k_pe_f32<<<kSMs * 8, kDiagThreads, 0, s>>>(g, p, cnt, masse, out);
    count_launches(1);
}

// ---------------------------------------------------------------------------
// Gauss residual
// ---------------------------------------------------------------------------
// The positive and the negative charge are summed apart (the residual wants
// their sum, the scale the positive one), so a particle adds to one array.
__device__ __forceinline__ void corner_weights(int dims, double dx, double dy, double dz, double w[8])
{
#pragma unroll
    for (int nn = 0; nn < 8; nn++)
        w[nn] = ((nn & 1) ? dx : 1.0 - dx) * ((nn & 2) ? dy : 1.0 - dy) * ((nn & 4) ? dz : 1.0 - dz);
}
__device__ __forceinline__ void deposit_rho(const GridP &g, double *rho, int i, int j, int k, double dx, double dy,
                                            double dz, double q)
{
    double w[8];
    corner_weights(g.dims, dx, dy, dz, w);
#pragma unroll
    for (int nn = 0; nn < 8; nn++) {
        if (nn >= 4 && g.dims == 2) break;
        const int a = wrap_index(i + (nn & 1), g.mx), b = wrap_index(j + ((nn >> 1) & 1), g.my);
        const int c = g.dims == 3 ? wrap_index(k + ((nn >> 2) & 1), g.mz) : 1;
        atomicAdd(rho + cidx(g, a, b, c), q * w[nn]);
    }
}

__global__ void k_rho_f64(GridP g, PartF64 p, const Counters *__restrict__ cnt, double *rho_neg, double *rho_pos)
{
    const long long n = cnt->used;
    for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x) {
        if (p.flv[t] == 0) continue;
        const double x = p.x[t], y = p.y[t], z = p.z[t];
        if (!(x >= 1.0 && x < g.mx && y >= 1.0 && y < g.my)) continue;
        const int i = (int)floor(x), j = (int)floor(y);
        const int k = g.dims == 3 ? (int)floor(z) : 1;
        if (g.dims == 3 && !(z >= 1.0 && z < g.mz)) continue;
        const double q = p.q[t] * g.qi;
        deposit_rho(g, q > 0 ? rho_pos : rho_neg, i, j, k, x - i, y - j, g.dims == 3 ? z - k : 0.0, q);
    }
}

__global__ void k_rho_f32(GridP g, PartF32 p, const Counters *__restrict__ cnt, double *rho_neg, double *rho_pos)
{
    const long long n = cnt->used;
    for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x) {
        const uint32_t key = p.key[t];
        if ((key >> kFlvShift) == 0) continue;
        int i, j, k;
        decode_cell(g, (int)(key & kCellMask), i, j, k);
        const double q = (double)p.w[t] * g.qi;
        deposit_rho(g, q > 0 ? rho_pos : rho_neg, i, j, k, (double)p.dx[t], (double)p.dy[t],
                    g.dims == 3 ? (double)p.dz[t] : 0.0, q);
    }
}

// The same after a reorder, one CTA per brick (bricks.cu): the brick's charge
// is summed in shared memory over the nodes of its box, and the box is added to
// the grid once.  A particle outside the box adds to the grid.  The sums are
// FP64 in any order, as in the grid: 64-bit fixed-point words would be faster
// (diagnostics of 268 M particles 6.0 ms), but hold fewer bits of light
// particles, and of any where a brick has over 4096, than FP64 does; with a
// 32-bit extension of those words 7.3 ms, so 8.4 ms as FP64 atomics of shared
// memory (11.3 ms into L2; 16.8 M particles in 2D 445 and 481 us).
constexpr int kRhoNodes = 3072;   // 48 KB, 4 CTAs per SM
template <int DIMS>
__global__ void __launch_bounds__(256) k_rho_f32_bricks(GridP g, PartF32 p, Bricks bk, double *rho_neg, double *rho_pos)
{
    extern __shared__ double s_rho[];   // positive, then negative charge
    const int b = blockIdx.x;
    const uint32_t p0 = bk.tile_start[b], p1 = bk.tile_start[b + 1];
    if (p0 >= p1) return;
    const int bx = b % bk.nb[0], byz = b / bk.nb[0], by = byz % bk.nb[1], bz = byz / bk.nb[1];
    const int n3[3] = {g.nx, g.ny, g.nz}, bi[3] = {bx, by, bz};
    int hc[3], lo[3], N[3];
#pragma unroll
    for (int d = 0; d < 3; d++) {
        hc[d] = d < DIMS ? 3 + bi[d] * bk.t[d] + (bk.t[d] >> 1) : 1;
        lo[d] = d < DIMS ? bk.box[8 * (size_t)b + d] : 0;
        N[d] = d < DIMS ? bk.box[8 * (size_t)b + 3 + d] - lo[d] + 2 : 1;   // nodes
    }
    const bool fits = N[0] > 1 && N[1] > 1 && (DIMS == 2 || N[2] > 1) && N[0] <= kBoxAxisMax && N[1] <= kBoxAxisMax &&
                      N[2] <= kBoxAxisMax && N[0] * N[1] * N[2] <= kRhoNodes;
    const int nn = fits ? N[0] * N[1] * N[2] : 0;
    for (int q = threadIdx.x; q < 2 * nn; q += 256) s_rho[q] = 0.0;
    __syncthreads();
    for (uint32_t t = p0 + threadIdx.x; t < p1; t += 256) {
        const uint32_t key = p.key[t];
        if ((key >> kFlvShift) == 0) continue;
        int i, j, k;
        decode_cell(g, (int)(key & kCellMask), i, j, k);
        const double q = (double)p.w[t] * g.qi;
        const double dx = p.dx[t], dy = p.dy[t], dz = DIMS == 3 ? (double)p.dz[t] : 0.0;
        auto un = [](int a, int c, int n) {
            int u = a - c;
            const int half = n >> 1;
            if (u >= n - half) u -= n;
            else if (u < -half) u += n;
            return u;
        };
        const int lx = un(i, hc[0], n3[0]) - lo[0], ly = un(j, hc[1], n3[1]) - lo[1],
                  lz = DIMS == 3 ? un(k, hc[2], n3[2]) - lo[2] : 0;
        if (!fits || (unsigned)lx >= (unsigned)(N[0] - 1) || (unsigned)ly >= (unsigned)(N[1] - 1) ||
            (DIMS == 3 && (unsigned)lz >= (unsigned)(N[2] - 1))) {
            deposit_rho(g, q > 0 ? rho_pos : rho_neg, i, j, k, dx, dy, dz, q);
            continue;
        }
        double w[8];
        corner_weights(DIMS, dx, dy, dz, w);
        double *at = s_rho + (q > 0 ? 0 : nn) + lx + N[0] * (ly + N[1] * lz);
#pragma unroll
        for (int c = 0; c < (DIMS == 3 ? 8 : 4); c++)
            atomicAdd(at + (c & 1) + ((c >> 1) & 1) * N[0] + ((c >> 2) & 1) * N[0] * N[1], q * w[c]);
    }
    __syncthreads();
    const uint32_t mX = 0xffffffffu / (uint32_t)N[0] + 1u, mY = 0xffffffffu / (uint32_t)N[1] + 1u;
    for (int q = threadIdx.x; q < nn; q += 256) {
        const double vp = s_rho[q], vn = s_rho[nn + q];
        if (vp == 0.0 && vn == 0.0) continue;
        const int r = (int)__umulhi((uint32_t)q, mX), xx = q - r * N[0];
        const int zz = (int)__umulhi((uint32_t)r, mY), yy = r - zz * N[1];
        const int c[3] = {hc[0] + lo[0] + xx, hc[1] + lo[1] + yy, DIMS == 3 ? hc[2] + lo[2] + zz : 1};
        int cc[3];
#pragma unroll
        for (int d = 0; d < 3; d++) {
            int a = c[d] - 3;
            if (d < DIMS) {
                a %= n3[d];
                if (a < 0) a += n3[d];
                cc[d] = 3 + a;
            } else {
                cc[d] = 1;
            }
        }
        const long long o = cidx(g, cc[0], cc[1], cc[2]);
        if (vp != 0.0) atomicAdd(rho_pos + o, vp);
        if (vn != 0.0) atomicAdd(rho_neg + o, vn);
    }
}

// rho_neg += rho_pos: the total density.
__global__ void k_rho_total(long long n, double *rho_neg, const double *__restrict__ rho_pos)
{
    for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x)
        rho_neg[t] += rho_pos[t];
}

template <typename T>
__global__ void __launch_bounds__(kDiagThreads) k_gauss_max(GridP g, const T *__restrict__ Ex, const T *__restrict__ Ey,
                                                            const T *__restrict__ Ez, const double *__restrict__ rho_neg,
                                                            const double *__restrict__ rho_pos, double *out2)
{
    double res = 0, rm = 0;
    for_interior_cells(g, [&](long long c, int) {
        double div = ((double)Ex[c] - (double)Ex[c - 1]) + ((double)Ey[c] - (double)Ey[c - g.sy]);
        if (g.dims == 3) div = div + ((double)Ez[c] - (double)Ez[c - g.sz]);
        const double rp = rho_pos[c];
        res = fmax(res, fabs(div - (rho_neg[c] + rp)));
        rm = fmax(rm, fabs(rp));
    });
    for (int o = 16; o > 0; o >>= 1) {
        res = fmax(res, __shfl_down_sync(0xffffffffu, res, o));
        rm = fmax(rm, __shfl_down_sync(0xffffffffu, rm, o));
    }
    if ((threadIdx.x & 31) == 0) {
        // non-negative doubles order like their bit patterns
        atomicMax((unsigned long long *)out2, (unsigned long long)__double_as_longlong(res));
        atomicMax((unsigned long long *)(out2 + 1), (unsigned long long)__double_as_longlong(rm));
    }
}

static void zero_rho(const GridP &g, double *rho, double *rho_pos, cudaStream_t s)
{
    const size_t bytes = (size_t)g.ncell * sizeof(double);
    if (rho_pos == rho + g.ncell) {   // the two arrays of one block
        cudaMemsetAsync(rho, 0, 2 * bytes, s);
    } else {
        cudaMemsetAsync(rho, 0, bytes, s);
        cudaMemsetAsync(rho_pos, 0, bytes, s);
    }
}
static void deposit_f64(const GridP &g, const PartF64 &p, const Counters *cnt, double *rho, double *rho_pos, cudaStream_t s)
{
    zero_rho(g, rho, rho_pos, s);
    k_rho_f64<<<kSMs * 8, 256, 0, s>>>(g, p, cnt, rho, rho_pos);
    count_launches(1);
}
static void deposit_f32(const GridP &g, const PartF32 &p, const Counters *cnt, const Bricks *bk, double *rho,
                        double *rho_pos, cudaStream_t s)
{
    zero_rho(g, rho, rho_pos, s);
    // fewer than two bricks per SM leave it too little in flight: with 24^3
    // cells and 27 bricks the diagnostics take 82 us, 61 without bricks, with
    // 218 to 256 bricks (0.9, 1 M particles) the same, with 870 170 and 234
    if (bk && bk->ntiles < 2 * kSMs) bk = nullptr;
    const size_t sm = 2 * kRhoNodes * sizeof(double);
    if (bk && g.dims == 3) k_rho_f32_bricks<3><<<bk->ntiles, 256, sm, s>>>(g, p, *bk, rho, rho_pos);
    else if (bk) k_rho_f32_bricks<2><<<bk->ntiles, 256, sm, s>>>(g, p, *bk, rho, rho_pos);
    else k_rho_f32<<<kSMs * 8, 256, 0, s>>>(g, p, cnt, rho, rho_pos);
    count_launches(1);
}
static void total_density(const GridP &g, double *rho, const double *rho_pos, cudaStream_t s)
{
    k_rho_total<<<kSMs * 8, 256, 0, s>>>(g.ncell, rho, rho_pos);
    count_launches(1);
}

// The CIC charge density alone (the initial Gauss solve, poisson.cu).
void launch_rho_f64(const GridP &g, const PartF64 &p, const Counters *cnt, double *rho, double *rho_pos, cudaStream_t s)
{
    deposit_f64(g, p, cnt, rho, rho_pos, s);
    total_density(g, rho, rho_pos, s);
}

void launch_rho_f32(const GridP &g, const PartF32 &p, const Counters *cnt, double *rho, double *rho_pos, cudaStream_t s)
{
    deposit_f32(g, p, cnt, nullptr, rho, rho_pos, s);
    total_density(g, rho, rho_pos, s);
}

// out2 must be zero.
void launch_gauss_f64(const GridP &g, const PartF64 &p, const Counters *cnt, const double *const E[3], double *rho,
                      double *rho_pos, double *out2, cudaStream_t s)
{
    deposit_f64(g, p, cnt, rho, rho_pos, s);
    k_gauss_max<double><<<field_energy_blocks(g), kDiagThreads, 0, s>>>(g, E[0], E[1], E[2], rho, rho_pos, out2);
    count_launches(1);
}

void launch_gauss_f32(const GridP &g, const PartF32 &p, const Counters *cnt, const Bricks *bk, const float *const E[3],
                      double *rho, double *rho_pos, double *out2, cudaStream_t s)
{
    deposit_f32(g, p, cnt, bk, rho, rho_pos, s);
    k_gauss_max<float><<<field_energy_blocks(g), kDiagThreads, 0, s>>>(g, E[0], E[1], E[2], rho, rho_pos, out2);
    count_launches(1);
}

}  // namespace pic
