// Electromagnetic (Lorentz) force of the welding current: kernels.py:1236-1513,
// driven by physics/weld_forces.py:196-281 solve_lorentz.
//
//   sigma map -> Gaussian current source normalised to I -> damped Jacobi
//   solve of div(sigma grad phi_e) = -source (the substrate below nz_solid
//   grounded, gas insulating) -> J = -sigma grad phi_e -> axial current binned
//   by radius per z slab, prefix-summed -> B_theta = mu0 I_enc / (2 pi r)
//   -> F += f_l (J x B) dt^2 / (rho dx).
//
// The Jacobi sweep optionally accumulates the L1 change and the L1 norm of its
// input (elec_l1_diff, kernels.py:1387-1398) in the same pass, so the host's
// convergence check every ten sweeps costs no extra grid read.  Grid sums are
// accumulated in double in a fixed block order (the reference's float atomics
// have no fixed order); the radial bins use double atomics and are rounded to
// float before the float prefix sum, as the oracle does.
#include <cmath>

#include "../../include/waam_b200.h"
#include "waam_common.cuh"
#include "waam_internal.cuh"

namespace waam {

#define STREAM(s) reinterpret_cast<cudaStream_t>(s)

namespace {

constexpr int kRedGridMax = kWsMaxPartials / 2;   // two sums share the partials
constexpr int kMaxBins = 1024;
constexpr int kOpScalarSourceScale = 16;          // ws.scalars slot of the source scale

// k slab of the arc current source (kernels.py:1261-1284): cells outside
// [k_min, k_max] get 0.  The same float arithmetic on host and device.
__host__ __device__ __forceinline__ void source_slab(float arc_k, float sigma_cells, int nz,
                                                     int& k_min, int& k_max) {
    k_max = imin(nz, (int)(arc_k + sigma_cells * 4.0f) + 1);
    k_min = imax(0, (int)(arc_k - sigma_cells));
}

// Reduction tiles: the 32 x 8 (k, j) tiles with loops over the tiles and i,
// so the grid stays at <= kRedGridMax blocks (one partial per block).
inline dim3 red_tile_grid(const Dims& d) {
    int gx = imin((d.nz + kTileK - 1) / kTileK, 16);
    int gy = imin((d.ny + kTileJ - 1) / kTileJ, 16);
    int gz = imax(1, imin(d.nx, kRedGridMax / (gx * gy)));
    return dim3(gx, gy, gz);
}

__device__ __forceinline__ double2 block_sum2(double a, double b) {
    __shared__ double sh[2][kTileK * kTileJ / 32];
    for (int o = 16; o > 0; o >>= 1) {
        a += __shfl_down_sync(0xffffffffu, a, o);
        b += __shfl_down_sync(0xffffffffu, b, o);
    }
    const int t = threadIdx.y * blockDim.x + threadIdx.x;
    const int lane = t & 31, wid = t >> 5;
    if (lane == 0) {
        sh[0][wid] = a;
        sh[1][wid] = b;
    }
    __syncthreads();
    double2 r = make_double2(0.0, 0.0);
    if (t == 0)
        for (int w = 0; w < kTileK * kTileJ / 32; ++w) {
            r.x += sh[0][w];
            r.y += sh[1][w];
        }
    __syncthreads();
    return r;   // valid in thread 0
}

// Last-block combine of two per-block sums: every thread of the last block
// adds a fixed strided subset of the partials in order, then the fixed tree
// of block_sum2 (the same order on every run).  Returns true in the thread
// that holds the totals.  Blocks of kTileK x kTileJ threads.
__device__ bool finish_sum2(Workspace ws, double2 part, double2& total) {
    __shared__ bool last;
    const int t = threadIdx.y * blockDim.x + threadIdx.x;
    const unsigned nb = gridDim.x * gridDim.y * gridDim.z;
    const unsigned b = (blockIdx.z * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x;
    if (t == 0) {
        ws.partials[b] = part.x;
        ws.partials[nb + b] = part.y;
        __threadfence();
        unsigned prev = atomicAdd(ws.counter, 1u);
        last = prev == nb - 1;
    }
    __syncthreads();
    if (!last) return false;
    __threadfence();
    double x = 0.0, y = 0.0;
    for (unsigned q = t; q < nb; q += kTileK * kTileJ) {
        x += ((volatile double*)ws.partials)[q];
        y += ((volatile double*)ws.partials)[nb + q];
    }
    const double2 r = block_sum2(x, y);
    if (t != 0) return false;
    total = r;
    *ws.counter = 0u;
    return true;
}

// kernels.py:1237-1251
__global__ void k_elec_sigma(float* sigma, const float* f_l, const int32_t* flags, int64_t n,
                             float s_liq, float s_sol) {
    for (int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; c < n;
         c += (int64_t)gridDim.x * blockDim.x) {
        int fl = flags[c];
        sigma[c] = fl == GAS ? 1e-8f : (f_l[c] > 0.55f ? s_liq : s_sol);
    }
}

// The arc source value of cell (i, j, k) (kernels.py:1261-1284).
__device__ __forceinline__ float elec_source_value(int i, int j, int k, float arc_i, float arc_j,
                                                  float arc_k, float inv2s2, float current,
                                                  float vol_eps, int k_min, int k_max) {
    if (k < k_min || k > k_max) return 0.0f;
    float di = (float)i - arc_i, dj = (float)j - arc_j, dk = (float)k - arc_k;
    float r2 = di * di + dj * dj + 0.25f * dk * dk;
    return current * waam_expf(-r2 * inv2s2) / vol_eps;
}

// kernels.py:1255-1284 (clear + inject in one pass)
__global__ void k_elec_source(Dims d, float* src, float arc_i, float arc_j, float arc_k,
                              float inv2s2, float current, float vol_eps, int k_min, int k_max) {
    int i, j, k, c;
    if (!tile_cell(d, i, j, k, c)) return;
    src[c] = elec_source_value(i, j, k, arc_i, arc_j, arc_k, inv2s2, current, vol_eps, k_min,
                               k_max);
}

// kernels.py:1288-1301, pass 1: sum(source * cell_vol) -> scale in ws scalars
__global__ void k_elec_source_sum(const float* src, int64_t n, float cell_vol, float current,
                                  Workspace ws) {
    double part = 0.0;
    for (int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; c < n;
         c += (int64_t)gridDim.x * blockDim.x)
        part += (double)(src[c] * cell_vol);
    __shared__ double sh[kThreads / 32];
    for (int o = 16; o > 0; o >>= 1) part += __shfl_down_sync(0xffffffffu, part, o);
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = part;
    __syncthreads();
    __shared__ bool last;
    if (threadIdx.x == 0) {
        double t = 0.0;
        for (int w = 0; w < kThreads / 32; ++w) t += sh[w];
        ws.partials[blockIdx.x] = t;
        __threadfence();
        last = atomicAdd(ws.counter, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last || threadIdx.x != 0) return;
    __threadfence();
    double t = 0.0;
    for (unsigned b = 0; b < gridDim.x; ++b) t += ((volatile double*)ws.partials)[b];
    float total = (float)t;
    ws.scalars[kOpScalarSourceScale] = current / fmax_(total, 1e-12f);
    *ws.counter = 0u;
}

// V consecutive cells of one column per thread: 4 where nz is a multiple of
// four (then a group never leaves its column) and every field is 16-byte
// aligned, so that a warp's access is 512 bytes; else 1.
template <int V>
__device__ __forceinline__ void load_cells(const float* p, float (&o)[V]) {
    if constexpr (V == 4) {
        const float4 x = *reinterpret_cast<const float4*>(p);
        o[0] = x.x, o[1] = x.y, o[2] = x.z, o[3] = x.w;
    } else {
        o[0] = *p;
    }
}
template <int V>
__device__ __forceinline__ void load_cells(const int32_t* p, int (&o)[V]) {
    if constexpr (V == 4) {
        const int4 x = *reinterpret_cast<const int4*>(p);
        o[0] = x.x, o[1] = x.y, o[2] = x.z, o[3] = x.w;
    } else {
        o[0] = *p;
    }
}
template <int V>
__device__ __forceinline__ void store_cells(float* p, const float (&o)[V]) {
    if constexpr (V == 4)
        *reinterpret_cast<float4*>(p) = make_float4(o[0], o[1], o[2], o[3]);
    else
        *p = o[0];
}

template <typename... P>
bool quads_ok(const Dims& d, const P*... p) {
    uintptr_t bits = 0;
    ((bits |= reinterpret_cast<uintptr_t>(p)), ...);
    return d.nz % 4 == 0 && bits % 16 == 0;
}
// A warp's share of the writing kernels: 32 consecutive k of V neighbouring
// columns, so that it stays within one material (metal below, gas above) and
// skips the arithmetic its cells do not need, while every thread still writes
// 16 bytes (with four columns' 128 cells in a row every warp holds metal:
// k_elec_J beside a step's pending stream 152 us on 512x256x160, 114 so).
struct RowGrid {
    FastDiv by_kt, by_ny;
    int kt, ny, nz, ncol;
};
inline RowGrid row_grid(const Dims& d) {
    const int kt = (d.nz + 31) / 32;
    return RowGrid{FastDiv::of((unsigned)kt), FastDiv::of((unsigned)d.ny), kt, d.ny, d.nz,
                   d.nx * d.ny};
}
template <int V>
inline unsigned row_blocks(const RowGrid& g) {
    const int64_t warps = (int64_t)((g.ncol + V - 1) / V) * g.kt;
    return (unsigned)((warps * 32 + kThreads - 1) / kThreads);
}
// The thread's first cell; false: none.
template <int V>
__device__ __forceinline__ bool row_cells(const RowGrid& g, int& i, int& j, int& k, int& c) {
    constexpr int kLanes = 32 / V;   // lanes per column
    // counted in warps: the threads of more than 2^27 of them pass 32 bits
    const unsigned w = blockIdx.x * (kThreads / 32) + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    const unsigned cg = g.by_kt.div(w);
    const int col = (int)cg * V + lane / kLanes;
    k = (int)(w - cg * (unsigned)g.kt) * 32 + (lane % kLanes) * V;
    if (col >= g.ncol || k >= g.nz) return false;
    i = (int)g.by_ny.div((unsigned)col);
    j = col - i * g.ny;
    c = col * g.nz + k;
    return true;
}
// x / y.  Most quotients here are of a zero (gas, grounded metal), which over a
// positive y is that same zero.
__device__ __forceinline__ float quotient(float x, float y) {
    return x == 0.0f && y > 0.0f ? x : x / y;
}

// Clear + inject + normalise in two passes that read nothing: pass 1 sums
// value * cell_vol over the slab k_min..k_max (every other cell is 0) in
// double, fixed order; pass 2 writes value * scale everywhere, the float the
// reference's in-place scaling leaves.
// Pass 1: one warp per column, lanes over the slab; a column so far from the
// arc that every exponential of it is 0 (waam_expf below -103.98) adds nothing
// and is left out.  A fixed grid, so the order of the sum never changes.
constexpr int kSourceBlocks = 592;
__global__ void __launch_bounds__(kTileK* kTileJ)
    k_elec_source_fused_sum(Dims d, float arc_i, float arc_j, float arc_k, const float* arc_k_dev,
                            float sigma_cells, float inv2s2, float current, float vol_eps,
                            float cell_vol, float target, Workspace ws) {
    if (arc_k_dev) arc_k = *arc_k_dev;
    int k_min, k_max;
    source_slab(arc_k, sigma_cells, d.nz, k_min, k_max);
    double part = 0.0;
    const int ks = imax(k_min, 0), ke = imin(k_max, d.nz - 1);
    const int lane = threadIdx.x;
    // unsigned: one stride past the last of nearly 2^31 columns is still above it
    const unsigned ncol = (unsigned)d.nx * (unsigned)d.ny;
    for (unsigned col = blockIdx.x * kTileJ + threadIdx.y; col < ncol; col += gridDim.x * kTileJ) {
        const int i = (int)(col / (unsigned)d.ny), j = (int)col - i * d.ny;
        const float di = (float)i - arc_i, dj = (float)j - arc_j;
        if (-(di * di + dj * dj) * inv2s2 < -104.0f) continue;
        for (int k = ks + lane; k <= ke; k += kTileK) {
            const float v = elec_source_value(i, j, k, arc_i, arc_j, arc_k, inv2s2, current,
                                              vol_eps, k_min, k_max);
            part += (double)(v * cell_vol);
        }
    }
    double2 tot;
    if (finish_sum2(ws, block_sum2(part, 0.0), tot)) {
        const float total = (float)tot.x;
        ws.scalars[kOpScalarSourceScale] = target / fmax_(total, 1e-12f);
    }
}

// Pass 2: bound by the exponential and the division of each cell in the slab
// (84 % of the SMs' issue slots at 6 % of the DRAM rate; pass 1 the same).
// 512x256x160, alone: 51 us, one cell per thread 71; pass 1 40 and 57.
template <int V>
__global__ void __launch_bounds__(kThreads)
    k_elec_source_fused_write(RowGrid g, float* src, float arc_i, float arc_j, float arc_k,
                              const float* arc_k_dev, float sigma_cells, float inv2s2,
                              float current, float vol_eps, Workspace ws) {
    int i, j, k, at;
    if (!row_cells<V>(g, i, j, k, at)) return;
    if (arc_k_dev) arc_k = *arc_k_dev;
    int k_min, k_max;
    source_slab(arc_k, sigma_cells, g.nz, k_min, k_max);
    const float s = ws.scalars[kOpScalarSourceScale];
    float o[V];
#pragma unroll
    for (int v = 0; v < V; ++v)
        o[v] = elec_source_value(i, j, k + v, arc_i, arc_j, arc_k, inv2s2, current, vol_eps, k_min,
                                 k_max) * s;
    store_cells<V>(src + at, o);
}

// kernels.py:1288-1301, pass 2
__global__ void k_elec_source_scale(float* src, int64_t n, Workspace ws) {
    const float s = ws.scalars[kOpScalarSourceScale];
    for (int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; c < n;
         c += (int64_t)gridDim.x * blockDim.x)
        src[c] *= s;
}

// kernels.py:1315-1355 elec_jacobi_step (+ kernels.py:1387-1398 elec_l1_diff
// of (phi_out, phi_in) when L1 is set).
template <bool L1>
__global__ void __launch_bounds__(kTileK* kTileJ)
    k_elec_jacobi(Dims d, const float* __restrict__ phi_in, float* __restrict__ phi_out,
                  const float* __restrict__ sigma, const float* __restrict__ src,
                  const int32_t* __restrict__ flags, float dx, float omega_j, int nz_solid,
                  float* diff_out, float* norm_out, Workspace ws) {
    const float eps = 1e-12f;
    const int sx = d.ny * d.nz, sy = d.nz;
    double dsum = 0.0, nsum = 0.0;
    for (int i = blockIdx.z; i < d.nx; i += gridDim.z)
        for (int jt = blockIdx.y; jt * kTileJ < d.ny; jt += gridDim.y)
            for (int kt = blockIdx.x; kt * kTileK < d.nz; kt += gridDim.x) {
                const int k = kt * kTileK + threadIdx.x, j = jt * kTileJ + threadIdx.y;
                if (k >= d.nz || j >= d.ny) continue;
                const int c = (i * d.ny + j) * d.nz + k;
                const int fl = flags[c];
                const float pin = phi_in[c];
                float out;
                if (fl == GAS || (k <= nz_solid && fl == SOLID)) {
                    out = 0.0f;
                } else {
                    const int ip = c + (i + 1 < d.nx ? sx : 0), im = c - (i > 0 ? sx : 0);
                    const int jp = c + (j + 1 < d.ny ? sy : 0), jm = c - (j > 0 ? sy : 0);
                    const int kp = c + (k + 1 < d.nz ? 1 : 0), km = c - (k > 0 ? 1 : 0);
                    const float sp = sigma[ip], sm = sigma[im], sn = sigma[jp], ss = sigma[jm];
                    const float st = sigma[kp], sb = sigma[km];
                    const float denom = sp + sm + sn + ss + st + sb + eps;
                    const float nb = sp * phi_in[ip] + sm * phi_in[im] + sn * phi_in[jp] +
                                     ss * phi_in[jm] + st * phi_in[kp] + sb * phi_in[km];
                    const float pn = (nb + src[c] * dx * dx) / denom;
                    out = (1.0f - omega_j) * pin + omega_j * pn;
                }
                phi_out[c] = out;
                if (L1) {
                    dsum += (double)fabsf(out - pin);
                    nsum += (double)fabsf(pin);
                }
            }
    if (L1) {
        double2 part = block_sum2(dsum, nsum);
        double2 tot;
        if (finish_sum2(ws, part, tot)) {
            *diff_out = (float)tot.x;
            *norm_out = (float)tot.y;
        }
    }
}

// The sweep of the fused solve: the same arithmetic as k_elec_jacobi, with
// the fixed cells (GAS, and SOLID at k <= nz_solid) read from a byte mask
// built with sigma, and the source read only inside its k slab (it is 0
// elsewhere).  A tile grid (one cell per thread) for the plain sweeps; the
// L1 sweep keeps the fixed reduction grid.
template <bool L1>
__global__ void __launch_bounds__(kTileK* kTileJ)
    k_elec_jacobi_m(Dims d, const float* __restrict__ phi_in, float* __restrict__ phi_out,
                    const float* __restrict__ sigma, const float* __restrict__ src,
                    const uint8_t* __restrict__ fixed, float dx, float omega_j, int k_src_lo,
                    int k_src_hi, float* diff_out, float* norm_out, Workspace ws) {
    const float eps = 1e-12f;
    const int sx = d.ny * d.nz, sy = d.nz;
    double dsum = 0.0, nsum = 0.0;
    const int i_step = L1 ? gridDim.z : d.nx, j_step = L1 ? gridDim.y : d.ny,
              k_step = L1 ? gridDim.x : d.nz;
    for (int i = blockIdx.z; i < d.nx; i += i_step)
        for (int jt = blockIdx.y; jt * kTileJ < d.ny; jt += j_step)
            for (int kt = blockIdx.x; kt * kTileK < d.nz; kt += k_step) {
                const int k = kt * kTileK + threadIdx.x, j = jt * kTileJ + threadIdx.y;
                if (k >= d.nz || j >= d.ny) continue;
                const int c = (i * d.ny + j) * d.nz + k;
                const float pin = phi_in[c];
                float out;
                if (fixed[c]) {
                    out = 0.0f;
                } else {
                    const int ip = c + (i + 1 < d.nx ? sx : 0), im = c - (i > 0 ? sx : 0);
                    const int jp = c + (j + 1 < d.ny ? sy : 0), jm = c - (j > 0 ? sy : 0);
                    const int kp = c + (k + 1 < d.nz ? 1 : 0), km = c - (k > 0 ? 1 : 0);
                    const float sp = sigma[ip], sm = sigma[im], sn = sigma[jp], ss = sigma[jm];
                    const float st = sigma[kp], sb = sigma[km];
                    const float sc = (k >= k_src_lo && k <= k_src_hi) ? src[c] : 0.0f;
                    const float denom = sp + sm + sn + ss + st + sb + eps;
                    const float nb = sp * phi_in[ip] + sm * phi_in[im] + sn * phi_in[jp] +
                                     ss * phi_in[jm] + st * phi_in[kp] + sb * phi_in[km];
                    const float pn = (nb + sc * dx * dx) / denom;
                    out = (1.0f - omega_j) * pin + omega_j * pn;
                }
                phi_out[c] = out;
                if (L1) {
                    dsum += (double)fabsf(out - pin);
                    nsum += (double)fabsf(pin);
                }
            }
    if (L1) {
        double2 part = block_sum2(dsum, nsum);
        double2 tot;
        if (finish_sum2(ws, part, tot)) {
            *diff_out = (float)tot.x;
            *norm_out = (float)tot.y;
        }
    }
}

// One cell of the masked sweep from its neighbour values, in the reference's
// expression order (kernels.py:1315-1355).
__device__ __forceinline__ float jacobi_cell(float pin, float sp, float sm, float sn, float ss,
                                            float st, float sb, float pp, float pm, float pn_,
                                            float ps, float pt, float pb, float sc, float dx,
                                            float omega_j) {
    const float eps = 1e-12f;
    const float denom = sp + sm + sn + ss + st + sb + eps;
    const float nb = sp * pp + sm * pm + sn * pn_ + ss * ps + st * pt + sb * pb;
    const float pn = (nb + sc * dx * dx) / denom;
    return (1.0f - omega_j) * pin + omega_j * pn;
}

// ---- the potential solve over its live cells ---------------------------------
// Only the cells the sweep does not hold at 0 (metal above the grounded
// plate) change: the sweeps walk a list of them.  The fixed cells stay exact
// because both potential buffers hold 0 at every fixed cell: k_elec_prepare
// zeroes the output buffer of the first sweep at cells that became fixed
// since the previous solve (old mask 0, new mask 1), the zero list zeroes the
// other buffer after that sweep, and every later sweep writes 0 there in the
// reference anyway.  Fixed cells then add exactly 0 to the L1 sums of every
// sweep after the first.  counts: [0] live cells, [1] newly fixed cells,
// [2 + b] live cells of unit b (kUnit consecutive cells), after the scan its
// list offset; after those one live bit per cell and the totals of the scan's
// 1024-unit groups.
constexpr int kCntLive = 0, kCntZero = 1, kCntBlocks = 2;
constexpr int kLiveBlocks = 148 * 8;
constexpr int kUnit = 1024, kUnitWords = kUnit / 32;
constexpr int kScanGroup = 1024;

inline int64_t live_units(const Dims& d) { return (d.n() + kUnit - 1) / kUnit; }
inline int64_t counts_bitmap_offset(int64_t nb) { return kCntBlocks + nb; }
inline int64_t counts_group_offset(int64_t nb) { return kCntBlocks + nb + nb * kUnitWords; }
inline int64_t counts_total_len(int64_t nb) {
    return counts_group_offset(nb) + (nb + kScanGroup - 1) / kScanGroup;
}

// sigma, the fixed-cell mask and one live bit per cell.  Bound by memory: the
// flags and the mask are read, sigma is written everywhere; f_l is read only
// where a group of cells holds metal (512x256x160, alone: 46 us at 57 % of the
// DRAM rate, 130 with one cell per thread and a block vote; beside a step's
// pending stream 50 and 152).  V cells per thread (see load_cells); the
// grid covers whole units, whose bits beyond the grid are 0.
template <int V>
__global__ void __launch_bounds__(kThreads)
    k_elec_prepare(Dims d, CellDecode dec, float* __restrict__ sigma, uint8_t* __restrict__ fixed,
                   float* __restrict__ phi_b, const float* __restrict__ f_l,
                   const int32_t* __restrict__ flags, float s_liq, float s_sol, int nz_solid,
                   int* __restrict__ zero_list, int* __restrict__ counts,
                   unsigned* __restrict__ bitmaps) {
    const unsigned at = (blockIdx.x * kThreads + threadIdx.x) * V;
    const bool in = at < (unsigned)d.n();
    const int lane = threadIdx.x & 31;
    unsigned live = 0u, newly = 0u;
    if (in) {
        int fl[V];
        load_cells<V>(flags + at, fl);
        unsigned of = 0u;   // the mask's V bytes
        if constexpr (V == 4)
            of = *reinterpret_cast<const unsigned*>(fixed + at);
        else
            of = fixed[at];
        bool metal = false;
#pragma unroll
        for (int v = 0; v < V; ++v) metal |= fl[v] != GAS;
        float sg[V];
        unsigned nf = 0u;
        if (!metal) {
#pragma unroll
            for (int v = 0; v < V; ++v) {
                sg[v] = 1e-8f;
                nf |= 1u << (8 * v);
            }
        } else {
            float liq[V];
            load_cells<V>(f_l + at, liq);
            int i, j, k;
            dec.ijk((int)at, i, j, k);
#pragma unroll
            for (int v = 0; v < V; ++v) {
                sg[v] = fl[v] == GAS ? 1e-8f : (liq[v] > 0.55f ? s_liq : s_sol);
                if (fl[v] == GAS || (k + v <= nz_solid && fl[v] == SOLID))
                    nf |= 1u << (8 * v);
                else
                    live |= 1u << v;
            }
        }
        store_cells<V>(sigma + at, sg);
        if (nf != of) {
            if constexpr (V == 4)
                *reinterpret_cast<unsigned*>(fixed + at) = nf;
            else
                fixed[at] = (uint8_t)nf;
        }
#pragma unroll
        for (int v = 0; v < V; ++v)
            if (((nf >> (8 * v)) & 1u) && !((of >> (8 * v)) & 0xffu)) {
                newly |= 1u << v;
                phi_b[at + v] = 0.0f;
            }
    }
    // newly fixed cells: one atomic per warp that has any
    if (__any_sync(0xffffffffu, newly != 0u)) {
        int incl = __popc(newly);
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += y;
        }
        int base = 0;
        if (lane == 31) base = atomicAdd(&counts[kCntZero], incl);
        base = __shfl_sync(0xffffffffu, base, 31) + incl - __popc(newly);
#pragma unroll
        for (int v = 0; v < V; ++v)
            if ((newly >> v) & 1u) zero_list[base++] = (int)at + v;
    }
    // the live bits, one word per 32 cells
    if constexpr (V == 4) {
        unsigned w = live << (4 * (lane & 7));
        for (int o = 1; o < 8; o <<= 1) w |= __shfl_xor_sync(0xffffffffu, w, o);
        if ((lane & 7) == 0) bitmaps[at >> 5] = w;
    } else {
        const unsigned w = __ballot_sync(0xffffffffu, live != 0u);
        if (lane == 0) bitmaps[at >> 5] = w;
    }
}

// Exclusive scan of the units' live counts in two levels: each block of 1024
// threads counts the bits of 1024 units, scans the counts and leaves the group
// total; k_elec_scan_groups scans the totals; k_elec_list adds both.
__device__ __forceinline__ int block_exclusive_scan_1024(int v, int& total) {
    __shared__ int warp_sums[32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    int incl = v;
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += y;
    }
    if (lane == 31) warp_sums[w] = incl;
    __syncthreads();
    if (w == 0) {
        int ws_ = warp_sums[lane], wincl = ws_;
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, wincl, o);
            if (lane >= o) wincl += y;
        }
        warp_sums[lane] = wincl - ws_;
        if (lane == 31) total = wincl;
    }
    __syncthreads();
    const int out = warp_sums[w] + incl - v;
    return out;
}

__global__ void __launch_bounds__(kScanGroup)
    k_elec_scan(int* counts, const unsigned* __restrict__ bitmaps, int nb, int* groups) {
    // a warp's 32 units: 32 words each, read row by row (coalesced)
    const int lane = threadIdx.x & 31;
    const int b0 = blockIdx.x * kScanGroup + (threadIdx.x & ~31), b = b0 + lane;
    int v = 0;
#pragma unroll 8
    for (int u = 0; u < 32; ++u) {
        const unsigned w = b0 + u < nb ? bitmaps[(int64_t)(b0 + u) * kUnitWords + lane] : 0u;
        const int c = (int)__reduce_add_sync(0xffffffffu, (unsigned)__popc(w));
        if (lane == u) v = c;
    }
    int t = 0;
    const int ex = block_exclusive_scan_1024(v, t);
    if (b < nb) counts[kCntBlocks + b] = ex;
    if (threadIdx.x == 31) groups[blockIdx.x] = t;   // thread 31 holds the group total
}

// Exclusive scan of the group totals (one block), total live count to counts[0].
__global__ void __launch_bounds__(kScanGroup) k_elec_scan_groups(int* counts, int* groups,
                                                                 int n_groups) {
    int running = 0;
    for (int g0 = 0; g0 < n_groups; g0 += kScanGroup) {
        const int g = g0 + threadIdx.x;
        const int v = g < n_groups ? groups[g] : 0;
        __shared__ int tot;
        int t = 0;
        const int ex = block_exclusive_scan_1024(v, t);
        if (threadIdx.x == 31) tot = t;
        __syncthreads();
        if (g < n_groups) groups[g] = running + ex;
        running += tot;
        __syncthreads();
    }
    if (threadIdx.x == 0) counts[kCntLive] = running;
}

// The live list in cell order, from the units' bits: one warp per unit
// (grid-stride), which leaves at once when the unit has no live cells.
__global__ void __launch_bounds__(256)
    k_elec_list(const int* __restrict__ counts, const unsigned* __restrict__ bitmaps,
                const int* __restrict__ groups, int nb, int* __restrict__ live_list) {
    const int lane = threadIdx.x & 31;
    const int nwarps = (gridDim.x * blockDim.x) >> 5;
    for (int b = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; b < nb; b += nwarps) {
        const int off = counts[kCntBlocks + b] + groups[b / kScanGroup];
        const int next = b + 1 < nb ? counts[kCntBlocks + b + 1] + groups[(b + 1) / kScanGroup]
                                    : counts[kCntLive];
        if (next == off) continue;
        const unsigned mine = bitmaps[(int64_t)b * kUnitWords + lane];
        int base = off;
        for (int w = 0; w < kUnitWords; ++w) {
            const unsigned m = __shfl_sync(0xffffffffu, mine, w);
            if ((m >> lane) & 1u)
                live_list[base + __popc(m & ((1u << lane) - 1u))] = b * kUnit + w * 32 + lane;
            base += __popc(m);
        }
    }
}

// One sweep over the live list (a fixed grid: the L1 sums in a fixed order).
template <bool L1>
__global__ void __launch_bounds__(256)
    k_elec_jacobi_live(Dims d, CellDecode dec, const float* __restrict__ phi_in, float* __restrict__ phi_out,
                       const float* __restrict__ sigma, const float* __restrict__ src,
                       const int* __restrict__ live_list, const int* __restrict__ counts,
                       float dx, float omega_j, const float* __restrict__ arc_k_dev,
                       float sigma_cells, float* diff_out, float* norm_out, Workspace ws) {
    const int cnt = counts[kCntLive];
    int k_src_lo, k_src_hi;
    source_slab(*arc_k_dev, sigma_cells, d.nz, k_src_lo, k_src_hi);
    const int sx = d.ny * d.nz, sy = d.nz;
    double dsum = 0.0, nsum = 0.0;
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < cnt; t += gridDim.x * blockDim.x) {
        const int c = live_list[t];
        int i, j, k;
        dec.ijk(c, i, j, k);
        const int ip = c + (i + 1 < d.nx ? sx : 0), im = c - (i > 0 ? sx : 0);
        const int jp = c + (j + 1 < d.ny ? sy : 0), jm = c - (j > 0 ? sy : 0);
        const int kp = c + (k + 1 < d.nz ? 1 : 0), km = c - (k > 0 ? 1 : 0);
        const float pin = phi_in[c];
        const float sc = (k >= k_src_lo && k <= k_src_hi) ? src[c] : 0.0f;
        const float out = jacobi_cell(pin, sigma[ip], sigma[im], sigma[jp], sigma[jm], sigma[kp],
                                      sigma[km], phi_in[ip], phi_in[im], phi_in[jp], phi_in[jm],
                                      phi_in[kp], phi_in[km], sc, dx, omega_j);
        phi_out[c] = out;
        if (L1) {
            dsum += (double)fabsf(out - pin);
            nsum += (double)fabsf(pin);
        }
    }
    if (L1) {
        double2 part = block_sum2(dsum, nsum);
        double2 tot;
        if (finish_sum2(ws, part, tot)) {
            *diff_out = (float)tot.x;
            *norm_out = (float)tot.y;
        }
    }
}

__global__ void k_elec_zero_list(const int* __restrict__ zero_list, const int* __restrict__ counts,
                                 float* phi) {
    const int cnt = counts[kCntZero];
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < cnt; t += gridDim.x * blockDim.x)
        phi[zero_list[t]] = 0.0f;
}

// kernels.py:1237-1251 elec_build_sigma, plus the byte mask of the cells the
// Jacobi sweep holds at 0 (kernels.py:1315-1355: GAS, SOLID at k <= nz_solid).
__global__ void k_elec_sigma_mask(Dims d, float* sigma, uint8_t* fixed, const float* f_l,
                                  const int32_t* flags, float s_liq, float s_sol, int nz_solid) {
    int i, j, k, c;
    if (!tile_cell(d, i, j, k, c)) return;
    const int fl = flags[c];
    sigma[c] = fl == GAS ? 1e-8f : (f_l[c] > 0.55f ? s_liq : s_sol);
    fixed[c] = (fl == GAS || (k <= nz_solid && fl == SOLID)) ? 1 : 0;
}

// kernels.py:1387-1398 elec_l1_diff as an operator
__global__ void __launch_bounds__(kTileK* kTileJ)
    k_elec_l1(Dims d, const float* __restrict__ a, const float* __restrict__ b, float* diff_out,
              float* norm_out, Workspace ws) {
    double dsum = 0.0, nsum = 0.0;
    for (int i = blockIdx.z; i < d.nx; i += gridDim.z)
        for (int jt = blockIdx.y; jt * kTileJ < d.ny; jt += gridDim.y)
            for (int kt = blockIdx.x; kt * kTileK < d.nz; kt += gridDim.x) {
                const int k = kt * kTileK + threadIdx.x, j = jt * kTileJ + threadIdx.y;
                if (k >= d.nz || j >= d.ny) continue;
                const int c = (i * d.ny + j) * d.nz + k;
                const float bv = b[c];
                dsum += (double)fabsf(a[c] - bv);
                nsum += (double)fabsf(bv);
            }
    double2 part = block_sum2(dsum, nsum);
    double2 tot;
    if (finish_sum2(ws, part, tot)) {
        *diff_out = (float)tot.x;
        *norm_out = (float)tot.y;
    }
}

// kernels.py:1358-1383 elec_compute_J.  Bound by latency: 58 registers keep 31 %
// of the warps active, at half the DRAM rate.  512x256x160, alone: 94 us, with
// one cell per thread 116 (beside a step's pending stream 114 and 125).
template <int V>
__global__ void __launch_bounds__(kThreads)
    k_elec_J(Dims d, RowGrid g, float* __restrict__ Jx, float* __restrict__ Jy,
             float* __restrict__ Jz, const float* __restrict__ phi,
             const float* __restrict__ sigma, const int32_t* __restrict__ flags, float dx) {
    int i, j, k, c;
    if (!row_cells<V>(g, i, j, k, c)) return;
    int fl[V];
    load_cells<V>(flags + c, fl);
    bool metal = false;
#pragma unroll
    for (int v = 0; v < V; ++v) metal |= fl[v] != GAS;
    float jx[V], jy[V], jz[V];
#pragma unroll
    for (int v = 0; v < V; ++v) jx[v] = jy[v] = jz[v] = 0.0f;
    if (metal) {
        const int sx = d.ny * d.nz, sy = d.nz;
        float sg[V], own[V], xp[V], xm[V], yp[V], ym[V];
        load_cells<V>(sigma + c, sg);
        load_cells<V>(phi + c, own);
        load_cells<V>(phi + c + (i + 1 < d.nx ? sx : 0), xp);
        load_cells<V>(phi + c - (i > 0 ? sx : 0), xm);
        load_cells<V>(phi + c + (j + 1 < d.ny ? sy : 0), yp);
        load_cells<V>(phi + c - (j > 0 ? sy : 0), ym);
        const float below = phi[c - (k > 0 ? 1 : 0)];
        const float above = phi[c + V - 1 + (k + V < d.nz ? 1 : 0)];
        const float two_dx = 2.0f * dx;
#pragma unroll
        for (int v = 0; v < V; ++v) {
            if (fl[v] == GAS) continue;
            const float zp = v + 1 < V ? own[v + 1 < V ? v + 1 : v] : above;
            const float zm = v > 0 ? own[v > 0 ? v - 1 : v] : below;
            jx[v] = -sg[v] * quotient(xp[v] - xm[v], two_dx);
            jy[v] = -sg[v] * quotient(yp[v] - ym[v], two_dx);
            jz[v] = -sg[v] * quotient(zp - zm, two_dx);
        }
    }
    store_cells<V>(Jx + c, jx);
    store_cells<V>(Jy + c, jy);
    store_cells<V>(Jz + c, jz);
}

__device__ __forceinline__ int radial_bin(float di, float dj, float bin_dr, int n_bins,
                                          float& r) {
    r = sqrtf(di * di + dj * dj);
    return imin((int)(r / bin_dr), n_bins - 1);
}

// kernels.py:1402-1421 elec_bin_axial_current: per z slab, sum of Jz dx^2 by
// radius bin.  Block (s, k) sums a strip of columns of slab k in shared
// double bins, then adds them to the slab's double accumulators.
__global__ void k_elec_bin(Dims d, const float* __restrict__ Jz, double* acc, float arc_i,
                           float arc_j, float dx2, float bin_dr, int n_bins) {
    extern __shared__ double sbin[];
    const int k = blockIdx.y;
    for (int b = threadIdx.x; b < n_bins; b += blockDim.x) sbin[b] = 0.0;
    __syncthreads();
    const int ncol = d.nx * d.ny;
    for (int col = blockIdx.x * blockDim.x + threadIdx.x; col < ncol;
         col += gridDim.x * blockDim.x) {
        const int i = col / d.ny, j = col - i * d.ny;
        float r;
        const int b = radial_bin((float)i - arc_i, (float)j - arc_j, bin_dr, n_bins, r);
        atomicAdd(&sbin[b], (double)(Jz[(int64_t)col * d.nz + k] * dx2));
    }
    __syncthreads();
    for (int b = threadIdx.x; b < n_bins; b += blockDim.x)
        if (sbin[b] != 0.0) atomicAdd(&acc[(int64_t)k * n_bins + b], sbin[b]);
}

// The same sums without atomics: block (kt, ch) is one warp that owns k in
// [32 kt, 32 kt + 32) of a contiguous chunk of columns and adds each column's
// Jz dx^2 into its private shared double bins (lane k touches only its own
// slots), column after column; the loads of 32 columns are in flight at a
// time, coalesced along k, and lane u finds the bin of the u-th of them.  The
// per-chunk bins go to partials[ch][b][k]; k_elec_bin_combine adds the chunks
// in a fixed order, so the bins are the same on every run.
constexpr int kBinUnroll = 32;

__global__ void __launch_bounds__(32) k_elec_bin_cols(Dims d, const float* __restrict__ Jz,
                                                      double* __restrict__ partials, float arc_i,
                                                      float arc_j, float dx2, float bin_dr,
                                                      int n_bins, int chunk) {
    extern __shared__ double sacc[];   // [n_bins][32]
    const int lane = threadIdx.x;
    const int k = blockIdx.x * 32 + lane;
    for (int b = 0; b < n_bins; ++b) sacc[b * 32 + lane] = 0.0;
    const int ncol = d.nx * d.ny;
    const int c0 = blockIdx.y * chunk, c1 = imin(ncol, c0 + chunk);
    const bool kin = k < d.nz;
    for (int col = c0; col < c1; col += kBinUnroll) {
        float v[kBinUnroll];
#pragma unroll
        for (int u = 0; u < kBinUnroll; ++u)
            v[u] = (kin && col + u < c1) ? Jz[(int64_t)(col + u) * d.nz + k] : 0.0f;
        int my_bin = 0;
        if (col + lane < c1) {
            const int i = (col + lane) / d.ny, j = (col + lane) - i * d.ny;
            float r;
            my_bin = radial_bin((float)i - arc_i, (float)j - arc_j, bin_dr, n_bins, r);
        }
#pragma unroll
        for (int u = 0; u < kBinUnroll; ++u) {
            const int b = __shfl_sync(0xffffffffu, my_bin, u);
            if (col + u < c1) sacc[b * 32 + lane] += (double)(v[u] * dx2);
        }
    }
    if (!kin) return;
    double* out = partials + (int64_t)blockIdx.y * n_bins * d.nz;
    for (int b = 0; b < n_bins; ++b) out[(int64_t)b * d.nz + k] = sacc[b * 32 + lane];
}

// Block (kt, b): the chunks of bin b for 32 consecutive k (coalesced); warp w
// adds chunks w, w + 8, ... in order, then the eight warps' sums in order.
__global__ void __launch_bounds__(256) k_elec_bin_combine(const double* __restrict__ partials,
                                                          float* bins, int nz, int n_bins,
                                                          int chunks) {
    __shared__ double sh[8][32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int k = blockIdx.x * 32 + lane, b = blockIdx.y;
    double s = 0.0;
    if (k < nz) {
#pragma unroll 8
        for (int ch = w; ch < chunks; ch += 8) s += partials[((int64_t)ch * n_bins + b) * nz + k];
    }
    sh[w][lane] = s;
    __syncthreads();
    if (w != 0 || k >= nz) return;
    double t = sh[0][lane];
    for (int q = 1; q < 8; ++q) t += sh[q][lane];
    bins[(int64_t)k * n_bins + b] = (float)t;
}

__global__ void k_elec_bin_store(const double* acc, float* bins, int64_t m) {
    for (int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; q < m;
         q += (int64_t)gridDim.x * blockDim.x)
        bins[q] = (float)acc[q];
}

// kernels.py:1424-1435 elec_prefix_bins (float, in place): one warp per k, the
// bins loaded 32 at a time and added one after another through shuffles (the
// float order of the reference).
__global__ void __launch_bounds__(256) k_elec_prefix(float* bins, int n_bins, int nz) {
    const int k = (int)(blockIdx.x * (blockDim.x / 32) + (threadIdx.x >> 5));
    const int lane = threadIdx.x & 31;
    if (k >= nz) return;
    float a = 0.0f;
    for (int b0 = 0; b0 < n_bins; b0 += 32) {
        const bool in = b0 + lane < n_bins;
        const float v = in ? bins[(int64_t)k * n_bins + b0 + lane] : 0.0f;
        const int m = imin(32, n_bins - b0);
        float mine = 0.0f;
        for (int o = 0; o < m; ++o) {
            a += __shfl_sync(0xffffffffu, v, o);
            if (o == lane) mine = a;
        }
        if (in) bins[(int64_t)k * n_bins + b0 + lane] = mine;
    }
}

// kernels.py:1438-1475 elec_B_axisymmetric: V cells of a column per thread,
// which share its radius, bin and r * dx; each cell takes the reference's
// three divisions in its order.  Bound by those divisions (81 % of the SMs'
// issue slots at 14 % of the DRAM rate).  512x256x160, alone: 106 us, 112 with
// a warp per column (beside a step's pending stream 118 and 127).
template <int V>
__global__ void __launch_bounds__(kThreads)
    k_elec_B_cols(RowGrid g, float* __restrict__ Bx, float* __restrict__ By,
                  float* __restrict__ Bz, const float* __restrict__ bins, float arc_i, float arc_j,
                  float dx, float bin_dr, float mu0, int n_bins) {
    int i, j, k, at;
    if (!row_cells<V>(g, i, j, k, at)) return;
    const float di = (float)i - arc_i, dj = (float)j - arc_j;
    float rc;
    const int b = radial_bin(di, dj, bin_dr, n_bins, rc);
    const bool on = rc > 1e-3f;
    const float rm = rc * dx;
    const float two_pi = 6.28318530717958647692f;
    float bx[V], by[V], bz[V];
#pragma unroll
    for (int v = 0; v < V; ++v) {
        bx[v] = by[v] = bz[v] = 0.0f;
        if (on) {
            const float I = bins[(int64_t)(k + v) * n_bins + b];
            const float Bt = quotient(mu0 * I, two_pi * rm);
            bx[v] = quotient(-Bt * dj, rc);
            by[v] = quotient(Bt * di, rc);
        }
    }
    store_cells<V>(Bx + at, bx);
    store_cells<V>(By + at, by);
    store_cells<V>(Bz + at, bz);
}

// kernels.py:1479-1513 apply_lorentz_JxB
__global__ void k_lorentz_JxB(float* Fx, float* Fy, float* Fz, const float* __restrict__ Jx,
                              const float* __restrict__ Jy, const float* __restrict__ Jz,
                              const float* __restrict__ Bx, const float* __restrict__ By,
                              const float* __restrict__ Bz, const float* __restrict__ f_l,
                              const int32_t* __restrict__ flags, int64_t n, float dt, float dx,
                              float rho_ref) {
    for (int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; c < n;
         c += (int64_t)gridDim.x * blockDim.x) {
        const float fl = f_l[c];
        if (flags[c] == GAS || fl < 0.05f) continue;
        const float jx = Jx[c], jy = Jy[c], jz = Jz[c], bx = Bx[c], by = By[c], bz = Bz[c];
        const float fxp = jy * bz - jz * by, fyp = jz * bx - jx * bz, fzp = jx * by - jy * bx;
        const float flw = fmin_(1.0f, fl);
        const float scale = flw * dt * dt / (rho_ref * dx);
        Fx[c] += fxp * scale;
        Fy[c] += fyp * scale;
        Fz[c] += fzp * scale;
    }
}

}  // namespace
}  // namespace waam

using namespace waam;


#define REQUIRE(cond, msg) \
    if (!(cond)) return waam::fail(WAAM_ERR_INVALID, msg)

extern "C" {

int waam_elec_build_sigma(float* sigma, const float* f_l, const int32_t* flags, int64_t n,
                          float sigma_liquid, float sigma_solid, void* stream) {
    REQUIRE(sigma && f_l && flags && n > 0, "elec_build_sigma: null field or empty grid");
    k_elec_sigma<<<elem_blocks(n), kThreads, 0, STREAM(stream)>>>(sigma, f_l, flags, n,
                                                                  sigma_liquid, sigma_solid);
    return check_launch("k_elec_sigma");
}

int waam_elec_inject_arc_source(float* source, int nx, int ny, int nz, float arc_i, float arc_j,
                                float arc_k, float sigma_cells, float current_A, float dx,
                                void* stream) {
    REQUIRE(dims_ok(nx, ny, nz), "elec_inject_arc_source: bad dims");
    REQUIRE(source, "elec_inject_arc_source: null field");
    REQUIRE(std::isfinite(arc_k) && std::isfinite(sigma_cells) && std::fabs(arc_k) < 1e6f &&
                std::fabs(sigma_cells) < 1e6f,
            "elec_inject_arc_source: arc k / sigma not finite");
    const float eps = 1e-6f;
    const float inv2s2 = 1.0f / (2.0f * sigma_cells * sigma_cells + eps);
    const float cell_vol = dx * dx * dx;
    int k_min, k_max;
    source_slab(arc_k, sigma_cells, nz, k_min, k_max);
    Dims d{nx, ny, nz};
    k_elec_source<<<tile_grid(d), tile_block(), 0, STREAM(stream)>>>(
        d, source, arc_i, arc_j, arc_k, inv2s2, current_A, cell_vol + eps, k_min, k_max);
    return check_launch("k_elec_source");
}

static int arc_source_impl(float* source, int nx, int ny, int nz, float arc_i, float arc_j,
                           float arc_k, const float* arc_k_dev, float sigma_cells,
                           float current_A, float dx, void* workspace, size_t workspace_bytes,
                           void* stream) {
    REQUIRE(dims_ok(nx, ny, nz), "elec_arc_source: bad dims");
    REQUIRE(source, "elec_arc_source: null field");
    REQUIRE(std::isfinite(arc_k) && std::isfinite(sigma_cells) && std::fabs(arc_k) < 1e6f &&
                std::fabs(sigma_cells) < 1e6f,
            "elec_arc_source: arc k / sigma not finite");
    Dims d{nx, ny, nz};
    REQUIRE(workspace_ok(workspace, workspace_bytes, d.n()),
            "elec_arc_source: workspace too small or misaligned");
    Workspace ws = Workspace::at(workspace);
    const float eps = 1e-6f;
    const float inv2s2 = 1.0f / (2.0f * sigma_cells * sigma_cells + eps);
    const float cell_vol = dx * dx * dx;
    k_elec_source_fused_sum<<<kSourceBlocks, tile_block(), 0, STREAM(stream)>>>(
        d, arc_i, arc_j, arc_k, arc_k_dev, sigma_cells, inv2s2, current_A, cell_vol + eps,
        cell_vol, current_A, ws);
    int rc = check_launch("k_elec_source_fused_sum");
    if (rc) return rc;
    const RowGrid g = row_grid(d);
    if (quads_ok(d, source))
        k_elec_source_fused_write<4><<<row_blocks<4>(g), kThreads, 0, STREAM(stream)>>>(
            g, source, arc_i, arc_j, arc_k, arc_k_dev, sigma_cells, inv2s2, current_A,
            cell_vol + eps, ws);
    else
        k_elec_source_fused_write<1><<<row_blocks<1>(g), kThreads, 0, STREAM(stream)>>>(
            g, source, arc_i, arc_j, arc_k, arc_k_dev, sigma_cells, inv2s2, current_A,
            cell_vol + eps, ws);
    return check_launch("k_elec_source_fused_write");
}

int waam_elec_arc_source(float* source, int nx, int ny, int nz, float arc_i, float arc_j,
                         float arc_k, float sigma_cells, float current_A, float dx,
                         void* workspace, size_t workspace_bytes, void* stream) {
    return arc_source_impl(source, nx, ny, nz, arc_i, arc_j, arc_k, nullptr, sigma_cells,
                           current_A, dx, workspace, workspace_bytes, stream);
}

int waam_elec_arc_source_dev(float* source, int nx, int ny, int nz, float arc_i, float arc_j,
                             const float* arc_k_dev, float sigma_cells, float current_A,
                             float dx, void* workspace, size_t workspace_bytes, void* stream) {
    REQUIRE(arc_k_dev, "elec_arc_source_dev: null arc k");
    return arc_source_impl(source, nx, ny, nz, arc_i, arc_j, 0.0f, arc_k_dev, sigma_cells,
                           current_A, dx, workspace, workspace_bytes, stream);
}

int waam_elec_normalize_source(float* source, int64_t n, float target_current_A, float dx,
                               void* workspace, size_t workspace_bytes, void* stream) {
    REQUIRE(source && n > 0, "elec_normalize_source: null field or empty grid");
    REQUIRE(workspace_ok(workspace, workspace_bytes, n),
            "elec_normalize_source: workspace too small or misaligned");
    Workspace ws = Workspace::at(workspace);
    const float cell_vol = dx * dx * dx;
    k_elec_source_sum<<<red_blocks(n), kThreads, 0, STREAM(stream)>>>(source, n, cell_vol,
                                                                      target_current_A, ws);
    int rc = check_launch("k_elec_source_sum");
    if (rc) return rc;
    k_elec_source_scale<<<elem_blocks(n), kThreads, 0, STREAM(stream)>>>(source, n, ws);
    return check_launch("k_elec_source_scale");
}

int waam_elec_init_ground(float* phi, int64_t n, void* stream) {
    REQUIRE(phi && n > 0, "elec_init_ground: null field or empty grid");
    cudaError_t e = cudaMemsetAsync(phi, 0, (size_t)n * sizeof(float), STREAM(stream));
    if (e != cudaSuccess) return fail(WAAM_ERR_CUDA, cudaGetErrorString(e));
    return WAAM_OK;
}

int waam_elec_jacobi_step(const float* phi_in, float* phi_out, const float* sigma,
                          const float* source, const int32_t* flags, int nx, int ny, int nz,
                          float dx, float omega_j, int nz_solid, void* stream) {
    REQUIRE(dims_ok(nx, ny, nz), "elec_jacobi_step: bad dims");
    REQUIRE(phi_in && phi_out && sigma && source && flags && phi_in != phi_out,
            "elec_jacobi_step: null or aliased field");
    Dims d{nx, ny, nz};
    k_elec_jacobi<false><<<red_tile_grid(d), tile_block(), 0, STREAM(stream)>>>(
        d, phi_in, phi_out, sigma, source, flags, dx, omega_j, nz_solid, nullptr, nullptr,
        Workspace{});
    return check_launch("k_elec_jacobi");
}

int waam_elec_jacobi_step_l1(const float* phi_in, float* phi_out, const float* sigma,
                             const float* source, const int32_t* flags, int nx, int ny, int nz,
                             float dx, float omega_j, int nz_solid, float* diff_buf,
                             float* norm_buf, void* workspace, size_t workspace_bytes,
                             void* stream) {
    REQUIRE(dims_ok(nx, ny, nz), "elec_jacobi_step_l1: bad dims");
    REQUIRE(phi_in && phi_out && sigma && source && flags && diff_buf && norm_buf &&
                phi_in != phi_out,
            "elec_jacobi_step_l1: null or aliased field");
    Dims d{nx, ny, nz};
    REQUIRE(workspace_ok(workspace, workspace_bytes, d.n()),
            "elec_jacobi_step_l1: workspace too small or misaligned");
    k_elec_jacobi<true><<<red_tile_grid(d), tile_block(), 0, STREAM(stream)>>>(
        d, phi_in, phi_out, sigma, source, flags, dx, omega_j, nz_solid, diff_buf, norm_buf,
        Workspace::at(workspace));
    return check_launch("k_elec_jacobi_l1");
}

int waam_elec_build_sigma_mask(float* sigma, uint8_t* fixed, const float* f_l,
                               const int32_t* flags, int nx, int ny, int nz, float sigma_liquid,
                               float sigma_solid, int nz_solid, void* stream) {
    REQUIRE(dims_ok(nx, ny, nz), "elec_build_sigma_mask: bad dims");
    REQUIRE(sigma && fixed && f_l && flags, "elec_build_sigma_mask: null field");
    Dims d{nx, ny, nz};
    k_elec_sigma_mask<<<tile_grid(d), tile_block(), 0, STREAM(stream)>>>(
        d, sigma, fixed, f_l, flags, sigma_liquid, sigma_solid, nz_solid);
    return check_launch("k_elec_sigma_mask");
}

int waam_elec_jacobi_chunk(float* phi_a, float* phi_b, const float* sigma, const float* source,
                           const uint8_t* fixed, int nx, int ny, int nz, float dx, float omega_j,
                           int n_sweeps, float arc_k, float sigma_cells, float* diff_buf,
                           float* norm_buf, void* workspace, size_t workspace_bytes,
                           void* stream) {
    REQUIRE(dims_ok(nx, ny, nz), "elec_jacobi_chunk: bad dims");
    REQUIRE(phi_a && phi_b && sigma && source && fixed && diff_buf && norm_buf && phi_a != phi_b,
            "elec_jacobi_chunk: null or aliased field");
    REQUIRE(n_sweeps >= 1, "elec_jacobi_chunk: n_sweeps must be >= 1");
    REQUIRE(std::isfinite(arc_k) && std::isfinite(sigma_cells) && std::fabs(arc_k) < 1e6f &&
                std::fabs(sigma_cells) < 1e6f,
            "elec_jacobi_chunk: arc k / sigma not finite");
    Dims d{nx, ny, nz};
    REQUIRE(workspace_ok(workspace, workspace_bytes, d.n()),
            "elec_jacobi_chunk: workspace too small or misaligned");
    int k_lo, k_hi;
    source_slab(arc_k, sigma_cells, nz, k_lo, k_hi);
    float* in = phi_a;
    float* out = phi_b;
    for (int s = 0; s < n_sweeps; ++s) {
        if (s + 1 < n_sweeps) {
            k_elec_jacobi_m<false><<<tile_grid(d), tile_block(), 0, STREAM(stream)>>>(
                d, in, out, sigma, source, fixed, dx, omega_j, k_lo, k_hi, nullptr, nullptr,
                Workspace{});
        } else {
            k_elec_jacobi_m<true><<<red_tile_grid(d), tile_block(), 0, STREAM(stream)>>>(
                d, in, out, sigma, source, fixed, dx, omega_j, k_lo, k_hi, diff_buf, norm_buf,
                Workspace::at(workspace));
        }
        int rc = check_launch("k_elec_jacobi_m");
        if (rc) return rc;
        float* t = in;
        in = out;
        out = t;
    }
    return WAAM_OK;
}

int64_t waam_elec_counts_len(int nx, int ny, int nz) {
    if (!dims_ok(nx, ny, nz)) return 0;
    return counts_total_len(live_units(Dims{nx, ny, nz}));
}

int waam_elec_prepare(float* sigma, uint8_t* fixed, float* phi_b, const float* f_l,
                      const int32_t* flags, int nx, int ny, int nz, float sigma_liquid,
                      float sigma_solid, int nz_solid, int32_t* live_list, int32_t* zero_list,
                      int32_t* counts, int64_t counts_len, void* stream) {
    REQUIRE(dims_ok(nx, ny, nz), "elec_prepare: bad dims");
    REQUIRE(sigma && fixed && phi_b && f_l && flags && live_list && zero_list && counts,
            "elec_prepare: null field");
    REQUIRE(counts_len >= waam_elec_counts_len(nx, ny, nz), "elec_prepare: counts too short");
    Dims d{nx, ny, nz};
    const int nb = (int)live_units(d);
    cudaError_t e = cudaMemsetAsync(counts, 0, kCntBlocks * sizeof(int32_t), STREAM(stream));
    if (e != cudaSuccess) return fail(WAAM_ERR_CUDA, cudaGetErrorString(e));
    unsigned* bitmaps = reinterpret_cast<unsigned*>(counts + counts_bitmap_offset(nb));
    int* groups = counts + counts_group_offset(nb);
    const int n_groups = (nb + kScanGroup - 1) / kScanGroup;
    const CellDecode dec = CellDecode::of(d);
    const unsigned cells = (unsigned)nb * kUnit;
    if (quads_ok(d, sigma, fixed, f_l, flags))
        k_elec_prepare<4><<<cells / (4 * kThreads), kThreads, 0, STREAM(stream)>>>(
            d, dec, sigma, fixed, phi_b, f_l, flags, sigma_liquid, sigma_solid, nz_solid,
            zero_list, counts, bitmaps);
    else
        k_elec_prepare<1><<<cells / kThreads, kThreads, 0, STREAM(stream)>>>(
            d, dec, sigma, fixed, phi_b, f_l, flags, sigma_liquid, sigma_solid, nz_solid,
            zero_list, counts, bitmaps);
    int rc = check_launch("k_elec_prepare");
    if (rc) return rc;
    k_elec_scan<<<n_groups, kScanGroup, 0, STREAM(stream)>>>(counts, bitmaps, nb, groups);
    rc = check_launch("k_elec_scan");
    if (rc) return rc;
    k_elec_scan_groups<<<1, kScanGroup, 0, STREAM(stream)>>>(counts, groups, n_groups);
    rc = check_launch("k_elec_scan_groups");
    if (rc) return rc;
    k_elec_list<<<kLiveBlocks, 256, 0, STREAM(stream)>>>(counts, bitmaps, groups, nb, live_list);
    return check_launch("k_elec_list");
}

int waam_elec_jacobi_live(float* phi_a, float* phi_b, const float* sigma, const float* source,
                          const int32_t* live_list, const int32_t* zero_list,
                          const int32_t* counts, int nx, int ny, int nz, float dx,
                          float omega_j, int n_sweeps, int first_chunk, const float* arc_k_dev,
                          float sigma_cells, float* diff_buf, float* norm_buf, void* workspace,
                          size_t workspace_bytes, void* stream) {
    REQUIRE(dims_ok(nx, ny, nz), "elec_jacobi_live: bad dims");
    REQUIRE(phi_a && phi_b && sigma && source && live_list && zero_list && counts && diff_buf &&
                norm_buf && phi_a != phi_b,
            "elec_jacobi_live: null or aliased field");
    REQUIRE(n_sweeps >= 1, "elec_jacobi_live: n_sweeps must be >= 1");
    REQUIRE(!first_chunk || n_sweeps >= 2,
            "elec_jacobi_live: the first chunk of a solve needs at least 2 sweeps");
    REQUIRE(arc_k_dev && std::isfinite(sigma_cells) && std::fabs(sigma_cells) < 1e6f,
            "elec_jacobi_live: null arc k or sigma not finite");
    Dims d{nx, ny, nz};
    REQUIRE(workspace_ok(workspace, workspace_bytes, d.n()),
            "elec_jacobi_live: workspace too small or misaligned");
    const CellDecode dec = CellDecode::of(d);
    float* in = phi_a;
    float* out = phi_b;
    for (int s = 0; s < n_sweeps; ++s) {
        if (s + 1 < n_sweeps)
            k_elec_jacobi_live<false><<<kLiveBlocks, 256, 0, STREAM(stream)>>>(
                d, dec, in, out, sigma, source, live_list, counts, dx, omega_j, arc_k_dev,
                sigma_cells, nullptr, nullptr, Workspace{});
        else
            k_elec_jacobi_live<true><<<kLiveBlocks, 256, 0, STREAM(stream)>>>(
                d, dec, in, out, sigma, source, live_list, counts, dx, omega_j, arc_k_dev,
                sigma_cells, diff_buf, norm_buf, Workspace::at(workspace));
        int rc = check_launch("k_elec_jacobi_live");
        if (rc) return rc;
        if (first_chunk && s == 0) {
            // the input of the first sweep: its newly fixed cells become 0
            k_elec_zero_list<<<kLiveBlocks, 256, 0, STREAM(stream)>>>(zero_list, counts, in);
            rc = check_launch("k_elec_zero_list");
            if (rc) return rc;
        }
        float* t = in;
        in = out;
        out = t;
    }
    return WAAM_OK;
}

int waam_elec_l1_diff(const float* a, const float* b, float* diff_buf, float* norm_buf, int nx,
                      int ny, int nz, void* workspace, size_t workspace_bytes, void* stream) {
    REQUIRE(dims_ok(nx, ny, nz), "elec_l1_diff: bad dims");
    REQUIRE(a && b && diff_buf && norm_buf, "elec_l1_diff: null field");
    Dims d{nx, ny, nz};
    REQUIRE(workspace_ok(workspace, workspace_bytes, d.n()),
            "elec_l1_diff: workspace too small or misaligned");
    k_elec_l1<<<red_tile_grid(d), tile_block(), 0, STREAM(stream)>>>(d, a, b, diff_buf, norm_buf,
                                                                     Workspace::at(workspace));
    return check_launch("k_elec_l1");
}

int waam_elec_compute_J(float* Jx, float* Jy, float* Jz, const float* phi, const float* sigma,
                        const int32_t* flags, int nx, int ny, int nz, float dx, void* stream) {
    REQUIRE(dims_ok(nx, ny, nz), "elec_compute_J: bad dims");
    REQUIRE(Jx && Jy && Jz && phi && sigma && flags, "elec_compute_J: null field");
    Dims d{nx, ny, nz};
    const RowGrid g = row_grid(d);
    if (quads_ok(d, Jx, Jy, Jz, phi, sigma, flags))
        k_elec_J<4><<<row_blocks<4>(g), kThreads, 0, STREAM(stream)>>>(d, g, Jx, Jy, Jz, phi,
                                                                      sigma, flags, dx);
    else
        k_elec_J<1><<<row_blocks<1>(g), kThreads, 0, STREAM(stream)>>>(d, g, Jx, Jy, Jz, phi,
                                                                      sigma, flags, dx);
    return check_launch("k_elec_J");
}

int waam_elec_bin_axial_current(const float* Jz, float* bins, int nx, int ny, int nz, float arc_i,
                                float arc_j, float dx, float bin_dr_cells, int n_bins,
                                void* workspace, size_t workspace_bytes, void* stream) {
    REQUIRE(dims_ok(nx, ny, nz), "elec_bin_axial_current: bad dims");
    REQUIRE(Jz && bins, "elec_bin_axial_current: null field");
    REQUIRE(n_bins >= 1 && n_bins <= kMaxBins, "elec_bin_axial_current: n_bins out of range");
    Dims d{nx, ny, nz};
    REQUIRE(workspace_ok(workspace, workspace_bytes, d.n()),
            "elec_bin_axial_current: workspace too small or misaligned");
    // double accumulators in the workspace's field scratch
    const int64_t m = (int64_t)nz * n_bins;
    REQUIRE((size_t)m * sizeof(double) <= (size_t)(d.n() + kFieldSlack) * sizeof(float),
            "elec_bin_axial_current: nz * n_bins accumulators exceed the workspace");
    Workspace ws = Workspace::at(workspace);
    double* acc = reinterpret_cast<double*>(ws.field);
    const int ncol = nx * ny;
    {
        // chunked per-warp bins in the field scratch, when they fit
        const size_t field_bytes = (size_t)(d.n() + kFieldSlack) * sizeof(float);
        const int ktiles = (nz + 31) / 32;
        int chunks = imax(1, (148 * 12) / ktiles);
        chunks = imin(chunks, ncol);
        chunks = (int)std::min<int64_t>(chunks, (int64_t)(field_bytes / ((size_t)m * sizeof(double))));
        if (chunks >= 1 && (size_t)n_bins * 32 * sizeof(double) <= 48 * 1024) {
            const int chunk = (ncol + chunks - 1) / chunks;
            chunks = (ncol + chunk - 1) / chunk;
            k_elec_bin_cols<<<dim3(ktiles, chunks), 32, (size_t)n_bins * 32 * sizeof(double),
                              STREAM(stream)>>>(d, Jz, acc, arc_i, arc_j, dx * dx, bin_dr_cells,
                                                n_bins, chunk);
            int rc = check_launch("k_elec_bin_cols");
            if (rc) return rc;
            k_elec_bin_combine<<<dim3(ktiles, n_bins), 256, 0, STREAM(stream)>>>(
                acc, bins, nz, n_bins, chunks);
            return check_launch("k_elec_bin_combine");
        }
    }
    cudaError_t e = cudaMemsetAsync(acc, 0, (size_t)m * sizeof(double), STREAM(stream));
    if (e != cudaSuccess) return fail(WAAM_ERR_CUDA, cudaGetErrorString(e));
    const int strips = imax(1, imin((ncol + kThreads - 1) / kThreads, imax(1, 1184 / nz)));
    k_elec_bin<<<dim3(strips, nz), kThreads, n_bins * sizeof(double), STREAM(stream)>>>(
        d, Jz, acc, arc_i, arc_j, dx * dx, bin_dr_cells, n_bins);
    int rc = check_launch("k_elec_bin");
    if (rc) return rc;
    k_elec_bin_store<<<elem_blocks(m), kThreads, 0, STREAM(stream)>>>(acc, bins, m);
    return check_launch("k_elec_bin_store");
}

int waam_elec_prefix_bins(float* bins, int n_bins, int nz, void* stream) {
    REQUIRE(bins && n_bins >= 1 && nz >= 1, "elec_prefix_bins: bad arguments");
    k_elec_prefix<<<(nz + 7) / 8, 256, 0, STREAM(stream)>>>(bins, n_bins, nz);
    return check_launch("k_elec_prefix");
}

int waam_elec_B_axisymmetric(float* Bx, float* By, float* Bz, const float* bins, int nx, int ny,
                             int nz, float arc_i, float arc_j, float dx, float bin_dr_cells,
                             float mu0, int n_bins, void* stream) {
    REQUIRE(dims_ok(nx, ny, nz), "elec_B_axisymmetric: bad dims");
    REQUIRE(Bx && By && Bz && bins, "elec_B_axisymmetric: null field");
    REQUIRE(n_bins >= 1, "elec_B_axisymmetric: n_bins out of range");
    Dims d{nx, ny, nz};
    const RowGrid g = row_grid(d);
    if (quads_ok(d, Bx, By, Bz))
        k_elec_B_cols<4><<<row_blocks<4>(g), kThreads, 0, STREAM(stream)>>>(
            g, Bx, By, Bz, bins, arc_i, arc_j, dx, bin_dr_cells, mu0, n_bins);
    else
        k_elec_B_cols<1><<<row_blocks<1>(g), kThreads, 0, STREAM(stream)>>>(
            g, Bx, By, Bz, bins, arc_i, arc_j, dx, bin_dr_cells, mu0, n_bins);
    return check_launch("k_elec_B_cols");
}

int waam_elec_fields(float* Jx, float* Jy, float* Jz, float* Bx, float* By, float* Bz,
                     float* bins, const float* phi, const float* sigma, const int32_t* flags,
                     int nx, int ny, int nz, float arc_i, float arc_j, float dx,
                     float bin_dr_cells, float mu0, int n_bins, void* workspace,
                     size_t workspace_bytes, void* stream) {
    int rc = waam_elec_compute_J(Jx, Jy, Jz, phi, sigma, flags, nx, ny, nz, dx, stream);
    if (rc) return rc;
    rc = waam_elec_bin_axial_current(Jz, bins, nx, ny, nz, arc_i, arc_j, dx, bin_dr_cells,
                                     n_bins, workspace, workspace_bytes, stream);
    if (rc) return rc;
    rc = waam_elec_prefix_bins(bins, n_bins, nz, stream);
    if (rc) return rc;
    return waam_elec_B_axisymmetric(Bx, By, Bz, bins, nx, ny, nz, arc_i, arc_j, dx, bin_dr_cells,
                                    mu0, n_bins, stream);
}

int waam_apply_lorentz_JxB(float* Fx, float* Fy, float* Fz, const float* Jx, const float* Jy,
                           const float* Jz, const float* Bx, const float* By, const float* Bz,
                           const float* f_l, const int32_t* flags, int64_t n, float dt, float dx,
                           float rho_ref, void* stream) {
    REQUIRE(Fx && Fy && Fz && Jx && Jy && Jz && Bx && By && Bz && f_l && flags && n > 0,
            "apply_lorentz_JxB: null field or empty grid");
    k_lorentz_JxB<<<elem_blocks(n), kThreads, 0, STREAM(stream)>>>(Fx, Fy, Fz, Jx, Jy, Jz, Bx, By,
                                                                   Bz, f_l, flags, n, dt, dx,
                                                                   rho_ref);
    return check_launch("k_lorentz_JxB");
}

}  // extern "C"
