// Esirkepov current deposition (Jx, Jy) -- new; the reference's "Esirkepov"
// deposits trajectory-averaged charge only (src/deposition/ngp.cpp:13-84).
//
// First-order (CIC-shape) charge-conserving current, Esirkepov, Comput. Phys.
// Commun. 135 (2001) 144, in 2D. For a particle moving by (dx_c, dy_c) cells
// (|d| < 1 on each axis, else PIC_ERR_COURANT), with S0/S1 the CIC weights of
// the old/new positions and DS = S1 - S0 on a 4-node frame (cell offsets -1..2
// around the old cell):
//     W1[j][i] = DSx[i] (S0y[j] + DSy[j]/2),  W2[j][i] = DSy[j] (S0x[i] + DSx[i]/2)
//     Jx(i+1/2, j) = -(q/dV)(dx/dt) sum_{i'<=i} W1[j][i'], Jy likewise along j.
// Jx[k] is stored at the node k of the cell edge's lower (left) end: the edge
// from node (i, j) to (i+1, j); Jy[k] at the edge from (i, j) to (i, j+1).
//
// Integer form (exact discrete continuity). A particle's old and new integer
// CIC charges R0, R1 use the charge deposit's rounding and remainder rule, W1 is
// rounded with row sums forced to 0 and column sums forced to those of R1 - R0,
// and W2 = (R1 - R0) - W1. Then (R1 - R0) + div J = 0 holds exactly in the
// int64 grids: the CIC charge of the pushed particles minus that of the old ones
// plus the integer divergence of J is zero at every node. J unit =
// max|q| inv_vol 2^-24 dx/dt (x), dy/dt (y). DS entries are formed from
// quantities of their own size (no S1 - S0 cancellation): no crossing
// DS = (0,-d,d,0); crossing up DS = (0, r-1, (1-r)-fr, fr); down DS = (-e, r+e, -r, 0).
//
// Kernels: cell-sorted particles, the lanes of a cell sum those that stay in it
// (current_cells) and the rest go through a list (current_listed); any order,
// the deposit's warp step (128 particles, 4 consecutive per lane via 128-bit
// loads), each lane summing its particles' 24 edge values while they share a
// cell (one rolled copy of the particle body), a segmented warp scan, and int64
// atomics from the run tails (deposit_current).
#include <cmath>

#include "cells.cuh"
#include "pic_internal.cuh"

namespace picgb {

constexpr int J_THREADS = 256;
constexpr int J_WARPS = J_THREADS / 32;
constexpr int NJ = 24;  // 12 Jx edges (rows j=0..3, i=0..2) + 12 Jy edges (j=0..2, i=0..3)
constexpr uint32_t J_NO_CELL = 0xffffffffu;

struct JArgs {
    const uint32_t* cell;
    const float *xr, *yr, *vx, *vy, *q;
    size_t n;
    int Nx, Ny;
    float dtdx, dtdy;
    float qc;  // nonzero: every particle's stored charge (the charge stream is not read)
    unsigned long long *jx, *jy;
    DevStats* st;
};

__device__ __forceinline__ void esk_ds(float r, float d, float (&s0)[4], float (&ds)[4]) {
    const float e = r + d;
    const float f = floorf(e);
    const float fr = e - f;
    s0[0] = 0.0f;
    s0[1] = 1.0f - r;
    s0[2] = r;
    s0[3] = 0.0f;
    if (f == 0.0f) {
        ds[0] = 0.0f;
        ds[1] = -d;
        ds[2] = d;
        ds[3] = 0.0f;
    } else if (f > 0.0f) {
        ds[0] = 0.0f;
        ds[1] = r - 1.0f;
        ds[2] = (1.0f - r) - fr;
        ds[3] = fr;
    } else {
        ds[0] = -e;
        ds[1] = r + e;
        ds[2] = -r;
        ds[3] = 0.0f;
    }
}

// The particle's integer CIC charges (a 2x2 block at frame offset (kx, ky)),
// exactly as the charge deposit rounds them.
__device__ __forceinline__ void cic_int(float a, int A, float rx, float ry, int (&v)[4]) {
    const float X0 = 1.0f - rx, X1 = rx, Y0 = 1.0f - ry, Y1 = ry;
    const float a0 = a * Y0, a1 = a * Y1;
    v[0] = __float2int_rn(a0 * X0);
    v[1] = __float2int_rn(a0 * X1);
    v[2] = __float2int_rn(a1 * X0);
    v[3] = __float2int_rn(a1 * X1);
    const int mx = X1 > X0 ? 1 : 0, my = Y1 > Y0 ? 1 : 0;
    const int rem = A - (v[0] + v[1] + v[2] + v[3]);
    const int km = my * 2 + mx;
#pragma unroll
    for (int k = 0; k < 4; ++k) v[k] += (k == km) ? rem : 0;
}

// 24 integer edge values of one particle (see the file header). Returns false
// (and flags PIC_ERR_COURANT) when the move is a cell or more.
__device__ __forceinline__ bool edge_values(const JArgs& a, float rx, float ry, float vxx, float vyy, float qn,
                                            size_t p, int (&out)[NJ]) {
    const float ddx = vxx * a.dtdx, ddy = vyy * a.dtdy;
    if (!(fabsf(ddx) < 1.0f && fabsf(ddy) < 1.0f)) {
        set_dev_error(a.st, DEV_COURANT, (unsigned)p);
        return false;
    }
    float s0x[4], dsx[4], s0y[4], dsy[4];
    esk_ds(rx, ddx, s0x, dsx);
    esk_ds(ry, ddy, s0y, dsy);
    const float aq = qn * 16777216.0f;
    const int A = __float2int_rn(aq);
    int r0[4], r1[4];
    cic_int(aq, A, rx, ry, r0);
    const float ex = rx + ddx, ey = ry + ddy;
    const float fx = floorf(ex), fy = floorf(ey);
    cic_int(aq, A, ex - fx, ey - fy, r1);
    const int kx = (int)fx + 1, ky = (int)fy + 1;
    // dR = R1 - R0 on the 4x4 frame; R0 sits at offset (1, 1)
    int dR[16];
#pragma unroll
    for (int k = 0; k < 16; ++k) dR[k] = 0;
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int i = 0; i < 2; ++i) dR[(1 + j) * 4 + (1 + i)] -= r0[j * 2 + i];
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int jj = j - ky, ii = i - kx;
            const bool in = jj >= 0 && jj < 2 && ii >= 0 && ii < 2;
            dR[j * 4 + i] += in ? r1[(jj & 1) * 2 + (ii & 1)] : 0;
        }
    int W1[16];
#pragma unroll
    for (int j = 0; j < 3; ++j) {
        const float ay = aq * (s0y[j] + 0.5f * dsy[j]);
        int row = 0;
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            W1[j * 4 + i] = __float2int_rn(ay * dsx[i]);
            row += W1[j * 4 + i];
        }
        W1[j * 4 + 3] = -row;
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        int col = 0, colR = 0;
#pragma unroll
        for (int j = 0; j < 3; ++j) col += W1[j * 4 + i];
#pragma unroll
        for (int j = 0; j < 4; ++j) colR += dR[j * 4 + i];
        W1[12 + i] = colR - col;
    }
    // Jx edges: out[j*3 + i] = -sum_{i'<=i} W1[j][i'], i = 0..2
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        int cum = 0;
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            cum += W1[j * 4 + i];
            out[j * 3 + i] = -cum;
        }
    }
    // Jy edges: out[12 + j*4 + i] = -sum_{j'<=j} (dR - W1)[j'][i], j = 0..2
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        int cum = 0;
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            cum += dR[j * 4 + i] - W1[j * 4 + i];
            out[12 + j * 4 + i] = -cum;
        }
    }
    return true;
}

__device__ __forceinline__ void flush_edges(const JArgs& a, uint32_t key, const int (&acc)[NJ]) {
    const int iy = (int)(key / (uint32_t)a.Nx), ix = (int)(key - (uint32_t)iy * (uint32_t)a.Nx);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const size_t row = (size_t)wrap_i(iy - 1 + j, a.Ny) * a.Nx;
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            const int v = acc[j * 3 + i];
            if (v) atomicAdd(a.jx + row + wrap_i(ix - 1 + i, a.Nx), (unsigned long long)(long long)v);
        }
    }
#pragma unroll
    for (int j = 0; j < 3; ++j) {
        const size_t row = (size_t)wrap_i(iy - 1 + j, a.Ny) * a.Nx;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int v = acc[12 + j * 4 + i];
            if (v) atomicAdd(a.jy + row + wrap_i(ix - 1 + i, a.Nx), (unsigned long long)(long long)v);
        }
    }
}

__device__ __forceinline__ float f4(const float4& v, int k) { return k == 0 ? v.x : k == 1 ? v.y : k == 2 ? v.z : v.w; }
__device__ __forceinline__ uint32_t u4(const uint4& v, int k) { return k == 0 ? v.x : k == 1 ? v.y : k == 2 ? v.z : v.w; }

__global__ void __launch_bounds__(J_THREADS) deposit_current(JArgs a) {
    const int lane = threadIdx.x & 31;
    const size_t gw = (size_t)blockIdx.x * J_WARPS + (threadIdx.x >> 5);
    const size_t stride = (size_t)gridDim.x * J_WARPS * 128;
    const uint32_t G = (uint32_t)a.Nx * (uint32_t)a.Ny;
    const unsigned upto = (lane == 31) ? 0xffffffffu : ((2u << lane) - 1u);
    for (size_t base = gw * 128; base < a.n; base += stride) {
        const size_t p0 = base + 4u * lane;
        uint4 cell = make_uint4(0, 0, 0, 0);
        float4 xr = make_float4(0, 0, 0, 0), yr = xr, vx = xr, vy = xr, q = xr;
        if (p0 < a.n) {
            cell = __ldcs(reinterpret_cast<const uint4*>(a.cell + p0));
            xr = __ldcs(reinterpret_cast<const float4*>(a.xr + p0));
            yr = __ldcs(reinterpret_cast<const float4*>(a.yr + p0));
            vx = __ldcs(reinterpret_cast<const float4*>(a.vx + p0));
            vy = __ldcs(reinterpret_cast<const float4*>(a.vy + p0));
            q = a.qc != 0.0f ? make_float4(a.qc, a.qc, a.qc, a.qc) : __ldcs(reinterpret_cast<const float4*>(a.q + p0));
        }
        uint32_t ckey = J_NO_CELL;
        int acc[NJ];
#pragma unroll
        for (int k = 0; k < NJ; ++k) acc[k] = 0;
        // rolled loops (one copy of the particle body and of the scan step): the
        // unrolled kernel thrashed the instruction cache (ncu: 18 cycles per issue
        // waiting for instructions; rolled, 2.1x faster)
#pragma unroll 1
        for (int k = 0; k < 4; ++k) {
            const size_t p = p0 + (size_t)k;
            if (p >= a.n) continue;
            const uint32_t key = u4(cell, k);
            if (key >= G) {
                set_dev_error(a.st, DEV_BAD_CELL, (unsigned)p);
                continue;
            }
            int v[NJ];
            if (!edge_values(a, f4(xr, k), f4(yr, k), f4(vx, k), f4(vy, k), f4(q, k), p, v)) continue;
            if (key != ckey) {
                if (ckey != J_NO_CELL) flush_edges(a, ckey, acc);
                ckey = key;
#pragma unroll
                for (int t = 0; t < NJ; ++t) acc[t] = v[t];
            } else {
#pragma unroll
                for (int t = 0; t < NJ; ++t) acc[t] += v[t];
            }
        }
        const uint32_t kprev = __shfl_up_sync(0xffffffffu, ckey, 1);
        // segments stop at lane 16: a run total covers <= 64 particles and fits int32
        const unsigned H = __ballot_sync(0xffffffffu, lane == 0 || lane == 16 || ckey != kprev);
        const int segstart = 31 - __clz(H & upto);
#pragma unroll 1
        for (int d = 1; d < 32; d <<= 1) {
            const bool take = lane - d >= segstart;
#pragma unroll
            for (int t = 0; t < NJ; ++t) {
                const int o = __shfl_up_sync(0xffffffffu, acc[t], d);
                if (take) acc[t] += o;
            }
        }
        const bool tail = (lane == 31) || ((H >> (lane + 1)) & 1u);
        if (tail && ckey != J_NO_CELL) flush_edges(a, ckey, acc);
    }
}

// Cell-sorted particles. A CTA owns a tile of 32 x tile_h cells (8 rows, fewer on grids
// that would not fill the SMs); its warps walk units of
// consecutive cells of a row, K lanes per cell, with the stream staged in shared
// memory (cells.cuh).
//  * A particle that stays in its cell (0 <= r + d < 1 on both axes) has
//    DS = (0, -d, d, 0) and its old and new charges on the same 2x2 nodes: of its
//    24 edge values seven are not zero, and they follow from five numbers that
//    add up over the cell's particles: W1[1][1], W1[2][1] and the changes of the
//    row 0, column 0 and diagonal sums of its integer charges. These are summed
//    in 32-bit registers (at most 64 particles per sum: |sum| <= 64 * 2^24).
//  * The others are listed (ballot compaction into a queue per warp, appended 32
//    at a time) for a second kernel, current_listed: 24 edge values in full, one particle per lane,
//    int64 atomics. Evaluating them in this kernel (queued, 32 at a time) cost it
//    half of its resident warps in registers.
// The sums go to the tile's Jx and Jy accumulators in shared memory (low 15 bits
// and the rest in two 32-bit words, a halo of one node left and below and two right
// and above), and the tile to the int64 grids once; tiles so full that the words
// could overflow add straight to the grids. Integer sums, so the grids equal those
// of deposit_current bit for bit.
// Bound by the staying particle's arithmetic (two rounded CIC charges and two
// edge values). Where many particles leave their cell the list's atomics cost more than
// evaluating every particle in full: current_begin looks at a sample, and current_full
// takes the particles instead.
constexpr int JC_TW = 32, JC_TH = 8, JC_WARPS = 4;
constexpr int JC_SW = JC_TW + 3, JC_SH = JC_TH + 3, JC_N = JC_SW * JC_SH;
constexpr int JC_RUN = 64;
constexpr int JC_FULL_CTAS = 10;  // current_full's CTAs per SM: two rounds of those that fit
constexpr int JC_SPLIT = 15;
constexpr unsigned JC_BATCH = 32;  // particles appended to the list at a time (one atomic on its length)
// A low word holds 2^17 additions; a run of at most JC_RUN particles of one lane
// adds to a node once, 32 lanes may share a cell, and five cells reach a node.
constexpr uint32_t JC_RUN_MAX = 1u << 17;  // particles of a tile whose runs use the tile's accumulators

// The particle stays in its cell. 0 <= e < 1 on both axes: the bits of non-negative
// floats are in their order.
__device__ __forceinline__ bool j_stays(float rx, float ry, float dx, float dy) {
    const float ex = rx + dx, ey = ry + dy;
    return fmaxf(fabsf(dx), fabsf(dy)) < 1.0f && max(__float_as_uint(ex), __float_as_uint(ey)) < 0x3F800000u;
}

// Zeroes the grids and the list, and chooses the kernel from a sample of the particles:
// current_full when at least `many` of them leave their cell in the move.
constexpr int J_SAMPLES = 4;  // per thread of the first block
__global__ void __launch_bounds__(J_THREADS) current_begin(JArgs a, size_t g, float many, unsigned* __restrict__ count) {
    if (blockIdx.x == 0) {
        const size_t step = a.n / (J_SAMPLES * J_THREADS) ? a.n / (J_SAMPLES * J_THREADS) : 1;
        float x[J_SAMPLES], y[J_SAMPLES], u[J_SAMPLES], w[J_SAMPLES];
        bool in[J_SAMPLES];
#pragma unroll
        for (int k = 0; k < J_SAMPLES; ++k) {
            const size_t p = (size_t)(k * J_THREADS + threadIdx.x) * step;
            in[k] = p < a.n;
            x[k] = y[k] = u[k] = w[k] = 0.0f;
            if (in[k]) {
                x[k] = a.xr[p];
                y[k] = a.yr[p];
                u[k] = a.vx[p];
                w[k] = a.vy[p];
            }
        }
        int leave = 0, all = 0;
#pragma unroll
        for (int k = 0; k < J_SAMPLES; ++k) {
            leave += __syncthreads_count(in[k] && !j_stays(x[k], y[k], u[k] * a.dtdx, w[k] * a.dtdy));
            all += __syncthreads_count(in[k]);
        }
        if (threadIdx.x == 0) {
            a.st->j_full = (float)leave >= many * (float)all ? 1u : 0u;
            *count = 0;
        }
    }
    for (size_t i = (size_t)blockIdx.x * J_THREADS + threadIdx.x; i < g; i += (size_t)gridDim.x * J_THREADS)
        a.jx[i] = a.jy[i] = 0ull;
}

// The listed particles with their values (the sort's spare arrays): reading them
// back from the particle arrays took a 64-byte DRAM access per value.
struct JList {
    unsigned* count;
    uint32_t *p, *cell;
    float *xr, *yr, *vx, *vy;
};

// All 24 edge values of the listed particles (also the Courant check).
__global__ void __launch_bounds__(J_THREADS) current_listed(JArgs a, JList l) {
    const unsigned n = *l.count;
    for (unsigned i = blockIdx.x * J_THREADS + threadIdx.x; i < n; i += gridDim.x * J_THREADS) {
        const uint32_t p = l.p[i];
        int v[NJ];
        if (edge_values(a, l.xr[i], l.yr[i], l.vx[i], l.vy[i], a.qc != 0.0f ? a.qc : a.q[p], p, v))
            flush_edges(a, l.cell[i], v);
    }
}

constexpr uint32_t JC_FULL_MAX = 1u << 21;  // particles of a tile whose sums use its accumulators in current_full

// A tile's accumulators to the grids.
__device__ __forceinline__ void tile_to_grids(const JArgs& a, const uint32_t* slo, const int* shi, int x0, int y0) {
    for (int i = threadIdx.x; i < 2 * JC_N; i += JC_WARPS * 32) {
        const long long v = (long long)shi[i] * (1ll << JC_SPLIT) + (long long)slo[i];
        if (v != 0) {
            const int li = i < JC_N ? i : i - JC_N;
            const int ly = li / JC_SW, lx = li - ly * JC_SW;
            const size_t g = (size_t)wrap_i(y0 - 1 + ly, a.Ny) * a.Nx + wrap_i(x0 - 1 + lx, a.Nx);
            atomicAdd((i < JC_N ? a.jx : a.jy) + g, (unsigned long long)v);
        }
    }
}

// All 24 edge values of every particle: one lane per cell of a tile row walks the cell's
// range (16-byte loads of 4 particles) and sums them in registers (at most 64 particles:
// |sum| <= 64 * 2^24), then adds the sums to the tile's accumulators, or to the grids in a
// tile whose high words could overflow (2^16 sums of 2^15 each). Takes the same time
// whatever the particles do. The CTAs walk the tiles: a launch that is not wanted costs
// little.
template <bool QC>
__global__ void __launch_bounds__(JC_WARPS * 32) current_full(JArgs a, const uint32_t* __restrict__ offsets, int tiles_x,
                                                               int tiles, int tile_h) {
    if (!a.st->j_full) return;
    __shared__ uint32_t slo[2 * JC_N];
    __shared__ int shi[2 * JC_N];
    __shared__ uint32_t s_count;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        const int tx = tile % tiles_x, ty = tile / tiles_x;
        const int x0 = tx * JC_TW, y0 = ty * tile_h;
        const int tw = min(JC_TW, a.Nx - x0), th = min(tile_h, a.Ny - y0);
        for (int i = threadIdx.x; i < 2 * JC_N; i += JC_WARPS * 32) {
            slo[i] = 0;
            shi[i] = 0;
        }
        if (threadIdx.x == 0) s_count = 0;
        __syncthreads();
        if ((int)threadIdx.x < th) {
            const uint32_t* row = offsets + (uint32_t)(y0 + (int)threadIdx.x) * (uint32_t)a.Nx + (uint32_t)x0;
            atomicAdd(&s_count, row[tw] - row[0]);
        }
        __syncthreads();
        const bool to_grids = s_count >= JC_FULL_MAX;
        int acc[NJ];
        // adds acc (the cell in column `lane`, tile row r) to the tile accumulators
        auto flush = [&](int r) {
            if (to_grids) {
                flush_edges(a, (uint32_t)(y0 + r) * (uint32_t)a.Nx + (uint32_t)(x0 + lane), acc);
#pragma unroll
                for (int t = 0; t < NJ; ++t) acc[t] = 0;
                return;
            }
#pragma unroll
            for (int t = 0; t < NJ; ++t) {
                const int v = acc[t];
                if (v != 0) {
                    // Jx edge (j, i) = t (j * 3 + i), Jy edge (j, i) = t - 12 (j * 4 + i): local node (lane + i, r + j)
                    const int j = t < 12 ? t / 3 : (t - 12) / 4, i = t < 12 ? t % 3 : (t - 12) % 4;
                    const int idx = (t < 12 ? 0 : JC_N) + (r + j) * JC_SW + lane + i;
                    atomicAdd(slo + idx, (uint32_t)v & ((1u << JC_SPLIT) - 1u));
                    atomicAdd(shi + idx, v >> JC_SPLIT);
                }
                acc[t] = 0;
            }
        };
        for (int r = warp; r < th; r += JC_WARPS) {
            uint32_t beg = 0, end = 0;
            if (lane < tw) {
                const uint32_t cell = (uint32_t)(y0 + r) * (uint32_t)a.Nx + (uint32_t)(x0 + lane);
                beg = offsets[cell];
                end = offsets[cell + 1];
            }
#pragma unroll
            for (int t = 0; t < NJ; ++t) acc[t] = 0;
            int cnt = 0;
            const uint32_t q0 = beg >> 2, q1 = end > beg ? (end + 3u) >> 2 : q0;
#pragma unroll 1
            for (uint32_t qd = q0; qd < q1; ++qd) {
                const float4 xr = __ldg(reinterpret_cast<const float4*>(a.xr) + qd);
                const float4 yr = __ldg(reinterpret_cast<const float4*>(a.yr) + qd);
                const float4 vx = __ldg(reinterpret_cast<const float4*>(a.vx) + qd);
                const float4 vy = __ldg(reinterpret_cast<const float4*>(a.vy) + qd);
                const float4 q = QC ? make_float4(a.qc, a.qc, a.qc, a.qc) : __ldg(reinterpret_cast<const float4*>(a.q) + qd);
#pragma unroll 1
                for (int k = 0; k < 4; ++k) {
                    const uint32_t p = 4u * qd + (uint32_t)k;
                    if (p < beg || p >= end) continue;
                    int v[NJ];
                    if (edge_values(a, f4(xr, k), f4(yr, k), f4(vx, k), f4(vy, k), f4(q, k), p, v)) {
#pragma unroll
                        for (int t = 0; t < NJ; ++t) acc[t] += v[t];
                    }
                    if (++cnt == JC_RUN) {
                        flush(r);
                        cnt = 0;
                    }
                }
            }
            if (cnt) flush(r);
        }
        __syncthreads();
        tile_to_grids(a, slo, shi, x0, y0);
        __syncthreads();
    }
}

template <bool QC>
__global__ void __launch_bounds__(JC_WARPS * 32, 5) current_cells(JArgs a, const uint32_t* __restrict__ offsets,
                                                                   int tiles_x, int tile_h, int klog, int cap, JList list) {
    if (a.st->j_full) return;
    constexpr int NF = QC ? 4 : 5;
    extern __shared__ __align__(16) uint32_t sbufs[];  // [JC_WARPS][NF][cap]
    __shared__ uint32_t soff[JC_TH * (JC_TW + 1)];
    __shared__ uint32_t slo[2 * JC_N];
    __shared__ int shi[2 * JC_N];
    __shared__ uint32_t s_count;
    __shared__ uint2 squeue[JC_WARPS][JC_BATCH + 32];   // particle, cell
    __shared__ float4 sqval[JC_WARPS][JC_BATCH + 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int tx = blockIdx.x % tiles_x, ty = blockIdx.x / tiles_x;
    const int x0 = tx * JC_TW, y0 = ty * tile_h;
    const int tw = min(JC_TW, a.Nx - x0), th = min(tile_h, a.Ny - y0);
    if (threadIdx.x == 0) s_count = 0;
    for (int i = threadIdx.x; i < 2 * JC_N; i += JC_WARPS * 32) {
        slo[i] = 0;
        shi[i] = 0;
    }
    for (int i = threadIdx.x; i < th * (tw + 1); i += JC_WARPS * 32) {
        const int r = i / (tw + 1);
        soff[i] = offsets[(uint32_t)(y0 + r) * (uint32_t)a.Nx + (uint32_t)x0 + (uint32_t)(i - r * (tw + 1))];
    }
    __syncthreads();
    if (threadIdx.x < th) atomicAdd(&s_count, soff[threadIdx.x * (tw + 1) + tw] - soff[threadIdx.x * (tw + 1)]);
    __syncthreads();
    const bool run_to_grid = s_count >= JC_RUN_MAX;
    uint2* queue = squeue[warp];
    float4* qval = sqval[warp];
    unsigned qn = 0;
    auto append = [&](unsigned m) {  // the first m queued particles to the list
        unsigned at = 0;
        if (lane == 0) at = atomicAdd(list.count, m);
        at = __shfl_sync(0xffffffffu, at, 0);
        for (unsigned i = (unsigned)lane; i < m; i += 32) {
            const uint2 id = queue[i];
            const float4 v = qval[i];
            list.p[at + i] = id.x;
            list.cell[at + i] = id.y;
            list.xr[at + i] = v.x;
            list.yr[at + i] = v.y;
            list.vx[at + i] = v.z;
            list.vy[at + i] = v.w;
        }
    };
    // one charge: values of +2^24 units, mirrored for a negative charge
    const int sgn = QC && a.qc < 0.0f ? -1 : 1;
    uint32_t* sbuf = sbufs + (size_t)warp * NF * cap;
    CellWalk<NF, JC_WARPS> walk;
    walk.init(tw, th, klog, cap);
    walk.soff = soff;
    walk.buf_addr = (uint32_t)__cvta_generic_to_shared(sbuf);
    walk.field[0] = reinterpret_cast<const uint32_t*>(a.xr);
    walk.field[1] = reinterpret_cast<const uint32_t*>(a.yr);
    walk.field[2] = reinterpret_cast<const uint32_t*>(a.vx);
    walk.field[3] = reinterpret_cast<const uint32_t*>(a.vy);
    if constexpr (!QC) walk.field[4] = reinterpret_cast<const uint32_t*>(a.q);
    CellPiece cw;
    for (walk.start(cw, warp); !walk.done(cw); walk.advance(cw)) {
        walk.stage(cw, lane);
        const float* sb = reinterpret_cast<const float*>(sbuf);
        const int r = cw.r, col = cw.c0 + (lane >> cw.klog);
        int m, first;
        uint32_t ncell;
        walk.share(cw, lane, first, m, ncell);
        // cells small enough that 32-bit sums hold all their lanes' particles
        const bool small = __all_sync(0xffffffffu, ncell <= 127u);
        // W1[1][1], W1[2][1]; changes of row 0, column 0 and the diagonal of the charges
        int e1 = 0, e2 = 0, drow = 0, dcol = 0, ddia = 0, cnt = 0;
        // value k of the cell's seven (edges below) to the tile, or to the grids
        auto add = [&](int k, long long x) {
            if (x == 0) return;
            // edges: Jx (1,1), (2,1), (3,1); Jy (1,1), (2,1), (1,2), (2,2), as (row j, column i)
            const int j = k == 0 || k == 3 || k == 5 ? 1 : k == 2 ? 3 : 2;
            const int i = k < 5 ? 1 : 2;
            if (!run_to_grid) {
                const int idx = (k < 3 ? 0 : JC_N) + (r + j) * JC_SW + col + i;
                atomicAdd(slo + idx, (uint32_t)x & ((1u << JC_SPLIT) - 1u));
                atomicAdd(shi + idx, (int)(x >> JC_SPLIT));
            } else {
                const size_t g = (size_t)wrap_i(y0 + r - 1 + j, a.Ny) * a.Nx + wrap_i(x0 + col - 1 + i, a.Nx);
                atomicAdd((k < 3 ? a.jx : a.jy) + g, (unsigned long long)x);
            }
        };
        auto flush = [&](int from, int step) {
            // change of node (0,0): exact, as the total does not change
            const long long d00 = ((long long)drow + dcol + ddia) / 2;
            const long long w = (long long)dcol - e1 - e2;  // W1[3][1] = -W1[3][2]
            const long long d01 = drow - d00;               // change of node (0,1)
            for (int k = from; k < 7; k += step) {
                const long long x = k == 0 ? -e1 : k == 1 ? -e2 : k == 2 || k == 4 ? -w : k == 3 ? e1 - d00 : k == 5 ? -(d01 + e1) : w;
                add(k, QC ? sgn * x : x);
            }
            e1 = e2 = drow = dcol = ddia = cnt = 0;
        };
        // warp-uniform trips of two particles per lane, cyclically from a pair that
        // differs from cell to cell (bank conflicts, as in deposit_cells)
        constexpr int UN = 2;
        const int ng = (m + UN - 1) / UN;
        const int trips = __reduce_max_sync(0xffffffffu, ng);
        int g = (lane >> cw.klog) < ng ? lane >> cw.klog : 0;
#pragma unroll 1
        for (int t = 0; t < trips; ++t) {
            const int left = t < ng ? m - g * UN : 0;
            const int i0 = first + g * UN;
            g = g + 1 >= ng ? 0 : g + 1;
#pragma unroll
            for (int k = 0; k < UN; ++k) {
                const bool valid = k < left;
                float rx = 0.0f, ry = 0.0f, vx = 0.0f, vy = 0.0f;
                if (valid) {
                    rx = sb[i0 + k];
                    ry = sb[cap + i0 + k];
                    vx = sb[2 * cap + i0 + k];
                    vy = sb[3 * cap + i0 + k];
                }
                const float dx = vx * a.dtdx, dy = vy * a.dtdy;
                const float ex = rx + dx, ey = ry + dy;
                const bool stays = j_stays(rx, ry, dx, dy);
                const unsigned out = __ballot_sync(0xffffffffu, valid && !stays);
                if (out) {
                    if (valid && !stays) {
                        const unsigned at = qn + __popc(out & ((1u << lane) - 1u));
                        queue[at] = make_uint2(cw.pos + (uint32_t)(i0 + k),
                                               (uint32_t)(y0 + r) * (uint32_t)a.Nx + (uint32_t)(x0 + col));
                        qval[at] = make_float4(rx, ry, vx, vy);
                    }
                    qn += __popc(out);
                    __syncwarp();
                    if (qn >= JC_BATCH) {
                        append(JC_BATCH);
                        const uint2 rest = queue[JC_BATCH + lane];
                        const float4 rval = qval[JC_BATCH + lane];
                        qn -= JC_BATCH;
                        __syncwarp();
                        if ((unsigned)lane < qn) {
                            queue[lane] = rest;
                            qval[lane] = rval;
                        }
                        __syncwarp();
                    }
                }
                if (valid && stays) {
                    if constexpr (QC) {
                        int r0, c0, g0, r1, c1, g1;
                        cic_unit(rx, ry, r0, c0, g0);
                        cic_unit(ex, ey, r1, c1, g1);
                        drow += r1 - r0;
                        dcol += c1 - c0;
                        ddia += g1 - g0;
                        e1 += __float2int_rn((16777216.0f * ((1.0f - ry) - 0.5f * dy)) * -dx);
                        e2 += __float2int_rn((16777216.0f * (ry + 0.5f * dy)) * -dx);
                    } else {
                        const float aq = sb[4 * cap + i0 + k] * 16777216.0f;
                        const int A = __float2int_rn(aq);
                        int v0[4], v1[4];
                        cic_int(aq, A, rx, ry, v0);
                        cic_int(aq, A, ex, ey, v1);
                        ddia += v1[0] + v1[3] - v0[0] - v0[3];
                        drow += v1[0] + v1[1] - v0[0] - v0[1];
                        dcol += v1[0] + v1[2] - v0[0] - v0[2];
                        e1 += __float2int_rn((aq * ((1.0f - ry) - 0.5f * dy)) * -dx);
                        e2 += __float2int_rn((aq * (ry + 0.5f * dy)) * -dx);
                    }
                    if (++cnt == JC_RUN && !small) flush(0, 1);
                }
            }
        }
        if (small) {
            // the cell's sums over its K lanes, which share the seven values
            const int K = 1 << cw.klog;
            for (int o = 1; o < K; o <<= 1) {
                e1 += __shfl_xor_sync(0xffffffffu, e1, o);
                e2 += __shfl_xor_sync(0xffffffffu, e2, o);
                drow += __shfl_xor_sync(0xffffffffu, drow, o);
                dcol += __shfl_xor_sync(0xffffffffu, dcol, o);
                ddia += __shfl_xor_sync(0xffffffffu, ddia, o);
                cnt += __shfl_xor_sync(0xffffffffu, cnt, o);
            }
            if (cnt) flush(lane & (K - 1), K);
        } else if (cnt) {
            flush(0, 1);
        }
        __syncwarp();
    }
    if (qn) append(qn);
    __syncthreads();
    tile_to_grids(a, slo, shi, x0, y0);
}

// The grids as FP64, four cells per thread: each block's first thread forms the units (FP64
// multiplications are slow on this part), the first block's also stores them.
__global__ void __launch_bounds__(256) current_to_f64(const long long* __restrict__ jx, const long long* __restrict__ jy,
                                                      size_t g, double inv_vol, double dxdt, double dydt,
                                                      const DevStats* st, double* __restrict__ units,
                                                      double* __restrict__ ox, double* __restrict__ oy) {
    const size_t i0 = (size_t)blockIdx.x * 1024 + threadIdx.x;
    __shared__ double s_units[2];
    if (threadIdx.x == 0) {
        const double u = charge_unit(st, inv_vol);
        s_units[0] = __dmul_rn(u, dxdt);
        s_units[1] = __dmul_rn(u, dydt);
        if (i0 == 0) {
            units[0] = s_units[0];
            units[1] = s_units[1];
        }
    }
    __syncthreads();
    const double ux = s_units[0], uy = s_units[1];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const size_t i = i0 + k * 256;
        if (i < g) {
            ox[i] = __dmul_rn((double)jx[i], ux);
            oy[i] = __dmul_rn((double)jy[i], uy);
        }
    }
}

static int ensure_current(pic_ctx* c) {
    int rc = PIC_OK;
    if (!c->accjx) c->accjx = (long long*)dalloc(c->G * 8, &rc);
    if (rc) return rc;
    if (!c->accjy) c->accjy = (long long*)dalloc(c->G * 8, &rc);
    if (rc) return rc;
    if (!c->jx) c->jx = (double*)dalloc(c->G * 8, &rc);
    if (rc) return rc;
    if (!c->jy) c->jy = (double*)dalloc(c->G * 8, &rc);
    if (rc) return rc;
    if (!c->junits) c->junits = (double*)dalloc(3 * 8, &rc);  // units, and the list's length
    return rc;
}

int deposit_current_async(pic_ctx* c, double dt) {
    if (!(dt > 0.0)) return fail(PIC_ERR_ARG, "deposit_current: dt must be > 0");
    PIC_TRY(ensure_current(c));
    JArgs a;
    a.cell = c->cell;
    a.xr = c->xr;
    a.yr = c->yr;
    a.vx = c->vx;
    a.vy = c->vy;
    a.q = c->q;
    a.n = c->n;
    a.Nx = c->Nx;
    a.Ny = c->Ny;
    a.dtdx = (float)(dt / c->dx);
    a.dtdy = (float)(dt / c->dy);
    a.qc = c->qn_uniform;
    a.jx = reinterpret_cast<unsigned long long*>(c->accjx);
    a.jy = reinterpret_cast<unsigned long long*>(c->accjy);
    a.st = c->dstats;
    int sms = 148;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, c->device);
    // Sets of less than a particle per two cells take the any-order kernel also when sorted:
    // a walk of empty cells costs more (2048^2, 0.01 per cell: 68 us against 190, 150 with one
    // lane per cell; 0.5: 207 to 297 against 293 to 366; 1.0: 348 to 518 against 316 to 496).
    if (c->sorted && 2 * c->n >= c->G && c->n) {
        const bool qc = a.qc != 0.0f;
        const int tiles_x = (c->Nx + JC_TW - 1) / JC_TW;
        // at least two tiles for every SM where the rows allow: a warp takes its units one
        // after the other (33 x 9: 48 us with tiles of 8 rows)
        int th = JC_TH;
        while (th > 1 && (long long)tiles_x * ((c->Ny + th - 1) / th) < 2 * sms) th /= 2;
        const unsigned tiles = (unsigned)(tiles_x * ((c->Ny + th - 1) / th));
        int klog, cap;
        cells_shape(c->n, c->G, qc ? 4 : 5, 1560, (size_t)tiles * JC_WARPS, &klog, &cap);
        PIC_TRY(ensure_sort_scratch(c));  // the list takes the sort's spare arrays
        unsigned* count = reinterpret_cast<unsigned*>(c->junits + 2);
        const JList list{count, c->idx_b, c->cell_alt, c->alt[0], c->alt[1], c->alt[2], c->alt[3]};
        const size_t smem = (size_t)JC_WARPS * (qc ? 4 : 5) * cap * 4;
        PIC_TRY(opt_in_dynamic_smem(qc ? (const void*)current_cells<true> : (const void*)current_cells<false>, smem));
        // current_full where each scheduler gets a warp of 32 cells (on smaller grids its
        // serial cells lose at any fraction: 64^2 x 64, 0.62 leaving: 107 us against 49) and
        // enough particles leave their cell; denser cells list more of them. Where the two
        // take the same time: above 0.63 leaving at 1 per cell, 0.38 at 4, 0.27 at 16, 0.2 at
        // 64 and 0.12 at 200 (512^2 and 1024^2). 1024^2 x 64, 0.62 leaving: 1.36 ms, 3.5 with
        // the list.
        const bool may_full = c->G >= (size_t)32 * 4 * sms;
        const float many = may_full ? (float)(0.1 + 0.58 / std::sqrt((double)c->n / (double)c->G)) : 2.0f;
        size_t zero = (c->G + J_THREADS * 4 - 1) / (J_THREADS * 4);
        if (zero > (size_t)sms * 8) zero = (size_t)sms * 8;
        current_begin<<<(unsigned)zero, J_THREADS, 0, c->stream>>>(a, c->G, many, count);
        PIC_TRY(check_launch(c, "current_begin"));
        prof_begin(c, "current");
        if (qc)
            current_cells<true><<<tiles, JC_WARPS * 32, smem, c->stream>>>(a, c->offsets, tiles_x, th, klog, cap, list);
        else
            current_cells<false><<<tiles, JC_WARPS * 32, smem, c->stream>>>(a, c->offsets, tiles_x, th, klog, cap, list);
        PIC_TRY(check_launch(c, "current_cells"));
        size_t blocks = (c->n + J_THREADS - 1) / J_THREADS;
        if (blocks > (size_t)sms * 4) blocks = (size_t)sms * 4;
        current_listed<<<(unsigned)blocks, J_THREADS, 0, c->stream>>>(a, list);
        PIC_TRY(check_launch(c, "current_listed"));
        if (may_full) {
            const int fh = th < JC_WARPS ? JC_WARPS : th;  // a row for every warp
            const int ftiles = tiles_x * ((c->Ny + fh - 1) / fh);
            const unsigned ctas = (unsigned)(ftiles < sms * JC_FULL_CTAS ? ftiles : sms * JC_FULL_CTAS);
            if (qc)
                current_full<true><<<ctas, JC_WARPS * 32, 0, c->stream>>>(a, c->offsets, tiles_x, ftiles, fh);
            else
                current_full<false><<<ctas, JC_WARPS * 32, 0, c->stream>>>(a, c->offsets, tiles_x, ftiles, fh);
            PIC_TRY(check_launch(c, "current_full"));
        }
        prof_end(c);
    } else {
        PIC_CUDA_TRY(cudaMemsetAsync(c->accjx, 0, c->G * 8, c->stream));
        PIC_CUDA_TRY(cudaMemsetAsync(c->accjy, 0, c->G * 8, c->stream));
        if (c->n) {
            size_t blocks = (c->n + J_THREADS * 4 - 1) / (J_THREADS * 4);
            if (blocks > (size_t)sms * 8) blocks = (size_t)sms * 8;
            prof_begin(c, "current");
            deposit_current<<<(unsigned)blocks, J_THREADS, 0, c->stream>>>(a);
            prof_end(c);
            PIC_TRY(check_launch(c, "deposit_current"));
        }
    }
    current_to_f64<<<(unsigned)((c->G + 1023) / 1024), 256, 0, c->stream>>>(
        c->accjx, c->accjy, c->G, 1.0 / (c->dx * c->dy), c->dx / dt, c->dy / dt, c->dstats, c->junits, c->jx, c->jy);
    PIC_TRY(check_launch(c, "current_to_f64"));
    c->has_current = 1;
    return PIC_OK;
}

void release_current(pic_ctx* c) {
    void* ptrs[] = {c->accjx, c->accjy, c->jx, c->jy, c->junits};
    for (void* p : ptrs) dfree(p);
}

}  // namespace picgb

using namespace picgb;

extern "C" {

int pic_gpu_deposit_current(pic_ctx* c, double dt, double* jx_out, double* jy_out) {
    if (!c) return fail(PIC_ERR_ARG, "NULL context");
    PIC_CUDA_TRY(cudaSetDevice(c->device));
    PIC_TRY(deposit_current_async(c, dt));
    if (jx_out) PIC_CUDA_TRY(cudaMemcpyAsync(jx_out, c->jx, c->G * 8, cudaMemcpyDeviceToHost, c->stream));
    if (jy_out) PIC_CUDA_TRY(cudaMemcpyAsync(jy_out, c->jy, c->G * 8, cudaMemcpyDeviceToHost, c->stream));
    if (jx_out || jy_out) return pic_gpu_synchronize(c);
    return PIC_OK;
}

int pic_gpu_get_current_fixed(pic_ctx* c, int64_t* jx, int64_t* jy, double* unit_x, double* unit_y) {
    if (!c) return fail(PIC_ERR_ARG, "NULL context");
    if (!c->has_current) return fail(PIC_ERR_STATE, "no current deposit has run");
    if (jx) PIC_CUDA_TRY(cudaMemcpyAsync(jx, c->accjx, c->G * 8, cudaMemcpyDeviceToHost, c->stream));
    if (jy) PIC_CUDA_TRY(cudaMemcpyAsync(jy, c->accjy, c->G * 8, cudaMemcpyDeviceToHost, c->stream));
    double u[2];
    PIC_CUDA_TRY(cudaMemcpyAsync(u, c->junits, sizeof(u), cudaMemcpyDeviceToHost, c->stream));
    PIC_TRY(pic_gpu_synchronize(c));
    if (unit_x) *unit_x = u[0];
    if (unit_y) *unit_y = u[1];
    return PIC_OK;
}

}  // extern "C"
