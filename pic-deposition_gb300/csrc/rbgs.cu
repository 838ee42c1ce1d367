// Red-black Gauss-Seidel Poisson solve (FP64).
//
// PoissonSolverGS::solve (src/pic/poisson_gs.cpp:11-61) is lexicographic,
// zeroes phi on every call and stops on max|dphi| < 1e-6. This solver keeps its
// 5-point stencil and sign, phi = ((phiW+phiE)/dx^2 + (phiS+phiN)/dy^2 + rho*dV)
// / (2(1/dx^2+1/dy^2)) (poisson_gs.cpp:32-38), and changes what a data-parallel
// solve with a learned warm start needs: red-black ordering (all points with (i+j) even, then odd; each
// colour is one data-parallel kernel), the right-hand side rho*dV with its mean
// removed (the periodic problem is singular), a warm start from the phi already
// in the context (the previous step's, or a learned guess), and the stop
// ||b - A phi||_2 / ||b||_2 <= tol checked every `check_every` sweeps. On exit
// phi has its mean removed and E is the forward difference of phi
// (poisson_gs.cpp:48-60). Multiplications by 1/dx^2, 1/dy^2 and 1/denom
// replace the reference's divisions (FP64 division is slow on this part); the
// oracle's restatement uses the same order of operations.
//
// Sums (mean, residual norms) use a fixed two-level tree, so results are
// identical run to run. Odd Nx or Ny is rejected: the colouring would not be a
// valid red-black split across the periodic seam.
#include <cstring>

#include "pic_internal.cuh"

namespace picgb {

constexpr int RB_THREADS = 256;
constexpr int RB_RED_BLOCKS = 1024;

struct RbArgs {
    double* phi;
    const double* b;
    int Nx, Ny;
    double ix2, iy2, inv_denom, denom;
};

__global__ void rbgs_half(RbArgs a, int color) {
    const int hx = a.Nx >> 1;
    const size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (size_t)hx * a.Ny) return;
    const int j = (int)(t / hx);
    const int i = 2 * (int)(t - (size_t)j * hx) + ((j + color) & 1);
    const int im = i == 0 ? a.Nx - 1 : i - 1, ip = i == a.Nx - 1 ? 0 : i + 1;
    const int jm = j == 0 ? a.Ny - 1 : j - 1, jp = j == a.Ny - 1 ? 0 : j + 1;
    const size_t id = (size_t)j * a.Nx + i;
    const double we = __dadd_rn(a.phi[(size_t)j * a.Nx + im], a.phi[(size_t)j * a.Nx + ip]);
    const double sn = __dadd_rn(a.phi[(size_t)jm * a.Nx + i], a.phi[(size_t)jp * a.Nx + i]);
    a.phi[id] = __dmul_rn(__dadd_rn(__dadd_rn(__dmul_rn(we, a.ix2), __dmul_rn(sn, a.iy2)), a.b[id]), a.inv_denom);
}

__device__ __forceinline__ double rb_block_sum(double v) {
    __shared__ double ws[RB_THREADS / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = __dadd_rn(v, __shfl_down_sync(0xffffffffu, v, o));
    if (lane == 0) ws[warp] = v;
    __syncthreads();
    double s = 0.0;
    if (threadIdx.x == 0)
        for (int w = 0; w < RB_THREADS / 32; ++w) s = __dadd_rn(s, ws[w]);
    __syncthreads();
    return s;
}

// partial[blk] = sum of rho*vol over a fixed chunk
__global__ void rb_sum_rhs(const double* __restrict__ rho, double vol, size_t g, double* __restrict__ partial) {
    const size_t chunk = (g + RB_RED_BLOCKS - 1) / RB_RED_BLOCKS;
    const size_t b = (size_t)blockIdx.x * chunk, e = b + chunk < g ? b + chunk : g;
    double s = 0.0;
    for (size_t i = b + threadIdx.x; i < e; i += RB_THREADS) s = __dadd_rn(s, __dmul_rn(rho[i], vol));
    const double t = rb_block_sum(s);
    if (threadIdx.x == 0) partial[blockIdx.x] = t;
}

// partial[2*blk] = sum r^2, partial[2*blk+1] = sum b^2 with r = b - A phi
__global__ void rb_resid_partials(RbArgs a, double* __restrict__ partial) {
    const size_t g = (size_t)a.Nx * a.Ny;
    const size_t chunk = (g + RB_RED_BLOCKS - 1) / RB_RED_BLOCKS;
    const size_t b0 = (size_t)blockIdx.x * chunk, e = b0 + chunk < g ? b0 + chunk : g;
    double rr = 0.0, bb = 0.0;
    for (size_t id = b0 + threadIdx.x; id < e; id += RB_THREADS) {
        const int j = (int)(id / a.Nx), i = (int)(id - (size_t)j * a.Nx);
        const int im = i == 0 ? a.Nx - 1 : i - 1, ip = i == a.Nx - 1 ? 0 : i + 1;
        const int jm = j == 0 ? a.Ny - 1 : j - 1, jp = j == a.Ny - 1 ? 0 : j + 1;
        const double we = __dadd_rn(a.phi[(size_t)j * a.Nx + im], a.phi[(size_t)j * a.Nx + ip]);
        const double sn = __dadd_rn(a.phi[(size_t)jm * a.Nx + i], a.phi[(size_t)jp * a.Nx + i]);
        const double ap = __dsub_rn(__dsub_rn(__dmul_rn(a.denom, a.phi[id]), __dmul_rn(we, a.ix2)), __dmul_rn(sn, a.iy2));
        const double r = __dsub_rn(a.b[id], ap);
        rr = __dadd_rn(rr, __dmul_rn(r, r));
        bb = __dadd_rn(bb, __dmul_rn(a.b[id], a.b[id]));
    }
    const double t1 = rb_block_sum(rr);
    const double t2 = rb_block_sum(bb);
    if (threadIdx.x == 0) {
        partial[2 * blockIdx.x] = t1;
        partial[2 * blockIdx.x + 1] = t2;
    }
}

// out[0] = sum of partial[0..n) (stride `stride`, offset `off`)
__global__ void rb_final(const double* __restrict__ partial, int n, int stride, int off, double* out) {
    double s = 0.0;
    for (int i = threadIdx.x; i < n; i += RB_THREADS) s = __dadd_rn(s, partial[(size_t)i * stride + off]);
    const double t = rb_block_sum(s);
    if (threadIdx.x == 0) *out = t;
}

// b = rho*vol - mean, mean = sum / g
__global__ void rb_make_rhs(const double* __restrict__ rho, double vol, size_t g, const double* __restrict__ sum,
                            double* __restrict__ b) {
    const double mean = __ddiv_rn(*sum, (double)g);
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < g) b[i] = __dsub_rn(__dmul_rn(rho[i], vol), mean);
}

__global__ void rb_sub_mean(double* __restrict__ phi, size_t g, const double* __restrict__ sum) {
    const double mean = __ddiv_rn(*sum, (double)g);
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < g) phi[i] = __dsub_rn(phi[i], mean);
}

static int ensure_rbgs(pic_ctx* c) {
    PIC_TRY(ensure_fields(c));
    int rc = PIC_OK;
    if (!c->rb_b) c->rb_b = (double*)dalloc(c->G * 8, &rc);
    if (rc) return rc;
    if (!c->rb_partial) c->rb_partial = (double*)dalloc(2 * RB_RED_BLOCKS * 8, &rc);
    if (rc) return rc;
    if (!c->rb_scalars) c->rb_scalars = (double*)dalloc(8 * 8, &rc);
    return rc;
}

static RbArgs rb_args(pic_ctx* c) {
    RbArgs a;
    a.phi = c->phi;
    a.b = c->rb_b;
    a.Nx = c->Nx;
    a.Ny = c->Ny;
    const double dx2 = c->dx * c->dx, dy2 = c->dy * c->dy;
    a.ix2 = 1.0 / dx2;
    a.iy2 = 1.0 / dy2;
    a.denom = 2.0 * (1.0 / dx2 + 1.0 / dy2);
    a.inv_denom = 1.0 / a.denom;
    return a;
}

static int rb_sweeps(pic_ctx* c, const RbArgs& a, int n) {
    const size_t half = (size_t)(c->Nx / 2) * c->Ny;
    const unsigned blocks = (unsigned)((half + RB_THREADS - 1) / RB_THREADS);
    for (int s = 0; s < n; ++s) {
        rbgs_half<<<blocks, RB_THREADS, 0, c->stream>>>(a, 0);
        PIC_TRY(check_launch(c, "rbgs_half"));
        rbgs_half<<<blocks, RB_THREADS, 0, c->stream>>>(a, 1);
        PIC_TRY(check_launch(c, "rbgs_half"));
    }
    return PIC_OK;
}

static int rb_residual_async(pic_ctx* c, const RbArgs& a) {
    rb_resid_partials<<<RB_RED_BLOCKS, RB_THREADS, 0, c->stream>>>(a, c->rb_partial);
    PIC_TRY(check_launch(c, "rb_resid_partials"));
    rb_final<<<1, RB_THREADS, 0, c->stream>>>(c->rb_partial, RB_RED_BLOCKS, 2, 0, c->rb_scalars + 1);
    PIC_TRY(check_launch(c, "rb_final"));
    rb_final<<<1, RB_THREADS, 0, c->stream>>>(c->rb_partial, RB_RED_BLOCKS, 2, 1, c->rb_scalars + 2);
    return check_launch(c, "rb_final");
}

// rhs b = rho*dV - mean into c->rb_b (queued).
static int rb_prepare(pic_ctx* c) {
    const unsigned blocks = (unsigned)((c->G + 255) / 256);
    rb_sum_rhs<<<RB_RED_BLOCKS, RB_THREADS, 0, c->stream>>>(c->rho, c->dx * c->dy, c->G, c->rb_partial);
    PIC_TRY(check_launch(c, "rb_sum_rhs"));
    rb_final<<<1, RB_THREADS, 0, c->stream>>>(c->rb_partial, RB_RED_BLOCKS, 1, 0, c->rb_scalars);
    PIC_TRY(check_launch(c, "rb_final"));
    rb_make_rhs<<<blocks, 256, 0, c->stream>>>(c->rho, c->dx * c->dy, c->G, c->rb_scalars, c->rb_b);
    return check_launch(c, "rb_make_rhs");
}

static int rb_finish(pic_ctx* c) {
    const unsigned blocks = (unsigned)((c->G + 255) / 256);
    rb_sum_rhs<<<RB_RED_BLOCKS, RB_THREADS, 0, c->stream>>>(c->phi, 1.0, c->G, c->rb_partial);
    PIC_TRY(check_launch(c, "rb_sum_rhs"));
    rb_final<<<1, RB_THREADS, 0, c->stream>>>(c->rb_partial, RB_RED_BLOCKS, 1, 0, c->rb_scalars + 3);
    PIC_TRY(check_launch(c, "rb_final"));
    rb_sub_mean<<<blocks, 256, 0, c->stream>>>(c->phi, c->G, c->rb_scalars + 3);
    PIC_TRY(check_launch(c, "rb_sub_mean"));
    return efield_from_phi(c, c->in_run || c->G <= (size_t)1 << 20);
}

// ---- one cooperative launch per solve ---------------------------------------
// The grid is cut into ntx x nty tiles (sizes differ by at most one cell), one
// CTA each, as many as fill the SMs. A CTA keeps its tile of phi, a halo of
// `halo` cells around it and the matching piece of b in shared memory for the
// whole solve, the two colours in separate arrays (neighbouring lanes touch
// neighbouring words). Between two exchanges it performs `halo` half-sweeps
// (halo / 2 full red-black sweeps) on the extended tile, the updated region
// shrinking by one cell per half-sweep, so the owned cells end with exactly the
// values the one-launch-per-colour path computes (same update, same operation
// order, same colour order). It then publishes the cells near its edge through
// one of two exchange buffers in turn and loads its halo from its neighbours'. Each
// 32-bit word travels with the exchange's number in one 64-bit word, so a value
// says itself whether it has arrived: no flag, no fence and no grid barrier between
// its store and its load. (A neighbour can be one exchange ahead at most, hence
// two buffers.) The residual is checked every check_every
// sweeps: per-CTA sums of r^2 and b^2, a grid-wide barrier, and every CTA adds
// the partials in the same order and takes the same decision. Waits give up
// after about one second (PIC_ERR_TIMEOUT).
//
// Bound by the exchange's latency (stores and loads through L2, a thread's halo words one
// after the other) and by FP64 arithmetic (a warp's FP64 instruction takes the SM 16
// cycles). rb_tiling picks tile counts and halo for the smallest sum of a model of the two;
// the model ranks the cuts, it does not give their times (256^2: 1,750 cycles a sweep,
// measured 3,300). With
// equal spacings that are powers of two (unit cells, say) an update is four FP64
// instructions instead of seven, with the same bits: the products are exact, so
// (we*s + sn*s + b)*inv is one fused multiply-add of we + sn and b*inv.
// 256^2, tol 1e-8, 57,920 sweeps from phi = 0: 92 ms in FP64 (1.6 us a sweep), 54 ms
// mixed; 515 and 208 ms with 64 x 32 tiles (32 CTAs), seven instructions, an index
// division per update and a grid-wide barrier per exchange. 64^2, 3,648 sweeps: 3.5
// ms, from 31. Flags with release and acquire instead of numbered words: 160 ms.
constexpr int PS_MAX_BLOCKS = 4096;
constexpr size_t PS_MAX_SMEM = 225 * 1024;
constexpr unsigned long long PS_WAIT_NS = 1000000000ull;

__device__ __forceinline__ uint64_t ps_time_ns() {
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// Limits a spin: true once wait_ns have passed since the first look at the clock.
// %globaltimer is slow to read (about a microsecond, as much as the whole wait), so
// only every 256th poll looks.
struct PsLimit {
    unsigned polls = 0;
    uint64_t t0 = 0;
    __device__ __forceinline__ bool over(unsigned long long wait_ns) {
        if ((++polls & 255u) != 0) return false;
        const uint64_t t = ps_time_ns();
        if (t0 == 0) t0 = t;
        return t - t0 > wait_ns;
    }
};

__device__ bool ps_barrier(unsigned* bar, int* err, unsigned long long wait_ns = PS_WAIT_NS) {
    __syncthreads();
    __shared__ int ok;
    if (threadIdx.x == 0) {
        ok = 1;
        volatile unsigned* vgen = bar + 1;
        const unsigned gen = *vgen;
        __threadfence();
        if (atomicAdd(bar, 1u) == gridDim.x - 1) {
            atomicExch(bar, 0u);
            __threadfence();
            atomicAdd(bar + 1, 1u);
        } else {
            PsLimit limit;
            while (*vgen == gen)
                if (limit.over(wait_ns)) {
                    atomicExch(err, 1);
                    ok = 0;
                    break;
                }
        }
        __threadfence();
    }
    __syncthreads();
    return ok != 0;
}

__device__ __forceinline__ int ps_wrap(int i, int n) {
    const int r = i % n;
    return r < 0 ? r + n : r;
}

// A value and its exchange's number: one 64-bit word, stored and loaded whole, per
// 32 bits of the value.
__device__ __forceinline__ unsigned long long ps_pack(unsigned word, unsigned epoch) {
    return (unsigned long long)epoch << 32 | word;
}
__device__ __forceinline__ void ps_publish(unsigned long long* x, size_t i, float v, unsigned epoch) {
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(x + i), "l"(ps_pack(__float_as_uint(v), epoch)) : "memory");
}
__device__ __forceinline__ void ps_publish(unsigned long long* x, size_t i, double v, unsigned epoch) {
    asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" ::"l"(x + 2 * i),
                 "l"(ps_pack((unsigned)__double2loint(v), epoch)), "l"(ps_pack((unsigned)__double2hiint(v), epoch))
                 : "memory");
}
__device__ __forceinline__ bool ps_receive(const unsigned long long* x, size_t i, unsigned epoch, float& v) {
    unsigned long long a;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(a) : "l"(x + i) : "memory");
    v = __uint_as_float((unsigned)a);
    return (unsigned)(a >> 32) == epoch;
}
__device__ __forceinline__ bool ps_receive(const unsigned long long* x, size_t i, unsigned epoch, double& v) {
    unsigned long long lo, hi;
    asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(lo), "=l"(hi) : "l"(x + 2 * i) : "memory");
    v = __hiloint2double((int)(unsigned)hi, (int)(unsigned)lo);
    return (unsigned)(lo >> 32) == epoch && (unsigned)(hi >> 32) == epoch;
}

template <typename T>
struct PsArgs {
    T* x;         // phi (FP64), or the correction (FP32); read at the start, written at the end
    const T* b;   // right-hand side
    unsigned long long* xb;  // exchange buffers, 2 * Nx * Ny values of sizeof(T) / 4 words (ps_pack); zeroed
    int Nx, Ny, ntx, nty;
    T ix2, iy2, inv_denom, denom;
    double tol;
    int max_iters, check_every;
    double* partial;  // [2][2 * PS_MAX_BLOCKS]
    unsigned* bar;    // [0] arrivals, [1] generation
    int* err;
    double* out;      // [0] sweeps, [1] residual, [2] first residual
    int absent_block; // -1, or a CTA that leaves at once (the timeout test hook)
    unsigned long long wait_ns;  // limit of one wait
};

// Sum over the block in a fixed order, the same value in every thread.
__device__ __forceinline__ double ps_block_sum(double v) {
    __shared__ double ws[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = __dadd_rn(v, __shfl_down_sync(0xffffffffu, v, o));
    if (lane == 0) ws[warp] = v;
    __syncthreads();
    double s = 0.0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) s = __dadd_rn(s, ws[w]);
    __syncthreads();
    return s;
}

__device__ __forceinline__ double ps_fma(double a, double b, double c) { return __fma_rn(a, b, c); }
__device__ __forceinline__ float ps_fma(float a, float b, float c) { return __fmaf_rn(a, b, c); }

// t / d for 0 <= t < 2^20, d < 2^10, with inv = 1 / d: the quotient of t + 0.5 is at
// least 1 / (2 d) away from an integer, far more than the rounding of the product.
__device__ __forceinline__ int ps_div(int t, float inv) { return (int)(((float)t + 0.5f) * inv); }

// POW2: equal spacings, a power of two; sb holds b * inv_denom (exact).
// The FP32 correction solve also stops when rounding stalls it.
// H: the halo. NPT: the updates of a thread in a half-sweep at most; their places
// are worked out once and kept in registers (a division, address arithmetic and a
// second round of latency per update otherwise, most of a half-sweep's time).
template <typename T, bool POW2, int H, int NPT>
__global__ void __launch_bounds__(1024) rbgs_persistent(PsArgs<T> p) {
    constexpr bool STALL = sizeof(T) == 4;
    extern __shared__ __align__(16) unsigned char psm[];
    __shared__ double tot[2];
    __shared__ int s_nh, s_nb, s_ok;
    if ((int)blockIdx.x == p.absent_block) return;
    const int nthr = blockDim.x;
    const int tx = blockIdx.x % p.ntx, ty = blockIdx.x / p.ntx;
    // tile t of n tiles over N cells starts at t * N / n
    const int xs = (int)((long long)tx * p.Nx / p.ntx), xe = (int)((long long)(tx + 1) * p.Nx / p.ntx);
    const int ys = (int)((long long)ty * p.Ny / p.nty), ye = (int)((long long)(ty + 1) * p.Ny / p.nty);
    const int tw = xe - xs, th = ye - ys, ew = tw + 2 * H, eh = th + 2 * H;
    const int ox = xs - H, oy = ys - H;
    const int hw = (ew + 1) >> 1, plane = hw * eh;  // one colour: eh rows of hw cells
    T* sx = reinterpret_cast<T*>(psm);              // [2 colours][plane]
    T* sb = sx + 2 * plane;
    uint2* list = reinterpret_cast<uint2*>(sb + 2 * plane);  // (shared index, global index): halo, then edge cells
    if (threadIdx.x == 0) s_nh = s_nb = 0;
    __syncthreads();
    // colour of the extended tile's cell (lx, ly), global parity of ox + lx + oy + ly
    const int par0 = (ox + oy) & 1;
    auto at = [&](int lx, int ly) { return (((par0 + lx + ly) & 1) ? plane : 0) + ly * hw + (lx >> 1); };
    const float inv_ew = 1.0f / (float)ew;
    const int E = ew * eh, nown = tw * th;
    auto in_halo = [&](int lx, int ly) { return lx < H || lx >= H + tw || ly < H || ly >= H + th; };
    for (int i = threadIdx.x; i < E; i += nthr) {
        const int ly = ps_div(i, inv_ew), lx = i - ly * ew;
        const size_t g = (size_t)ps_wrap(oy + ly, p.Ny) * p.Nx + ps_wrap(ox + lx, p.Nx);
        const int k = at(lx, ly);
        sb[k] = POW2 ? p.b[g] * p.inv_denom : p.b[g];
        sx[k] = p.x[g];
        if (in_halo(lx, ly)) list[atomicAdd(&s_nh, 1)] = make_uint2((unsigned)k, (unsigned)g);
    }
    __syncthreads();
    const int nh = s_nh;
    for (int i = threadIdx.x; i < E; i += nthr) {  // owned cells within H of the tile's edge
        const int ly = ps_div(i, inv_ew), lx = i - ly * ew;
        if (in_halo(lx, ly) || !(lx < 2 * H || lx >= tw || ly < 2 * H || ly >= th)) continue;
        const unsigned g = (unsigned)((oy + ly) * p.Nx + ox + lx);
        list[nh + atomicAdd(&s_nb, 1)] = make_uint2((unsigned)at(lx, ly), g);
    }
    __syncthreads();
    const int nb = s_nb;
    const uint2* edge = list + nh;
    const size_t G = (size_t)p.Nx * p.Ny;
    const float inv_tw = 1.0f / (float)tw;
    auto own_b = [&](int k) { return POW2 ? sb[k] * p.denom : sb[k]; };  // exact
    double bb = 0.0;
    for (int t = threadIdx.x; t < nown; t += nthr) {
        const int r = ps_div(t, inv_tw);
        const double v = (double)own_b(at(H + t - r * tw, H + r));
        bb = __dadd_rn(bb, __dmul_rn(v, v));
    }
    bb = ps_block_sum(bb);
    // half-sweep k updates colour k & 1 in rows and columns k + 1 .. of the extended
    // tile: (index << 1 | column parity), or -1
    int place[H][NPT];
#pragma unroll
    for (int k = 0; k < H; ++k) {
        const int lo = k + 1, rows = eh - 2 * lo, half = (ew - 2 * lo + 1) >> 1;
        const float inv_half = 1.0f / (float)half;
#pragma unroll
        for (int n = 0; n < NPT; ++n) {
            const int t = threadIdx.x + n * nthr;
            const int r = ps_div(t, inv_half), ly = lo + r;
            const int lx = lo + ((par0 + lo + ly + (k & 1)) & 1) + 2 * (t - r * half);
            place[k][n] = t < rows * half && lx < ew - lo ? ((ly * hw + (lx >> 1)) << 1) | (lx & 1) : -1;
        }
    }
    int it = 0;
    unsigned epoch = 0, check = 0;
    double res = 0.0, res0 = -1.0, prev = 1e300;
    const T c4 = p.ix2 * p.inv_denom;  // POW2: exact
    bool failed = false;
    for (;;) {
        if (it % p.check_every == 0 || it >= p.max_iters) {
            double rr = 0.0;
            for (int t = threadIdx.x; t < nown; t += nthr) {
                const int r = ps_div(t, inv_tw);
                const int ly = H + r, lx = H + t - r * tw, k = at(lx, ly), odd = lx & 1;
                const int o = (k < plane ? plane : 0) + ly * hw + (lx >> 1);  // the other colour, same row and pair
                const T we = sx[o - 1 + odd] + sx[o + odd], sn = sx[o - hw] + sx[o + hw];
                const T ap = p.denom * sx[k] - we * p.ix2 - sn * p.iy2;
                const double q = (double)(own_b(k) - ap);
                rr = __dadd_rn(rr, __dmul_rn(q, q));
            }
            rr = ps_block_sum(rr);
            // two sets in turn: a CTA far away can reach its next check before this
            // one has read the set of this check, but not the one after
            double* partial = p.partial + (check++ & 1u) * 2 * PS_MAX_BLOCKS;
            if (threadIdx.x == 0) {
                partial[2 * blockIdx.x] = rr;
                partial[2 * blockIdx.x + 1] = bb;
            }
            if (!ps_barrier(p.bar, p.err, p.wait_ns)) {
                failed = true;
                break;
            }
            if (threadIdx.x < 32) {
                double s1 = 0.0, s2 = 0.0;
                for (unsigned k = threadIdx.x; k < gridDim.x; k += 32) {
                    s1 = __dadd_rn(s1, __ldcg(partial + 2 * k));
                    s2 = __dadd_rn(s2, __ldcg(partial + 2 * k + 1));
                }
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) {
                    s1 = __dadd_rn(s1, __shfl_down_sync(0xffffffffu, s1, o));
                    s2 = __dadd_rn(s2, __shfl_down_sync(0xffffffffu, s2, o));
                }
                if (threadIdx.x == 0) {
                    tot[0] = s1;
                    tot[1] = s2;
                }
            }
            __syncthreads();
            res = tot[1] > 0.0 ? sqrt(tot[0] / tot[1]) : STALL ? 0.0 : sqrt(tot[0]);
            if (res0 < 0.0) res0 = res;
            if (res <= p.tol || it >= p.max_iters || (STALL && res > 0.999 * prev)) break;
            prev = res;
        }
#pragma unroll
        for (int k = 0; k < H; ++k) {
            T* own = sx + ((k & 1) ? plane : 0);
            const T* oth = sx + ((k & 1) ? 0 : plane);
            const T* rhs = sb + ((k & 1) ? plane : 0);
#pragma unroll
            for (int n = 0; n < NPT; ++n) {
                const int e = place[k][n];
                if (e >= 0) {
                    const int o = e >> 1, w = o - 1 + (e & 1);
                    const T we = oth[w] + oth[w + 1], sn = oth[o - hw] + oth[o + hw];
                    own[o] = POW2 ? ps_fma(we + sn, c4, rhs[o]) : (we * p.ix2 + sn * p.iy2 + rhs[o]) * p.inv_denom;
                }
            }
            __syncthreads();
        }
        it += H / 2;
        unsigned long long* xb = p.xb + (epoch & 1u) * G * (sizeof(T) / 4);
        ++epoch;
        if (threadIdx.x == 0) s_ok = 1;
        for (int i = threadIdx.x; i < nb; i += nthr) ps_publish(xb, edge[i].y, sx[edge[i].x], epoch);
        __syncthreads();  // the edge cells are read, s_ok is set
        PsLimit limit;
        for (int i = threadIdx.x; i < nh; i += nthr) {
            const uint2 h = list[i];
            T v;
            while (!ps_receive(xb, h.y, epoch, v))
                if (limit.over(p.wait_ns)) {
                    atomicExch(p.err, 1);
                    s_ok = 0;
                    break;
                }
            sx[h.x] = v;
            if (!s_ok) break;
        }
        __syncthreads();
        if (!s_ok) {
            failed = true;
            break;
        }
    }
    if (failed) return;
    for (int t = threadIdx.x; t < nown; t += nthr) {
        const int r = ps_div(t, inv_tw), c = t - r * tw;
        p.x[(size_t)(ys + r) * p.Nx + xs + c] = sx[at(H + c, H + r)];
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        p.out[0] = (double)it;
        p.out[1] = res;
        p.out[2] = res0;
    }
}

// How the one-launch solve cuts the grid.
struct RbTiling {
    int ntx = 0, nty = 0, halo = 0, npt = 0, threads = 0;
    size_t smem = 0;
};
constexpr int PS_MAX_NPT = 8;

// Tile counts and halo for the least estimated time per sweep: the half-sweeps'
// updates at `op_cycles` per warp (never below `min_cycles`, the latency of one
// update and its barrier) and one exchange per halo / 2 sweeps. A tile is at
// least as wide as the halo (or the whole grid), so that only the eight
// neighbours' cells are needed; `step`: the sweeps between checks are a multiple
// of it, so halo / 2 must divide it.
static RbTiling rb_tiling(int Nx, int Ny, int max_blocks, int step, size_t bytes, double op_cycles, double min_cycles) {
    constexpr double EXCHANGE = 1000.0;  // fitted, not measured: 2,000 chose longer halos at 256^2 (101 ms), 500 shorter ones at 222 x 106 (41 against 38)
    RbTiling best;
    double best_cost = 1e300;
    for (int H = 4; H <= 8; H += 4) {
        if (step % (H / 2)) continue;
        for (int nx = 1; nx <= max_blocks && nx <= Nx; ++nx) {
            if (nx > 1 && Nx / nx < H) break;
            for (int ny = 1; ny <= max_blocks / nx && ny <= Ny; ++ny) {
                if (ny > 1 && Ny / ny < H) break;
                const int w = (Nx + nx - 1) / nx, h = (Ny + ny - 1) / ny;
                const size_t ew = w + 2 * H, eh = h + 2 * H;
                const size_t plane = (ew + 1) / 2 * eh;
                const size_t inner = (size_t)(w > 2 * H ? w - 2 * H : 0) * (h > 2 * H ? h - 2 * H : 0);
                const size_t need = 4 * plane * bytes + (ew * eh - inner) * sizeof(uint2);
                const size_t most = (ew - 1) / 2 * (eh - 2);  // updates of the first half-sweep, at most
                if (need > PS_MAX_SMEM || ew >= 1024 || most > (size_t)1024 * PS_MAX_NPT) continue;
                double cost = EXCHANGE;
                for (int k = 0; k < H; ++k) {
                    const double upd = 0.5 * (w + 2 * (H - 1 - k)) * (h + 2 * (H - 1 - k));
                    const double c = (double)(long long)((upd + 31.0) / 32.0) * op_cycles;
                    cost += c > min_cycles ? c : min_cycles;
                }
                cost /= H / 2;
                if (cost < best_cost) {
                    best_cost = cost;
                    best.ntx = nx;
                    best.nty = ny;
                    best.halo = H;
                    best.smem = need;
                    best.npt = 1;
                    while (most > (size_t)512 * best.npt && best.npt < PS_MAX_NPT) best.npt *= 2;
                    best.threads = (int)((most + best.npt - 1) / best.npt + 31) / 32 * 32;
                    if (best.threads < 64) best.threads = 64;
                }
            }
        }
    }
    return best;
}

// Whether 2^k * 2^k = x for the operator's coefficients: equal spacings, powers of two.
static bool rb_pow2(const RbArgs& a) {
    return a.ix2 == a.iy2 && exact_reciprocal(a.ix2) != 0.0 && exact_reciprocal(a.denom) != 0.0 && a.ix2 > 1e-30 && a.ix2 < 1e30;
}

template <typename T, bool POW2, int H>
static const void* rb_kernel_npt(int npt) {
    switch (npt) {
        case 1:
            return (const void*)rbgs_persistent<T, POW2, H, 1>;
        case 2:
            return (const void*)rbgs_persistent<T, POW2, H, 2>;
        case 4:
            return (const void*)rbgs_persistent<T, POW2, H, 4>;
        default:
            return (const void*)rbgs_persistent<T, POW2, H, 8>;
    }
}
template <typename T>
static const void* rb_kernel(bool pow2, int halo, int npt) {
    return pow2 ? (halo == 4 ? rb_kernel_npt<T, true, 4>(npt) : rb_kernel_npt<T, true, 8>(npt))
                : (halo == 4 ? rb_kernel_npt<T, false, 4>(npt) : rb_kernel_npt<T, false, 8>(npt));
}

template <typename T>
static int rb_launch(pic_ctx* c, const RbTiling& t, const PsArgs<T>& p, bool pow2) {
    const void* k = rb_kernel<T>(pow2, t.halo, t.npt);
    PIC_TRY(opt_in_dynamic_smem(k, t.smem));
    // exchange numbers start again from 1
    PIC_CUDA_TRY(cudaMemsetAsync(p.xb, 0, 2 * c->G * 2 * sizeof(T), c->stream));
    PsArgs<T> q = p;
    void* args[] = {&q};
    PIC_CUDA_TRY(cudaLaunchCooperativeKernel(k, dim3(t.ntx * t.nty), dim3(t.threads), args, t.smem, c->stream));
    c->launches++;
    return PIC_OK;
}

// Buffers of the one-launch solves: partial sums, out[0..3], the barrier and the error
// flag; the exchange buffers; with `mixed` the residuals and the correction. False when the
// device has no room for them: the launches per colour need none.
static bool ensure_ps(pic_ctx* c, bool mixed) {
    int rc = PIC_OK;
    if (!c->rb_ps) c->rb_ps = (double*)dalloc((4 * PS_MAX_BLOCKS + 8) * sizeof(double), &rc);
    if (!rc && !c->rb_xb) c->rb_xb = dalloc(2 * c->G * 2 * sizeof(double), &rc);
    if (!rc && mixed && !c->rb_mix) c->rb_mix = (double*)dalloc(c->G * (8 + 4 + 4), &rc);
    return rc == PIC_OK;
}

static int sm_count(pic_ctx* c) {
    int sms = 0;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, c->device);
    return sms > PS_MAX_BLOCKS ? PS_MAX_BLOCKS : sms;
}

static int largest_divisor_tile(int n, const int* cand, int ncand) {
    for (int k = 0; k < ncand; ++k)
        if (cand[k] <= n && n % cand[k] == 0) return cand[k];
    return 0;
}

// Solves in one cooperative launch when the tiles fit the SMs' shared memory and its
// buffers the device's; returns PIC_ERR_UNSUPPORTED (nothing queued) otherwise.
// absent_block >= 0 makes that CTA leave before its first barrier, so that every
// other CTA's wait runs out after wait_ns (the timeout test hook; -1 in solves).
static int rbgs_solve_persistent(pic_ctx* c, const RbArgs& a, double tol, int max_iters, int check_every, int* it,
                                 double* res, int absent_block = -1, unsigned long long wait_ns = PS_WAIT_NS) {
    if ((check_every & 1) || (max_iters & 1)) return PIC_ERR_UNSUPPORTED;
    const bool pow2 = rb_pow2(a);
    const int step = (check_every % 4 == 0 && max_iters % 4 == 0) ? 4 : 2;
    const RbTiling t = rb_tiling(c->Nx, c->Ny, sm_count(c), step, sizeof(double), pow2 ? 64.0 : 112.0, 400.0);
    if (!t.ntx) return PIC_ERR_UNSUPPORTED;
    if (!ensure_ps(c, false)) return PIC_ERR_UNSUPPORTED;
    double* out = c->rb_ps + 4 * PS_MAX_BLOCKS;
    unsigned* bar = reinterpret_cast<unsigned*>(out + 4);
    int* err = reinterpret_cast<int*>(out + 5);
    PIC_CUDA_TRY(cudaMemsetAsync(bar, 0, 2 * sizeof(unsigned), c->stream));
    PIC_CUDA_TRY(cudaMemsetAsync(err, 0, sizeof(int), c->stream));
    const PsArgs<double> p{c->phi, c->rb_b, static_cast<unsigned long long*>(c->rb_xb), c->Nx, c->Ny, t.ntx, t.nty, a.ix2, a.iy2,
                           a.inv_denom, a.denom, tol, max_iters, check_every, c->rb_ps, bar, err, out,
                           absent_block, wait_ns};
    PIC_TRY(rb_launch<double>(c, t, p, pow2));
    double h[6];
    PIC_CUDA_TRY(cudaMemcpyAsync(h, out, sizeof(h), cudaMemcpyDeviceToHost, c->stream));
    PIC_CUDA_TRY(cudaStreamSynchronize(c->stream));
    int herr = 0;
    std::memcpy(&herr, &h[5], sizeof(int));
    if (herr) return fail(PIC_ERR_TIMEOUT, "red-black Gauss-Seidel: a neighbour's exchange or the grid-wide barrier timed out");
    *it = (int)h[0];
    *res = h[1];
    c->first_rbgs_resid = h[2];
    return PIC_OK;
}

// ---- mixed precision: FP32 sweeps on the correction, FP64 residual --------
// Iterative refinement: r = b - A phi in FP64; A e = r is relaxed in FP32 by the
// same red-black sweeps (one cooperative launch) until ||r - A e|| <= itol ||r||; phi += e in FP64; repeat until the
// FP64 relative residual meets tol. The answer meets the same FP64 test as the
// FP64 solve; sweeps are counted over all corrections.
__global__ void rb_residual_field(RbArgs a, const double* __restrict__ phi, double* __restrict__ r);

__global__ void rb_to_f32(const double* __restrict__ r, size_t n, float* __restrict__ r32, float* __restrict__ e) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) {
        r32[i] = __double2float_rn(r[i]);
        e[i] = 0.0f;
    }
}

__global__ void rb_add_correction(double* __restrict__ phi, const float* __restrict__ e, size_t n) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) phi[i] = __dadd_rn(phi[i], (double)e[i]);
}

// The mixed-precision solve; PIC_ERR_UNSUPPORTED (nothing queued) when the
// grid does not tile evenly or the tiles cannot all be resident.
static int rbgs_solve_mixed(pic_ctx* c, const RbArgs& a, double tol, int max_iters, int check_every, int* it_out,
                            double* res_out) {
    // Which grids refine in FP32 is part of the results (the two modes agree to the
    // tolerance, not bit for bit): those that divide into 64 x 32 or smaller
    // power-of-two tiles, few enough of them, as pic_gpu_set_rbgs_precision states.
    static const int cw[] = {64, 32, 16, 8, 4, 2};
    static const int ch[] = {32, 16, 8, 4, 2};
    const int dw = largest_divisor_tile(c->Nx, cw, 6), dh = largest_divisor_tile(c->Ny, ch, 5);
    if (!dw || !dh) return PIC_ERR_UNSUPPORTED;
    const long long blocks = (long long)(c->Nx / dw) * (c->Ny / dh);
    if (blocks > PS_MAX_BLOCKS || blocks > (long long)(dw * dh == 2048 ? 7 : 8) * sm_count(c)) return PIC_ERR_UNSUPPORTED;
    const bool pow2 = rb_pow2(a);
    const RbTiling t = rb_tiling(c->Nx, c->Ny, sm_count(c), 4, sizeof(float), 14.0, 200.0);
    if (!t.ntx) return PIC_ERR_UNSUPPORTED;
    if (!ensure_ps(c, true)) return PIC_ERR_UNSUPPORTED;
    double* r64 = c->rb_mix;
    float* r32 = reinterpret_cast<float*>(r64 + c->G);
    float* e32 = r32 + c->G;
    unsigned long long* xb32 = static_cast<unsigned long long*>(c->rb_xb);
    double* out = c->rb_ps + 4 * PS_MAX_BLOCKS;
    unsigned* bar = reinterpret_cast<unsigned*>(out + 4);
    int* err = reinterpret_cast<int*>(out + 5);
    PIC_CUDA_TRY(cudaMemsetAsync(bar, 0, 2 * sizeof(unsigned), c->stream));
    PIC_CUDA_TRY(cudaMemsetAsync(err, 0, sizeof(int), c->stream));
    const unsigned gb = (unsigned)((c->G + 255) / 256);
    const int ce = check_every < 4 ? 4 : (check_every / 4) * 4;
    int it = 0;
    double res = 0.0, prev_res = 0.0;
    for (int outer = 0;; ++outer) {
        PIC_TRY(rb_residual_async(c, a));
        double s[3];
        PIC_CUDA_TRY(cudaMemcpyAsync(s, c->rb_scalars, sizeof(s), cudaMemcpyDeviceToHost, c->stream));
        PIC_CUDA_TRY(cudaStreamSynchronize(c->stream));
        res = s[2] > 0.0 ? std::sqrt(s[1] / s[2]) : std::sqrt(s[1]);
        if (outer == 0) c->first_rbgs_resid = res;
        if (res <= tol || it >= max_iters) break;
        const int left = max_iters - it;
        if (left < 4) {  // the FP32 sweeps come in fours, as the check interval does: the last few in FP64
            PIC_TRY(rb_sweeps(c, a, left));
            it += left;
            continue;
        }
        rb_residual_field<<<gb, 256, 0, c->stream>>>(a, c->phi, r64);
        PIC_TRY(check_launch(c, "rb_residual_field"));
        rb_to_f32<<<gb, 256, 0, c->stream>>>(r64, c->G, r32, e32);
        PIC_TRY(check_launch(c, "rb_to_f32"));
        // reduce the residual by what is left to reach tol; FP32 rounding of the
        // correction limits one pass to about cond(A) * 2^-24 of the residual, so a
        // pass aims at 1e-2 at most and the passes repeat
        double itol = 0.5 * tol / res;
        if (itol < 1e-2) itol = 1e-2;
        if (itol > 0.5) itol = 0.5;
        if (outer > 0 && res > 0.5 * prev_res) {  // a pass that no longer helps: finish in FP64
            int it64 = 0;
            double r64v = 0.0;
            const double first = c->first_rbgs_resid;
            const int prc = rbgs_solve_persistent(c, a, tol, left & ~1, check_every & ~1 ? check_every & ~1 : 2,
                                                  &it64, &r64v);
            c->first_rbgs_resid = first;
            if (prc == PIC_OK) {
                it += it64;
                res = r64v;
                if (res <= tol || it >= max_iters) break;
                continue;
            }
            if (prc != PIC_ERR_UNSUPPORTED) return prc;
        }
        prev_res = res;
        const PsArgs<float> p{e32, r32, xb32, c->Nx, c->Ny, t.ntx, t.nty, (float)a.ix2, (float)a.iy2,
                              (float)a.inv_denom, (float)a.denom, (double)(float)itol, left & ~3, ce,
                              c->rb_ps, bar, err, out, -1, PS_WAIT_NS};
        PIC_TRY(rb_launch<float>(c, t, p, pow2));
        rb_add_correction<<<gb, 256, 0, c->stream>>>(c->phi, e32, c->G);
        PIC_TRY(check_launch(c, "rb_add_correction"));
        double h[6];
        PIC_CUDA_TRY(cudaMemcpyAsync(h, out, sizeof(h), cudaMemcpyDeviceToHost, c->stream));
        PIC_CUDA_TRY(cudaStreamSynchronize(c->stream));
        int herr = 0;
        std::memcpy(&herr, &h[5], sizeof(int));
        if (herr) return fail(PIC_ERR_TIMEOUT, "red-black Gauss-Seidel: a neighbour's exchange or the grid-wide barrier timed out");
        const int sw = (int)h[0];
        it += sw > 0 ? sw : 1;  // a pass that made no sweep still counts, so the loop ends
    }
    *it_out = it;
    *res_out = res;
    return PIC_OK;
}

// Solves with the residual checked every `check_every` sweeps: in one
// cooperative launch where possible, else one launch per colour with the
// residual read on the host; with the mixed-precision option, FP32 sweeps on
// FP64-refined corrections.
int rbgs_solve(pic_ctx* c, double tol, int max_iters, int check_every, int* iters_out, double* resid_out) {
    if ((c->Nx & 1) || (c->Ny & 1)) return fail(PIC_ERR_UNSUPPORTED, "red-black Gauss-Seidel needs even Nx and Ny");
    if (max_iters < 0) return fail(PIC_ERR_ARG, "max_iters < 0");
    if (check_every < 1) check_every = 1;
    PIC_TRY(ensure_rbgs(c));
    PIC_TRY(rb_prepare(c));
    const RbArgs a = rb_args(c);
    int it = 0;
    double res = 0.0;
    prof_begin(c, "rbgs");
    int prc = PIC_ERR_UNSUPPORTED;
    if (c->rbgs_mixed) prc = rbgs_solve_mixed(c, a, tol, max_iters, check_every, &it, &res);
    if (prc == PIC_ERR_UNSUPPORTED && c->rbgs_persistent)
        prc = rbgs_solve_persistent(c, a, tol, max_iters, check_every, &it, &res);
    if (prc != PIC_OK && prc != PIC_ERR_UNSUPPORTED) {
        prof_end(c);
        return prc;
    }
    for (; prc == PIC_ERR_UNSUPPORTED;) {
        PIC_TRY(rb_residual_async(c, a));
        double s[3];
        PIC_CUDA_TRY(cudaMemcpyAsync(s, c->rb_scalars, sizeof(s), cudaMemcpyDeviceToHost, c->stream));
        PIC_CUDA_TRY(cudaStreamSynchronize(c->stream));
        res = s[2] > 0.0 ? std::sqrt(s[1] / s[2]) : std::sqrt(s[1]);
        if (it == 0) c->first_rbgs_resid = res;
        if (res <= tol || it >= max_iters) break;
        const int n = (max_iters - it) < check_every ? (max_iters - it) : check_every;
        PIC_TRY(rb_sweeps(c, a, n));
        it += n;
    }
    prof_end(c);
    PIC_TRY(rb_finish(c));
    if (iters_out) *iters_out = it;
    if (resid_out) *resid_out = res;
    c->last_rbgs_iters = it;
    c->last_rbgs_resid = res;
    return PIC_OK;
}

// r = b - A phi for the right-hand side prepared by rbgs_prepare.
__global__ void rb_residual_field(RbArgs a, const double* __restrict__ phi, double* __restrict__ r) {
    const size_t id = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (id >= (size_t)a.Nx * a.Ny) return;
    const int j = (int)(id / a.Nx), i = (int)(id - (size_t)j * a.Nx);
    const int im = i == 0 ? a.Nx - 1 : i - 1, ip = i == a.Nx - 1 ? 0 : i + 1;
    const int jm = j == 0 ? a.Ny - 1 : j - 1, jp = j == a.Ny - 1 ? 0 : j + 1;
    const double we = __dadd_rn(phi[(size_t)j * a.Nx + im], phi[(size_t)j * a.Nx + ip]);
    const double sn = __dadd_rn(phi[(size_t)jm * a.Nx + i], phi[(size_t)jp * a.Nx + i]);
    const double ap = __dsub_rn(__dsub_rn(__dmul_rn(a.denom, phi[id]), __dmul_rn(we, a.ix2)), __dmul_rn(sn, a.iy2));
    r[id] = __dsub_rn(a.b[id], ap);
}

int rbgs_prepare(pic_ctx* c) {
    if ((c->Nx & 1) || (c->Ny & 1)) return fail(PIC_ERR_UNSUPPORTED, "red-black Gauss-Seidel needs even Nx and Ny");
    PIC_TRY(ensure_rbgs(c));
    return rb_prepare(c);
}

int rbgs_residual_field(pic_ctx* c, const double* phi, double* r) {
    const RbArgs a = rb_args(c);
    rb_residual_field<<<(unsigned)((c->G + 255) / 256), 256, 0, c->stream>>>(a, phi, r);
    return check_launch(c, "rb_residual_field");
}

void rbgs_operator(pic_ctx* c, double* ix2, double* iy2, double* denom) {
    const RbArgs a = rb_args(c);
    *ix2 = a.ix2;
    *iy2 = a.iy2;
    *denom = a.denom;
}

int rbgs_solve_async(pic_ctx* c, double tol, int max_iters, int check_every) {
    return rbgs_solve(c, tol, max_iters, check_every, nullptr, nullptr);
}

void release_rbgs(pic_ctx* c) {
    dfree(c->rb_mix);
    dfree(c->rb_xb);
    dfree(c->rb_ps);
    dfree(c->rb_b);
    dfree(c->rb_partial);
    dfree(c->rb_scalars);
}

}  // namespace picgb

using namespace picgb;

extern "C" int pic_gpu_set_rbgs_precision(pic_ctx* c, int mixed) {
    if (!c) return fail(PIC_ERR_ARG, "NULL context");
    if (mixed != 0 && mixed != 1) return fail(PIC_ERR_ARG, "precision must be 0 (FP64) or 1 (mixed)");
    c->rbgs_mixed = mixed;
    return PIC_OK;
}

// Runs the persistent FP64 solve on the context's rho with CTA `absent_block`
// leaving at once and every barrier wait limited to wait_ms: the other CTAs give
// up, set the error flag and return, and the call reports PIC_ERR_TIMEOUT.
extern "C" int pic_gpu_test_rbgs_barrier_timeout(pic_ctx* c, int absent_block, double wait_ms) {
    if (!c) return fail(PIC_ERR_ARG, "NULL context");
    if (absent_block < -1) return fail(PIC_ERR_ARG, "absent_block < -1");
    if (!(wait_ms > 0.0 && wait_ms <= 1000.0)) return fail(PIC_ERR_ARG, "wait_ms must be in (0, 1000]");
    if ((c->Nx & 1) || (c->Ny & 1)) return fail(PIC_ERR_UNSUPPORTED, "red-black Gauss-Seidel needs even Nx and Ny");
    PIC_CUDA_TRY(cudaSetDevice(c->device));
    PIC_TRY(ensure_fields(c));
    PIC_TRY(ensure_rbgs(c));
    PIC_TRY(rb_prepare(c));
    PIC_CUDA_TRY(cudaMemsetAsync(c->phi, 0, c->G * 8, c->stream));
    const RbArgs a = rb_args(c);
    int it = 0;
    double res = 0.0;
    const int rc = rbgs_solve_persistent(c, a, 0.0, 64, 2, &it, &res, absent_block,
                                         (unsigned long long)(wait_ms * 1e6));
    if (rc == PIC_ERR_UNSUPPORTED) return fail(rc, "the grid does not fit one cooperative launch");
    if (rc != PIC_OK) return rc;
    return pic_gpu_synchronize(c);
}

extern "C" int pic_gpu_poisson_rbgs(pic_ctx* c, double tol, int max_iters, int warm_start, int check_every,
                                    int* iters_out, double* resid_out) {
    if (!c) return fail(PIC_ERR_ARG, "NULL context");
    PIC_CUDA_TRY(cudaSetDevice(c->device));
    PIC_TRY(ensure_fields(c));
    if (!warm_start) PIC_CUDA_TRY(cudaMemsetAsync(c->phi, 0, c->G * 8, c->stream));
    PIC_TRY(rbgs_solve(c, tol, max_iters, check_every, iters_out, resid_out));
    return pic_gpu_synchronize(c);
}
