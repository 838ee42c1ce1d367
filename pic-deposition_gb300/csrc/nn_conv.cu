// 3x3 periodic convolutions as implicit GEMMs on the 5th-generation tensor cores.
//
// Forward / input-gradient kernel (conv3x3_kernel): one CTA owns a 128-pixel
// segment of a run of image rows, taken in blocks of 4 output rows. The GEMM of a
// block is
//     D[128 px][row r, cout] = sum over input rows m and dx of
//                              A_(m,dx)[128 px][cin] * B_(m-r,dx)[cin][cout]
// with D in tensor memory (FP32), issued as tcgen05.mma kind::f16 (BF16 x BF16,
// M = 128, K = 16, N = cout times the up to three output rows that an input row
// reaches) by one thread. An MMA of N = 32 spends its time on reading A (64 cycles,
// measured, where its products are 16), one of N = 96 no more than that: a row at a
// time takes 18 of them per row (cin = 32), a block 39 per 4 rows. An output's
// products are added in the same order either way.
// The input rows are staged in shared
// memory as "planes" of 8 channels: pixel slot s of plane j holds the 16 bytes of
// channels 8j..8j+7 of pixel x0-1+s. In the K-major no-swizzle operand layout
// (8-row core matrices of 16-byte rows, stride between row groups SBO = 128 B,
// between the two K halves LBO = one plane) row r of A sits at r*16 bytes, so
// the operand of tap dx is the same staged row with its start moved by
// (dx+1)*16 bytes: im2col costs nothing. The weight image holds the three dy of a
// dx side by side along N, the last first: output rows r, r+1, .. want m-r, m-r-1, ..
// Warp-specialised: two warps stage rows
// into a ring of 7 slots or more, one thread issues the MMAs of a block into one TMEM
// buffer while eight warps drain the block before from the other (bias + ReLU, or the
// ReLU mask of the backward pass), handing over through mbarriers.
// 32 to 32 channels, 512^2, batch 16: forward 104 us (171 a row at a time), 537 MB;
// input gradient 122 us (194), 805 MB, where a copy of as many bytes takes 80 and 120.
//
// Weight-gradient kernel (wgrad_kernel): D[(x row, ci)][(dy row, co)] = sum over
// pixels of x[row, px + dx][ci] * dy[row, px][co], K = pixels, both operands MN-major as
// they sit in NHWC memory (see the kernel's comment); the bias gradient is an
// MMA against an all-ones operand. Each CTA accumulates its blocks
// of pixels in TMEM and writes one partial sum; reduce_wgrad adds the partials
// in a fixed order, so gradients are identical run to run.
//
// Every wait on the tensor cores is bounded (about one second of %globaltimer);
// on expiry the kernel records an error, skips the remaining work, frees its
// tensor memory and returns.
#include <cuda_bf16.h>

#include <climits>

#include "nn_conv.cuh"
#include "pic_internal.cuh"

namespace picnn {

namespace {

constexpr int SLOTS = 130;             // pixels x0-1 .. x0+128
constexpr int PLANE = SLOTS * 16;      // bytes per 8-channel plane

__device__ __forceinline__ uint32_t smem_addr(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// tcgen05 shared-memory matrix descriptor, no swizzle.
__device__ __forceinline__ uint64_t umma_desc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
    return (uint64_t)((addr & 0x3FFFFu) >> 4) | ((uint64_t)((lbo >> 4) & 0x3FFFu) << 16) |
           ((uint64_t)((sbo >> 4) & 0x3FFFu) << 32) | (1ull << 46);
}

// Instruction descriptor of kind::f16: D FP32, A and B BF16, both K-major.
__host__ __device__ constexpr uint32_t idesc_bf16(int m, int n) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}

// Through L1 (.ca): the two halves of a 32-byte sector go to different planes, and .cg
// asks L2 for each (twice the L2 reads; forward 131 us against 112, both with rings of 9).
__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait_group() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

__device__ __forceinline__ void mbar_init(uint32_t a, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(a), "r"(count) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ bool mbar_try(uint32_t a, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n}"
        : "=r"(ok)
        : "r"(a), "r"(parity)
        : "memory");
    return ok != 0;
}
__device__ __forceinline__ uint64_t globaltimer_ns() {
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
// Waits for phase `parity` of the barrier; false after about one second.
__device__ bool mbar_wait(uint32_t a, uint32_t parity) {
    if (mbar_try(a, parity)) return true;
    const uint64_t t0 = globaltimer_ns();
    while (!mbar_try(a, parity))
        if (globaltimer_ns() - t0 > 1000000000ull) return false;
    return true;
}

__device__ __forceinline__ void tmem_alloc(uint32_t slot, uint32_t ncols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(slot), "r"(ncols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void mma_bf16(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}" ::"r"(d),
        "l"(a), "l"(b), "r"(idesc), "r"(accumulate)
        : "memory");
}
// One lane of the warp. The issuing warp computes descriptors in all its lanes and only
// the MMA itself is the elected lane's: they stay in uniform registers, where the
// instruction takes them from (an MMA issued from one lane's branch took about 95
// cycles whatever its size: weight gradient, with 7 staging warps, 159 us against 148,
// with 16 channels on one side 152 against 108 and 120).
__device__ __forceinline__ bool elect_one() {
    uint32_t r;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n}" : "=r"(r));
    return r != 0;
}
__device__ __forceinline__ void mma_commit(uint32_t mbar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(mbar) : "memory");
}

// 16 consecutive FP32 columns of this thread's TMEM lane.
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t* r) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
}
// 16 consecutive columns of this thread's TMEM lane set to zero
__device__ __forceinline__ void tmem_zero16(uint32_t taddr) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1};" ::"r"(taddr),
                 "r"(0)
                 : "memory");
}
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

template <int N>
__device__ __forceinline__ void tmem_load(uint32_t taddr, float* v) {
    uint32_t r[N];
#pragma unroll
    for (int c = 0; c < N; c += 16) tmem_ld16(taddr + c, r + c);
    tmem_wait_ld();
#pragma unroll
    for (int c = 0; c < N; ++c) v[c] = __uint_as_float(r[c]);
}

__device__ __forceinline__ uint32_t pack_bf16x2(float lo, float hi) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&h);
}

__host__ __device__ constexpr uint32_t tmem_cols(int n) {
    return n <= 32 ? 32u : n <= 64 ? 64u : n <= 128 ? 128u : n <= 256 ? 256u : 512u;
}

// ---------------------------------------------------------------------------
// forward / input gradient
// ---------------------------------------------------------------------------
__device__ __forceinline__ void bulk_store(void* dst, uint32_t src, uint32_t bytes) {
    asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(dst), "r"(src), "r"(bytes) : "memory");
    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
}
template <int N>
__device__ __forceinline__ void bulk_wait_read() {
    asm volatile("cp.async.bulk.wait_group.read %0;" ::"n"(N) : "memory");
}

// Which of the 8 BF16 values are above zero, bit e for value e.
__device__ __forceinline__ uint32_t positive8(uint4 m) {
    const uint32_t w[4] = {m.x, m.y, m.z, m.w};
    uint32_t x = 0;
#pragma unroll
    for (int q = 0; q < 4; ++q) x |= __vcmpgts2(w[q], 0u) & (1u << (2 * q) | 1u << (17 + 2 * q));
    return (x | x >> 16) & 0xFFu;
}

// A warp's 32 pixels of a row, in both directions as one contiguous range of
// 32 * COUT * 2 bytes: the ReLU mask is loaded 16 bytes per lane, a row ahead, and
// its signs handed to the pixels' lanes by shuffles; the outputs are put together in
// shared memory (each lane its pixel, the 16-byte pieces in an order that keeps 8
// lanes off one another's banks) and stored by one bulk copy. (Each lane loading and
// storing its own pixel's 64 bytes in four pieces, half a sector each: 231 us against
// 175 for the input gradient of 32 channels at 512^2, batch 16, 172 against 145
// forward.)
template <int COUT, int EPI>
struct RowEpilogue {
    static constexpr int P = COUT / 8;         // 16-byte pieces per pixel
    static constexpr int BYTES = 32 * COUT * 2;
    uint4 next[P];

    __device__ __forceinline__ void prefetch(const ConvLaunch& a, size_t pix0, int lane) {
        if (EPI != EPI_MASK) return;
        const uint4* m = reinterpret_cast<const uint4*>(a.mask + pix0 * COUT);
#pragma unroll
        for (int q = 0; q < P; ++q) next[q] = m[q * 32 + lane];
    }
    // The mask of the lane's pixel, bit c for channel c. Piece q * 32 + lane is piece
    // lane % P of pixel q * 32 / P + lane / P.
    __device__ __forceinline__ uint32_t mask_bits(int lane) const {
        uint32_t bits = 0;
#pragma unroll
        for (int q = 0; q < P; ++q) {
            uint32_t v = positive8(next[q]) << (8 * (lane % P));
#pragma unroll
            for (int o = 1; o < P; o *= 2) v |= __shfl_xor_sync(0xffffffffu, v, o);
            v = __shfl_sync(0xffffffffu, v, lane % (32 / P) * P);
            if (lane / (32 / P) == q) bits = v;
        }
        return bits;
    }
    // v: the accumulators of the lane's pixel. stage: the warp's buffer of BYTES, free
    __device__ __forceinline__ void finish(const ConvLaunch& a, size_t pix0, float (&v)[COUT], uint32_t bits, uint8_t* stage,
                                           const float* sbias, int lane) const {
        if constexpr (EPI == EPI_BIAS_OUT) {
            reinterpret_cast<float*>(a.y)[pix0 + lane] = v[0] + sbias[0];
            return;
        } else {
            uint4 o[P];
#pragma unroll
            for (int q = 0; q < P; ++q) {
                uint32_t w[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const int c = q * 8 + 2 * e;
                    if (EPI == EPI_BIAS_RELU)
                        w[e] = pack_bf16x2(fmaxf(v[c] + sbias[c], 0.0f), fmaxf(v[c + 1] + sbias[c + 1], 0.0f));
                    else
                        w[e] = pack_bf16x2(bits >> c & 1u ? v[c] : 0.0f, bits >> (c + 1) & 1u ? v[c + 1] : 0.0f);
                }
                o[q] = make_uint4(w[0], w[1], w[2], w[3]);
            }
            // pieces in the order (q + rot) % P
            const int rot = lane * P / 8 % P;
#pragma unroll
            for (int step = 1; step < P; step *= 2) {
                uint4 t[P];
#pragma unroll
                for (int q = 0; q < P; ++q) {
                    const uint4 x = o[q], y = o[(q + step) % P];
                    const bool r = (rot & step) != 0;
                    t[q] = make_uint4(r ? y.x : x.x, r ? y.y : x.y, r ? y.z : x.z, r ? y.w : x.w);
                }
#pragma unroll
                for (int q = 0; q < P; ++q) o[q] = t[q];
            }
            uint4* row = reinterpret_cast<uint4*>(stage) + lane * P;
#pragma unroll
            for (int q = 0; q < P; ++q) row[(q + rot) % P] = o[q];
            fence_async_smem();
            __syncwarp();
            if (lane == 0) bulk_store(reinterpret_cast<uint16_t*>(a.y) + pix0 * COUT, smem_addr(stage), BYTES);
        }
    }
};

constexpr int CONV_ROWS = 4;  // output rows per block

template <int CIN, int COUT>
struct ConvSmem {
    // Staged rows: a block's 6 and AHEAD of the next one's 4. AHEAD rows' copies are in
    // flight behind the newest. Copies go through L1, of which shared memory leaves 60
    // KB with two CTAs of 7 rows and 28 with more (32 to 32 channels, 512^2, batch 16:
    // forward 105 us, input gradient 126, with 8 or 9 rows 112 and 154); the 16-channel
    // outputs' CTAs are smaller (32 to 16: 82 us with 9, 112 with 7).
    static constexpr int AHEAD = COUT == 32 ? 1 : 3;
    static constexpr int NRING = 6 + AHEAD;
    static constexpr int PLANES = CIN / 8;
    static constexpr int SLOT = PLANES * PLANE;
    static constexpr int WBYTES = 9 * CIN * COUT * 2;
    static constexpr int OFF_BIAS = WBYTES;
    static constexpr int OFF_OUT = ((WBYTES + COUT * 4) + 127) / 128 * 128;
    static constexpr int OFF_RING = OFF_OUT + 4 * 2 * 32 * COUT * 2;  // a buffer per epilogue warp
    // no more CTAs on an SM than its 512 TMEM columns serve at once
    static constexpr int TCOLS = (int)tmem_cols(2 * CONV_ROWS * COUT);
    static constexpr int LEAST = 228 * 1024 / (512 / TCOLS + 1) + 1024;
    static constexpr int BYTES = OFF_RING + NRING * SLOT > LEAST ? OFF_RING + NRING * SLOT : LEAST;
    static constexpr int CTAS = 227 * 1024 / (BYTES + 1024);
};

__device__ __forceinline__ void mbar_arrive_cta(uint32_t a) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(a) : "memory");
}

// A ring's place: slot and the parity of its present use.
struct RingPos {
    int slot = 0;
    uint32_t parity = 0;
    __device__ __forceinline__ void advance(int n) {
        if (++slot == n) {
            slot = 0;
            parity ^= 1u;
        }
    }
};

// The persistent CTAs take work items (128 pixels x a.rows output rows of an image)
// blockIdx.x, blockIdx.x + gridDim.x, ... in one unbroken pipeline: loading the
// weights, allocating TMEM and filling and draining the pipeline anew for every item
// took 64 us of 139 at 512^2, batch 16.
// Warp-specialised: warps 9 and 10 stage input rows into the ring (cp.async), lane 0
// of warp 8 issues each block's MMAs, warps 0-7 (a TMEM lane quarter and every
// other row each) run the epilogue of the previous block from the other TMEM buffer.
// Barriers: full[s] (the producers' arrivals: the row in slot s has landed),
// rowfree[s] (an MMA commit: the last block that reads slot s is done with it),
// tfull[b] (an MMA commit: accumulator b holds a block), tempty[b] (the
// epilogue's arrivals: accumulator b has been read). A block needs staged rows
// 4i .. 4i+5 of its item; row 4i+5 is handed over once the copies AHEAD rows on are
// issued, into the slot of row 4i-1, which the block before frees. Every wait is
// bounded and no role waits at a CTA barrier inside the loop.
constexpr int PRODUCERS = 64;
constexpr int EPI_WARPS = 8;
constexpr int CONV_THREADS = EPI_WARPS * 32 + 32 + PRODUCERS;

struct ConvItem {
    int b, x0, y0, nout;  // image, first pixel and row, output rows (nout + 2 staged rows from y0 - 1)
};
__device__ __forceinline__ ConvItem conv_item(const ConvLaunch& a, int k) {
    const int segs = a.W / 128, runs = (a.H + a.rows - 1) / a.rows;
    ConvItem it;
    it.x0 = k % segs * 128;
    it.y0 = k / segs % runs * a.rows;
    it.b = k / segs / runs;
    it.nout = min(a.rows, a.H - it.y0);
    return it;
}

template <int CIN, int COUT, int EPI>
__global__ void __launch_bounds__(CONV_THREADS, 2) conv3x3_kernel(ConvLaunch a) {
    using L = ConvSmem<CIN, COUT>;
    constexpr int KSTEPS = CIN / 16;
    constexpr uint32_t TCOLS = (uint32_t)L::TCOLS;
    constexpr int NRING = L::NRING, AHEAD = L::AHEAD;
    extern __shared__ __align__(1024) uint8_t smem[];
    __shared__ __align__(8) uint64_t full[NRING], rowfree[NRING], tfull[2], tempty[2];
    __shared__ uint32_t tmem_slot;

    const int tid = threadIdx.x, lane = tid & 31;
    const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);  // the same in all lanes, for the compiler too
    const int items = a.batch * ((a.H + a.rows - 1) / a.rows) * (a.W / 128);
    const uint32_t s_w = smem_addr(smem);
    const uint32_t s_ring = s_w + L::OFF_RING;
    float* sbias = reinterpret_cast<float*>(smem + L::OFF_BIAS);

    for (int i = tid; i < L::WBYTES / 16; i += CONV_THREADS)
        cp_async16(s_w + i * 16, reinterpret_cast<const uint8_t*>(a.wimg) + (size_t)i * 16);
    if (EPI != EPI_MASK && tid < COUT) sbias[tid] = a.bias[tid];
    cp_async_wait_all();
    fence_async_smem();
    if (tid == 0) {
        for (int i = 0; i < NRING; ++i) {
            mbar_init(smem_addr(&full[i]), PRODUCERS);
            mbar_init(smem_addr(&rowfree[i]), 1);
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(smem_addr(&tfull[i]), 1);
            mbar_init(smem_addr(&tempty[i]), EPI_WARPS * 32);
        }
    }
    if (warp == 0) tmem_alloc(smem_addr(&tmem_slot), TCOLS);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = __shfl_sync(0xffffffffu, tmem_slot, 0);
    auto slot_addr = [&](int slot) { return s_ring + (uint32_t)(slot * L::SLOT); };

    int ok = 1;
    if (warp > EPI_WARPS) {
        // producers: input row y0 - 1 + rr of the item; a thread copies the same
        // 16-byte pieces of every row
        constexpr int PLANES = CIN / 8, PIECES = SLOTS * PLANES, PER = (PIECES + PRODUCERS - 1) / PRODUCERS;
        RingPos put, give;  // the next slot to fill; the next to hand over
        int filled = 0, given = 0;
        for (int k = blockIdx.x; k < items && ok; k += gridDim.x) {
            const ConvItem it = conv_item(a, k);
            uint32_t src[PER];
#pragma unroll
            for (int u = 0; u < PER; ++u) {
                const int t = u * PRODUCERS + tid - (EPI_WARPS + 1) * 32, sl = t / PLANES, j = t - sl * PLANES;
                int xx = it.x0 - 1 + sl;
                if (xx < 0) xx += a.W;
                if (xx >= a.W) xx -= a.W;
                src[u] = (uint32_t)(xx * CIN + j * 8);
            }
            int yy = it.y0 == 0 ? a.H - 1 : it.y0 - 1;
            for (int rr = 0; rr < it.nout + 2; ++rr) {
                if (filled >= NRING && !mbar_wait(smem_addr(&rowfree[put.slot]), put.parity ^ 1u)) {
                    ok = 0;
                    break;
                }
                const uint16_t* row = a.x + ((size_t)it.b * a.H + yy) * (size_t)a.W * CIN;
                if (++yy == a.H) yy = 0;
                const uint32_t slot = slot_addr(put.slot);
#pragma unroll
                for (int u = 0; u < PER; ++u) {
                    const int t = u * PRODUCERS + tid - (EPI_WARPS + 1) * 32, sl = t / PLANES, j = t - sl * PLANES;
                    if (u + 1 < PER || t < PIECES) cp_async16(slot + (uint32_t)(j * PLANE + sl * 16), row + src[u]);
                }
                cp_async_commit();
                put.advance(NRING);
                if (++filled > AHEAD) {  // that row's copies have landed: hand it over
                    cp_async_wait_group<AHEAD>();
                    fence_async_smem();
                    mbar_arrive_cta(smem_addr(&full[give.slot]));
                    give.advance(NRING);
                    ++given;
                }
            }
        }
        if (ok) {
            cp_async_wait_group<0>();
            fence_async_smem();
            for (; given < filled; ++given) {
                mbar_arrive_cta(smem_addr(&full[give.slot]));
                give.advance(NRING);
            }
        }
    } else if (warp == EPI_WARPS) {
        const bool leader = elect_one();
        // MMA issuer: output row r of a block reads its staged rows r, r+1, r+2
        RingPos top;           // the slot of the block's first staged row
        int blk = 0;           // blocks issued
        for (int k = blockIdx.x; k < items && ok; k += gridDim.x) {
            const int nout = conv_item(a, k).nout;
            for (int done = 0; done < nout && ok; done += CONV_ROWS, ++blk) {
                const int nb = min(CONV_ROWS, nout - done);
                const bool last = done + nb == nout;
                if (blk >= 2 && !__all_sync(0xffffffffu, mbar_wait(smem_addr(&tempty[blk & 1]), ((blk >> 1) - 1) & 1))) ok = 0;
                const uint32_t d = tmem + (uint32_t)((blk & 1) * CONV_ROWS * COUT);
                RingPos at = top;
                for (int m = 0; m < nb + 2 && ok; ++m) {
                    // staged row m, of output rows r0 .. r1
                    if ((done == 0 || m >= 2) && !__all_sync(0xffffffffu, mbar_wait(smem_addr(&full[at.slot]), at.parity))) {
                        ok = 0;
                        break;
                    }
                    tc_fence_after();
                    const int r0 = max(0, m - 2), r1 = min(m, nb - 1);
                    // descriptors advance by (bytes >> 4) in their start-address field
                    const uint64_t ad0 = umma_desc(slot_addr(at.slot), PLANE, 128);
                    const uint64_t bd0 = umma_desc(s_w + (uint32_t)((2 - m + r0) * COUT * 16), 3 * COUT * 16, 128);
                    // row m's accumulator starts with its first product
                    const int old = min(r1 + 1, m) - r0;
#pragma unroll
                    for (int q = 0; q < 3 * KSTEPS; ++q) {
                        const int dx = q / KSTEPS, ks = q % KSTEPS;
                        const uint64_t ad = ad0 + (uint64_t)(dx + 2 * ks * (PLANE >> 4));
                        const uint64_t bd = bd0 + (uint64_t)((dx * L::PLANES + 2 * ks) * 3 * COUT);
                        if (q == 0) {
                            if (old > 0 && leader) mma_bf16(d + r0 * COUT, ad, bd, idesc_bf16(128, old * COUT), 1u);
                            if (r1 == m && leader) mma_bf16(d + m * COUT, ad, bd + old * COUT, idesc_bf16(128, COUT), 0u);
                        } else {
                            if (leader) mma_bf16(d + r0 * COUT, ad, bd, idesc_bf16(128, (r1 - r0 + 1) * COUT), 1u);
                        }
                    }
                    if ((m < CONV_ROWS || last) && leader) mma_commit(smem_addr(&rowfree[at.slot]));  // its last reader
                    at.advance(NRING);
                    if (m < CONV_ROWS || last) top = at;
                }
                if (ok && leader) mma_commit(smem_addr(&tfull[blk & 1]));
            }
        }
        __syncwarp();
    } else {
        // epilogue warps: TMEM lanes 32*(warp%4) .. + 31 = pixels, rows warp/4, warp/4 + 2
        const int quarter = warp & 3, half = warp >> 2;
        const uint32_t lane_base = tmem + ((uint32_t)(quarter * 32) << 16);
        using E = RowEpilogue<COUT, EPI>;
        E epi;
        uint8_t* stage = smem + L::OFF_OUT + warp * E::BYTES;
        // the warp's first pixel of row y of an item
        auto pixel = [&](const ConvItem& it, int y) { return ((size_t)it.b * a.H + it.y0 + y) * a.W + it.x0 + quarter * 32; };
        // first pixel of the warp's first row of item k, if there is one
        auto first = [&](int k, size_t otherwise) {
            if (k >= items) return otherwise;
            const ConvItem it = conv_item(a, k);
            return half < it.nout ? pixel(it, half) : otherwise;
        };
        int blk = 0;
        size_t held = first(blockIdx.x, 0);  // the pixels whose mask is in registers
        epi.prefetch(a, held, lane);
        for (int k = blockIdx.x; k < items && ok; k += gridDim.x) {
            const ConvItem it = conv_item(a, k);
            for (int done = 0; done < it.nout; done += CONV_ROWS, ++blk) {
                // the TMEM load below is warp-aligned: the warp decides together
                if (!__all_sync(0xffffffffu, mbar_wait(smem_addr(&tfull[blk & 1]), (blk >> 1) & 1))) {
                    ok = 0;
                    break;
                }
                tc_fence_after();
                const int nb = min(CONV_ROWS, it.nout - done);
                for (int r = half; r < nb; r += 2) {
                    const size_t pix0 = pixel(it, done + r);
                    float v[COUT];
                    tmem_load<COUT>(lane_base + (uint32_t)(((blk & 1) * CONV_ROWS + r) * COUT), v);
                    uint32_t bits = 0;
                    if (EPI == EPI_MASK) {
                        if (held != pix0) epi.prefetch(a, pix0, lane);
                        bits = epi.mask_bits(lane);
                        held = done + r + 2 < it.nout ? pix0 + 2 * (size_t)a.W : first(k + gridDim.x, pix0);
                        epi.prefetch(a, held, lane);
                    }
                    if (EPI != EPI_BIAS_OUT) {  // the buffer's last copy has been read
                        if (lane == 0) bulk_wait_read<0>();
                        __syncwarp();
                    }
                    epi.finish(a, pix0, v, bits, stage, sbias, lane);
                }
                tc_fence_before();
                mbar_arrive_cta(smem_addr(&tempty[blk & 1]));
            }
        }
        if (lane == 0) bulk_wait_read<0>();
    }
    cp_async_wait_all();
    ok = __syncthreads_and(ok);
    if (!ok && tid == 0) atomicExch(a.err, 1);
    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        tc_fence_after();
        tmem_dealloc(tmem, TCOLS);
    }
}

// ---------------------------------------------------------------------------
// weight gradient
// ---------------------------------------------------------------------------
// Both operands are MN-major: A[m][k] = x with m = (row, channel) and
// k = pixel, B[k][n] = dy with n = (row, output channel). Staged as 8-channel planes
// (16 bytes per pixel slot) they are the canonical MN-major no-swizzle layout:
// a core matrix is 8 pixels (K, 16 B apart) of 8 channels (MN, contiguous); K
// core matrices are 128 B apart (LBO), MN core matrices one plane apart (SBO).
// With the staged rows of a block one after the other, the 16 MN core
// matrices of an M = 128 operand starting at x row i are rows i .. i + 128/CIN - 1,
// and those of an N = 2 COUT operand dy rows i and i + 1: with a the x row and b the
// dy row of the product, a - b = 0, 1, 2 are the taps dy = -1, 0, 1 (the rest is
// discarded). The tap dx moves A's start by one 16-byte pixel slot.
// Bias gradient: an all-ones A against all the dy rows of the block, N = 256
// (COUT = 32). A block is 26 MMAs where one dy row at a time took 64.
// Planes are an odd number of 16-byte slots apart, so that the core matrices of an
// operand do not share banks (little matters: 182 to 176 us at 32 x 32 channels,
// 512^2, batch 16, together with bias MMAs over all rows instead of four).
// TMEM starts at zero: an odd last row's MMAs write the first dy row's columns alone.
//
// Staging: cp.async, whole 64-byte pixels per four lanes. (TMA boxes of 8 channels x 34
// pixels x planes read L2 in 16-byte pieces: 2.1 GB of sectors for 0.64 GB.)
constexpr int WG_ROWS = 8;           // output rows per block
constexpr int WG_XROWS = WG_ROWS + 2;
constexpr int WG_PX = 32;            // output pixels per block (one K segment)
constexpr int WG_SLOTS = 34;         // x pixels: x0-1 .. x0+32
constexpr int WG_XPLANE = 35 * 16;
constexpr int WG_DPLANE = 33 * 16;
constexpr int WG_NBUF = 3;           // blocks in the shared-memory ring
constexpr int WG_LAG = 1;            // blocks whose copies are in flight behind the newest
constexpr int WG_ONES = 16 * 256;    // all-ones A operand: 16 MN x 2 K core matrices
constexpr int WG_THREADS = 512;
constexpr int WG_PRODUCERS = WG_THREADS - 32;

template <int CIN, int COUT>
struct WgSmem {
    static constexpr int XROW = (CIN / 8) * WG_XPLANE;  // bytes per staged x row
    static constexpr int DROW = (COUT / 8) * WG_DPLANE;
    static constexpr int XBYTES = WG_XROWS * XROW;
    static constexpr int DBYTES = WG_ROWS * DROW;
    static constexpr int BUF = (XBYTES + DBYTES + 127) / 128 * 128;
    static constexpr int OFF_ONES = WG_NBUF * BUF;
    // one CTA on an SM: with 32 channels it takes all 512 TMEM columns
    static constexpr int BYTES = OFF_ONES + WG_ONES > 116 * 1024 ? OFF_ONES + WG_ONES : 116 * 1024;
    static constexpr int BIAS_COL = 6 * COUT;           // columns before: 2 * COUT per dx
    static constexpr int COLS = BIAS_COL + WG_ROWS * COUT;
    static constexpr uint32_t TCOLS = tmem_cols(COLS);
    // an M = 128 operand at the last pair's row ends inside the allocation
    static_assert((WG_ROWS - 2 + 128 / CIN) * XROW <= BUF + WG_ONES, "A operand");
};

// Instruction descriptor of kind::f16 with both operands MN-major.
__host__ __device__ constexpr uint32_t idesc_bf16_mn(int m, int n) {
    return idesc_bf16(m, n) | (1u << 15) | (1u << 16);
}

// A block of the CTA's range: 32-pixel segments fastest, then rows, then images.
struct WgBlock {
    int b, y0, x0, rows;
    __device__ __forceinline__ WgBlock(const WgradLaunch& a, long long blk) {
        const int segs = a.W / WG_PX, yblocks = (a.H + WG_ROWS - 1) / WG_ROWS;
        x0 = (int)(blk % segs) * WG_PX;
        y0 = (int)(blk / segs % yblocks) * WG_ROWS;
        b = (int)(blk / segs / yblocks);
        rows = min(WG_ROWS, a.H - y0);
    }
    __device__ __forceinline__ void advance(const WgradLaunch& a) {
        x0 += WG_PX;
        if (x0 < a.W) return;
        x0 = 0;
        y0 += WG_ROWS;
        if (y0 >= a.H) {
            y0 = 0;
            ++b;
        }
        rows = min(WG_ROWS, a.H - y0);
    }
};

// Copies of a block by producer thread pt: x rows y0 - 1 .. y0 + rows, dy rows y0 ..
template <int CIN, int COUT>
__device__ __forceinline__ void wg_stage(const WgradLaunch& a, const WgBlock& k, uint32_t buf, int pt) {
    using L = WgSmem<CIN, COUT>;
    constexpr int XP = CIN / 8, DP = COUT / 8;
    const size_t img = (size_t)k.b * a.H;
    for (int u = pt; u < (k.rows + 2) * WG_SLOTS * XP; u += WG_PRODUCERS) {
        const int r = u / (WG_SLOTS * XP), p = u - r * (WG_SLOTS * XP), sl = p / XP, j = p % XP;
        int xx = k.x0 - 1 + sl;
        if (xx < 0) xx += a.W;
        if (xx >= a.W) xx -= a.W;
        int yy = k.y0 - 1 + r;
        if (yy < 0) yy += a.H;
        if (yy >= a.H) yy %= a.H;
        cp_async16(buf + (uint32_t)(r * L::XROW + j * WG_XPLANE + sl * 16),
                   a.x + ((img + yy) * (size_t)a.W + xx) * CIN + j * 8);
    }
    const uint16_t* dy = a.dy + ((img + k.y0) * (size_t)a.W + k.x0) * COUT;
    for (int u = pt; u < k.rows * WG_PX * DP; u += WG_PRODUCERS) {
        const int r = u / (WG_PX * DP), p = u % (WG_PX * DP), sl = p / DP, j = p % DP;
        cp_async16(buf + (uint32_t)(L::XBYTES + r * L::DROW + j * WG_DPLANE + sl * 16), dy + (size_t)r * a.W * COUT + p * 8);
    }
}

// One CTA per SM. Warps 1-15 are the producers; lane 0 of warp 0 issues the MMAs.
// full[b] takes one arrival from every producer thread for every block (after its
// copies landed, WG_LAG blocks later) and says buffer b
// holds a block; empty[b] (the MMAs' commit) says the tensor cores are done with
// it. Every producer thread waits on empty and arrives on full for every block,
// so no thread is ever more than one phase away from a barrier it waits on (a
// parity wait needs that), and no producer waits for another, so a wait that
// runs out cannot strand the rest.
// 32 x 32 channels, 512^2, batch 16: 124 us, 185 with TMA staging and one dy row per MMA
// (when the MMAs took 181 us and the staging 172 by themselves; now the MMAs take 98).
// Bound by staging through L1, 0.6 GB: 15 producer warps (7: 142 us, 23: 130); three
// buffers leave L1 more room than four (131 us; with 7 warps 148, five 160).
template <int CIN, int COUT>
__global__ void __launch_bounds__(WG_THREADS) wgrad_kernel(WgradLaunch a) {
    using L = WgSmem<CIN, COUT>;
    constexpr int MPAD = 9 * CIN + 1;
    extern __shared__ __align__(1024) uint8_t smem[];
    __shared__ __align__(8) uint64_t full[WG_NBUF], empty[WG_NBUF];
    __shared__ uint32_t tmem_slot;

    const int tid = threadIdx.x, lane = tid & 31;
    const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);  // the same in all lanes, for the compiler too
    const long long total = (long long)a.batch * ((a.H + WG_ROWS - 1) / WG_ROWS) * (a.W / WG_PX);
    const long long k_begin = (long long)blockIdx.x * a.units_per_cta;
    const int nk = (int)max(0ll, min(total, k_begin + a.units_per_cta) - k_begin);
    const uint32_t s0 = smem_addr(smem);
    float* part = a.partials + (size_t)blockIdx.x * MPAD * COUT;

    {  // the all-ones operand of the bias MMAs (BF16 1.0)
        uint4* o = reinterpret_cast<uint4*>(smem + L::OFF_ONES);
        for (int i = tid; i < WG_ONES / 16; i += WG_THREADS) o[i] = make_uint4(0x3F803F80u, 0x3F803F80u, 0x3F803F80u, 0x3F803F80u);
    }
    fence_async_smem();
    if (tid == 0) {
        for (int i = 0; i < WG_NBUF; ++i) {
            mbar_init(smem_addr(&full[i]), WG_PRODUCERS);
            mbar_init(smem_addr(&empty[i]), 1);
        }
    }
    if (warp == 0) tmem_alloc(smem_addr(&tmem_slot), L::TCOLS);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = __shfl_sync(0xffffffffu, tmem_slot, 0);
    const uint32_t lanes = tmem + ((uint32_t)((warp & 3) * 32) << 16);
    if (warp < 4) {
#pragma unroll 4
        for (int c = 0; c < L::COLS; c += 16) tmem_zero16(lanes + c);
        tmem_wait_st();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();

    int ok = 1;
    if (warp > 0) {
        const int pt = tid - 32;
        WgBlock blk(a, k_begin);
        for (int k = 0; k < nk; ++k, blk.advance(a)) {
            const int bsel = k % WG_NBUF;
            if (k >= WG_NBUF && !mbar_wait(smem_addr(&empty[bsel]), ((k / WG_NBUF) - 1) & 1)) {
                ok = 0;
                break;
            }
            wg_stage<CIN, COUT>(a, blk, s0 + (uint32_t)(bsel * L::BUF), pt);
            cp_async_commit();
            if (k >= WG_LAG) {
                cp_async_wait_group<WG_LAG>();
                fence_async_smem();
                mbar_arrive_cta(smem_addr(&full[(k - WG_LAG) % WG_NBUF]));
            }
        }
        if (ok) {
            cp_async_wait_group<0>();
            fence_async_smem();
            for (int k = max(0, nk - WG_LAG); k < nk; ++k) mbar_arrive_cta(smem_addr(&full[k % WG_NBUF]));
        }
    } else {
        const bool leader = elect_one();
        const uint64_t ones = umma_desc(s0 + (uint32_t)L::OFF_ONES, 128, 256);
        WgBlock blk(a, k_begin);
        for (int k = 0; k < nk; ++k, blk.advance(a)) {
            const int bsel = k % WG_NBUF;
            const uint32_t buf = s0 + (uint32_t)(bsel * L::BUF);
            if (!__all_sync(0xffffffffu, mbar_wait(smem_addr(&full[bsel]), (k / WG_NBUF) & 1))) {
                ok = 0;
                break;
            }
            tc_fence_after();
            const int rows = blk.rows;
            // descriptors advance by (bytes >> 4) in their start-address field
            const uint64_t a0 = umma_desc(buf, 128, WG_XPLANE);
            const uint64_t b0 = umma_desc(buf + (uint32_t)L::XBYTES, 128, WG_DPLANE);
            for (int i = 0; i < rows; i += 2) {
                const uint32_t idesc = idesc_bf16_mn(128, i + 1 < rows ? 2 * COUT : COUT);
#pragma unroll
                for (int kk = 0; kk < WG_PX / 16; ++kk) {
                    const uint64_t bd = b0 + (uint64_t)((i * L::DROW + 16 * kk * 16) >> 4);
#pragma unroll
                    for (int dx = 0; dx < 3; ++dx) {
                        const uint64_t ad = a0 + (uint64_t)((i * L::XROW + (16 * kk + dx) * 16) >> 4);
                        if (leader) mma_bf16(tmem + (uint32_t)(dx * 2 * COUT), ad, bd, idesc, 1u);
                    }
                }
            }
#pragma unroll
            for (int kk = 0; kk < WG_PX / 16; ++kk)
                if (leader)
                    mma_bf16(tmem + (uint32_t)L::BIAS_COL, ones, b0 + (uint64_t)((16 * kk * 16) >> 4),
                             idesc_bf16_mn(128, rows * COUT), 1u);
            if (leader) mma_commit(smem_addr(&empty[bsel]));
        }
    }
    cp_async_wait_all();
    __syncwarp();
    ok = __syncthreads_and(ok);
    if (ok && nk > 0) {
        const int last = nk - 1;
        ok = __syncthreads_and(mbar_wait(smem_addr(&empty[last % WG_NBUF]), (last / WG_NBUF) & 1));
        if (ok) {
            tc_fence_after();
            // TMEM lane m = (x row a, channel ci), columns dx * 2 COUT + b * COUT + co:
            // tap row dyi is a = dyi, b = 0 plus a = dyi + 1, b = 1, which goes
            // through shared memory (the ring is free)
            float* other = reinterpret_cast<float*>(smem);  // [dyi][ci][co]
            const int m = warp * 32 + lane, xr = m / CIN, ci = m % CIN;
            for (int dx = 0; dx < 3; ++dx) {
                float v[COUT];
                if (warp * 32 < 4 * CIN) {  // warps of x rows 0 .. 3
                    tmem_load<COUT>(lanes + (uint32_t)((dx * 2 + 1) * COUT), v);
                    if (xr >= 1 && xr <= 3) {
#pragma unroll
                        for (int c = 0; c < COUT; ++c) other[((xr - 1) * CIN + ci) * (COUT + 1) + c] = v[c];
                    }
                }
                __syncthreads();
                if (warp * 32 < 4 * CIN) {
                    tmem_load<COUT>(lanes + (uint32_t)(dx * 2 * COUT), v);
                    if (xr < 3) {
                        float* row = part + (size_t)((xr * 3 + dx) * CIN + ci) * COUT;
#pragma unroll
                        for (int c = 0; c < COUT; ++c) row[c] = v[c] + other[(xr * CIN + ci) * (COUT + 1) + c];
                    }
                }
                __syncthreads();
            }
            if (warp == 0) {  // every lane the same: columns (dy row, channel)
                float s[COUT] = {};
                for (int r = 0; r < WG_ROWS; ++r) {
                    float v[COUT];
                    tmem_load<COUT>(tmem + (uint32_t)(L::BIAS_COL + r * COUT), v);
#pragma unroll
                    for (int c = 0; c < COUT; ++c) s[c] += v[c];
                }
                if (lane == 0) {
#pragma unroll
                    for (int c = 0; c < COUT; ++c) part[(size_t)9 * CIN * COUT + c] = s[c];
                }
            }
        }
    } else if (ok) {
        for (int i = tid; i < MPAD * COUT; i += WG_THREADS) part[i] = 0.0f;
    }
    if (!ok && tid == 0) atomicExch(a.err, 1);
    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        tc_fence_after();
        tmem_dealloc(tmem, L::TCOLS);
    }
}

__global__ void weight_image_kernel(const float* __restrict__ w, int cin, int cout, int transpose,
                                    uint16_t* __restrict__ img) {
    const int kcin = transpose ? cout : cin, kcout = transpose ? cin : cout;
    const int total = 9 * kcin * kcout;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= total) return;
    // img[(((dx*(kcin/8) + j)*3 + 2 - dy)*kcout + n)*8 + e] holds kernel weight
    // (tap 3*dy + dx, out n, in 8j+e)
    const int e = i & 7;
    const int r = i >> 3;
    const int n = r % kcout;
    const int r2 = r / kcout;
    const int j = r2 / 3 % (kcin / 8);
    const int dx = r2 / 3 / (kcin / 8);
    const int tap = 3 * (2 - r2 % 3) + dx;
    const int kc = 8 * j + e;
    const float v = transpose ? w[((size_t)(8 - tap) * cout + kc) * cin + n] : w[((size_t)tap * cout + n) * cin + kc];
    const __nv_bfloat16 h = __float2bfloat16_rn(v);
    img[i] = *reinterpret_cast<const uint16_t*>(&h);
}

// Sums of the CTAs' partials: a warp per 32 consecutive values of their layout
// ([row m][cout]: coalesced) and every RW_WARPS-th partial, then the warps' sums in
// order. (One thread per value in dw's order, all partials: 53 us for 304 partials
// of 32 x 32 channels, 37 blocks of scattered loads; bound now by reading 11 MB.)
constexpr int RW_WARPS = 8;
__global__ void __launch_bounds__(RW_WARPS * 32) reduce_wgrad_kernel(const float* __restrict__ partials, int grid, int cin,
                                                                     int cout, int mpad, float* __restrict__ dw,
                                                                     float* __restrict__ db) {
    __shared__ float sums[RW_WARPS][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int i = blockIdx.x * 32 + lane, n = mpad * cout;
    float s = 0.0f;
    if (i < n) {
#pragma unroll 4
        for (int g = warp; g < grid; g += RW_WARPS) s += partials[(size_t)g * n + i];
    }
    sums[warp][lane] = s;
    __syncthreads();
    if (warp != 0 || i >= n) return;
#pragma unroll
    for (int w = 1; w < RW_WARPS; ++w) s += sums[w][lane];
    const int m = i / cout, co = i - m * cout;
    if (m < 9 * cin) {  // dw[tap][co][ci]
        const int tap = m / cin, ci = m - tap * cin;
        dw[((size_t)tap * cout + co) * cin + ci] = s;
    } else {
        db[co] = s;
    }
}

template <int CIN, int COUT, int EPI>
int launch_conv_t(const ConvLaunch& a0, cudaStream_t s) {
    using L = ConvSmem<CIN, COUT>;
    const int attr = picgb::opt_in_dynamic_smem((const void*)conv3x3_kernel<CIN, COUT, EPI>, L::BYTES);
    if (attr != PIC_OK) return attr;
    // Rows of an item: a CTA stages two more than it puts out and computes, so long
    // items are better, unless they leave CTAs without one.
    const long long segs = (long long)a0.batch * (a0.W / 128), slots = 152 * L::CTAS;
    ConvLaunch a = a0;
    long long best = 0, items = 0;
    for (int rows = CONV_ROWS; rows <= 64; rows += CONV_ROWS) {
        const long long n = segs * ((a.H + rows - 1) / rows), cost = (n + slots - 1) / slots * (rows + 3);
        if (best == 0 || cost < best) {
            best = cost;
            items = n;
            a.rows = rows;
        }
        if (rows >= a.H) break;
    }
    if (items > INT_MAX) return picgb::fail(PIC_ERR_ARG, "convolution: too many pixels");
    conv3x3_kernel<CIN, COUT, EPI><<<(unsigned)(items < slots ? items : slots), CONV_THREADS, L::BYTES, s>>>(a);
    const cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? PIC_OK : picgb::cuda_fail(e, "conv3x3_kernel launch");
}

template <int CIN, int COUT>
int launch_wgrad_t(const WgradLaunch& a, int grid, cudaStream_t s) {
    using L = WgSmem<CIN, COUT>;
    const int attr = picgb::opt_in_dynamic_smem((const void*)wgrad_kernel<CIN, COUT>, L::BYTES);
    if (attr != PIC_OK) return attr;
    wgrad_kernel<CIN, COUT><<<grid, WG_THREADS, L::BYTES, s>>>(a);
    const cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? PIC_OK : picgb::cuda_fail(e, "wgrad_kernel launch");
}

template <int CIN, int COUT>
int launch_conv_epi(const ConvLaunch& a, int epi, cudaStream_t s) {
    switch (epi) {
        case EPI_BIAS_RELU:
            return launch_conv_t<CIN, COUT, EPI_BIAS_RELU>(a, s);
        case EPI_BIAS_OUT:
            return launch_conv_t<CIN, COUT, EPI_BIAS_OUT>(a, s);
        case EPI_MASK:
            return launch_conv_t<CIN, COUT, EPI_MASK>(a, s);
    }
    return picgb::fail(PIC_ERR_ARG, "unknown convolution epilogue");
}

}  // namespace

int build_weight_image(const float* w_math, int cin, int cout, int transpose, uint16_t* img, cudaStream_t s) {
    const int total = 9 * cin * cout;
    weight_image_kernel<<<(total + 255) / 256, 256, 0, s>>>(w_math, cin, cout, transpose, img);
    const cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? PIC_OK : picgb::cuda_fail(e, "weight_image_kernel launch");
}

int launch_conv(const ConvLaunch& a, int kcin, int kcout, int epi, cudaStream_t s) {
    if (a.W % 128 != 0 || a.W <= 0 || a.H <= 0 || a.batch <= 0)
        return picgb::fail(PIC_ERR_ARG, "convolution needs W a multiple of 128 and H, batch > 0");
    if (kcin == 16 && kcout == 16) return launch_conv_epi<16, 16>(a, epi, s);
    if (kcin == 16 && kcout == 32) return launch_conv_epi<16, 32>(a, epi, s);
    if (kcin == 32 && kcout == 16) return launch_conv_epi<32, 16>(a, epi, s);
    if (kcin == 32 && kcout == 32) return launch_conv_epi<32, 32>(a, epi, s);
    return picgb::fail(PIC_ERR_ARG, "convolution channels must be 16 or 32");
}

int wgrad_grid(long long units) {
    const long long g = units < 152 ? units : 152;
    return (int)(g < 1 ? 1 : g);
}

int launch_wgrad(const WgradLaunch& a, int cin, int cout, int grid, cudaStream_t s) {
    if (a.W % WG_PX != 0 || a.W <= 0 || a.H <= 0 || a.batch <= 0 || grid <= 0)
        return picgb::fail(PIC_ERR_ARG, "weight gradient needs W a multiple of 32");
    if (cin == 16 && cout == 16) return launch_wgrad_t<16, 16>(a, grid, s);
    if (cin == 16 && cout == 32) return launch_wgrad_t<16, 32>(a, grid, s);
    if (cin == 32 && cout == 16) return launch_wgrad_t<32, 16>(a, grid, s);
    if (cin == 32 && cout == 32) return launch_wgrad_t<32, 32>(a, grid, s);
    return picgb::fail(PIC_ERR_ARG, "convolution channels must be 16 or 32");
}

int reduce_wgrad(const float* partials, int grid, int cin, int cout, float* dw, float* db, cudaStream_t s) {
    const int total = wgrad_mpad(cin) * cout;
    reduce_wgrad_kernel<<<(total + 31) / 32, RW_WARPS * 32, 0, s>>>(partials, grid, cin, cout, wgrad_mpad(cin), dw, db);
    const cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? PIC_OK : picgb::cuda_fail(e, "reduce_wgrad_kernel launch");
}

}  // namespace picnn
