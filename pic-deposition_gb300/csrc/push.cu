// Field gather and leapfrog push on the resident particles.
//
//  gather   = pic::gatherFieldsSoA (src/deposition/deposition.cpp:335-356): CIC
//             interpolation of Ex, Ey at the particle with the deposit's
//             weights, then v += -(q/m) * E * dt.
//  push     = pic::pushParticlesSoA (deposition.cpp:367-374): x += v * dt with
//             periodic wrap (Domain::wrapPosition, src/pic/domain.hpp:27-32).
//  fused    = gather then push in one pass over the particles (kick of step n
//             and drift of step n+1 in the reference's loop order,
//             src/pic/simulation.cpp:82-131): reads cell, offsets, v, q
//             (24 B) and writes cell, offsets, v (20 B) per particle.
//
// Positions stay cell-relative in FP32: r' = r + v*dt/dx, the integer part moves
// the cell key (wrapped) and the fraction stays in [0,1]. Operation order
// follows the reference:
//   e  = ((E00*(1-wx))*(1-wy) + (E10*wx)*(1-wy)) + (E01*(1-wx))*wy + (E11*wx)*wy
//   v  = v + ((-q/m)*e)*dt
// with E the FP32 copies of the FP64 fields. Compiled with --fmad=false, so the
// oracle reproduces every bit.
#include "pic_internal.cuh"

namespace picgb {

struct MoveArgs {
    double* ke_partial;  // KE: per-block sums of vx^2 + vy^2 after the gather
    uint32_t* cell;
    float *xr, *yr, *vx, *vy;
    const float* q;
    const float* m;  // null when every mass is 1
    const float* Exf;
    const float* Eyf;
    size_t n;
    int Nx, Ny;
    float dtf, dtdx, dtdy;
    float qc;  // nonzero: every particle's stored charge (the charge stream is not read)
    const DevStats* st;
};


// KE (with GATHER, every mass 1): the sum of vx^2 + vy^2 of the updated
// velocities in the arithmetic of fields.cu's sum_v2_partials (exact FP32
// squares, double-FP32 per thread, FP64 across the block in a fixed order),
// one partial per block (as many as the particles fill, at most MOVE_KE_BLOCKS): the time
// step's kinetic energy without another pass over the velocities.
// A thread takes two consecutive particles at a time: 8-byte loads and stores, and
// both particles' field reads in flight together. Bound by memory: 0.75 ms for 105 M
// particles on 1024^2 with gather, push and kinetic sums, 0.84 of the measured copy
// rate at 40 bytes per particle (0.80 with one at a time and the next one's values
// prefetched). Four at a time spread a warp's field reads over more cells: 10 % slower
// when the particles are out of order.
// Few particles are one wave of threads either way, and two per thread only lengthen each
// one's chain: NP = 1 there (not with the kinetic sums, whose chains would change).
template <int NP, bool GATHER, bool PUSH, bool KE = false>
__global__ void __launch_bounds__(256, 5) move_particles(MoveArgs a) {
    static_assert(NP == 2 || (NP == 1 && !KE), "");
    float ke_hi = 0.0f, ke_lo = 0.0f;
    const float maxq = load_maxq(a.st);
    const float inv_nx = 1.0f / (float)a.Nx;
    const size_t stride = (size_t)gridDim.x * blockDim.x, nq = (a.n + NP - 1) / NP;
    for (size_t qi = (size_t)blockIdx.x * blockDim.x + threadIdx.x; qi < nq; qi += stride) {
        const size_t p = qi * NP;
        const int cnt = a.n - p < NP ? (int)(a.n - p) : NP;
        uint32_t key[NP];
        float rx[NP], ry[NP], vx[NP], vy[NP];
        if constexpr (NP == 2) {  // the arrays are aligned and padded past the last particle
            const uint2 kv = *reinterpret_cast<const uint2*>(a.cell + p);
            const float2 xv = *reinterpret_cast<const float2*>(a.xr + p), yv = *reinterpret_cast<const float2*>(a.yr + p);
            const float2 uv = *reinterpret_cast<const float2*>(a.vx + p), wv = *reinterpret_cast<const float2*>(a.vy + p);
            key[0] = kv.x, key[1] = kv.y;
            rx[0] = xv.x, rx[1] = xv.y;
            ry[0] = yv.x, ry[1] = yv.y;
            vx[0] = uv.x, vx[1] = uv.y;
            vy[0] = wv.x, vy[1] = wv.y;
        } else {
            key[0] = a.cell[p];
            rx[0] = a.xr[p];
            ry[0] = a.yr[p];
            vx[0] = a.vx[p];
            vy[0] = a.vy[p];
        }
        int ix[NP], iy[NP];
#pragma unroll
        for (int k = 0; k < NP; ++k) {
            if (k >= cnt) key[k] = 0;  // past the end: any cell will do
            split_key(key[k], a.Nx, inv_nx, iy[k], ix[k]);
        }
        if constexpr (GATHER) {
            float e[NP][8];
#pragma unroll
            for (int k = 0; k < NP; ++k) {
                const int ixp = ix[k] + 1 == a.Nx ? 0 : ix[k] + 1, iyp = iy[k] + 1 == a.Ny ? 0 : iy[k] + 1;
                const size_t r0 = (size_t)iy[k] * a.Nx, r1 = (size_t)iyp * a.Nx;
                const size_t at[4] = {r0 + ix[k], r0 + ixp, r1 + ix[k], r1 + ixp};
#pragma unroll
                for (int m = 0; m < 4; ++m) {
                    e[k][m] = __ldg(a.Exf + at[m]);
                    e[k][4 + m] = __ldg(a.Eyf + at[m]);
                }
            }
#pragma unroll
            for (int k = 0; k < NP; ++k) {
                if (k < cnt) {
                    const float ex = interp_nodes(e[k][0], e[k][1], e[k][2], e[k][3], rx[k], ry[k]);
                    const float ey = interp_nodes(e[k][4], e[k][5], e[k][6], e[k][7], rx[k], ry[k]);
                    const float qf = (a.qc != 0.0f ? a.qc : a.q[p + k]) * maxq;
                    const float coef = a.m ? __fdiv_rn(-qf, a.m[p + k]) : -qf;
                    vx[k] = vx[k] + (coef * ex) * a.dtf;
                    vy[k] = vy[k] + (coef * ey) * a.dtf;
                    if constexpr (KE) ke_add(ke_hi, ke_lo, vx[k], vy[k]);
                }
            }
        }
        if constexpr (PUSH) {
#pragma unroll
            for (int k = 0; k < NP; ++k) {
                drift(rx[k], ix[k], vx[k], a.dtdx, a.Nx);
                drift(ry[k], iy[k], vy[k], a.dtdy, a.Ny);
                key[k] = (uint32_t)iy[k] * (uint32_t)a.Nx + (uint32_t)ix[k];
            }
        }
        if (NP == 2 && cnt == NP) {
            if constexpr (GATHER) {
                *reinterpret_cast<float2*>(a.vx + p) = make_float2(vx[0], vx[NP - 1]);
                *reinterpret_cast<float2*>(a.vy + p) = make_float2(vy[0], vy[NP - 1]);
            }
            if constexpr (PUSH) {
                *reinterpret_cast<float2*>(a.xr + p) = make_float2(rx[0], rx[NP - 1]);
                *reinterpret_cast<float2*>(a.yr + p) = make_float2(ry[0], ry[NP - 1]);
                *reinterpret_cast<uint2*>(a.cell + p) = make_uint2(key[0], key[NP - 1]);
            }
        } else {
            if constexpr (GATHER) {
                a.vx[p] = vx[0];
                a.vy[p] = vy[0];
            }
            if constexpr (PUSH) {
                a.xr[p] = rx[0];
                a.yr[p] = ry[0];
                a.cell[p] = key[0];
            }
        }
    }
    if constexpr (KE) {
        __shared__ double ws[8];
        double v = __dadd_rn((double)ke_hi, (double)ke_lo);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v = __dadd_rn(v, __shfl_down_sync(0xffffffffu, v, o));
        if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = v;
        __syncthreads();
        if (threadIdx.x == 0) {
            double t = 0.0;
            for (int w = 0; w < 8; ++w) t = __dadd_rn(t, ws[w]);
            a.ke_partial[blockIdx.x] = t;
        }
    }
}

// ke: with the gather and unit masses, also leave the kinetic sums of the
// updated velocities in c->ke_partials (c->ke_count blocks' sums).
int move(pic_ctx* c, double dt, bool gather, bool push, bool ke) {
    c->ke_ready = 0;
    if (c->n == 0) return PIC_OK;
    if (gather) PIC_TRY(ensure_fields(c));
    ke = ke && gather && !c->has_mass;
    MoveArgs a;
    a.ke_partial = c->ke_partials;
    a.cell = c->cell;
    a.xr = c->xr;
    a.yr = c->yr;
    a.vx = c->vx;
    a.vy = c->vy;
    a.q = c->q;
    a.m = c->has_mass ? c->m : nullptr;
    a.Exf = c->Exf;
    a.Eyf = c->Eyf;
    a.n = c->n;
    a.Nx = c->Nx;
    a.Ny = c->Ny;
    a.dtf = (float)dt;
    a.dtdx = (float)(dt / c->dx);
    a.dtdy = (float)(dt / c->dy);
    a.qc = c->qn_uniform;
    a.st = c->dstats;
    int sms = 148;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, c->device);
    const size_t filled = (c->n + 511) / 512;  // blocks of 256 threads, two particles each
    size_t blocks = filled;
    if (blocks > (size_t)sms * 32) blocks = (size_t)sms * 32;
    // the partition of the sums depends on the particle count alone; no more blocks
    // than the particles fill (4096 nearly empty blocks took 18 us at 65,536 particles)
    if (ke) blocks = filled < (size_t)MOVE_KE_BLOCKS ? filled : (size_t)MOVE_KE_BLOCKS;
    // One particle per thread up to the counts where two become as fast: 256 per SM for a
    // push alone, 4,096 where fields are gathered (262,144 particles out of order on 512^2,
    // gather: 10.3 us against 11.3; 1,001: 4.1 against 6.2).
    const bool one = !ke && c->n <= (size_t)sms * (gather ? 4096 : 256);
    if (one) blocks = (c->n + 255) / 256;
    auto launch = [&](auto kernel) { kernel<<<(unsigned)blocks, 256, 0, c->stream>>>(a); };
    prof_begin(c, gather && push ? "gather_push" : gather ? "gather" : "push");
    if (gather && push)
        launch(ke ? move_particles<2, true, true, true> : one ? move_particles<1, true, true> : move_particles<2, true, true>);
    else if (gather)
        launch(ke ? move_particles<2, true, false, true> : one ? move_particles<1, true, false> : move_particles<2, true, false>);
    else
        launch(one ? move_particles<1, false, true> : move_particles<2, false, true>);
    prof_end(c);
    PIC_TRY(check_launch(c, "move_particles"));
    if (push) c->sorted = 0;
    c->ke_ready = ke ? 1 : 0;
    c->ke_count = (int)blocks;
    return PIC_OK;
}

int move(pic_ctx* c, double dt, bool gather, bool push) { return move(c, dt, gather, push, false); }

}  // namespace picgb

using namespace picgb;

extern "C" {

int pic_gpu_gather(pic_ctx* c, double dt) {
    if (!c) return fail(PIC_ERR_ARG, "NULL context");
    PIC_CUDA_TRY(cudaSetDevice(c->device));
    return move(c, dt, true, false);
}

int pic_gpu_push(pic_ctx* c, double dt) {
    if (!c) return fail(PIC_ERR_ARG, "NULL context");
    PIC_CUDA_TRY(cudaSetDevice(c->device));
    return move(c, dt, false, true);
}

int pic_gpu_gather_push(pic_ctx* c, double dt) {
    if (!c) return fail(PIC_ERR_ARG, "NULL context");
    PIC_CUDA_TRY(cudaSetDevice(c->device));
    return move(c, dt, true, true);
}

}  // extern "C"
