// The last stage of the diagnostics, run by one block of RED_THREADS threads: a kernel
// of its own (fields.cu), or, in a time step, one more block of the deposit's last
// kernel (deposit.cu).
#pragma once

namespace picgb {

constexpr int RED_THREADS = 256;

// Block sums of K values at once (one exchange); valid in thread 0.
template <int K>
__device__ __forceinline__ void block_sums(double (&v)[K]) {
    __shared__ double ws[K][RED_THREADS / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int k = 0; k < K; ++k) v[k] = __dadd_rn(v[k], __shfl_down_sync(0xffffffffu, v[k], o));
    if (lane == 0)
#pragma unroll
        for (int k = 0; k < K; ++k) ws[k][warp] = v[k];
    __syncthreads();
    if (threadIdx.x == 0)
#pragma unroll
        for (int k = 0; k < K; ++k) {
            double s = 0.0;
            for (int w = 0; w < RED_THREADS / 32; ++w) s = __dadd_rn(s, ws[k][w]);
            v[k] = s;
        }
}
__device__ __forceinline__ double block_sum(double v) {
    double a[1] = {v};
    block_sums(a);
    return a[0];
}

// The last stage of the diagnostics in one block: up to three partial sums
// (kinetic, rho, E^2; rho and E^2 interleaved), the particle set's charge sums,
// and, with a history, the step's pic_diag from them (the formulas of
// read_diagnostics) and the step counter.
struct FinalArgs {
    const double* ke;    // null: r[3] already holds the kinetic energy
    const double* grid;  // pairs (sum rho, sum E^2)
    int ke_count, grid_count;
    double* r;           // red_out
    double vol;
    double* hist;
    int* step;
    int steps;
};

__device__ __forceinline__ void diag_block(const FinalArgs& a) {
    double ke = 0.0, rho = 0.0, ee = 0.0;
    if (a.ke)
        for (int i = threadIdx.x; i < a.ke_count; i += RED_THREADS) ke = __dadd_rn(ke, a.ke[i]);
    for (int i = threadIdx.x; i < a.grid_count; i += RED_THREADS) {
        const double2 g = reinterpret_cast<const double2*>(a.grid)[i];
        rho = __dadd_rn(rho, g.x);
        ee = __dadd_rn(ee, g.y);
    }
    double sums[3] = {ke, rho, ee};
    block_sums(sums);
    if (threadIdx.x != 0) return;
    ke = sums[0];
    rho = sums[1];
    ee = sums[2];
    double* r = a.r;
    r[1] = r[8];
    r[6] = r[9];
    r[2] = rho;
    if (a.ke) r[3] = __dmul_rn(0.5, ke);
    r[4] = ee;
    if (!a.hist) return;
    const int s = *a.step;
    if (s < a.steps) {
        double* d = a.hist + (size_t)s * 6;
        const double total_charge = r[1];
        const double integrated = __dmul_rn(rho, a.vol);
        const double den = r[6] > 1e-12 ? r[6] : 1e-12;
        const double kin = r[3];
        const double fe = __dmul_rn(__dmul_rn(0.5, ee), a.vol);
        d[0] = __ddiv_rn(fabs(__dsub_rn(integrated, total_charge)), den);
        d[1] = total_charge;
        d[2] = integrated;
        d[3] = kin;
        d[4] = fe;
        d[5] = __dadd_rn(kin, fe);
    }
    *a.step = s + 1;
}

}  // namespace picgb
