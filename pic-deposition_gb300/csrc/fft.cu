// FP64 transforms of the FFT Poisson solve (pic::PoissonSolverFFT,
// src/pic/poisson_fft.cpp:45-94) for grids whose sides are powers of two from 8 to
// 2048: three kernels instead of a library's four and a pass over the spectrum.
//   fft_rows_forward: a row of nx real values each of two rows as one complex
//     transform (row 2p + i row 2p+1), separated into their nx/2 + 1 frequencies;
//   fft_columns: every frequency column: transform, the factor of each frequency
//     (fields.cu fft_scale: volume / k^2 / (nx ny)), inverse transform;
//   fft_rows_inverse: the two rows' frequencies back into one complex transform,
//     its real and imaginary parts the two rows of phi.
// A transform is the autosorting (Stockham) form of Govindaraju et al.,
// "High performance discrete Fourier transforms on graphics processors", SC 2008, of
// radix E = 8 or 4: thread j of n/E holds elements j + m n/E, a step is a butterfly in
// registers and an exchange through shared memory, and a last step of a smaller radix
// completes n. Twiddles come from a table of exp(-2 pi i k / n).
//
// Bound by FP64 arithmetic, of which an SM does two multiply-adds per cycle: about
// 35 instructions per point and transform at n = 512, 38 at 1024.
#include "pic_internal.cuh"

namespace picgb {

namespace {

struct C2 {
    double x, y;
};
__device__ __forceinline__ C2 cadd(C2 a, C2 b) { return {__dadd_rn(a.x, b.x), __dadd_rn(a.y, b.y)}; }
__device__ __forceinline__ C2 csub(C2 a, C2 b) { return {__dsub_rn(a.x, b.x), __dsub_rn(a.y, b.y)}; }
__device__ __forceinline__ C2 cmul(C2 a, double2 w) {
    return {__fma_rn(a.x, w.x, -__dmul_rn(a.y, w.y)), __fma_rn(a.x, w.y, __dmul_rn(a.y, w.x))};
}
// times -i (forward) or i (inverse)
template <bool INV>
__device__ __forceinline__ C2 quarter(C2 a) {
    return INV ? C2{-a.y, a.x} : C2{a.y, -a.x};
}
__device__ __forceinline__ void pair2(C2& a, C2& b) {
    const C2 t = a;
    a = cadd(t, b);
    b = csub(t, b);
}
// four-point transform in place, natural order
template <bool INV>
__device__ __forceinline__ void four(C2& a0, C2& a1, C2& a2, C2& a3) {
    pair2(a0, a2);
    pair2(a1, a3);
    a3 = quarter<INV>(a3);
    const C2 s0 = a0, s1 = a2, s2 = a1, s3 = a3;
    a0 = cadd(s0, s2);
    a2 = csub(s0, s2);
    a1 = cadd(s1, s3);
    a3 = csub(s1, s3);
}
// eight-point transform in place, natural order
template <bool INV>
__device__ __forceinline__ void eight(C2 (&v)[8]) {
    constexpr double H = 0.70710678118654752440;
    pair2(v[0], v[4]);
    pair2(v[1], v[5]);
    pair2(v[2], v[6]);
    pair2(v[3], v[7]);
    // v5, v6, v7 times exp(-+ i pi m / 4), m = 1, 2, 3
    const C2 q5 = quarter<INV>(v[5]), q7 = quarter<INV>(v[7]);
    v[5] = {__dmul_rn(H, __dadd_rn(v[5].x, q5.x)), __dmul_rn(H, __dadd_rn(v[5].y, q5.y))};
    v[6] = quarter<INV>(v[6]);
    v[7] = {__dmul_rn(H, __dsub_rn(q7.x, v[7].x)), __dmul_rn(H, __dsub_rn(q7.y, v[7].y))};
    four<INV>(v[0], v[1], v[2], v[3]);  // outputs 0, 2, 4, 6
    four<INV>(v[4], v[5], v[6], v[7]);  // outputs 1, 3, 5, 7
    const C2 o1 = v[4], o2 = v[1], o3 = v[5], o4 = v[2], o5 = v[6], o6 = v[3];
    v[1] = o1;
    v[2] = o2;
    v[3] = o3;
    v[4] = o4;
    v[5] = o5;
    v[6] = o6;
}

// A transform's place in shared memory, one element of padding in nine: the radix-8
// writes (stride 8) and the reads (stride 1) both miss no bank twice.
__device__ __forceinline__ int padded(int i) { return i + (i >> 3); }
__host__ __device__ constexpr int region(int n) { return n + n / 8 + 2; }

// N-point transform of the elements j + m N/E in v (N/E threads, j < N/E; E is 8 or 4,
// the radix), in natural order in the same places; NS: what the steps so far cover. sm:
// this transform's region (free when the call begins).
template <int N, bool INV, int NS = 1, int E>
__device__ __forceinline__ void transform(C2 (&v)[E], int j, double2* sm, const double2* __restrict__ tw) {
    constexpr int T = N / E;
    if constexpr (N / NS >= E) {
        if constexpr (NS > 1) {
            const int step = (j & (NS - 1)) * (N / (NS * E));
#pragma unroll
            for (int r = 1; r < E; ++r) {
                double2 w = __ldg(tw + step * r);
                if (INV) w.y = -w.y;
                v[r] = cmul(v[r], w);
            }
        }
        if constexpr (E == 8)
            eight<INV>(v);
        else
            four<INV>(v[0], v[1], v[2], v[3]);
        if constexpr (NS * E < N) {
            const int base = (j / NS) * NS * E + (j & (NS - 1));
            __syncthreads();
#pragma unroll
            for (int r = 0; r < E; ++r) sm[padded(base + r * NS)] = make_double2(v[r].x, v[r].y);
            __syncthreads();
#pragma unroll
            for (int m = 0; m < E; ++m) {
                const double2 e = sm[padded(j + m * T)];
                v[m] = {e.x, e.y};
            }
            transform<N, INV, NS * E>(v, j, sm, tw);
        }
    } else {
        // radix 4 (two butterflies per thread) or 2 (four, of E = 4 two): butterfly
        // j + b N/E of elements v[b + r E/R], back into the same places
        constexpr int R = N / NS, B = E / R;
#pragma unroll
        for (int b = 0; b < B; ++b) {
#pragma unroll
            for (int r = 1; r < R; ++r) {
                double2 w = __ldg(tw + (j + b * T) * r);
                if (INV) w.y = -w.y;
                v[b + r * B] = cmul(v[b + r * B], w);
            }
            if constexpr (R == 4)
                four<INV>(v[b], v[b + B], v[b + 2 * B], v[b + 3 * B]);
            else
                pair2(v[b], v[b + B]);
        }
    }
}

// Where the transforms are few (up to four per SM) and of at most 1024 elements, each is
// a block of its own with four elements per thread, radix 4: a warp's FP64 instruction
// takes its SM 16 cycles however many of its lanes work, a transform's chain of them is
// the kernel's time, and in radix 8 with fewer threads the chain is twice as long. Many
// transforms fill the SMs either way and radix 8 has less to do. us per step, radix 8
// against radix 4: 64^2 53 and 44, 256^2 (TSC) 86 and 71, 512^2 121 and 105, 64 x 1024 90
// and 67; with sides of 2048 taking it too, or more transforms, 100 and 102 at 2048 x 64,
// 98 and 99 at 64 x 2048.
constexpr int SMALL_MAX = 1024, SMALL_COUNT = 608;

// transforms of a block: whole warps of small ones
__host__ __device__ constexpr int row_batch(int n) { return n / 8 >= 32 ? 1 : 32 / (n / 8); }

template <int N, int E, int RB>
__global__ void __launch_bounds__(RB * (N / E)) fft_rows_forward(const double* __restrict__ in, int pairs,
                                                                           const double2* __restrict__ tw,
                                                                           double2* __restrict__ spec) {
    constexpr int T = N / E, NH = N / 2 + 1;
    __shared__ double2 smem[RB * region(N)];
    const int j = threadIdx.x % T, f = blockIdx.x * RB + threadIdx.x / T;
    double2* sm = smem + (threadIdx.x / T) * region(N);
    const bool on = f < pairs;
    const double* r0 = in + (size_t)f * 2 * N;
    C2 v[E];
#pragma unroll
    for (int m = 0; m < E; ++m) v[m] = on ? C2{r0[j + m * T], r0[N + j + m * T]} : C2{0.0, 0.0};
    transform<N, false>(v, j, sm, tw);
    __syncthreads();
#pragma unroll
    for (int m = 0; m < E; ++m) sm[padded(j + m * T)] = make_double2(v[m].x, v[m].y);
    __syncthreads();
    if (!on) return;
    // twice the rows' frequencies: Z[k] + conj Z[-k] and -i (Z[k] - conj Z[-k]); the
    // half is in the frequency factors
    double2* s0 = spec + (size_t)f * 2 * NH;
    for (int k = j; k < NH; k += T) {
        const double2 a = sm[padded(k)], b = sm[padded((N - k) & (N - 1))];
        s0[k] = make_double2(__dadd_rn(a.x, b.x), __dsub_rn(a.y, b.y));
        s0[NH + k] = make_double2(__dadd_rn(a.y, b.y), __dsub_rn(b.x, a.x));
    }
}

template <int N, int E, int RB>
__global__ void __launch_bounds__(RB * (N / E)) fft_rows_inverse(const double2* __restrict__ spec, int pairs,
                                                                           const double2* __restrict__ tw,
                                                                           double* __restrict__ out) {
    constexpr int T = N / E, NH = N / 2 + 1;
    __shared__ double2 smem[RB * region(N)];
    const int j = threadIdx.x % T, f = blockIdx.x * RB + threadIdx.x / T;
    double2* sm = smem + (threadIdx.x / T) * region(N);
    const bool on = f < pairs;
    const double2* s0 = spec + (size_t)f * 2 * NH;
    C2 v[E];
#pragma unroll
    for (int m = 0; m < E; ++m) {
        const int k = j + m * T, kk = k <= N / 2 ? k : N - k;
        double2 a = make_double2(0.0, 0.0), b = a;
        if (on) {
            a = s0[kk];
            b = s0[NH + kk];
        }
        if (kk == 0 || kk == N / 2) a.y = b.y = 0.0;  // a real row's
        // X0 + i X1, or of the conjugates above the middle
        v[m] = k <= N / 2 ? C2{__dsub_rn(a.x, b.y), __dadd_rn(a.y, b.x)} : C2{__dadd_rn(a.x, b.y), __dsub_rn(b.x, a.y)};
    }
    transform<N, true>(v, j, sm, tw);
    if (!on) return;
    double* r0 = out + (size_t)f * 2 * N;
#pragma unroll
    for (int m = 0; m < E; ++m) {
        r0[j + m * T] = v[m].x;
        r0[N + j + m * T] = v[m].y;
    }
}

// columns of a block: 64-byte row segments, less where a transform needs 128 threads or more
__host__ __device__ constexpr int col_batch(int n) { return n <= 512 ? 4 : n <= 1024 ? 2 : 1; }

template <int N, int E, int CB>
__global__ void __launch_bounds__(CB * (N / E)) fft_columns(double2* __restrict__ spec, int nh,
                                                                      const double2* __restrict__ tw,
                                                                      const double* __restrict__ scale) {
    constexpr int T = N / E;
    extern __shared__ double2 csm[];
    const int c = threadIdx.x % CB, j = threadIdx.x / CB, col = blockIdx.x * CB + c;
    double2* sm = csm + c * region(N);
    const bool on = col < nh;
    double2* s = spec + col;
    C2 v[E];
#pragma unroll
    for (int m = 0; m < E; ++m) {
        const double2 e = on ? s[(size_t)(j + m * T) * nh] : make_double2(0.0, 0.0);
        v[m] = {e.x, e.y};
    }
    double f[E];
#pragma unroll
    for (int m = 0; m < E; ++m) f[m] = on ? scale[(size_t)(j + m * T) * nh + col] : 0.0;
    transform<N, false>(v, j, sm, tw);
#pragma unroll
    for (int m = 0; m < E; ++m) v[m] = {__dmul_rn(v[m].x, f[m]), __dmul_rn(v[m].y, f[m])};
    transform<N, true>(v, j, sm, tw);
    if (!on) return;
#pragma unroll
    for (int m = 0; m < E; ++m) s[(size_t)(j + m * T) * nh] = make_double2(v[m].x, v[m].y);
}

__global__ void make_twiddles(double2* __restrict__ tw, int n) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    double s, c;
    sincospi(2.0 * (double)k / (double)n, &s, &c);
    tw[k] = make_double2(c, -s);
}

template <int N, int E, int RB>
int rows_as(pic_ctx* c, const double2* tw, const double* in, double2* spec, double* out) {
    const int pairs = c->Ny / 2;
    const unsigned blocks = (unsigned)((pairs + RB - 1) / RB);
    if (in)
        fft_rows_forward<N, E, RB><<<blocks, RB * (N / E), 0, c->stream>>>(in, pairs, tw, spec);
    else
        fft_rows_inverse<N, E, RB><<<blocks, RB * (N / E), 0, c->stream>>>(spec, pairs, tw, out);
    return check_launch(c, in ? "fft_rows_forward" : "fft_rows_inverse");
}
template <int N>
int rows(pic_ctx* c, const double2* tw, const double* in, double2* spec, double* out) {
    if constexpr (N <= SMALL_MAX)
        if (c->Ny / 2 <= SMALL_COUNT) return rows_as<N, 4, 1>(c, tw, in, spec, out);
    return rows_as<N, 8, row_batch(N)>(c, tw, in, spec, out);
}

template <int N, int E, int CB>
int columns_as(pic_ctx* c, const double2* tw, double2* spec) {
    const int nh = c->Nx / 2 + 1;
    const size_t smem = (size_t)CB * region(N) * sizeof(double2);
    PIC_TRY(opt_in_dynamic_smem((const void*)fft_columns<N, E, CB>, smem));
    fft_columns<N, E, CB><<<(unsigned)((nh + CB - 1) / CB), CB * (N / E), smem, c->stream>>>(spec, nh, tw, c->fft_scale);
    return check_launch(c, "fft_columns");
}
template <int N>
int columns(pic_ctx* c, const double2* tw, double2* spec) {
    if constexpr (N <= SMALL_MAX)
        if (c->Nx / 2 + 1 <= SMALL_COUNT) return columns_as<N, 4, 1>(c, tw, spec);
    return columns_as<N, 8, col_batch(N)>(c, tw, spec);
}

#define PIC_FFT_SIZES(X) X(8) X(16) X(32) X(64) X(128) X(256) X(512) X(1024) X(2048)

}  // namespace

bool own_fft_size(int n) { return n >= 8 && n <= 2048 && (n & (n - 1)) == 0; }

int make_own_fft(pic_ctx* c) {
    int rc = PIC_OK;
    if (!c->fft_tw) c->fft_tw = dalloc((size_t)(c->Nx + c->Ny) * sizeof(double2), &rc);
    if (rc) return rc;
    double2* tw = static_cast<double2*>(c->fft_tw);
    make_twiddles<<<(unsigned)((c->Nx + 255) / 256), 256, 0, c->stream>>>(tw, c->Nx);
    PIC_TRY(check_launch(c, "make_twiddles"));
    make_twiddles<<<(unsigned)((c->Ny + 255) / 256), 256, 0, c->stream>>>(tw + c->Nx, c->Ny);
    return check_launch(c, "make_twiddles");
}

// phi = the inverse transform of fft_scale times the transform of rho (both grids of the context).
int own_fft_solve(pic_ctx* c) {
    double2* spec = static_cast<double2*>(c->spec);
    const double2 *tx = static_cast<const double2*>(c->fft_tw), *ty = tx + c->Nx;
    switch (c->Nx) {
#define X(n) case n: PIC_TRY(rows<n>(c, tx, c->rho, spec, nullptr)); break;
        PIC_FFT_SIZES(X)
#undef X
    }
    switch (c->Ny) {
#define X(n) case n: PIC_TRY(columns<n>(c, ty, spec)); break;
        PIC_FFT_SIZES(X)
#undef X
    }
    switch (c->Nx) {
#define X(n) case n: PIC_TRY(rows<n>(c, tx, nullptr, spec, c->phi)); break;
        PIC_FFT_SIZES(X)
#undef X
    }
    return PIC_OK;
}

}  // namespace picgb
