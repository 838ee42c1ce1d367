// Walking a tile's cells over the cell-sorted stream (deposit_cells, current_cells).
//
// A tile's rows are cut into units of U = 32 / K consecutive cells, K lanes per
// cell; a warp takes units w, w + NW, ... A unit's particles are one contiguous
// range of the stream. It is copied to shared memory with cp.async, coalesced, 16
// bytes per lane and field, into the warp's buffer of `cap` particles
// (the other warps sum theirs meanwhile: a second buffer per warp halved the warps
// that fit and took 5 to 15 % longer); a longer range (dense cells) is taken in pieces, and
// all the warp's lanes share the cells that a piece reaches (one lane for each of three
// cells of 166,667 particles among empty ones, one after the other: 1000 x 700, half of 3 M
// particles in nine cells, mixed charges, CIC: 21 ms, 13 before units were staged). Then
// each lane walks its share of its own cell in shared memory. (Copying each lane's own cell instead
// touched 32 lines per copy instruction.)
#pragma once

#include <cstdint>

namespace picgb {

__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// A piece of a unit: particles [pos, pos + cap) up to the unit's end (the same in
// every lane of the warp). pos is a multiple of 4.
struct CellPiece {
    int r, ch;          // tile row, unit of the row
    int c0, cn, klog;   // the piece's first column, columns, log2 lanes per cell
    uint32_t pos, end;  // first particle staged, end of the unit's range
    bool pieces;        // the range is longer than the buffer, and of several cells
};

// NF fields of 4 bytes per particle; field f of the buffer's particle i is word
// f * cap + i. The field arrays are 16-byte aligned and padded past the last particle.
template <int NF, int NW>
struct CellWalk {
    const uint32_t* field[NF];
    const uint32_t* soff;  // the tile rows' cell offsets in shared memory, rows of tw + 1
    uint32_t buf_addr;     // shared address of the warp's buffer
    int tw, th, nch, klog, cap;

    __device__ __forceinline__ void init(int tw_, int th_, int klog_, int cap_) {
        tw = tw_;
        th = th_;
        klog = klog_;
        cap = cap_;
        nch = (tw + (32 >> klog) - 1) >> (5 - klog);
    }
    __device__ __forceinline__ bool done(const CellPiece& w) const { return w.r >= th; }
    // the warp's first non-empty unit
    __device__ __forceinline__ void start(CellPiece& w, int warp) const {
        w.r = 0;
        w.ch = warp;
        seek(w);
    }
    // the first non-empty unit at or after (w.r, w.ch), the row's unit number taken past its end
    __device__ __forceinline__ void seek(CellPiece& w) const {
        for (;; w.ch += NW) {
            while (w.ch >= nch) {
                w.ch -= nch;
                ++w.r;
            }
            if (w.r >= th) return;
            w.c0 = w.ch << (5 - klog);
            w.cn = min(32 >> klog, tw - w.c0);
            w.klog = klog;
            const uint32_t beg = soff[w.r * (tw + 1) + w.c0];
            w.end = soff[w.r * (tw + 1) + w.c0 + w.cn];
            w.pos = beg & ~3u;
            w.pieces = klog < 5 && w.end - w.pos > (uint32_t)cap;  // a unit of one cell has all lanes already
            if (w.end > beg) return;
        }
    }
    // of a unit that is taken in pieces: the columns that the piece reaches and the lanes for each
    __device__ __forceinline__ void narrow(CellPiece& w) const {
        const int lane = threadIdx.x & 31, c0 = w.ch << (5 - klog), cn = min(32 >> klog, tw - c0);
        bool in = false;
        if (lane < cn) {
            const uint32_t b = soff[w.r * (tw + 1) + c0 + lane], e = soff[w.r * (tw + 1) + c0 + lane + 1];
            in = e > b && e > w.pos && b < w.pos + (uint32_t)cap;
        }
        const unsigned m = __ballot_sync(0xffffffffu, in);  // not empty: the piece has particles
        const int first = __ffs(m) - 1;
        w.c0 = c0 + first;
        w.cn = 32 - __clz(m) - first;
        w.klog = w.cn == 1 ? 5 : __clz(w.cn - 1) - 27;  // 32 over the next power of two
    }
    // all lanes are at one cell, and so they are in the next piece: their sums may go on
    __device__ __forceinline__ bool same_cell(const CellPiece& w) const {
        if (__builtin_expect(w.cn != 1 || w.end - w.pos <= (uint32_t)cap, 1)) return false;
        return soff[w.r * (tw + 1) + w.c0 + 1] >= min(w.end, w.pos + 2u * (uint32_t)cap);
    }
    __device__ __forceinline__ void advance(CellPiece& w) const {
        w.pos += (uint32_t)cap;
        if (w.pos >= w.end) {
            w.ch += NW;
            seek(w);
        }
    }
    // copies the piece; returns when it has arrived, in every lane
    __device__ __forceinline__ void stage(CellPiece& w, int lane) const {
        if (__builtin_expect(w.pieces, 0)) narrow(w);
        const uint32_t n4 = (min(w.end - w.pos, (uint32_t)cap) + 3u) >> 2;
        for (uint32_t i = (uint32_t)lane; i < n4; i += 32)
#pragma unroll
            for (int f = 0; f < NF; ++f)
                cp_async16(buf_addr + (uint32_t)(f * cap) * 4u + i * 16u, field[f] + w.pos + 4u * i);
        cp_async_wait_all();
        __syncwarp();
    }
    // the lane's share of the piece: m consecutive particles of its cell (column
    // w.c0 + (lane >> w.klog)) from buffer index `first`
    // `count`: the cell's particles
    __device__ __forceinline__ void share(const CellPiece& w, int lane, int& first, int& m, uint32_t& count) const {
        const int cl = lane >> w.klog, sub = lane & ((1 << w.klog) - 1);
        m = first = 0;
        count = 0;
        if (cl >= w.cn) return;
        const int o = w.r * (tw + 1) + w.c0 + cl;
        count = soff[o + 1] - soff[o];
        const uint32_t b = max(soff[o], w.pos), e = min(soff[o + 1], min(w.end, w.pos + (uint32_t)cap));
        if (e <= b) return;
        int per = (int)(e - b + (1u << w.klog) - 1u) >> w.klog;
        per |= w.pieces ? 1 : 0;  // many lanes of one cell start in different banks
        first = (int)(b - w.pos) + sub * per;
        m = max(0, min(per, (int)(e - b) - sub * per));
    }
};

// Lanes per cell (as its logarithm) and the buffer's particles: units of up to
// `words` staged words over the fields at the mean density (a buffer an eighth
// longer, and at least half of `words`, for cells denser than the mean: 200 x 130, half of
// 26,000 particles in nine cells, NGP 48 us against 109 with a buffer of the mean alone; all
// of `words` left sparse grids fewer CTAs on an SM, 2000 x 1500 x 4 139 us against 111).
// Larger units cost less to set up and write out, smaller ones leave room
// for more warps; where one cell fills a unit, smaller pieces of it do as well.
// Small grids take smaller units, so that every warp of the launch has one, but no more
// than that: a warp takes its units one after the other (tiles of 64 x 32 asked for on
// 64^2, 16 per cell, CIC: 139 us with four cells to a unit, 40 with 32).
inline void cells_shape(size_t n, size_t cells, int fields, int words, size_t warps, int* klog, int* cap) {
    const double ppc = (double)n / (double)cells;
    const double unit = (double)words / fields;
    int k = 0;
    while (k < 5 && (32 >> k) * ppc > unit) ++k;
    const double most_units = warps < 1800 ? (double)warps : 1800.0;
    while (k < 3 && (double)cells / (32 >> k) < most_units) ++k;
    double want = (32 >> k) * ppc * 1.125 + 64.0;
    const double most = unit * (k == 5 ? 0.625 : 1.25), least = unit * 0.5;
    if (want < least) want = least;
    if (want > most) want = most;
    *klog = k;
    *cap = ((int)want + 3) & ~3;
}

}  // namespace picgb
