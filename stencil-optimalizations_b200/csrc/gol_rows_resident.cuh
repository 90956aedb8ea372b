// Shared-memory-resident run: every generation of a grid that fits in the
// GPU's shared memory, in one cooperative launch.
//
// A grid whose rows fit in the SMs' shared memory (8192^2 bits is 8 MiB;
// 148 SMs hold up to 33 MiB) need not go through HBM or L2 between passes:
// CTA c keeps rows [y0, y1) of the grid (its band) in two shared-memory
// buffers and advances them K generations per epoch. An epoch needs K rows
// above and K below the band (cells within K of the band's edge depend on
// them), which the neighbouring CTAs publish through global memory.
//
// The exchange is overlapped with the band's interior. The first ni
// generations of an epoch (ni = kResidentInterior, at most K) are first
// computed on the rows at least g away from the band's edges (they depend on
// the band only) while the neighbours' rows arrive. Then the CTA waits for
// them (bounded polls: GOL_E_TIMEOUT in *status and the CTA stops), copies
// them into its halo and completes generations g = 1..ni near the two edges:
// rows [K - kk + g, K + g) and the mirror rows at the bottom. Those read
// generation g - 1 rows that the interior pass of generation g + 1 (same
// buffer) left alone, since the interior shrinks by one row per side per
// generation. Generations ni+1..K are then computed whole (the band and the
// K - g halo rows each side that the halo still determines). Rows outside
// the grid are never computed and stay dead (zero).
//
// Epoch e publishes the band's top and bottom K rows into slot e & 1, every
// word with the epoch's tag e + 1 beside it in one 64-bit store: the
// neighbours poll the words themselves, so an exchange costs one trip through
// L2 and no fence, counter or barrier of its own. Launches on the same slots
// count their epochs on, so that no tag comes twice (a memset of the slots
// before each took 3 to 6 us). A CTA rewrites a slot two epochs later, after both neighbours
// have published the epoch in between, i.e. after they read it.
//
// Within a pass a thread owns four words of a row (128 cells; the CTA's
// threads are lanes across the row times row groups) and walks a range of
// rows two at a time (pair_sum, next_word_pair in gol_word_ops.cuh), the sums
// of the two rows above in registers. The run is bound by the integer pipe,
// so shared memory holds the lane's cells interleaved: bit i of its word j is
// cell 4i + j. The cells left and right of a word's are then the words before
// and after it, and only the outer two neighbours of a lane's four words take
// a shift: 8.5 operations a word and generation, against 12 for rows as they
// are, one at a time (9.4 -> 7.6 ms for 8192^2, 4096 generations). A band is
// interleaved when it is loaded and restored when it is stored, some 8
// operations a word each way; the exchange slots hold interleaved rows. The
// four words are kept in planes (word j of all lanes in a run), so every
// access takes one wavefront: ten for a warp's 128 words of a row, where the
// integer pipe takes 17 cycles. (With the four words of a lane side by side
// the two neighbour loads alone take eight.) Cells at or past column W are
// masked by the warps that hold some.
//
// The band algorithm (resident_band) serves two kernels: one grid, CTA c
// running band c (rows_resident_kernel), and many grids, persistent CTAs
// taking bands of a batch in ticket order (batch_resident_kernel). All
// CTAs of a launch must be resident at once (they wait on each other): the
// launches are cooperative.
#pragma once

#include <cstdint>

#include "gol_internal.h"
#include "gol_rows_temporal.cuh"
#include "gol_word_ops.cuh"

namespace golb200 {

#ifndef GOL_RESIDENT_MAX_THREADS
#define GOL_RESIDENT_MAX_THREADS 512
#endif
constexpr int kResidentMaxThreads = GOL_RESIDENT_MAX_THREADS;
#ifndef GOL_RESIDENT_INTERIOR
#define GOL_RESIDENT_INTERIOR 1
#endif
// Generations of an epoch computed on the interior alone, before the wait
// for the neighbours' rows.
constexpr int kResidentInterior = GOL_RESIDENT_INTERIOR;

struct ResidentLaunch {   // one grid (rows_resident_kernel)
    const uint32_t* src;   // the grid at generation 0 (W words per row, Y rows)
    uint32_t* dst;         // the grid after `gens` generations (not src)
    unsigned long long* pub;   // [nbands][2 parities][2 sides][K rows][4 planes][lanes], tags up to epoch0
    int* status;           // GOL_E_TIMEOUT if a wait gave up
    int W, Y;
    int K;                 // generations per epoch
    int lanes;             // lanes across a row, four words each: ceil(W / 4)
    int groups;            // row groups (blockDim.x = lanes * groups)
    long long gens;
    long long spin_limit;
    int epoch0;            // number of the launch's first epoch
};

// A published word: the value below, the epoch's tag above, stored and loaded
// at once.
__device__ __forceinline__ void st_tagged(unsigned long long* p, uint32_t v, uint32_t tag) {
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"((unsigned long long)tag << 32 | v)
                 : "memory");
}

__device__ __forceinline__ unsigned long long ld_tagged(const unsigned long long* p) {
    unsigned long long v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}

// A shared-memory row: a zero word, plane 3 of the lanes, planes 1 and 2,
// plane 0, a zero word. The words beyond a row's ends that a pass reads are
// plane 3 before lane 0 and plane 0 after the last lane: the zero words. Rows
// whose lanes do not fill warps have an odd stride, so that the row groups of
// one warp fall into different banks.
__host__ __device__ inline int resident_stride(int lanes) {
    return 4 * lanes + 2 + (lanes % 32 ? 1 : 0);
}
__host__ __device__ constexpr int resident_plane(int j) { return j == 3 ? 0 : j == 0 ? 3 : j; }

// Shared memory of one CTA: two buffers of (band + 2K) rows.
__host__ __device__ inline size_t resident_smem_bytes(int band, int K, int lanes) {
    return 2ull * (size_t)(band + 2 * K) * (size_t)resident_stride(lanes) * sizeof(uint32_t);
}

// Exchanges index bit B of the bit position with the upper bit of the register
// index (v[0], v[1] against v[2], v[3]).
template <int B>
__device__ __forceinline__ void swap_index_bit(uint32_t (&v)[4]) {
    constexpr uint32_t m = B == 4 ? 0x0000ffffu : B == 3 ? 0x00ff00ffu : B == 2 ? 0x0f0f0f0fu
                           : B == 1 ? 0x33333333u : 0x55555555u;   // positions whose bit B is 0
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const uint32_t x = v[i], y = v[i + 2];
        v[i] = (x & m) | ((y & m) << (1 << B));
        v[i + 2] = ((x >> (1 << B)) & m) | (y & ~m);
    }
}

__device__ __forceinline__ void swap_registers(uint32_t (&v)[4]) {   // the register index's two bits
    const uint32_t t = v[1];
    v[1] = v[2];
    v[2] = t;
}

// Cell c of the lane's 128 from bit c % 32 of word c / 32 to bit c / 4 of word
// c % 4, and back: the index (w1 w0 a2 a1 a0 j1 j0) rotated by two, one bit
// at a time through the register index.
__device__ __forceinline__ void interleave4(uint32_t (&v)[4]) {
    swap_index_bit<4>(v);
    swap_index_bit<2>(v);
    swap_index_bit<0>(v);
    swap_registers(v);
    swap_index_bit<3>(v);
    swap_index_bit<1>(v);
}

__device__ __forceinline__ void deinterleave4(uint32_t (&v)[4]) {
    swap_index_bit<1>(v);
    swap_index_bit<3>(v);
    swap_registers(v);
    swap_index_bit<0>(v);
    swap_index_bit<2>(v);
    swap_index_bit<4>(v);
}

// One row of a lane: its four words, and their horizontal sums.
struct ResidentRow {
    uint32_t c[4], h0[4], h1[4];
};

// Reads the row whose first plane's entry of this lane is at p (planes PL
// words apart).
__device__ __forceinline__ void resident_row(const uint32_t* p, int PL, ResidentRow& r) {
#pragma unroll
    for (int j = 0; j < 4; ++j) r.c[j] = p[resident_plane(j) * PL];
    const uint32_t lw = p[-1];           // plane 3 of the lane before
    const uint32_t rw = p[3 * PL + 1];   // plane 0 of the lane after
    const uint32_t left = __funnelshift_l(lw, r.c[3], 1);
    const uint32_t right = __funnelshift_r(r.c[0], rw, 1);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const uint32_t l = j == 0 ? left : r.c[j - 1];
        const uint32_t q = j == 3 ? right : r.c[j + 1];
        r.h0[j] = lop3<LUT_XOR3>(l, r.c[j], q);
        r.h1[j] = lop3<LUT_MAJ>(l, r.c[j], q);
    }
}

// The next state of rows b and p (a above b, q below p), to d and d + stride.
template <bool RAG>
__device__ __forceinline__ void resident_pair(const ResidentRow& a, const ResidentRow& b,
                                              const ResidentRow& p, const ResidentRow& q,
                                              uint32_t* d, int stride, int PL, uint32_t mask) {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const PairSum s = pair_sum(b.h0[j], b.h1[j], p.h0[j], p.h1[j]);
        uint32_t x = next_word_pair(a.h0[j], a.h1[j], s, b.c[j]);
        uint32_t y = next_word_pair(q.h0[j], q.h1[j], s, p.c[j]);
        if (RAG) {
            x &= mask;
            y &= mask;
        }
        d[resident_plane(j) * PL] = x;
        d[stride + resident_plane(j) * PL] = y;
    }
}

// Rows [r0, r1) of one generation, S -> D (S and D point at this lane's entry
// of row 0's first plane). Four rows per turn, so that the rows' sums change
// roles by name.
template <bool RAG>
__device__ __forceinline__ void resident_rows(const uint32_t* S, uint32_t* D, int r0, int r1,
                                              int stride, int PL, uint32_t mask) {
    if (r0 >= r1) return;
    ResidentRow a, b, p, q;
    const uint32_t* s = S + (size_t)(r0 - 1) * stride;
    uint32_t* d = D + (size_t)r0 * stride;
    resident_row(s, PL, a);
    resident_row(s + stride, PL, b);
    s += 2 * stride;
    int n = r1 - r0;
    for (; n >= 4; n -= 4) {
        resident_row(s, PL, p);
        resident_row(s + stride, PL, q);
        resident_pair<RAG>(a, b, p, q, d, stride, PL, mask);
        resident_row(s + 2 * stride, PL, a);
        resident_row(s + 3 * stride, PL, b);
        resident_pair<RAG>(p, q, a, b, d + 2 * stride, stride, PL, mask);
        s += 4 * stride;
        d += 4 * stride;
    }
    if (n >= 2) {
        resident_row(s, PL, p);
        resident_row(s + stride, PL, q);
        resident_pair<RAG>(a, b, p, q, d, stride, PL, mask);
        a = p;
        b = q;
        s += 2 * stride;
        d += 2 * stride;
        n -= 2;
    }
    if (n == 1) {   // one row: its pair's other half is not wanted
        resident_row(s, PL, p);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const PairSum x = pair_sum(b.h0[j], b.h1[j], p.h0[j], p.h1[j]);
            uint32_t y = next_word_pair(a.h0[j], a.h1[j], x, b.c[j]);
            if (RAG) y &= mask;
            d[resident_plane(j) * PL] = y;
        }
    }
}

// Rows [lo, hi) split over groups [g0, g0 + ng) (this thread's group is g).
// Rows of whole warps are split evenly: sizes differ by at most one row, so
// the schedulers' shares do not drift apart (whole pairs per group left two of
// them 10 % more). Narrower ones, several groups to a warp, lie as many rows
// apart, and with the odd stride they share banks where that number has more
// factors of two than the lanes: then they take a row more (256 x 2048: 12.7
// thousand cycles a generation without, 4.4 with).
__device__ __forceinline__ void resident_pass(const uint32_t* S, uint32_t* D, int lo, int hi,
                                              int g, int g0, int ng, int stride, int PL,
                                              uint32_t mask, bool rag) {
    if (g < g0 || g >= g0 + ng || hi <= lo) return;
    const int n = hi - lo;
    int r0, r1;
    if (PL >= 32) {
        const int q = n / ng, extra = n - q * ng;   // the first `extra` groups one more
        r0 = lo + (g - g0) * q + min(g - g0, extra);
        r1 = r0 + q + (g - g0 < extra ? 1 : 0);
    } else {
        int q = (n + ng - 1) / ng;
        if (q % (2 * (PL & -PL)) == 0) ++q;
        r0 = lo + (g - g0) * q;
        r1 = min(hi, r0 + q);
    }
    if (rag)   // the same for every lane of a warp
        resident_rows<true>(S, D, r0, r1, stride, PL, mask);
    else
        resident_rows<false>(S, D, r0, r1, stride, PL, mask);
}

// Global <-> register copies of a lane's four words: vector accesses where
// they are whole and aligned, else word by word up to W.
__device__ __forceinline__ void band_load(const uint32_t* p, bool vec, int n, uint32_t (&v)[4]) {
    if (vec) {
        load_words<4>(p, v);
    } else {
#pragma unroll
        for (int w = 0; w < 4; ++w) v[w] = w < n ? __ldg(p + w) : 0u;
    }
}

__device__ __forceinline__ void band_store(uint32_t* p, bool vec, int n, const uint32_t (&v)[4]) {
    if (vec) {
        store_words<4>(p, v);
    } else {
#pragma unroll
        for (int w = 0; w < 4; ++w)
            if (w < n) p[w] = v[w];
    }
}

// Runs band j.b of its grid: returns false if a wait gave up (GOL_E_TIMEOUT
// in *status; the caller ends the CTA). Every thread of the CTA calls it;
// smem holds 2 * (B + 2K) rows of the stride. LANES: the lanes across a row
// when known at compile time (0: j.lanes), so the shared-memory row stride
// is a constant and row addresses are immediate offsets.
template <int LANES>
__device__ __forceinline__ bool resident_band(const ResidentBand& j, uint32_t* smem, int* stop,
                                              int* status, long long spin_limit) {
    const int K = j.K;
    const int PL = LANES ? LANES : j.lanes;
    const int stride = resident_stride(PL);
    const int lane_in_row = threadIdx.x % PL;
    const int group = threadIdx.x / PL;   // >= j.groups: idle in the passes
    const int col = lane_in_row * 4;
    const int W = j.W;
    const int nw = W - col;               // words of this lane inside the row
    // Warps with cells past column W mask their results: word j holds cells
    // 4i + j, so a lane of nw words keeps the lower 8 nw bits of each.
    const uint32_t mask = nw >= 4 ? 0xffffffffu : (1u << (8 * max(nw, 0))) - 1u;
    const bool rag = __any_sync(0xffffffffu, mask != 0xffffffffu);
    const bool top = j.b == 0, bottom = j.b == j.nb - 1;
    // Bands split the rows evenly (sizes differ by at most one row; with
    // several bands every band is at least K rows).
    const int y0 = (int)((long long)j.b * j.Y / j.nb);
    const int B = (int)((long long)(j.b + 1) * j.Y / j.nb) - y0;
    const int rows = B + 2 * K;                 // shared-memory rows: K halo each side
    const size_t side_words = (size_t)K * 4 * PL;
    const int ng_top = j.groups > 1 ? j.groups / 2 : 1;
    const int g_bot = j.groups > 1 ? ng_top : 0;
    const int ng_bot = j.groups > 1 ? j.groups - ng_top : 1;
    const bool mover = group < j.groups;        // moves words between global and shared
    const bool whole = nw >= 4 && (j.pitch & 3) == 0;
    const bool svec = whole && ((uintptr_t)j.src & 15u) == 0;
    const bool dvec = whole && ((uintptr_t)j.dst & 15u) == 0;

    // Buffers zero (halo rows, the rows' outer words), then the band rows
    // into buffer 0 (shared row K + i = grid row y0 + i). Copies between
    // global and shared rows go by row group and lane: each thread moves its
    // lane's four words of every groups-th row.
    for (int i = threadIdx.x; i < 2 * rows * stride; i += blockDim.x) smem[i] = 0u;
    __syncthreads();
    uint32_t* const lane0 = smem + 1 + lane_in_row;   // this lane's entry of row 0's first plane
    if (mover) {
        for (int r = group; r < B; r += j.groups) {
            uint32_t v[4];
            band_load(j.src + (size_t)(y0 + r) * j.pitch + col, svec, nw, v);
            interleave4(v);
            uint32_t* d = lane0 + (size_t)(K + r) * stride;
#pragma unroll
            for (int i = 0; i < 4; ++i) d[resident_plane(i) * PL] = v[i];
        }
    }
    if (threadIdx.x == 0) *stop = 0;
    __syncthreads();

    int cur = 0;
    long long left = j.gens;
    for (int e = j.epoch0; left > 0; ++e) {
        const int kk = (int)min((long long)K, left);
        // Publish the band's top and bottom K rows (the state at epoch start).
        const uint32_t tag = (uint32_t)e + 1u;
        unsigned long long* mine = j.pub + ((size_t)j.b * 4 + (e & 1) * 2) * side_words + lane_in_row;
        uint32_t* const Aw = lane0 + (cur ? (size_t)rows * stride : 0);
        if (mover) {
            for (int r = group; r < K; r += j.groups) {
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const size_t at = ((size_t)r * 4 + i) * PL;
                    if (!top) st_tagged(mine + at, Aw[(size_t)(K + r) * stride + i * PL], tag);
                    if (!bottom)
                        st_tagged(mine + side_words + at, Aw[(size_t)(B + r) * stride + i * PL], tag);
                }
            }
        }
        // The interior: generation g's rows at least g from the band's edges,
        // for the first ni generations (enough to cover the exchange).
        const int ni = min(kk, kResidentInterior);
        for (int g = 1; g <= ni; ++g) {
            const int sb = (cur + g - 1) & 1;
            const uint32_t* S = lane0 + (sb ? (size_t)rows * stride : 0);
            uint32_t* D = lane0 + (sb ? 0 : (size_t)rows * stride);
            resident_pass(S, D, K + g, K + B - g, group, 0, j.groups, stride, PL, mask, rag);
            __syncthreads();
        }
        // The neighbours' rows of this epoch, polled word by word (bounded):
        // the upper one's bottom rows, the lower one's top rows. At the grid's
        // edges the halo stays zero (never written).
        if (mover) {
            const unsigned long long* up =
                j.pub + ((size_t)(j.b - 1) * 4 + (e & 1) * 2 + 1) * side_words + lane_in_row;
            const unsigned long long* dn =
                j.pub + ((size_t)(j.b + 1) * 4 + (e & 1) * 2) * side_words + lane_in_row;
            for (int r = group; r < K; r += j.groups) {
                unsigned long long u[4], v[4];
                long long spins = 0;
                for (;;) {
                    bool here = true;
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const size_t at = ((size_t)r * 4 + i) * PL;
                        u[i] = top ? (unsigned long long)tag << 32 : ld_tagged(up + at);
                        v[i] = bottom ? (unsigned long long)tag << 32 : ld_tagged(dn + at);
                    }
#pragma unroll
                    for (int i = 0; i < 4; ++i)
                        here = here && (uint32_t)(u[i] >> 32) == tag && (uint32_t)(v[i] >> 32) == tag;
                    if (here) break;
                    if (++spins > spin_limit || *(volatile int*)status != 0) {
                        atomicCAS(status, 0, GOL_E_TIMEOUT);
                        atomicExch(stop, 1);
                        break;
                    }
                }
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    if (!top) Aw[(size_t)r * stride + i * PL] = (uint32_t)u[i];
                    if (!bottom) Aw[(size_t)(K + B + r) * stride + i * PL] = (uint32_t)v[i];
                }
            }
        }
        __syncthreads();
        if (*(volatile int*)stop) return false;   // the same for every thread of the CTA
        // Generations 1..ni near the edges: rows within g of the band's
        // edges, and the halo rows the later generations still need.
        for (int g = 1; g <= ni; ++g) {
            const int sb = (cur + g - 1) & 1;
            const uint32_t* S = lane0 + (sb ? (size_t)rows * stride : 0);
            uint32_t* D = lane0 + (sb ? 0 : (size_t)rows * stride);
            const int bhi = bottom ? K + B : K + B + kk - g;
            const int tlo = top ? K : K - kk + g, thi = min(K + g, bhi);   // (a band under g rows)
            const int blo = max(K + g, K + B - g);
            resident_pass(S, D, tlo, thi, group, 0, ng_top, stride, PL, mask, rag);
            resident_pass(S, D, blo, bhi, group, g_bot, ng_bot, stride, PL, mask, rag);
            __syncthreads();
        }
        // Generations ni+1..kk whole: the band and what the halo still
        // determines.
        for (int g = ni + 1; g <= kk; ++g) {
            const int sb = (cur + g - 1) & 1;
            const uint32_t* S = lane0 + (sb ? (size_t)rows * stride : 0);
            uint32_t* D = lane0 + (sb ? 0 : (size_t)rows * stride);
            const int lo = top ? K : K - kk + g, hi = bottom ? K + B : K + B + kk - g;
            resident_pass(S, D, lo, hi, group, 0, j.groups, stride, PL, mask, rag);
            __syncthreads();
        }
        cur = (cur + kk) & 1;
        left -= kk;
    }
    // The band after the last generation.
    if (mover) {
        const uint32_t* A = lane0 + (cur ? (size_t)rows * stride : 0);
        for (int r = group; r < B; r += j.groups) {
            uint32_t v[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) v[i] = A[(size_t)(K + r) * stride + resident_plane(i) * PL];
            deinterleave4(v);
            band_store(j.dst + (size_t)(y0 + r) * j.pitch + col, dvec, nw, v);
        }
    }
    return true;
}

// One grid: CTA c runs band c.
template <int LANES>
__global__ void __launch_bounds__(kResidentMaxThreads, 1) rows_resident_kernel(ResidentLaunch a) {
    extern __shared__ __align__(16) uint32_t smem[];
    __shared__ int stop;
    ResidentBand j;
    j.src = a.src;
    j.dst = a.dst;
    j.pub = a.pub;
    j.pitch = a.W;
    j.W = a.W;
    j.Y = a.Y;
    j.K = a.K;
    j.lanes = a.lanes;
    j.groups = a.groups;
    j.b = blockIdx.x;
    j.nb = gridDim.x;
    j.gens = a.gens;
    j.epoch0 = a.epoch0;
    resident_band<LANES>(j, smem, &stop, a.status, a.spin_limit);
}

} // namespace golb200
