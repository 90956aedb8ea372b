// Row-pair pipeline: K generations per pass of large grids, two rows a step.
//
// A CTA owns a band of rows across the width (up to 256 lanes of four words;
// wider rows in x-slices with a halo lane each side) and streams down it, two
// rows per step. Stage g turns pairs of generation g - 1 rows into pairs of
// generation g rows, one row higher and one step later: it takes in the pair
// (r, r + 1) that stage g - 1 put out in the step before and, with the sums of
// rows r - 2 and r - 1 from its own last step, puts out rows r - 1 and r
// (pair_sum, next_word_pair in gol_word_ops.cuh). Two rows a step halve the
// barriers and edge accesses per row, and the shared sum takes the word from
// 12 operations to 10. All state is in registers (28 words per stage for a
// lane's four words); row pairs arrive through a cp.async ring in shared
// memory; the words beyond a lane's own come from its neighbours' edge words,
// published two rows at a time in shared memory, one barrier per step.
//
// INTER: rows are interleaved by four (bit i of a lane's word j is its cell
// 4i + j, interleave4 in gol_rows_resident.cuh), which leaves two shifts per
// four words: 8.5 operations a word. A run of many passes converts the grid
// once before and once after (interleave_kernel, a pass over memory each).
//
// Bound by the integer pipe, with two CTAs of four warps per SM (the state
// takes 236 registers; held to 168 or 128 it spills: 33 and 25 T). 16384^2,
// K = 4, 56-row bands: 25.4 us a pass interleaved (42.4 T cell-updates/s), 28.7
// as rows are, against 31.4 for the K-stage kernel of gol_rows_temporal.cuh and
// 33.5 for the register-block kernel at this depth (63 at depth 8); at depths
// 3, 5 and 6 40, 41 and 35 T. It wants bands of about 40 rows or more, since
// 4 K rows' worth of steps fill and drain the stages.
#pragma once

#include <cstdint>

#include "gol_rows_resident.cuh"
#include "gol_rows_temporal.cuh"
#include "gol_word_ops.cuh"

namespace golb200 {

constexpr int kPairK = 4;
constexpr int kPairRing = 4;   // row pairs in the ring, three in flight

struct PairCtx {
    const uint32_t* src;
    uint32_t* dst;
    int Y, y0, y1, steps_end;   // band rows, last step + 1
    int pitch, base;
    bool lane_ok, own;
    uint2* eb;                  // edge table: this lane's entry (first words)
    uint32_t ring;              // shared address of this lane's words in ring slot 0
};

template <int K>
struct PairRegs {
    uint32_t h0[K][2][2][4], h1[K][2][2][4];   // sums: stage, step parity, row of the pair
    uint32_t cen[K][4];                        // the last row taken in
    uint32_t o[K][2][4];                       // the pair put out (index 0: loaded rows)
};

// Edge table: [2 sides][K producers][2 step parities][threads + 2] entries of
// a row pair's words, lane t at t + 1; the outer entries and those of lanes
// outside the grid are never written and stay zero.
constexpr int kPairEdgeStride = kTemporalMaxThreads + 2;
__host__ __device__ constexpr int pair_edge(int g, int parity) { return (2 * g + parity) * kPairEdgeStride; }
template <int K>
__host__ __device__ constexpr int pair_last_side() { return 2 * K * kPairEdgeStride; }
__host__ __device__ inline size_t pair_smem_bytes(int K) {
    return (size_t)kPairRing * 2 * kTemporalMaxThreads * 16 + (size_t)4 * K * kPairEdgeStride * sizeof(uint2);
}

// Copies the row pair of step s into its ring slot (zeros outside the grid),
// as one group.
template <int K>
__device__ __forceinline__ void pair_issue(const PairCtx& c, int s) {
    constexpr uint32_t SB = kTemporalMaxThreads * 16u;
    const uint32_t slot = c.ring + (uint32_t)(s & (kPairRing - 1)) * 2u * SB;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const int r = c.y0 - K + 2 * s + i;
        const bool v = c.lane_ok && (unsigned)r < (unsigned)c.Y;
        cp_async_words<4>(slot + i * SB, v ? c.src + (size_t)r * c.pitch + c.base : c.src, v);
    }
    cp_async_commit();
}

// TEST: warm-up and drain steps (stages outside their rows skip). MASK: bands
// at the grid's top or bottom (rows outside it stay dead, rows past the band
// are not stored).
template <int K, bool INTER, int PH, bool TEST, bool MASK>
__device__ __forceinline__ void pair_step(PairRegs<K>& s, const PairCtx& c, int i) {
    constexpr int WAS = PH ^ 1;
#pragma unroll
    for (int g = K; g >= 1; --g) {
        // stage g's rows at this step: o_g, o_g + 1
        const int row = c.y0 - K + 2 * i - 3 * g;
        if (TEST && (i < 2 * g - 1 || row > c.y1 - 1 + K - g)) continue;
        const uint2 lw = c.eb[pair_last_side<K>() + pair_edge(g - 1, WAS)];
        const uint2 rw = c.eb[2 + pair_edge(g - 1, WAS)];
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const uint32_t(&x)[4] = s.o[g - 1][q];
            const uint32_t l = q ? lw.y : lw.x, r = q ? rw.y : rw.x;
            if (INTER) {
                const uint32_t left = __funnelshift_l(l, x[3], 1);
                const uint32_t right = __funnelshift_r(x[0], r, 1);
#pragma unroll
                for (int w = 0; w < 4; ++w) {
                    const uint32_t a = w == 0 ? left : x[w - 1], b = w == 3 ? right : x[w + 1];
                    s.h0[g - 1][PH][q][w] = lop3<LUT_XOR3>(a, x[w], b);
                    s.h1[g - 1][PH][q][w] = lop3<LUT_MAJ>(a, x[w], b);
                }
            } else {
#pragma unroll
                for (int w = 0; w < 4; ++w)
                    hsum(w == 0 ? l : x[w - 1], x[w], w == 3 ? r : x[w + 1], s.h0[g - 1][PH][q][w],
                         s.h1[g - 1][PH][q][w]);
            }
        }
        uint32_t up[4], down[4];
#pragma unroll
        for (int w = 0; w < 4; ++w) {
            const PairSum t = pair_sum(s.h0[g - 1][WAS][1][w], s.h1[g - 1][WAS][1][w],
                                       s.h0[g - 1][PH][0][w], s.h1[g - 1][PH][0][w]);
            up[w] = next_word_pair(s.h0[g - 1][WAS][0][w], s.h1[g - 1][WAS][0][w], t, s.cen[g - 1][w]);
            down[w] = next_word_pair(s.h0[g - 1][PH][1][w], s.h1[g - 1][PH][1][w], t, s.o[g - 1][0][w]);
            s.cen[g - 1][w] = s.o[g - 1][1][w];
            if (MASK) {
                up[w] = (unsigned)row < (unsigned)c.Y ? up[w] : 0u;
                down[w] = (unsigned)(row + 1) < (unsigned)c.Y ? down[w] : 0u;
            }
        }
        if (g == K) {
            uint32_t* d = c.dst + (long long)row * c.pitch + c.base;
            if (c.own && (!TEST || row >= c.y0) && (!(TEST || MASK) || row < c.y1)) store_words<4>(d, up);
            if (c.own && (!TEST || row + 1 >= c.y0) && (!(TEST || MASK) || row + 1 < c.y1))
                store_words<4>(d + c.pitch, down);
        } else {
#pragma unroll
            for (int w = 0; w < 4; ++w) {
                s.o[g][0][w] = up[w];
                s.o[g][1][w] = down[w];
            }
            if (c.lane_ok) {
                c.eb[1 + pair_edge(g, PH)] = make_uint2(up[0], down[0]);
                c.eb[1 + pair_last_side<K>() + pair_edge(g, PH)] = make_uint2(up[3], down[3]);
            }
        }
    }
    // Stage 0: this step's pair out of the ring, and the next copy into the
    // slot read a step ago.
    constexpr uint32_t SB = kTemporalMaxThreads * 16u;
    cp_async_wait<kPairRing - 2>();
    const uint32_t slot = c.ring + (uint32_t)(i & (kPairRing - 1)) * 2u * SB;
    lds_words_at<4>(slot, s.o[0][0]);
    lds_words_at<4>(slot + SB, s.o[0][1]);
    if (c.lane_ok) {
        c.eb[1 + pair_edge(0, PH)] = make_uint2(s.o[0][0][0], s.o[0][1][0]);
        c.eb[1 + pair_last_side<K>() + pair_edge(0, PH)] = make_uint2(s.o[0][0][3], s.o[0][1][3]);
    }
    pair_issue<K>(c, i + kPairRing - 1);
    __syncthreads();
}

template <int K, bool INTER, bool TEST, bool MASK>
__device__ __forceinline__ void pair_steps(PairRegs<K>& s, const PairCtx& c, int i0, int i1) {
    for (int i = i0; i < i1; i += 2) {   // i0 even
        pair_step<K, INTER, 0, TEST, MASK>(s, c, i);
        pair_step<K, INTER, 1, TEST, MASK>(s, c, i + 1);
    }
}

template <int K, bool INTER>
__global__ void __launch_bounds__(kTemporalMaxThreads, 1) rows_pair_kernel(RowsLaunch a) {
    extern __shared__ __align__(16) uint32_t smem[];
    PairCtx c;
    c.src = a.src;
    c.dst = a.dst;
    c.Y = a.Y;
    c.pitch = a.pitch;
    c.y0 = blockIdx.x * a.band;
    c.y1 = min(c.y0 + a.band, a.Y);
    const int xs = blockIdx.y * a.slice;
    c.base = xs - a.halo + (int)threadIdx.x * 4;
    c.lane_ok = c.base >= 0 && c.base < a.W;
    c.own = c.lane_ok && c.base >= xs && c.base < xs + a.slice;
    uint2* edges = reinterpret_cast<uint2*>(smem + kPairRing * 2 * kTemporalMaxThreads * 4);
    c.eb = edges + threadIdx.x;
    c.ring = (uint32_t)__cvta_generic_to_shared(smem + threadIdx.x * 4);
    for (int t = threadIdx.x; t < 2 * pair_last_side<K>(); t += blockDim.x) edges[t] = make_uint2(0u, 0u);
    PairRegs<K> s;
#pragma unroll
    for (int g = 0; g < K; ++g)
#pragma unroll
        for (int w = 0; w < 4; ++w) {
            s.cen[g][w] = 0u;
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                s.o[g][q][w] = 0u;
                s.h0[g][0][q][w] = s.h0[g][1][q][w] = 0u;
                s.h1[g][0][q][w] = s.h1[g][1][q][w] = 0u;
            }
        }
    __syncthreads();
    asm volatile("griddepcontrol.wait;" ::: "memory");
    for (int j = 0; j < kPairRing - 1; ++j) pair_issue<K>(c, j);
    // The last row is y1 - 1 = o_K + 1 at the latest at step (B + 1) / 2 + 2K - 1.
    const int B = c.y1 - c.y0;
    const int end = ((B + 1) / 2 + 2 * K + 1) & ~1;
    if (c.y0 - K >= 0 && c.y1 + K <= c.Y) {
        // Steady steps: every stage active and its rows wanted, i.e. from 2K
        // while o_K + 1 < y1 and stage 1's rows end at y1 - 1 + K - 1.
        const int f0 = 2 * K, f1 = max(f0, f0 + (((B - 2 * K) / 2) & ~1));
        pair_steps<K, INTER, true, false>(s, c, 0, f0);
        pair_steps<K, INTER, false, false>(s, c, f0, f1);
        asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
        pair_steps<K, INTER, true, false>(s, c, f1, end);
    } else {
        pair_steps<K, INTER, true, true>(s, c, 0, end);
        asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    }
    asm volatile("cp.async.wait_all;\n" ::: "memory");
}

// Interleaves a grid of whole lanes (n groups of four words) by four, in
// place, or restores it.
template <bool BACK>
__global__ void __launch_bounds__(256) interleave_kernel(uint4* grid, size_t n) {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
         i += (size_t)gridDim.x * blockDim.x) {
        const uint4 q = grid[i];
        uint32_t v[4] = {q.x, q.y, q.z, q.w};
        if (BACK)
            deinterleave4(v);
        else
            interleave4(v);
        grid[i] = make_uint4(v[0], v[1], v[2], v[3]);
    }
}

} // namespace golb200
