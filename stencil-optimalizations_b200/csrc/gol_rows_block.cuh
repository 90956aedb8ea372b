// Register-block pass: K generations of a block of rows held in registers.
//
// One warp advances 32 adjacent words of a row by R rows (R a compile-time
// constant): each lane keeps its word of every row in a register, loaded
// once, advanced K generations in place and stored once. There is no shared
// memory and no barrier, and the rows of a generation are independent of
// each other, so a warp alone keeps its scheduler three quarters busy. What
// bounds it is the integer pipe: ten operations per word and generation
// (two shifts, two for the horizontal sum, six for the rule, which two rows
// at a time share; gol_word_ops.cuh).
//
//   * Rows: a block of B output rows loads B + 2K rows; each generation the
//     rows still correct shrink by one at either end (about 9 % more rows
//     computed than stored at K = 8, R = 96). Generation g writes row i to
//     register i - 1, so the rows that count always start at register 0:
//     one loop body serves every generation and every K, leaving early once
//     the rows that still count are done.
//   * Columns: the words beyond a lane's own come from its neighbours by
//     shuffle. The outer two lanes are context (errors from the words beyond
//     them move one cell per generation and stay inside them for K <= 32),
//     so a warp stores 30 of its 32 columns.
//   * A row's columns need not be a multiple of 30: the columns of all blocks
//     of rows stand in one line, a dead column after each row, and warp w
//     takes columns 30 w - 1 .. 30 w + 30 of it, each lane in its own block.
//     Only warps that hold a dead column, or rows outside the grid, mask
//     their words after each generation.
//   * One warp per CTA, and the next pass is let in only when the block is
//     about to be stored: passes are programmatic dependents, and CTAs of the
//     next pass that became resident earlier took the place of this pass's
//     on some SMs (8.2 against 11.3 us per pass of 8 generations at
//     5024 x 3001, R = 32, B = 16).
// Measured (K = 8): 16384^2 63 us per pass (34 T cell-updates/s, R = 96,
// B = 80), 10240 x 6001 18.5 us (55.6 for the K-stage kernel of
// gol_rows_temporal.cuh), 5024 x 3001 7.6 us (two K-stage passes of 4: 20.8),
// 2048^2 4.4 us.
#pragma once

#include <cstdint>

#include "gol_rows_temporal.cuh"
#include "gol_word_ops.cuh"

namespace golb200 {

constexpr int kBlockOwn = 30;   // columns a warp stores

struct BlockLaunch {
    const uint32_t* src;   // gen-0 grid (row r at src + r * pitch)
    uint32_t* dst;         // gen-K grid (must not alias src)
    int W, Y, pitch;
    int B;                 // rows stored per block (even, B + 2K <= R)
    int K;
    int nblocks;           // blocks of rows
};

template <int R>
constexpr int block_min_ctas() { return R <= 32 ? 32 : R <= 48 ? 24 : R <= 64 ? 20 : 16; }

// Horizontal sum of this lane's word of one row (bit planes 0 and 1).
__device__ __forceinline__ void block_hsum(uint32_t c, uint32_t& h0, uint32_t& h1) {
    const uint32_t lw = __shfl_up_sync(0xffffffffu, c, 1);
    const uint32_t rw = __shfl_down_sync(0xffffffffu, c, 1);
    hsum(lw, c, rw, h0, h1);
}

// Rows that block_load reads for n wanted ones.
__host__ __device__ constexpr int block_rows(int n) { return (n + 7) & ~7; }

// Rows y0 .. y0 + n - 1 of one column into registers, eight at a time (p
// points at row y0 of it; it is dereferenced inside the grid only). inside:
// every row read and every column of the warp lies in the grid; ok: this
// lane's column does. CG: through L2 only, for rows that other CTAs of the
// same launch write.
template <int R, bool CG = false>
__device__ __forceinline__ void block_load(uint32_t (&w)[R], const uint32_t* p, int pitch,
                                           bool inside, bool ok, int y0, int Y, int n) {
    if (inside) {
#pragma unroll
        for (int r0 = 0; r0 < R; r0 += 8) {
            if (r0 < n) {
#pragma unroll
                for (int r = r0; r < r0 + 8 && r < R; ++r, p += pitch)
                    w[r] = CG ? __ldcg(p) : __ldg(p);
            } else {
#pragma unroll
                for (int r = r0; r < r0 + 8 && r < R; ++r) w[r] = 0u;
            }
        }
    } else {
#pragma unroll
        for (int r = 0; r < R; ++r, p += pitch) {
            const bool v = r < n && ok && (unsigned)(y0 + r) < (unsigned)Y;
            w[r] = !v ? 0u : CG ? __ldcg(p) : __ldg(p);
        }
    }
}

// K generations of the block in w (rows y0 ..): afterwards w[0 .. B-1] are
// rows y0 + K .. y0 + K + B - 1 (B + 2K <= R).
template <int R>
__device__ __forceinline__ void block_generations(uint32_t (&w)[R], int B, int K, bool inside,
                                                  bool ok, int y0, int Y) {
    static_assert(R % 4 == 0, "rows are taken two at a time, the exit tested every four");
    for (int g = 1; g <= K; ++g) {
        const int n = B + 2 * (K - g);   // rows that count after this generation
        uint32_t a0, a1, b0, b1;
        block_hsum(w[0], a0, a1);
        block_hsum(w[1], b0, b1);
#pragma unroll
        for (int j = 0; j + 3 < R; j += 2) {   // rows j + 1 and j + 2 of the block
            if (j % 4 == 0 && j >= 8 && j >= n) break;
            uint32_t p0, p1, q0, q1;
            block_hsum(w[j + 2], p0, p1);
            block_hsum(w[j + 3], q0, q1);
            const PairSum s = pair_sum(b0, b1, p0, p1);
            const uint32_t up = next_word_pair(a0, a1, s, w[j + 1]);
            const uint32_t down = next_word_pair(q0, q1, s, w[j + 2]);
            w[j] = up;
            w[j + 1] = down;
            a0 = p0;
            a1 = p1;
            b0 = q0;
            b1 = q1;
        }
        if (!inside) {   // columns and rows outside the grid stay dead
#pragma unroll
            for (int r0 = 0; r0 < R; r0 += 8) {
                if (r0 >= 8 && r0 >= n) break;
#pragma unroll
                for (int r = r0; r < r0 + 8 && r < R; ++r)
                    w[r] = ok && (unsigned)(y0 + g + r) < (unsigned)Y ? w[r] : 0u;
            }
        }
    }
}

// Stores rows [0, rows) of a block of the change-tracking pass: load(p) reads
// the word before the pass, diff(r, x) gets its difference from row r's.
// Eight words are read before any of theirs is stored, and a whole group of
// eight takes no test per row (6000 generations of a sparse 16384^2 grid 12.4
// -> 12.0 ms, 1200 of a random one 15.2 -> 14.9, against row by row; groups of
// four the same; a test per row kept in predicates spills).
constexpr int kBlockAhead = 8;

template <int R, class Load, class Diff>
__device__ __forceinline__ void block_store_tracked(const uint32_t (&w)[R], int rows,
                                                    const uint32_t* old, uint32_t* out,
                                                    long long pitch, Load load, Diff diff) {
#pragma unroll
    for (int r0 = 0; r0 < R - 2; r0 += kBlockAhead, old += kBlockAhead * pitch, out += kBlockAhead * pitch) {
        if (r0 + kBlockAhead <= R - 2 && r0 + kBlockAhead <= rows) {
            uint32_t before[kBlockAhead];
#pragma unroll
            for (int i = 0; i < kBlockAhead; ++i) before[i] = load(old + i * pitch);
#pragma unroll
            for (int i = 0; i < kBlockAhead && r0 + i < R; ++i) {
                diff(r0 + i, before[i] ^ w[r0 + i]);
                out[i * pitch] = w[r0 + i];
            }
        } else {
#pragma unroll
            for (int i = 0; i < kBlockAhead && r0 + i < R - 2; ++i)
                if (r0 + i < rows) {
                    diff(r0 + i, load(old + i * pitch) ^ w[r0 + i]);
                    out[i * pitch] = w[r0 + i];
                }
        }
    }
}

template <int R>
__global__ void __launch_bounds__(32, block_min_ctas<R>()) rows_block_kernel(BlockLaunch a) {
    const int lane = threadIdx.x;
    const long long line = a.W + 1;
    const long long idx = (long long)blockIdx.x * kBlockOwn - 1 + lane;
    const int block = idx < 0 ? 0 : (int)(idx / line);
    const int col = (int)(idx - block * line);   // -1: before the first column, W: a dead column
    const bool ok = idx >= 0 && block < a.nblocks && col < a.W;
    const int y0 = block * a.B - a.K;            // row of w[0]
    const bool inside = __all_sync(0xffffffffu, ok && y0 >= 0 && y0 + block_rows(a.B + 2 * a.K) <= a.Y);
    asm volatile("griddepcontrol.wait;" ::: "memory");
    uint32_t w[R];
    block_load<R>(w, a.src + (long long)y0 * a.pitch + col, a.pitch, inside, ok, y0, a.Y,
                  a.B + 2 * a.K);
    block_generations<R>(w, a.B, a.K, inside, ok, y0, a.Y);
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    if (ok && lane >= 1 && lane <= kBlockOwn) {
        const int ys = block * a.B;
        const int rows = min(a.B, a.Y - ys);
        uint32_t* d = a.dst + (long long)ys * a.pitch + col;
#pragma unroll
        for (int r = 0; r < R - 2; ++r, d += a.pitch)
            if (r < rows) *d = w[r];
    }
}

} // namespace golb200
