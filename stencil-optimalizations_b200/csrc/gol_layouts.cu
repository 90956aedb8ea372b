// Column and tile word layouts as input / output formats beside the rows
// layout the engine computes in: GeneralBitGrid<uintW_t, BitColumnsMode |
// BitTileMode> (src/algorithms/_shared/bitwise/general_bit_grid.hpp:171-246,
// bit_modes.hpp:10-125, 165-177), the layouts of the reference's
// columns-based (Fujita) and tiled ("Core Tiled 64") kernels.
//
//   columns (W = 16/32/64): a word holds W cells of one column; cell (x, y)
//     is bit y % W (lowest bit = top cell) of word (y / W) * X + x.
//   tiles: 4x4 cells in 16-bit words, 8x4 in 32-bit, 8x8 in 64-bit; cell
//     (x, y) is bit W-1 - ((y % YB) * XB + x % XB) (top-left cell in the
//     highest bit, x fastest) of word (y / YB) * (X / XB) + x / XB.
//   rows (W = 16/32/64): cell (x, y) is bit x % W of word y * (X / W) + x / W;
//     the same bytes for every W on a little-endian host.
//
// Host conversions (cells <-> any layout; layout words <-> the engine's
// rows) run over row bands on all host threads. Device conversions between
// rows and the other layouts, for grids kept on the device:
//   columns: one warp per 128-column x 32- (or 64-) row block: lane i holds
//            four words of row y0 + i (one 16-byte access), and each 32 x 32
//            block is transposed across the lanes in five exchange steps.
//   tiles:   one thread per row word (32 columns) of a tile row: it reads the
//            rows' words, reverses their bits and moves their bytes (or
//            nibbles) into the tile words, 16 or 32 bytes in a run (and back).
// Both are bound by memory: a grid is read and written once. 16384^2 from
// columns to rows and from rows to tiles (64-bit words) takes 31 us together
// (4.3 TB/s), against 123 us with a ballot and a select per bit and a byte per
// load and store.
#include <algorithm>
#include <cstdint>
#include <cstring>
#include <thread>
#include <vector>

#include <cuda_runtime.h>

#include "gol_b200.h"
#include "gol_internal.h"

namespace golb200 {

bool layout_geom(int layout, uint32_t wb, uint32_t* xb, uint32_t* yb) {
    if (wb != 16 && wb != 32 && wb != 64) return false;
    switch (layout) {
        case GOL_LAYOUT_ROWS: *xb = wb; *yb = 1; return true;
        case GOL_LAYOUT_COLUMNS: *xb = 1; *yb = wb; return true;
        case GOL_LAYOUT_TILES:
            *xb = wb == 16 ? 4 : 8;
            *yb = wb == 64 ? 8 : 4;
            return true;
        default: return false;
    }
}

namespace {

// Bit position of cell (bx, by) inside its word.
inline uint32_t bit_of(int layout, uint32_t wb, uint32_t xb, uint32_t bx, uint32_t by) {
    switch (layout) {
        case GOL_LAYOUT_ROWS: return bx;
        case GOL_LAYOUT_COLUMNS: return by;
        default: return wb - 1 - (by * xb + bx);
    }
}

inline uint64_t get_word(const void* w, uint32_t wb, size_t i) {
    if (wb == 64) return static_cast<const uint64_t*>(w)[i];
    if (wb == 32) return static_cast<const uint32_t*>(w)[i];
    return static_cast<const uint16_t*>(w)[i];
}

inline void set_word(void* w, uint32_t wb, size_t i, uint64_t v) {
    if (wb == 64) static_cast<uint64_t*>(w)[i] = v;
    else if (wb == 32) static_cast<uint32_t*>(w)[i] = static_cast<uint32_t>(v);
    else static_cast<uint16_t*>(w)[i] = static_cast<uint16_t>(v);
}

// Runs body(r0, r1) over word rows [0, n) split across host threads.
template <typename F>
void parallel_word_rows(size_t n, size_t cells_per_row, F&& body) {
    unsigned hw = std::max(1u, usable_cpus());
    size_t nt = std::min<size_t>(hw, std::max<size_t>(1, n * cells_per_row / (1u << 20)));
    nt = std::min(nt, n ? n : 1);
    if (nt <= 1) {
        body(size_t(0), n);
        return;
    }
    std::vector<std::thread> ts;
    const size_t per = (n + nt - 1) / nt;
    for (size_t t = 0; t < nt; ++t) {
        const size_t r0 = t * per, r1 = std::min(n, r0 + per);
        if (r0 >= r1) break;
        ts.emplace_back([=, &body] { body(r0, r1); });
    }
    for (auto& th : ts) th.join();
}

} // namespace

void host_cells_to_layout(const uint8_t* cells, size_t x, size_t y, int layout, uint32_t wb,
                          uint32_t xb, uint32_t yb, void* words) {
    const size_t wx = x / xb;
    parallel_word_rows(y / yb, x * yb, [=](size_t r0, size_t r1) {
        for (size_t wy = r0; wy < r1; ++wy)
            for (size_t i = 0; i < wx; ++i) {
                uint64_t w = 0;
                for (uint32_t by = 0; by < yb; ++by) {
                    const uint8_t* row = cells + (wy * yb + by) * x + i * xb;
                    for (uint32_t bx = 0; bx < xb; ++bx)
                        if (row[bx]) w |= uint64_t(1) << bit_of(layout, wb, xb, bx, by);
                }
                set_word(words, wb, wy * wx + i, w);
            }
    });
}

void host_layout_to_cells(const void* words, size_t x, size_t y, int layout, uint32_t wb,
                          uint32_t xb, uint32_t yb, uint8_t* cells) {
    const size_t wx = x / xb;
    parallel_word_rows(y / yb, x * yb, [=](size_t r0, size_t r1) {
        for (size_t wy = r0; wy < r1; ++wy)
            for (size_t i = 0; i < wx; ++i) {
                const uint64_t w = get_word(words, wb, wy * wx + i);
                for (uint32_t by = 0; by < yb; ++by) {
                    uint8_t* row = cells + (wy * yb + by) * x + i * xb;
                    for (uint32_t bx = 0; bx < xb; ++bx)
                        row[bx] = (w >> bit_of(layout, wb, xb, bx, by)) & 1u;
                }
            }
    });
}

// Layout words -> rows words (32-bit, x % 32 == 0) and back, without a cell
// buffer: each rows word gathers its 32 cells from the layout words.
void host_layout_to_rows(const void* words, size_t x, size_t y, int layout, uint32_t wb,
                         uint32_t xb, uint32_t yb, uint32_t* rows) {
    const size_t wx = x / xb, rw = x / 32;
    parallel_word_rows(y, x, [=](size_t r0, size_t r1) {
        for (size_t cy = r0; cy < r1; ++cy) {
            const size_t wy = cy / yb;
            const uint32_t by = static_cast<uint32_t>(cy % yb);
            for (size_t j = 0; j < rw; ++j) {
                uint32_t out = 0;
                for (uint32_t b = 0; b < 32; ++b) {
                    const size_t cx = j * 32 + b;
                    const uint64_t w = get_word(words, wb, wy * wx + cx / xb);
                    out |= static_cast<uint32_t>((w >> bit_of(layout, wb, xb, cx % xb, by)) & 1u) << b;
                }
                rows[cy * rw + j] = out;
            }
        }
    });
}

void host_rows_to_layout(const uint32_t* rows, size_t x, size_t y, int layout, uint32_t wb,
                         uint32_t xb, uint32_t yb, void* words) {
    const size_t wx = x / xb, rw = x / 32;
    parallel_word_rows(y / yb, x * yb, [=](size_t r0, size_t r1) {
        for (size_t wy = r0; wy < r1; ++wy)
            for (size_t i = 0; i < wx; ++i) {
                uint64_t w = 0;
                for (uint32_t by = 0; by < yb; ++by) {
                    const uint32_t* row = rows + (wy * yb + by) * rw;
                    for (uint32_t bx = 0; bx < xb; ++bx) {
                        const size_t cx = i * xb + bx;
                        if ((row[cx / 32] >> (cx % 32)) & 1u)
                            w |= uint64_t(1) << bit_of(layout, wb, xb, bx, by);
                    }
                }
                set_word(words, wb, wy * wx + i, w);
            }
    });
}

namespace {

constexpr int kLayoutThreads = 256;

// Bit transpose of a 32 x 32 block, one row per lane: afterwards bit i of
// lane j is what bit j of lane i was. Step s exchanges with lane ^ s the
// halves that differ in index bit s: a shuffle, a rotation and a select.
// (Five steps of three instructions; a ballot and select per bit, as before,
// took about 100.)
__device__ __forceinline__ uint32_t transpose32(uint32_t v, int lane) {
#pragma unroll
    for (int s = 16; s >= 1; s >>= 1) {
        const uint32_t low = s == 16 ? 0x0000ffffu : s == 8 ? 0x00ff00ffu : s == 4 ? 0x0f0f0f0fu
                             : s == 2 ? 0x33333333u : 0x55555555u;   // bits whose index bit s is 0
        const bool up = lane & s;
        const uint32_t o = __shfl_xor_sync(0xffffffffu, v, s);
        const uint32_t r = __funnelshift_l(o, o, up ? 32 - s : s);
        const uint32_t keep = up ? ~low : low;
        v = (v & keep) | (r & ~keep);
    }
    return v;
}

// Up to four words at p, those from n on zero; vec: one 16-byte access.
__device__ __forceinline__ uint4 load_row4(const uint32_t* p, int n, bool vec) {
    if (vec) return __ldg(reinterpret_cast<const uint4*>(p));
    uint4 v = make_uint4(0u, 0u, 0u, 0u);
    if (n > 0) v.x = __ldg(p);
    if (n > 1) v.y = __ldg(p + 1);
    if (n > 2) v.z = __ldg(p + 2);
    if (n > 3) v.w = __ldg(p + 3);
    return v;
}

__device__ __forceinline__ void store_row4(uint32_t* p, const uint32_t (&v)[4], int n, bool vec) {
    if (vec) {
        *reinterpret_cast<uint4*>(p) = make_uint4(v[0], v[1], v[2], v[3]);
        return;
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
        if (i < n) p[i] = v[i];
}

// Rows -> columns. A warp takes four word columns (wx .. wx + 3) of the row
// group g of R = max(W, 32) rows; lane j ends with columns 32 * (wx + i) + j.
// vec: every row's words start on a 16-byte boundary.
template <int WB>
__global__ void __launch_bounds__(kLayoutThreads)
rows_to_columns_kernel(const uint32_t* __restrict__ rows, void* __restrict__ cols, int X, int Y,
                       bool vec) {
    constexpr int R = WB > 32 ? WB : 32;
    const int Wx = X / 32, quads = (Wx + 3) / 4;
    const long long w = (long long)blockIdx.x * (kLayoutThreads / 32) + (threadIdx.x >> 5);
    const int groups = (Y + R - 1) / R;
    if (w >= (long long)quads * groups) return;   // whole warp
    const int lane = threadIdx.x & 31;
    const int g = (int)(w / quads), wx = (int)(w - (long long)g * quads) * 4, y0 = g * R;
    const int n = min(4, Wx - wx);
    uint32_t m[R / 32][4];
#pragma unroll
    for (int h = 0; h < R / 32; ++h) {
        const int r = y0 + 32 * h + lane;
        const uint4 v = load_row4(rows + (size_t)r * Wx + wx, r < Y ? n : 0, vec && r < Y);
        m[h][0] = v.x;
        m[h][1] = v.y;
        m[h][2] = v.z;
        m[h][3] = v.w;
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        if (i >= n) break;   // the same for the whole warp
        uint32_t t[R / 32];
#pragma unroll
        for (int h = 0; h < R / 32; ++h) t[h] = transpose32(m[h][i], lane);
        const size_t x = (size_t)(wx + i) * 32 + lane;
        if (WB == 64) {
            static_cast<uint64_t*>(cols)[(size_t)(y0 / 64) * X + x] =
                (uint64_t)t[0] | ((uint64_t)t[R / 32 - 1] << 32);
        } else if (WB == 32) {
            static_cast<uint32_t*>(cols)[(size_t)(y0 / 32) * X + x] = t[0];
        } else {
            uint16_t* c = static_cast<uint16_t*>(cols);
            c[(size_t)(y0 / 16) * X + x] = (uint16_t)t[0];
            if (y0 + 16 < Y) c[(size_t)(y0 / 16 + 1) * X + x] = (uint16_t)(t[0] >> 16);
        }
    }
}

template <int WB>
__global__ void __launch_bounds__(kLayoutThreads)
columns_to_rows_kernel(const void* __restrict__ cols, uint32_t* __restrict__ rows, int X, int Y,
                       bool vec) {
    constexpr int R = WB > 32 ? WB : 32;
    const int Wx = X / 32, quads = (Wx + 3) / 4;
    const long long w = (long long)blockIdx.x * (kLayoutThreads / 32) + (threadIdx.x >> 5);
    const int groups = (Y + R - 1) / R;
    if (w >= (long long)quads * groups) return;
    const int lane = threadIdx.x & 31;
    const int g = (int)(w / quads), wx = (int)(w - (long long)g * quads) * 4, y0 = g * R;
    const int n = min(4, Wx - wx);
    uint32_t m[R / 32][4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const size_t x = (size_t)(wx + i) * 32 + lane;
        uint32_t lo = 0u, hi = 0u;
        if (i < n) {
            if (WB == 64) {
                const uint64_t c =
                    __ldg(static_cast<const unsigned long long*>(cols) + (size_t)(y0 / 64) * X + x);
                lo = (uint32_t)c;
                hi = (uint32_t)(c >> 32);
            } else if (WB == 32) {
                lo = __ldg(static_cast<const uint32_t*>(cols) + (size_t)(y0 / 32) * X + x);
            } else {
                const uint16_t* c = static_cast<const uint16_t*>(cols);
                lo = __ldg(c + (size_t)(y0 / 16) * X + x);
                if (y0 + 16 < Y) lo |= (uint32_t)__ldg(c + (size_t)(y0 / 16 + 1) * X + x) << 16;
            }
        }
        m[0][i] = lo;
        if (R > 32) m[R / 32 - 1][i] = hi;
    }
#pragma unroll
    for (int h = 0; h < R / 32; ++h) {
#pragma unroll
        for (int i = 0; i < 4; ++i) m[h][i] = transpose32(m[h][i], lane);
        const int r = y0 + 32 * h + lane;
        if (r < Y) store_row4(rows + (size_t)r * Wx + wx, m[h], n, vec);
    }
}

// 4 x 4 byte transpose: byte i of v[j] becomes byte j of v[i].
__device__ __forceinline__ void transpose_bytes(uint32_t (&v)[4]) {
    const uint32_t a = __byte_perm(v[0], v[1], 0x5140), b = __byte_perm(v[2], v[3], 0x5140);
    const uint32_t c = __byte_perm(v[0], v[1], 0x7362), d = __byte_perm(v[2], v[3], 0x7362);
    v[0] = __byte_perm(a, b, 0x5410);
    v[1] = __byte_perm(a, b, 0x7632);
    v[2] = __byte_perm(c, d, 0x5410);
    v[3] = __byte_perm(c, d, 0x7632);
}

// Four rows of 32 cells (bits reversed, last row first) <-> eight 4 x 4 tiles
// in four words: the tile at nibble t from the left takes nibble 7 - t of
// every reversed row, the first row's in its highest nibble.
__device__ __forceinline__ void nibble_pairs(uint32_t a, uint32_t b, uint32_t& even, uint32_t& odd) {
    even = (a & 0x0f0f0f0fu) | ((b << 4) & 0xf0f0f0f0u);
    odd = ((a >> 4) & 0x0f0f0f0fu) | (b & 0xf0f0f0f0u);
}

// Rows -> tiles and back, one thread per (row word, tile row): the 32 cells
// of a row word are four 8-cell tile rows or eight 4-cell ones. A tile row's
// byte is the row's byte with its bits reversed, the first row's highest, so
// reversed words in reverse row order, transposed by bytes, are the tiles from
// right to left. vec: the tile words of a thread start on a 16-byte boundary.
template <int WB>
__global__ void __launch_bounds__(kLayoutThreads)
rows_to_tiles_kernel(const uint32_t* __restrict__ rows, uint32_t* __restrict__ tiles, int X, int Y,
                     bool vec) {
    constexpr int YB = WB == 64 ? 8 : 4;
    const int Wx = X / 32;
    const long long t = (long long)blockIdx.x * kLayoutThreads + threadIdx.x;
    if (t >= (long long)Wx * (Y / YB)) return;
    const int ty = (int)(t / Wx), c = (int)(t - (long long)ty * Wx);
    uint32_t v[YB];
#pragma unroll
    for (int y = 0; y < YB; ++y) v[y] = __ldg(rows + (size_t)(ty * YB + y) * Wx + c);
    uint32_t out[YB];   // the thread's tile words, 32 bits at a time
    uint32_t q[4];
#pragma unroll
    for (int y = 0; y < 4; ++y) q[y] = __brev(v[YB - 1 - y]);
    if (WB == 16) {
        uint32_t x, y, u, w;
        nibble_pairs(q[0], q[1], x, y);   // rows 3 and 2
        nibble_pairs(q[2], q[3], u, w);   // rows 1 and 0
        const uint32_t yh = __byte_perm(y, w, 0x6273), xh = __byte_perm(x, u, 0x6273);
        const uint32_t yl = __byte_perm(y, w, 0x4051), xl = __byte_perm(x, u, 0x4051);
        out[0] = __byte_perm(yh, xh, 0x5410);
        out[1] = __byte_perm(yh, xh, 0x7632);
        out[2] = __byte_perm(yl, xl, 0x5410);
        out[YB - 1] = __byte_perm(yl, xl, 0x7632);
    } else {
        transpose_bytes(q);
        if (WB == 32) {
#pragma unroll
            for (int i = 0; i < 4; ++i) out[i] = q[3 - i];
        } else {
            uint32_t p[4];
#pragma unroll
            for (int y = 0; y < 4; ++y) p[y] = __brev(v[3 - y]);
            transpose_bytes(p);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                out[(2 * i) % YB] = q[3 - i];
                out[(2 * i + 1) % YB] = p[3 - i];
            }
        }
    }
    uint32_t* d = tiles + (size_t)t * YB;
    if (vec) {
#pragma unroll
        for (int i = 0; i < YB; i += 4)
            *reinterpret_cast<uint4*>(d + i) = make_uint4(out[i], out[i + 1], out[i + 2], out[i + 3]);
    } else {
#pragma unroll
        for (int i = 0; i < YB; ++i) d[i] = out[i];
    }
}

template <int WB>
__global__ void __launch_bounds__(kLayoutThreads)
tiles_to_rows_kernel(const uint32_t* __restrict__ tiles, uint32_t* __restrict__ rows, int X, int Y,
                     bool vec) {
    constexpr int YB = WB == 64 ? 8 : 4;
    const int Wx = X / 32;
    const long long t = (long long)blockIdx.x * kLayoutThreads + threadIdx.x;
    if (t >= (long long)Wx * (Y / YB)) return;
    const int ty = (int)(t / Wx), c = (int)(t - (long long)ty * Wx);
    const uint32_t* s = tiles + (size_t)t * YB;
    uint32_t in[YB];
    if (vec) {
#pragma unroll
        for (int i = 0; i < YB; i += 4) {
            const uint4 f = __ldg(reinterpret_cast<const uint4*>(s + i));
            in[i] = f.x;
            in[i + 1] = f.y;
            in[i + 2] = f.z;
            in[i + 3] = f.w;
        }
    } else {
#pragma unroll
        for (int i = 0; i < YB; ++i) in[i] = __ldg(s + i);
    }
    uint32_t v[YB];
    uint32_t q[4];
    if (WB == 16) {
        const uint32_t yh = __byte_perm(in[0], in[1], 0x5410), xh = __byte_perm(in[0], in[1], 0x7632);
        const uint32_t yl = __byte_perm(in[2], in[3], 0x5410), xl = __byte_perm(in[2], in[3], 0x7632);
        // bytes 3, 2 (upper half) and 1, 0 of the four pair words
        const uint32_t y = __byte_perm(yh, yl, 0x0246), w = __byte_perm(yh, yl, 0x1357);
        const uint32_t x = __byte_perm(xh, xl, 0x0246), u = __byte_perm(xh, xl, 0x1357);
        q[0] = (x & 0x0f0f0f0fu) | ((y << 4) & 0xf0f0f0f0u);
        q[1] = ((x >> 4) & 0x0f0f0f0fu) | (y & 0xf0f0f0f0u);
        q[2] = (u & 0x0f0f0f0fu) | ((w << 4) & 0xf0f0f0f0u);
        q[3] = ((u >> 4) & 0x0f0f0f0fu) | (w & 0xf0f0f0f0u);
    } else {
#pragma unroll
        for (int i = 0; i < 4; ++i) q[3 - i] = in[WB == 64 ? (2 * i) % YB : i];
        transpose_bytes(q);
        if (WB == 64) {
            uint32_t p[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) p[3 - i] = in[(2 * i + 1) % YB];
            transpose_bytes(p);
#pragma unroll
            for (int y = 0; y < 4; ++y) v[3 - y] = __brev(p[y]);
        }
    }
#pragma unroll
    for (int y = 0; y < 4; ++y) v[YB - 1 - y] = __brev(q[y]);
#pragma unroll
    for (int y = 0; y < YB; ++y) rows[(size_t)(ty * YB + y) * Wx + c] = v[y];
}

template <int WB>
cudaError_t launch_convert(bool to_rows, int layout, const void* src, void* dst, int X, int Y,
                           cudaStream_t s) {
    if (layout == GOL_LAYOUT_COLUMNS) {
        constexpr int R = WB > 32 ? WB : 32;
        const long long warps = (long long)((X / 32 + 3) / 4) * ((Y + R - 1) / R);
        const long long blocks = (warps + kLayoutThreads / 32 - 1) / (kLayoutThreads / 32);
        const bool vec = X % 128 == 0 && ((uintptr_t)(to_rows ? dst : src) & 15u) == 0;
        if (to_rows)
            columns_to_rows_kernel<WB><<<(unsigned)blocks, kLayoutThreads, 0, s>>>(
                src, static_cast<uint32_t*>(dst), X, Y, vec);
        else
            rows_to_columns_kernel<WB><<<(unsigned)blocks, kLayoutThreads, 0, s>>>(
                static_cast<const uint32_t*>(src), dst, X, Y, vec);
    } else {
        constexpr int YB = WB == 64 ? 8 : 4;
        const long long threads = (long long)(X / 32) * (Y / YB);
        const long long blocks = (threads + kLayoutThreads - 1) / kLayoutThreads;
        const bool vec = ((uintptr_t)(to_rows ? src : dst) & 15u) == 0;
        if (to_rows)
            tiles_to_rows_kernel<WB><<<(unsigned)blocks, kLayoutThreads, 0, s>>>(
                static_cast<const uint32_t*>(src), static_cast<uint32_t*>(dst), X, Y, vec);
        else
            rows_to_tiles_kernel<WB><<<(unsigned)blocks, kLayoutThreads, 0, s>>>(
                static_cast<const uint32_t*>(src), static_cast<uint32_t*>(dst), X, Y, vec);
    }
    return cudaPeekAtLastError();
}

int device_convert(bool to_rows, const void* src, void* dst, uint64_t x, uint64_t y, int layout,
                   uint32_t wb, void* stream) {
    uint32_t xb, yb;
    if (!layout_geom(layout, wb, &xb, &yb) || layout == GOL_LAYOUT_ROWS) return GOL_E_INVALID;
    if ((!src || !dst) && x * y) return GOL_E_INVALID;
    if (x % 32 || y % yb || x > (1u << 30) || y > (1u << 30)) return GOL_E_INVALID;
    if (((uintptr_t)src | (uintptr_t)dst) & (wb / 8 - 1) || ((uintptr_t)src | (uintptr_t)dst) & 3u)
        return GOL_E_INVALID;
    if (x * y == 0) return GOL_OK;
    auto s = static_cast<cudaStream_t>(stream);
    cudaError_t ce;
    switch (wb) {
        case 64: ce = launch_convert<64>(to_rows, layout, src, dst, (int)x, (int)y, s); break;
        case 32: ce = launch_convert<32>(to_rows, layout, src, dst, (int)x, (int)y, s); break;
        default: ce = launch_convert<16>(to_rows, layout, src, dst, (int)x, (int)y, s); break;
    }
    return ce == cudaSuccess ? GOL_OK : GOL_E_CUDA;
}

} // namespace
} // namespace golb200

extern "C" {

int gol_pack_layout(const uint8_t* cells, uint64_t x, uint64_t y, int layout, uint32_t word_bits,
                    void* words) {
    uint32_t xb, yb;
    if (!golb200::layout_geom(layout, word_bits, &xb, &yb)) return GOL_E_INVALID;
    if (x % xb || y % yb || ((!cells || !words) && x * y)) return GOL_E_INVALID;
    golb200::host_cells_to_layout(cells, x, y, layout, word_bits, xb, yb, words);
    return GOL_OK;
}

int gol_unpack_layout(const void* words, uint64_t x, uint64_t y, int layout, uint32_t word_bits,
                      uint8_t* cells) {
    uint32_t xb, yb;
    if (!golb200::layout_geom(layout, word_bits, &xb, &yb)) return GOL_E_INVALID;
    if (x % xb || y % yb || ((!cells || !words) && x * y)) return GOL_E_INVALID;
    golb200::host_layout_to_cells(words, x, y, layout, word_bits, xb, yb, cells);
    return GOL_OK;
}

int gol_layout_to_rows_device(const void* d_src, void* d_rows, uint64_t x, uint64_t y, int layout,
                              uint32_t word_bits, void* stream) {
    return golb200::device_convert(true, d_src, d_rows, x, y, layout, word_bits, stream);
}

int gol_rows_to_layout_device(const void* d_rows, void* d_dst, uint64_t x, uint64_t y, int layout,
                              uint32_t word_bits, void* stream) {
    return golb200::device_convert(false, d_rows, d_dst, x, y, layout, word_bits, stream);
}

} // extern "C"
