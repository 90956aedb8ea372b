// Kernel instantiations and launch dispatch for the row-band temporal
// kernel, plus device-side pack/unpack between uint8 cells and row words.
#include <algorithm>
#include <climits>
#include <cmath>

#include "gol_b200.h"
#include "gol_internal.h"
#include "gol_rows_block.cuh"
#include "gol_rows_pair.cuh"
#include "gol_rows_resident.cuh"
#include "gol_rows_stream.cuh"
#include "gol_rows_temporal.cuh"
#include "gol_word_ops.cuh"

#ifndef GOL_STREAM_THREADS
#define GOL_STREAM_THREADS 128   // CTA size of the one-generation streaming kernel
#endif

namespace golb200 {

namespace {

// Launched as a programmatic dependent of the previous kernel in the
// stream: its CTAs may be scheduled while that kernel drains and wait in
// griddepcontrol.wait (full completion and memory flush of the previous
// grid) before touching global memory, which hides the launch gap between
// consecutive passes.
template <int WPL, int K>
cudaError_t launch_one(const RowsLaunch& a, const RowsPlan& p, cudaStream_t stream) {
    // Deep passes need more than the default 48 KB of dynamic shared memory
    // (the edge table grows with K).
    static std::atomic<uint64_t> raised{0};
    const cudaError_t e = raise_smem_limit((const void*)rows_temporal_kernel<WPL, K>,
                                           temporal_smem_bytes(K, kTemporalMaxThreads, WPL), raised);
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(p.nbands, p.nslices);
    cfg.blockDim = dim3(p.threads);
    cfg.dynamicSmemBytes = temporal_smem_bytes(K, p.threads, WPL);
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, rows_temporal_kernel<WPL, K>, a);
}

// The one-generation streaming kernel, also a programmatic dependent.
template <int WPL>
cudaError_t launch_stream(const RowsLaunch& a, const RowsPlan& p, cudaStream_t stream) {
    cudaLaunchConfig_t cfg = {};
    const long long ctas = (long long)p.nslices * p.nbands;
    if (ctas > 0x7fffffffLL) return cudaErrorInvalidConfiguration;
    cfg.gridDim = dim3((unsigned)ctas);
    cfg.blockDim = dim3(p.threads);
    cfg.dynamicSmemBytes = 0;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, p.once ? rows_once_kernel<WPL> : rows_stream_kernel<WPL>, a);
}

// The register-block kernel, a programmatic dependent too.
template <int R>
cudaError_t launch_block(const BlockLaunch& a, cudaStream_t stream) {
    const long long warps = ((long long)a.nblocks * (a.W + 1) + kBlockOwn - 1) / kBlockOwn;
    if (warps > 0x7fffffffLL) return cudaErrorInvalidConfiguration;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)warps);
    cfg.blockDim = dim3(32);
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, rows_block_kernel<R>, a);
}

// The row-pair pipeline, a programmatic dependent too.
template <bool INTER>
cudaError_t launch_pair(const RowsLaunch& a, const RowsPlan& p, cudaStream_t stream) {
    static std::atomic<uint64_t> raised{0};
    const cudaError_t e = raise_smem_limit((const void*)rows_pair_kernel<kPairK, INTER>,
                                           pair_smem_bytes(kPairK), raised);
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(p.nbands, p.nslices);
    cfg.blockDim = dim3(p.threads);
    cfg.dynamicSmemBytes = pair_smem_bytes(kPairK);
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, rows_pair_kernel<kPairK, INTER>, a);
}

// Estimated time (us) of a register-block pass and its best block. Fitted to
// passes at 256^2 .. 16384^2, K = 4 and 8, to about 10 %: a warp takes
// `rows` row-generations (plus about 2.5 a generation for the exits every
// four rows and the first two rows' sums) at 28.5 cycles each when it has its
// scheduler to itself, 25.5 beside one other and 23.5 beside more (the
// integer pipe alone: 20), a few cycles a row for loads and stores, and a
// pass a fixed part for its launch and first loads. Short blocks waste rows,
// tall ones leave schedulers idle, so the block's height is searched.
struct BlockChoice {
    int R = 0, B = 0;
    double us = 0;
};

BlockChoice best_block(int W, int Y, int k, int num_sms) {
    // A caller's passes are mostly of one shape: the thread's last choice is
    // kept (the search takes about a microsecond, a launch two).
    thread_local int last[4] = {0, 0, 0, 0};
    thread_local BlockChoice kept;
    const int shape[4] = {W, Y, k, num_sms};
    if (std::equal(shape, shape + 4, last)) return kept;
    BlockChoice best;
    for (int R : {32, 48, 64, 96}) {
        for (int B = std::min(R - 2 * k, (Y + 1) / 2 * 2); B >= 2; B -= B > 4 ? 4 : 2) {
            const long long nblocks = ((long long)Y + B - 1) / B;
            const double warps = (double)(nblocks * (W + 1)) / kBlockOwn;
            double n = warps / (4.0 * num_sms);   // warps per scheduler
            if (n < 8) n = std::ceil(n);
            const double cycles = n <= 1 ? 28.5 : n <= 2 ? 25.5 : 23.5;
            const double rows = (double)k * (B + k - 1 + 2.5);
            const double us = 0.9 + 0.018 * R + n * (0.0083 * R + rows * cycles / 1965.0);
            if (!best.R || us < best.us) best = {R, B, us};
        }
    }
    std::copy(shape, shape + 4, last);
    kept = best;
    return best;
}

template <int WPL, int K>
cudaError_t dispatch_k(int k, const RowsLaunch& a, const RowsPlan& p, cudaStream_t stream) {
    if constexpr (K > kMaxKForWpl(WPL)) {
        return cudaErrorInvalidValue;
    } else {
        if (k == K) return launch_one<WPL, K>(a, p, stream);
        return dispatch_k<WPL, K + 1>(k, a, p, stream);
    }
}

} // namespace

int device_sm_count(int device) {
    int n = 0;
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, device) != cudaSuccess) n = 148;
    return n > 0 ? n : 148;
}

// Plans the row-pair pipeline and estimates a pass on interleaved rows (us; 0
// where rows are not whole lanes): whole waves of CTAs (two of up to four
// warps per SM, or one), each taking its rows and the K that fill its stages
// at 0.42 us per two rows and warp on the fullest scheduler, 0.57 for a warp
// alone there. Against 16384^2 (25.4 us), 12288^2 (20.5), 32768^2 (89) and
// 8192 x 16384 (18.3) it is 1, -1, 9 and 0 % off.
static double plan_pair(int W, int Y, int num_sms, RowsPlan* p) {
    if (W % 4 || W <= 0) return 0;
    const int lanes = W / 4;
    int slice = lanes, nslices = 1, halo = 0;
    if (lanes > kTemporalMaxThreads) {
        const int per = kTemporalMaxThreads - 2;   // one halo lane each side
        nslices = (lanes + per - 1) / per;
        slice = (lanes + nslices - 1) / nslices;
        nslices = (lanes + slice - 1) / slice;
        halo = 4;
    }
    const int threads = (slice + (halo ? 2 : 0) + 31) / 32 * 32;
    const int per_sm = threads <= 128 ? 2 : 1;
    const int target = std::max(1, per_sm * num_sms / nslices);   // CTAs along y per wave
    double best = 0;
    const int warps = (per_sm * threads / 32 + 3) / 4;   // per scheduler
    for (int waves = 1;; ++waves) {   // the fewest waves of bands of up to 120 rows (taller
                                      // ones leave a long tail: 32768^2 102 us at 222, 89 at 112)
        int band = (int)(((long long)Y + (long long)target * waves - 1) / ((long long)target * waves));
        band = std::max(8, (band + 1) / 2 * 2);
        if (band > 120) continue;
        best = 1.0 + waves * 0.5 * (band + kPairK) * (warps == 1 ? 0.57 : 0.42 * warps);
        p->wpl = 4;
        p->threads = threads;
        p->band = band;
        p->nbands = (Y + band - 1) / band;
        p->slice = slice * 4;
        p->nslices = nslices;
        p->halo = halo;
        break;
    }
    p->stream = false;
    p->block = 0;
    p->pair = true;
    return best;
}

// CTAs per SM that the K-stage pipeline's bands are cut for.
static int stage_ctas_per_sm(int warps) { return warps >= 4 ? 2 : 2 * ((4 + warps - 1) / warps); }

// The K-stage pipeline's CTAs (p->wpl words per lane).
static void plan_stage(int W, int Y, int k, int band_rows, int num_sms, RowsPlan* p) {
    const int wpl = p->wpl, lanes = W / wpl;
    if (lanes <= kTemporalMaxThreads) {
        p->slice = W;
        p->nslices = 1;
        p->halo = 0;
        p->threads = std::max(32, (lanes + 31) / 32 * 32);
    } else {
        const int per = kTemporalMaxThreads - 2;               // one halo lane each side
        const int ns = (lanes + per - 1) / per;
        const int slice_lanes = (lanes + ns - 1) / ns;
        p->slice = slice_lanes * wpl;
        p->nslices = (W + p->slice - 1) / p->slice;
        p->halo = wpl;
        p->threads = (slice_lanes + 2 + 31) / 32 * 32;
    }
    int band = band_rows;
    if (band <= 0) {
        // About two CTAs per SM, or more when a CTA has fewer than four
        // warps (narrow grids: at 8192^2, k = 4, 2-warp CTAs with 16-row
        // bands ran at 18.9 T cell-updates/s against 16.0 T with 28-row
        // ones); never thinner than a few times the depth, whose y-halo
        // costs ~k extra rows per stage per band.
        const int per_sm = stage_ctas_per_sm(p->threads / 32);
        const int target = std::max(1, per_sm * num_sms / p->nslices);
        band = (Y + target - 1) / target;
        band = std::max(band, std::max(8, 4 * k));
    }
    band = std::min(band, std::max(Y, 1));
    p->band = band;
    p->nbands = (Y + band - 1) / band;
}

// How many times as fast as the other forms the K-stage pipeline with geometry
// p is at a pass of k generations, where it is the fastest (0 elsewhere).
// On grids whose two buffers fill L2 or more it can be: it reads
// each row about once, the blocks of 30 columns their halos again, and CTAs of
// whole warps waste nothing. What it gains over the register blocks there
// depends on the words per lane, the depth and the warps per CTA, and falls
// with the share of its threads that own words (part; whole: rows of whole
// warps, which start on a line) and by the halo lanes of slices. Some pay only
// where the CTAs fill every SM alike, most of these with no short band among
// them: the next pass's CTAs, let in early, land unevenly otherwise. Measured
// from 24 to 256 MiB a buffer, us a pass, pipeline / blocks: 32768^2 64 / 74 and
// 88 / 97 (k = 2, 3), 32640 x 32768 67 / 74 and 30720 x 32768 66 / 71 (k = 2),
// 16384 x 65536 68 / 79 (k = 2; at k = 3, a short last band, 118 / 103),
// 4096 x 262144 114 / 158 and 8192 x 65536 57 / 72 (k = 4), 7936 x 67650 60 / 68
// (k = 4); in L2 the blocks win: 16384 x 12288 18 / 16 (k = 2).
static double stage_gain(const RowsPlan& p, int W, int Y, int k, int num_sms) {
    enum Fill { kAny, kEven, kNoShort };
    struct Gain {
        int wpl, k, warps;
        Fill fill;
        int words;   // least size of the grid, 2^20 words
        double whole, part;
    };
    static constexpr Gain kGains[] = {
        {4, 2, 1, kAny, 15, 1.14, 1.14},     {4, 2, 2, kNoShort, 15, 1.25, 1.25},
        {4, 2, 4, kEven, 15, 1.16, 1.13},    {4, 2, 6, kAny, 18, 1.02, 0.0},
        {4, 2, 7, kAny, 15, 1.05, 0.0},      {4, 2, 8, kAny, 15, 1.15, 1.13},
        {4, 3, 1, kAny, 12, 1.07, 1.25},
        {4, 3, 4, kNoShort, 12, 1.18, 1.13}, {4, 3, 8, kAny, 12, 1.09, 1.04},
        {4, 4, 1, kAny, 12, 1.35, 1.24},     {4, 4, 2, kAny, 8, 1.30, 1.20},
        {2, 5, 1, kAny, 12, 1.15, 0.0},      {2, 5, 4, kNoShort, 12, 1.05, 0.0},
        {2, 6, 1, kAny, 12, 1.10, 0.0},      {2, 6, 2, kAny, 8, 1.18, 1.08},
        {2, 6, 4, kNoShort, 12, 1.03, 0.0},  {2, 7, 1, kAny, 12, 1.15, 0.0},
        {2, 7, 2, kAny, 8, 1.18, 1.08},      {2, 7, 4, kAny, 12, 1.05, 0.0},
        {2, 8, 2, kAny, 32, 1.05, 0.0},      {2, 8, 4, kAny, 16, 1.05, 0.0},
        {1, 15, 4, kAny, 24, 1.04, 0.0},     {1, 16, 4, kAny, 16, 1.04, 0.0},
    };
    const int warps = p.threads / 32, lanes = p.slice / p.wpl;
    const bool even = (long long)p.nbands * p.nslices == (long long)stage_ctas_per_sm(warps) * num_sms;
    const bool no_short = even && 3ll * (Y - (p.nbands - 1) * p.band) >= p.band;
    for (const Gain& g : kGains) {
        if (g.wpl != p.wpl || g.k != k || g.warps != warps) continue;
        if ((long long)W * Y < (long long)g.words << 20) return 0;
        if (g.fill == kEven ? !even : g.fill == kNoShort && !no_short) return 0;
        const double gain =
            (p.nslices > 1 ? 0.95 : 1.0) * (lanes == p.threads ? g.whole : g.part * lanes / p.threads);
        return gain > 1.015 ? gain : 0;
    }
    return 0;
}

// The depth at which a generation costs least, a tie going to the row-pair
// pipeline (its interleaved passes against the register-block ones). Tall
// narrow grids on which the K-stage pipeline beats the blocks at depth 4 by
// more than they gain from 4 to 8 (1.2 times) take it: 4096 x 131072 15.6 us a
// generation against 17.2 at depth 8, 8192 x 65536 14.0 against 15.1.
int best_depth(int W, int Y, int num_sms) {
    int best = 4;
    double t = 0;
    RowsPlan pair, stage;
    if (W % 4 == 0 && W > 0) {
        stage.wpl = 4;
        plan_stage(W, Y, 4, 0, num_sms, &stage);
        if (stage_gain(stage, W, Y, 4, num_sms) > 1.2) return 4;
    }
    for (int k : {4, 6, 8, 12, 16}) {
        const double u = best_block(W, std::max(Y, 1), k, num_sms).us / k;
        if (t == 0 || u < t) {
            t = u;
            best = k;
        }
    }
    const double u = plan_pair(W, Y, num_sms, &pair) / kPairK;
    return u > 0 && u <= t ? kPairK : best;
}

bool plan_rows(int W, int Y, int k, int band_rows, int wpl, int num_sms, RowsPlan* plan,
               bool k_stage) {
    if (k < 1 || k > kMaxTemporalSteps || W <= 0) return false;
    const bool forced = wpl != 0 || band_rows > 0;
    if (wpl != 0) {
        if ((wpl != 1 && wpl != 2 && wpl != 4) || W % wpl || k > kMaxKForWpl(wpl)) return false;
    } else {
        // Widest lane access whose register rings fit this depth.
        for (int cand : {4, 2, 1}) {
            if (W % cand == 0 && k <= kMaxKForWpl(cand)) {
                wpl = cand;
                break;
            }
        }
        if (wpl == 0) return false;
    }
    plan->wpl = wpl;
    const int lanes = W / wpl;
    plan->stream = k == 1 && !k_stage;
    plan->block = 0;
    plan->pair = false;
    if (plan->stream) {
        // One generation: lanes of wpl words across the row, each thread
        // loading its short band whole, or with a forced band walking that.
        plan->once = band_rows <= 0;
        plan->threads = std::min(plan->once ? kOnceThreads : GOL_STREAM_THREADS, (lanes + 31) / 32 * 32);
        // Rows of an odd number of warps: CTAs of one (with two, a row of
        // three has a CTA half idle: 12288 x 32768 20.1 us, 17.6 so).
        if (plan->once && (lanes + 31) / 32 % 2) plan->threads = 32;
        plan->nslices = (lanes + plan->threads - 1) / plan->threads;
        plan->slice = plan->threads * wpl;
        plan->halo = 0;
        const int band = plan->once ? wpl == 4 ? once_rows<4>() : wpl == 2 ? once_rows<2>() : once_rows<1>()
                                    : std::min(band_rows, std::max(Y, 1));
        plan->band = band;
        plan->nbands = (Y + band - 1) / band;
        return true;
    }
    plan_stage(W, Y, k, band_rows, num_sms, plan);
    if (k > 1 && !k_stage && !forced && stage_gain(*plan, W, Y, k, num_sms) == 0) {
        const BlockChoice c = best_block(W, std::max(Y, 1), k, num_sms);
        if (k == kPairK) {   // rows as they are take the pipeline an eighth longer
            const double us = 1.13 * plan_pair(W, Y, num_sms, plan);
            if (us > 0 && us <= c.us) return true;
            plan->pair = false;
        }
        plan->wpl = 1;
        plan->threads = 32;
        plan->block = c.R;
        plan->band = c.B;
        plan->nbands = (int)(((long long)Y + c.B - 1) / c.B);
        plan->slice = kBlockOwn;
        plan->nslices = (W + kBlockOwn - 1) / kBlockOwn;
        plan->halo = 1;
    }
    return true;
}

#ifndef GOL_RESIDENT_K
#define GOL_RESIDENT_K 8   // generations per epoch of the resident run
#endif
#ifndef GOL_RESIDENT_THREADS
#define GOL_RESIDENT_THREADS 512   // threads per CTA (lanes across a row x row groups)
#endif

// Row groups of a resident run's CTA (bands of `band` rows of `lanes` lanes). A
// generation is a chain (barrier, row loads, the thread's rows) on narrow
// bands, and integer work of the fullest scheduler on wide ones. Measured over
// 100 shapes, every count of groups, us per 1024 generations:
//   under 16 lanes a row a group, up to 256 threads or so (544 x 700: 824 with
//   two rows a group, 698 so; 512^2 747, 630), with 8 lanes half of them on
//   short bands (bank conflicts between the groups of a warp: 1024 x 4096 811,
//   748);
//   16 lanes, rows of whole half-warps and wide rows: counts that load the four
//   schedulers alike (2048^2 784 with 11 groups, 757 with 8; 12288 x 1024 1447
//   with 5, 1366 with 4; 4096^2 1030 with 16, 943 with 8; 8192 x 1024 1025 with
//   8, 960 with 4; 8192^2 1948 with 8, 1978 with 4, 1927 with 6);
//   others two rows or more a group, up to the CTA's threads.
static int resident_groups(int lanes, int band, int K) {
    const int most = std::min(GOL_RESIDENT_THREADS, kResidentMaxThreads) / lanes;
    int n = (band + K + 1) / 2;
    if (lanes < 16) {
        n = std::min(lanes > 12 ? 20 : std::min(32, 256 / lanes), band + 2 * K);
        if (lanes == 8 && band < 40) n = std::min(n, 16);
    } else if (lanes == 16) {
        n = band < 20 ? 8 : 20;
    } else if (lanes > 80 && lanes <= 112) {
        n = 4;
    } else if (lanes % 16 == 0 && lanes >= 32 && lanes <= 80) {
        n = lanes < 64 ? 8 : band < 28 ? 4 : 6;
    }
    return std::max(1, std::min(n, most));
}

bool plan_resident(int W, int Y, int k_epoch, int device, ResidentPlan* p) {
    const int K = k_epoch > 0 ? k_epoch : GOL_RESIDENT_K;
    if (K < 1 || K > 64 || W <= 0 || Y <= 0) return false;
    const int lanes = (W + 3) / 4;
    // The grids a resident run takes (gol_init refuses the others): rows of up
    // to 1024 words, 512 when odd, and bands whose two buffers fit with rows
    // of `accepted` words (the rows themselves are shorter).
    const int unit = W % 2 ? 1 : 2;
    const int accepted = (W / unit + 31) / 32 * 32 * unit + 8;
    if ((W / unit + 31) / 32 * 32 > kResidentMaxThreads) return false;
    int sms = 0, smem_max = 0, coop = 0;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess ||
        cudaDeviceGetAttribute(&smem_max, cudaDevAttrMaxSharedMemoryPerBlockOptin, device) != cudaSuccess ||
        cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, device) != cudaSuccess || !coop)
        return false;
    // Every band at least K rows (a band's halo comes from its neighbours
    // only), at most one CTA per SM; the largest band's two buffers must fit.
    // A grid of fewer than K rows is one band with no neighbours.
    const int nbands = std::max(1, std::min(sms, Y / K));
    const int band = (Y + nbands - 1) / nbands;
    if (2ull * (band + 2 * K) * accepted * sizeof(uint32_t) + 1024 > (size_t)smem_max) return false;
    const size_t smem = resident_smem_bytes(band, K, lanes);
    p->lanes = lanes;
    p->groups = resident_groups(lanes, band, K);
    p->K = K;
    p->band = band;
    p->nbands = nbands;
    p->smem = smem;
    p->pub_words = (size_t)nbands * 4 * K * 4 * lanes;
    return true;
}

template <int LANES>
static cudaError_t launch_resident_lanes(const ResidentLaunch& a, const ResidentPlan& p,
                                         cudaStream_t stream) {
    cudaError_t e = cudaFuncSetAttribute(rows_resident_kernel<LANES>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, (int)p.smem);
    if (e != cudaSuccess) return e;
    ResidentLaunch arg = a;
    void* args[] = {&arg};
    // whole warps: the threads past the last row group are idle in the passes
    return cudaLaunchCooperativeKernel((const void*)rows_resident_kernel<LANES>, dim3(p.nbands),
                                       dim3((p.lanes * p.groups + 31) / 32 * 32), args, p.smem,
                                       stream);
}

cudaError_t launch_resident(const uint32_t* src, uint32_t* dst, int W, int Y, long long gens,
                            const ResidentPlan& p, unsigned long long* pub, int* epochs_done,
                            int* status, cudaStream_t stream, long long spin_limit) {
    const long long epochs = (gens + p.K - 1) / p.K;
    int epoch0 = *epochs_done;
    cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
    cudaError_t e = cudaStreamIsCapturing(stream, &capture);
    // Numbers about to run out, or a launch that may be replayed: from zero. (A
    // replay leaves tags up to its epochs, which later launches count on from.)
    const bool full = epoch0 + epochs >= INT_MAX;
    if (full || capture != cudaStreamCaptureStatusNone) {
        if (e == cudaSuccess) e = cudaMemsetAsync(pub, 0, p.pub_words * sizeof(unsigned long long), stream);
        if (full) *epochs_done = 0;
        epoch0 = 0;
    }
    if (e == cudaSuccess) e = cudaMemsetAsync(status, 0, sizeof(int), stream);
    if (e != cudaSuccess) return e;
    *epochs_done = std::max(*epochs_done, (int)(epoch0 + epochs));
    ResidentLaunch a{src, dst, pub, status, W, Y, p.K, p.lanes, p.groups, gens,
                     spin_limit > 0 ? spin_limit : (1ll << 24), epoch0};
    // Rows of 4096, 8192 and 16384 cells get a compile-time row stride.
    switch (p.lanes) {
        case 32: return launch_resident_lanes<32>(a, p, stream);
        case 64: return launch_resident_lanes<64>(a, p, stream);
        case 128: return launch_resident_lanes<128>(a, p, stream);
        default: return launch_resident_lanes<0>(a, p, stream);
    }
}

cudaError_t launch_rows_pass(const uint32_t* src, uint32_t* dst, int W, int Y, int k,
                             const RowsPlan& p, cudaStream_t stream, int pitch, bool interleaved) {
    if (Y <= 0 || W <= 0) return cudaSuccess;
    if (p.block) {
        if (k < 1 || p.band + 2 * k > p.block) return cudaErrorInvalidValue;
        const BlockLaunch b{src, dst, W, Y, pitch ? pitch : W, p.band, k, p.nbands};
        switch (p.block) {
            case 32: return launch_block<32>(b, stream);
            case 48: return launch_block<48>(b, stream);
            case 64: return launch_block<64>(b, stream);
            case 96: return launch_block<96>(b, stream);
            default: return cudaErrorInvalidValue;
        }
    }
    RowsLaunch a{src, dst, W, Y, p.band, p.slice, p.halo, pitch ? pitch : W};
    if (p.pair) {
        if (k != kPairK || a.pitch % 4) return cudaErrorInvalidValue;
        return interleaved ? launch_pair<true>(a, p, stream) : launch_pair<false>(a, p, stream);
    }
    if (interleaved) return cudaErrorInvalidValue;
    if (p.stream) {
        if (k != 1) return cudaErrorInvalidValue;
        switch (p.wpl) {
            case 4: return launch_stream<4>(a, p, stream);
            case 2: return launch_stream<2>(a, p, stream);
            case 1: return launch_stream<1>(a, p, stream);
            default: return cudaErrorInvalidValue;
        }
    }
    switch (p.wpl) {
        case 4: return dispatch_k<4, 1>(k, a, p, stream);
        case 2: return dispatch_k<2, 1>(k, a, p, stream);
        case 1: return dispatch_k<1, 1>(k, a, p, stream);
        default: return cudaErrorInvalidValue;
    }
}

cudaError_t launch_interleave(uint32_t* grid, int W, int Y, bool back, cudaStream_t stream) {
    const size_t n = (size_t)W / 4 * Y;
    if (n == 0) return cudaSuccess;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)std::min<size_t>((n + 255) / 256, 148 * 16));
    cfg.blockDim = dim3(256);
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    auto* g = reinterpret_cast<uint4*>(grid);
    return back ? cudaLaunchKernelEx(&cfg, interleave_kernel<true>, g, n)
                : cudaLaunchKernelEx(&cfg, interleave_kernel<false>, g, n);
}

// ---------------------------------------------------------------------------
// Device pack / unpack (uint8 cell grid <-> row words), the device-side form
// of GeneralBitGrid::fill_grid / to_grid (general_bit_grid.hpp:171-246).
// ---------------------------------------------------------------------------

namespace {

// Both directions are bound by HBM (1.125 bytes a cell). A lane moves 16 cells
// (one 16-byte access, a warp's accesses contiguous) against 16 bits of words,
// kCellsAhead of them in flight, and works on four cells at a time in 32-bit
// registers. A 16384^2 grid packed and unpacked takes 102 us (5.9 TB/s; 2 and 8
// accesses in flight 102 and 101), against 135 us with a lane per 32-cell
// word (two accesses 32 bytes apart, 64-bit arithmetic).
constexpr int kCellsAhead = 4;

// Four cells (one byte each, nonzero = alive) -> bits 28..31, cell i at bit
// 28 + i: bit 7 of each byte says nonzero, and the product moves byte i's to
// bit 28 + i (its other terms stay below bit 28 or leave the word).
__device__ __forceinline__ uint32_t pack4_top(uint32_t v) {
    const uint32_t t = ((v & 0x7f7f7f7fu) + 0x7f7f7f7fu) | v;
    return (t & 0x80808080u) * 0x00204081u;
}

// 16 cells -> 16 bits in the upper half, cell i at bit 16 + i.
__device__ __forceinline__ uint32_t pack16(const uint4& c) {
    uint32_t h = pack4_top(c.w);
    h = (h & 0xf0000000u) | (pack4_top(c.z) >> 28 << 24);
    h |= pack4_top(c.y) >> 28 << 20;
    return h | (pack4_top(c.x) >> 28 << 16);
}

// Bits 0..3 -> four cells of 0/1.
__device__ __forceinline__ uint32_t unpack4(uint32_t b) {
    return ((b & 15u) * 0x00204081u) & 0x01010101u;
}

__global__ void __launch_bounds__(256) pack_cells_kernel(const uint4* __restrict__ cells,
                                                         uint16_t* __restrict__ halves, size_t n) {
    const size_t step = (size_t)gridDim.x * blockDim.x;
    size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    for (; i + (kCellsAhead - 1) * step < n; i += kCellsAhead * step) {
        uint4 c[kCellsAhead];
#pragma unroll
        for (int u = 0; u < kCellsAhead; ++u) c[u] = __ldcs(cells + i + u * step);
#pragma unroll
        for (int u = 0; u < kCellsAhead; ++u)
            halves[i + u * step] = (uint16_t)(pack16(c[u]) >> 16);
    }
    for (; i < n; i += step) halves[i] = (uint16_t)(pack16(__ldcs(cells + i)) >> 16);
}

__device__ __forceinline__ uint4 unpack16(uint32_t h) {
    return make_uint4(unpack4(h), unpack4(h >> 4), unpack4(h >> 8), unpack4(h >> 12));
}

__global__ void __launch_bounds__(256) unpack_cells_kernel(const uint16_t* __restrict__ halves,
                                                           uint4* __restrict__ cells, size_t n) {
    const size_t step = (size_t)gridDim.x * blockDim.x;
    size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    for (; i + (kCellsAhead - 1) * step < n; i += kCellsAhead * step) {
        uint32_t h[kCellsAhead];
#pragma unroll
        for (int u = 0; u < kCellsAhead; ++u) h[u] = __ldg(halves + i + u * step);
#pragma unroll
        for (int u = 0; u < kCellsAhead; ++u) __stcs(cells + i + u * step, unpack16(h[u]));
    }
    for (; i < n; i += step) __stcs(cells + i, unpack16(__ldg(halves + i)));
}

// Counter-based Bernoulli cells: cell i (raster order) of a grid with seed s
// is alive iff (mix64(s + (i + 1) * 0x9E3779B97F4A7C15) >> 11) * 2^-53 <
// density, mix64 the SplitMix64 finaliser. Each thread writes one word.
__host__ __device__ __forceinline__ unsigned long long mix64(unsigned long long z) {
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}

__global__ void hash_bernoulli_kernel(uint32_t* __restrict__ words, size_t nwords,
                                      unsigned long long seed, unsigned long long threshold) {
    for (size_t w = blockIdx.x * (size_t)blockDim.x + threadIdx.x; w < nwords;
         w += (size_t)gridDim.x * blockDim.x) {
        uint32_t v = 0;
        const unsigned long long base = (unsigned long long)w * 32ull;
#pragma unroll 8
        for (int b = 0; b < 32; ++b) {
            const unsigned long long h = mix64(seed + (base + b + 1ull) * 0x9E3779B97F4A7C15ull);
            v |= (uint32_t)((h >> 11) < threshold) << b;
        }
        words[w] = v;
    }
}

int grid_for(size_t n, int threads) {
    size_t blocks = (n + threads - 1) / threads;
    return (int)std::min<size_t>(std::max<size_t>(blocks, 1), 148 * 16);
}

} // namespace

cudaError_t launch_pack_cells(const uint8_t* cells, uint32_t* words, size_t x, size_t y,
                              cudaStream_t stream) {
    const size_t n = x / 16 * y;   // x % 32 == 0
    if (n == 0) return cudaSuccess;
    pack_cells_kernel<<<grid_for(n, 256), 256, 0, stream>>>(
        reinterpret_cast<const uint4*>(cells), reinterpret_cast<uint16_t*>(words), n);
    return cudaPeekAtLastError();
}

unsigned long long bernoulli_threshold(double density) {
    if (!(density > 0)) return 0ull;
    if (density >= 1) return 1ull << 53;
    return (unsigned long long)(density * 9007199254740992.0);   // density * 2^53
}

cudaError_t launch_hash_bernoulli(uint32_t* words, size_t x, size_t y, uint64_t seed,
                                  double density, cudaStream_t stream) {
    const size_t n = x / 32 * y;
    if (n == 0) return cudaSuccess;
    hash_bernoulli_kernel<<<grid_for(n, 256), 256, 0, stream>>>(words, n, seed,
                                                                  bernoulli_threshold(density));
    return cudaPeekAtLastError();
}

void host_hash_bernoulli(uint8_t* cells, size_t n, uint64_t seed, double density) {
    const unsigned long long t = bernoulli_threshold(density);
    for (size_t i = 0; i < n; ++i)
        cells[i] = (mix64(seed + (i + 1ull) * 0x9E3779B97F4A7C15ull) >> 11) < t ? 1 : 0;
}

cudaError_t launch_unpack_cells(const uint32_t* words, uint8_t* cells, size_t x, size_t y,
                                cudaStream_t stream) {
    const size_t n = x / 16 * y;
    if (n == 0) return cudaSuccess;
    unpack_cells_kernel<<<grid_for(n, 256), 256, 0, stream>>>(
        reinterpret_cast<const uint16_t*>(words), reinterpret_cast<uint4*>(cells), n);
    return cudaPeekAtLastError();
}

// ---------------------------------------------------------------------------
// Integer-pipe peak probe: independent LOP3 chains (8 per thread) with no
// memory traffic, to measure the lane-ops/s ceiling the temporal kernel's
// bit-sliced arithmetic is bounded by.
// ---------------------------------------------------------------------------

namespace {

__global__ void lop3_rate_kernel(uint32_t* sink, int iters, uint32_t seed) {
    uint32_t v[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] = (threadIdx.x + 1u) * (2u * j + 3u) ^ seed;
    for (int i = 0; i < iters; ++i) {
#pragma unroll
        for (int r = 0; r < 16; ++r) {
#pragma unroll
            for (int j = 0; j < 8; ++j)
                v[j] = lop3<LUT_XOR3>(v[j], v[(j + 1) & 7], v[(j + 3) & 7]);
        }
    }
    uint32_t acc = 0;
#pragma unroll
    for (int j = 0; j < 8; ++j) acc ^= v[j];
    if (acc == 0x9e3779b9u) sink[blockIdx.x] = acc;   // keeps the chains live
}

} // namespace

cudaError_t probe_lop3_rate(int device, cudaStream_t stream, double* lane_ops_per_s) {
    const int sms = device_sm_count(device);
    const int blocks = sms * 8, threads = 256, iters = 4096;
    uint32_t* sink = nullptr;
    cudaEvent_t a = nullptr, b = nullptr;
    cudaError_t e = cudaMalloc(&sink, sizeof(uint32_t) * blocks);
    if (e == cudaSuccess) e = cudaEventCreate(&a);
    if (e == cudaSuccess) e = cudaEventCreate(&b);
    if (e == cudaSuccess) {
        lop3_rate_kernel<<<blocks, threads, 0, stream>>>(sink, iters / 8, 1u);   // warm-up
        cudaEventRecord(a, stream);
        lop3_rate_kernel<<<blocks, threads, 0, stream>>>(sink, iters, 2u);
        cudaEventRecord(b, stream);
        e = cudaEventSynchronize(b);
    }
    if (e == cudaSuccess) {
        float ms = 0.f;
        e = cudaEventElapsedTime(&ms, a, b);
        const double ops = (double)blocks * threads * iters * 16.0 * 8.0;
        *lane_ops_per_s = ops / (ms * 1e-3);
    }
    if (a) cudaEventDestroy(a);
    if (b) cudaEventDestroy(b);
    if (sink) cudaFree(sink);
    return e;
}

} // namespace golb200
