// The GEMM of this library whose accumulation stays in tensor memory, for decode-sized M on sm_100a:
//
//   C[M, N] = A[M, K] x W[N, K]^T,   M <= 256
//
// in four operand kinds: FP8 or 4-bit weights with power-of-two scales applied by the tensor core (gemm_fp8_mx.cu),
// NVFP4 (gemm_nvfp4.cu) and BF16 (gemm_bf16.cu); those files describe the formats and hold the entry points.  The FP8
// GEMM with general scales promotes every K block on CUDA cores and is a kernel of its own (gemm_fp8.cu).
//
// What bounds it: the weight stream.  A unit is one weight tile, 128 rows x 128 bytes of K, and the activation rows of
// the same K range.  A probe that only streams units (TMA, no MMA) brings 24576 x 7168 bytes in 28-30 us (5.8-6.2 TB/s)
// beside 0 to 128 activation rows and in 32.8 us beside 256: an SM takes in up to 110 bytes per ns, so re-reading the
// activations from L2 with every weight tile is cheap and nothing is kept resident or shared between CTAs.
//
//   * swap-AB: weight rows are the MMA's M = 128, activation rows (rounded up to 16, not to a power of two) its N.
//   * one elected thread fetches (as many stages as fit, 4 to 12), one issues the MMAs into an accumulator that is
//     double-buffered where tensor memory has the room; all rows up to 256 go in ONE pass over the weights.
//   * block scales of the FP8 / 4-bit kinds are exponent bytes in tensor memory.  A 32-bit scale column holds four
//     consecutive K blocks (the MMA's scale id picks one), so two warps build ONE image per four units, from scales
//     they requested sixteen units earlier; the fetching and the issuing thread never wait for scale arithmetic.
//   * work split: stream-K, i.e. the flat unit list in equal contiguous ranges, at most max_split() of them to a tile.
//     Tiles enough for every SM: a range that starts inside a tile leaves its partial sums in its scratch slot and the
//     CTA with the tile's start adds them in CTA order - it comes to that tile last, the partial was finished first.
//     Few tiles ("sliced"): every CTA leaves the partial sums of its one or two tiles, and once a tile's counter is
//     complete each of its CTAs adds one slice of it over all partials - instead of one CTA adding up to fifteen whole
//     partials one after the other (with few rows the CTA that completes the counter adds the tile, last_arrival_adds()).  The order of the additions is CTA order either way and part of the results (it
//     moves single roundings of the fp32 sums, and 4-bit quantisation behind them makes 4e-3 of a layer's output of
//     that): it depends on the shape and the SM count alone, not on timing.
//   * before it waits for the kernel ahead (programmatic launch) a CTA asks L2 for its first weight tiles, so a chain
//     of small kernels hides the start of the weight stream.  A prefetch into L2 is a hint: it reads nothing into the
//     SM, so weights written by an earlier kernel of the chain are still seen.
// Every wait is bounded.  A CTA whose wait ran out records it, fills its partial sums with NaN and takes every step that
// other CTAs count on all the same, so that all flags and counters are zero again when the launch ends: the next launch
// must not take what an aborted one left behind for an arrival of its own.
// Times of the GEMM files, where they say "as in gemm_tc.cuh": CUDA graphs of one call each on three sets of operands, replayed
// in turn back to back (weights from HBM; every graph has a scratch of its own), mean per replay.  Replays of 10 to 16 us come
// in steps of 2 us.
#pragma once
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "host.h"
#include "ptx.cuh"

namespace wuda {
namespace gemmtc {

enum class Kind { kMx8, kMx8W4, kNv4, kBf16 };

constexpr int kTileN = 128;                   // weight rows per tile (UMMA M)
constexpr int kRowBytes = 128;                // K bytes of a unit: 128 e4m3, 256 e2m1, 64 bf16
constexpr int kWBytes = kTileN * kRowBytes;   // 16 KB
constexpr int kMaxStages = 12;
// The grouped form streams for hundreds of microseconds, and there more copies in flight cost bandwidth: routed experts of
// 64 tokens (5.65 GB) 924 us with 10 stages, 892 with 8, 877 with 6, 905 with 5, 939 with 4.  The dense calls are too short
// for that (24576 x 7168 NVFP4 at 8 rows 20.8 us with 8 to 10 stages, 21.8 with 6).
constexpr int kGroupedStages = 6;
constexpr int kImgSlots = 4;
constexpr int kImgBlock = 512;                // scale bytes of 128 rows, four bytes each: [row % 32][row / 32]
constexpr int kNvSfBytes = 2048;              // NVFP4: packed scales of 128 rows x 256 K
constexpr int kMaxGrid = 192;
constexpr int kMaxEvenSplit = 32;
constexpr int64_t kFlagBytes = 1024;          // the flags lead the scratch, whatever the shape (kernels share scratches)

struct Params {
    void* c;
    int c_is_fp32;
    float* scratch;            // partial-tile slots, fp32 [M_PAD / 4][128 weight rows][4 activation rows]: [grid], sliced also [n_tiles]
    int32_t* flags;            // one flag per CTA; sliced: one counter per weight tile
    int32_t* status;
    int M, N, kb, n_tiles;     // kb = units per weight tile
    int a_rows;                // M rounded up to 16
    int stages;
    int sliced;                // a tile's partial sums are added by all of its CTAs, a slice each (even slices: how many CTAs)
    int last_adds;             // .. or by the one that completes the tile's counter
    // power-of-two scaled kinds
    const float* a_scales;     // [M, scale_cols]
    const float* w_scales;     // [n_tiles, kb] (FP8 weights)
    const uint8_t* w_sf;       // 4-bit weights: [N, sf_stride] exponent bytes, one per weight row and 32 K-elements
    int sf_stride;
    int tiles_per_group;       // tile t reads the activations from K block (t / tiles_per_group) * kb on
    int scale_cols;
    int vec_scales;            // rows of a_scales (and w_sf) can be read 16 bytes at a time
    // NVFP4
    float out_scale;
    const int32_t* group_expert;   // grouped form (routed experts): [num_groups], else NULL; see gemm_nvfp4.cu
    const int32_t* row_token;
    const int32_t* num_groups;
    const float* expert_scale;
};

template <Kind KIND, int M_PAD>
struct Layout {
    static constexpr bool kMx = KIND == Kind::kMx8 || KIND == Kind::kMx8W4;
    static constexpr int kBlocks = (M_PAD + 127) / 128;               // 128-row blocks of activation scales
    // FP8 x FP8 and BF16 up to 128 rows keep two sums, of the even and of the odd units of a range, added at the end.  The
    // order of the additions is part of the layer's results: another order moves single roundings of the projections, and
    // the 4-bit activations of the experts behind them turn those into 4e-3 of the layer's output.
    static constexpr int kAccs = (KIND == Kind::kMx8 || KIND == Kind::kBf16) && M_PAD <= 128 ? 2 : 1;
    // Beyond 128 rows there is no earlier order to keep (those were two passes), and a CTA's partial sums are 128 KB per tile, so
    // few tiles are cut evenly and no CTA holds parts of two (4096 x 7168 FP8 at 200 rows 29.8 -> 20.5 us).
    static constexpr bool kEvenSlices = M_PAD > 128;
    static constexpr int kBuffers = kAccs * M_PAD <= 128 ? 2 : 1;
    // Epilogue warps: behind the last copy they move partial sums and results with the bytes in flight that they have, so
    // 256 rows take sixteen (7168 x 16384 FP8 43.8 -> 40.4 us; not with 4-bit weights, whose scale images need the
    // registers).  At 128 rows sixteen are slower: NVFP4 24576 x 7168 28.8 -> 31.4 us, the layer at batch 128 1498 -> 1519.
    static constexpr int kEpiWarps = M_PAD == 256 && KIND != Kind::kMx8W4 ? 16 : (M_PAD >= 64 ? 8 : 4);
    static constexpr int kThreads = 32 * (4 + kEpiWarps);
    static constexpr int kCols = M_PAD / (kEpiWarps / 4);             // accumulator columns per epilogue thread
    // scale columns of one set (two sets alternate)
    static constexpr int kSfwCols = kMx ? 4 : (KIND == Kind::kNv4 ? 16 : 0);
    static constexpr int kSfaCols = kSfwCols * kBlocks;
    static constexpr int kAccCols = kBuffers * kAccs * M_PAD;
    static constexpr int kUsedCols = kAccCols + 2 * (kSfwCols + kSfaCols);
    static constexpr int kTmemCols = kUsedCols <= 32 ? 32 : (kUsedCols <= 64 ? 64 : (kUsedCols <= 128 ? 128 : (kUsedCols <= 256 ? 256 : 512)));
    static constexpr int kImgW = KIND == Kind::kMx8W4 ? 4 * kImgBlock : kImgBlock;    // weight part of an image slot
    static constexpr int kImgBytes = kMx ? kImgW + kBlocks * kImgBlock : 0;
    static __host__ __device__ constexpr int stage_bytes(int a_rows) {
        return kWBytes + a_rows * kRowBytes + (KIND == Kind::kNv4 ? kNvSfBytes * (1 + kBlocks) : 0);
    }
    static __host__ __device__ constexpr int img_off(int stages, int a_rows) { return stages * stage_bytes(a_rows); }
    static __host__ __device__ constexpr int bar_off(int stages, int a_rows) { return img_off(stages, a_rows) + kImgSlots * kImgBytes; }
    // barriers: full[12] empty[12] img_full[4] img_empty[4] full_tm[2] empty_tm[2]
    static constexpr int kBars = 2 * kMaxStages + 2 * kImgSlots + 4;
    static __host__ __device__ constexpr int misc_off(int stages, int a_rows) { return bar_off(stages, a_rows) + kBars * 8; }
    static __host__ __device__ constexpr int total(int stages, int a_rows) { return misc_off(stages, a_rows) + 16 + 1024; }
};

// A CTA's flag goes up when its partial sums are complete and down when the CTA that adds them has done so.  Both flip it,
// and both always do: in whichever order (the one that adds may have given up waiting), the flag ends at zero.
__device__ __forceinline__ void raise_flag(int32_t* flag) {
    asm volatile("red.release.gpu.global.inc.u32 [%0], %1;" ::"l"(flag), "r"(1) : "memory");
}
// (nobody reads it any more in this launch, so nothing has to be ordered: a release would hold up the results behind it, the
// layer at batch 1 by 3 us)
__device__ __forceinline__ void lower_flag(int32_t* flag) {
    asm volatile("red.relaxed.gpu.global.inc.u32 [%0], %1;" ::"l"(flag), "r"(1) : "memory");
}
__device__ __forceinline__ void st_release_gpu(int32_t* p, int v) {
    asm volatile("st.release.gpu.global.s32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ int ld_acquire_gpu(const int32_t* p) {
    int v;
    asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
// old >= limit ? 0 : old + 1
__device__ __forceinline__ int inc_acq_rel_gpu(int32_t* p, int limit) {
    int old;
    asm volatile("atom.acq_rel.gpu.global.inc.u32 %0, [%1], %2;" : "=r"(old) : "l"(p), "r"(limit) : "memory");
    return old;
}
// floor(units * c / grid) for fewer than 2^32 units (16 KB each), in 32-bit divisions: a launch's prologue is on the critical
// path of a short call, and a 64-bit division takes a few hundred cycles
__device__ __forceinline__ uint32_t range_begin(uint32_t units, uint32_t c, uint32_t grid) {
    const uint32_t q = units / grid, rest = units - q * grid;
    return q * c + rest * c / grid;
}
__device__ __forceinline__ int cta_of(uint32_t units, uint32_t u, int grid) {
    int c = static_cast<int>(static_cast<uint64_t>(u) * static_cast<uint32_t>(grid) / units);
    while (c + 1 < grid && range_begin(units, c + 1, grid) <= u) ++c;
    while (c > 0 && range_begin(units, c, grid) > u) --c;
    return c;
}

// Exponent byte of a power-of-two fp32 scale; anything else is reported and truncated to the power of two below.
__device__ __forceinline__ uint32_t exponent_byte(float scale, int32_t* status) {
    const uint32_t bits = __float_as_uint(scale);
    if (((bits & 0x807fffffu) != 0u || (bits >> 23) == 0xffu) && scale != 0.f && status)
        atomicCAS(status, 0, static_cast<int>(kDevScaleNotPow2));
    const uint32_t e = (bits >> 23) & 0xffu;
    return e == 0xffu ? 0xfeu : e;
}

__device__ __forceinline__ void umma_mxf8(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t sfa_tmem,
                                          uint32_t sfb_tmem, uint32_t accumulate) {
    asm volatile(
        "{\n\t"
        ".reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::mxf8f6f4.block_scale.scale_vec::1X "
        "[%0], %1, %2, %3, [%5], [%6], p;\n\t"
        "}\n"
        ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate), "r"(sfa_tmem), "r"(sfb_tmem)
        : "memory");
}

__device__ __forceinline__ uint32_t to_bf16x2(float a, float b) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
    return reinterpret_cast<const uint32_t&>(v);
}
// Four lanes (rows r = lane & 3) hold columns 0..3 as two pairs of 16 bits; lane r leaves with column r of the four rows.
__device__ __forceinline__ void transpose4(uint32_t c01, uint32_t c23, uint32_t lane, uint32_t& rows01, uint32_t& rows23) {
    const bool up = (lane & 2u) != 0u, odd = (lane & 1u) != 0u;
    const uint32_t got = __shfl_xor_sync(0xffffffffu, up ? c01 : c23, 2);
    const uint32_t near = up ? got : c01, far = up ? c23 : got;     // this lane's column pair of rows (r & 1) and (r & 1) + 2
    const uint32_t low = __byte_perm(near, far, 0x5410), high = __byte_perm(near, far, 0x7632);
    const uint32_t other = __shfl_xor_sync(0xffffffffu, odd ? low : high, 1);
    const uint32_t even_rows = odd ? other : low, odd_rows = odd ? high : other;   // rows (0, 2) and (1, 3) of the lane's column
    rows01 = __byte_perm(even_rows, odd_rows, 0x5410);
    rows23 = __byte_perm(even_rows, odd_rows, 0x7632);
}

// One thread's bounded wait for a word in global memory (another CTA's flag or a tile's counter); SLEEP_NS > 0 where the wait
// runs beside the stream and must not take its issue slots.
template <unsigned SLEEP_NS = 0, typename Pred>
__device__ __forceinline__ void await_word(const int32_t* word, Pred done, volatile int* abort_flag, int32_t* status) {
    if (done(ld_acquire_gpu(word))) return;
    const unsigned long long start = globaltimer_ns();
    uint32_t spins = 0;
    while (!done(ld_acquire_gpu(word))) {
        if ((++spins & 255u) == 0u && (*abort_flag || globaltimer_ns() - start > kWaitLimitNs)) {
            *abort_flag = 1;
            if (status) atomicCAS(status, 0, static_cast<int>(kDevTimeoutPeerFlag));
            break;
        }
        if (SLEEP_NS) __nanosleep(SLEEP_NS);
    }
}

// The CTAs that hold units of a sliced tile.  A CTA has at most two tiles: its range is at most a third of one.
struct Holders {
    int first, last;
    __device__ __forceinline__ int count() const { return last - first + 1; }
};
// .. as one word (there are fewer than 256 CTAs): two tiles' stay in registers until the end of a range
__device__ __forceinline__ uint32_t holders_of(uint32_t units, int tile, int kb, int grid) {
    const uint32_t begin = static_cast<uint32_t>(tile) * static_cast<uint32_t>(kb);
    return static_cast<uint32_t>(cta_of(units, begin, grid)) | static_cast<uint32_t>(cta_of(units, begin + kb - 1, grid)) << 8;
}
__device__ __forceinline__ Holders unpack_holders(uint32_t both, int i) {
    return {static_cast<int>(both >> (16 * i) & 0xffu), static_cast<int>(both >> (16 * i + 8) & 0xffu)};
}
// Slot of this CTA's partial sums.  Those that start a sliced tile go behind the CTAs' own (their CTA may hold the end of the
// tile before, too).
__device__ __forceinline__ int start_slot(int tile) { return static_cast<int>(gridDim.x) + tile; }
__device__ __forceinline__ int slot_index(int sliced, bool from_zero, int tile) {
    return sliced && from_zero ? start_slot(tile) : static_cast<int>(blockIdx.x);
}

// Slice j of `slices` of a weight tile: the sum over all partials, in CTA order, scaled and stored.
// A thread adds four activation rows of a weight row, eight partials in flight.
template <Kind KIND>
__device__ __forceinline__ void add_slice(const float* scratch, int64_t slot_floats, int tile, Holders h, int first_slot, int j, int slices,
                                          int thread, int threads, int M, int N, float out_scale, int c_is_fp32, void* c) {
    const int parts = h.count(), quads = (M + 3) / 4 * kTileN;
    const float4* start = reinterpret_cast<const float4*>(scratch + static_cast<int64_t>(first_slot) * slot_floats);
    const float4* part = reinterpret_cast<const float4*>(scratch + static_cast<int64_t>(h.first) * slot_floats);   // [1], [2], ..
    const int end = quads * (j + 1) / slices;
    for (int e = quads * j / slices + thread; e < end; e += threads) {
        float4 v = __ldcg(start + e);
        for (int q0 = 1; q0 < parts; q0 += 8) {
            float4 x[8];
#pragma unroll
            for (int q = 0; q < 8; ++q) x[q] = __ldcg(part + min(q0 + q, parts - 1) * (slot_floats / 4) + e);
#pragma unroll
            for (int q = 0; q < 8; ++q)
                if (q0 + q < parts) v.x += x[q].x, v.y += x[q].y, v.z += x[q].z, v.w += x[q].w;
        }
        const float out[4] = {v.x, v.y, v.z, v.w};
        const int m = e / kTileN * 4, nr = tile * kTileN + e % kTileN;
        if (nr < N) {
#pragma unroll
            for (int i = 0; i < 4; ++i)
                if (m + i < M) {
                    const int64_t at = static_cast<int64_t>(m + i) * N + nr;
                    const float o = KIND == Kind::kNv4 ? out[i] * out_scale : out[i];
                    if (KIND == Kind::kBf16 && c_is_fp32) static_cast<float*>(c)[at] = o;
                    else static_cast<__nv_bfloat16*>(c)[at] = __float2bfloat16_rn(o);
                }
        }
    }
}

template <Kind KIND, int M_PAD>
__global__ void __launch_bounds__(Layout<KIND, M_PAD>::kThreads, 1)
gemm_tc_kernel(const __grid_constant__ CUtensorMap w_map, const __grid_constant__ CUtensorMap a_map,
               const __grid_constant__ CUtensorMap wsf_map, const __grid_constant__ CUtensorMap asf_map, const Params p) {
    using L = Layout<KIND, M_PAD>;
    constexpr bool kMx = L::kMx;
    constexpr int kBuffers = L::kBuffers;
    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw_addr = smem_u32(smem_raw);
    const uint32_t base = (raw_addr + 1023u) & ~1023u;
    uint8_t* base_ptr = smem_raw + (base - raw_addr);
    const int S = p.stages;
    const uint32_t stage_bytes = L::stage_bytes(p.a_rows);
    const uint32_t bars = base + L::bar_off(S, p.a_rows);
    const uint32_t full = bars, empty = full + kMaxStages * 8, img_full = empty + kMaxStages * 8, img_empty = img_full + kImgSlots * 8,
                   full_tm = img_empty + kImgSlots * 8, empty_tm = full_tm + 16;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(base_ptr + L::misc_off(S, p.a_rows));
    volatile int* abort_flag = reinterpret_cast<volatile int*>(base_ptr + L::misc_off(S, p.a_rows) + 4);
    volatile int* arrived_last = reinterpret_cast<volatile int*>(base_ptr + L::misc_off(S, p.a_rows) + 8);

    const int warp = __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x >> 5), 0);
    const uint32_t lane = lane_id();

    if (threadIdx.x == 0) {
        *abort_flag = 0;
        for (int i = 0; i < S; ++i) {
            mbar_init(full + i * 8, 1);
            mbar_init(empty + i * 8, 1);
        }
        for (int i = 0; i < kImgSlots; ++i) {
            mbar_init(img_full + i * 8, 1);
            mbar_init(img_empty + i * 8, 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(full_tm + b * 8, 1);               // a segment's accumulator is complete
            mbar_init(empty_tm + b * 8, L::kEpiWarps);   // the epilogue has read it
        }
        fence_mbar_init();
    }
    if (warp == 1) {
        tmem_alloc(smem_u32(tmem_slot), L::kTmemCols);
        tmem_relinquish();
    }
    const bool grouped = KIND == Kind::kNv4 && p.group_expert != nullptr;
    // the unit range of this CTA (the grouped form learns its number of units from the kernel ahead)
    uint32_t units = static_cast<uint32_t>(p.n_tiles) * static_cast<uint32_t>(p.kb), u0 = 0;
    int grid = static_cast<int>(gridDim.x), count = 0;
    if (!grouped) {
        u0 = range_begin(units, blockIdx.x, grid);
        count = static_cast<int>(range_begin(units, blockIdx.x + 1, grid) - u0);
    }
    int tile0 = static_cast<int>(u0 / static_cast<uint32_t>(p.kb)), kb0 = static_cast<int>(u0) - tile0 * p.kb;
    if (warp == 0 && elect_one()) {
        prefetch_tmap(&w_map);
        prefetch_tmap(&a_map);
        if constexpr (KIND == Kind::kNv4) {
            prefetch_tmap(&wsf_map);
            prefetch_tmap(&asf_map);
        }
        if constexpr (KIND != Kind::kMx8W4) {
            int tile = tile0, kb = kb0;
            for (int n = 0; n < count && n < S; ++n) {
                tma_prefetch_2d(&w_map, kb * (KIND == Kind::kBf16 ? kRowBytes / 2 : kRowBytes), tile * kTileN);
                if (++kb == p.kb) kb = 0, ++tile;
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    // all of the above ran while the kernel ahead was still finishing; its results are read from here on
    pdl_launch_dependents();
    pdl_wait();

    if (grouped) {
        // Only the first min(grid, units) CTAs take part: every participating CTA then owns at least one unit, which
        // the fix-up relies on when it waits for the CTAs that share a tile.
        units *= *p.num_groups;
        if (units < static_cast<uint32_t>(grid)) grid = static_cast<int>(units);
        if (static_cast<int>(blockIdx.x) < grid) {
            u0 = range_begin(units, blockIdx.x, grid);
            count = static_cast<int>(range_begin(units, blockIdx.x + 1, grid) - u0);
            tile0 = static_cast<int>(u0 / static_cast<uint32_t>(p.kb)), kb0 = static_cast<int>(u0) - tile0 * p.kb;
        }
    }

    if (warp == 0) {
        // ------------------------------------------------------------ copies
        if (elect_one()) {
            const uint64_t stream_policy = policy_evict_first();
            const uint64_t keep_policy = policy_evict_last();
            const uint32_t tx = stage_bytes - (KIND == Kind::kMx8W4 ? kWBytes / 2 : 0);   // packed weights: the padding is not counted
            int s = 0;
            uint32_t phase = 1;
            int tile = tile0, kb = kb0;
            int seen_tile = -1, grp = grouped ? -1 : 0, expert = 0, wtile = 0;
            for (int n = 0; n < count; ++n) {
                // grouped: `tile` is the flat index; the weight tile is the expert's, the activations the group's
                // (looked up only when the tile changes)
                if (grouped && tile != seen_tile) {
                    seen_tile = tile;
                    const int g_now = tile / p.n_tiles;
                    if (g_now != grp) {
                        grp = g_now;
                        expert = __ldcg(p.group_expert + grp);   // written by the dispatch kernel of the same chain
                    }
                    wtile = expert * p.n_tiles + (tile - grp * p.n_tiles);
                } else if (!grouped) {
                    wtile = tile;
                }
                if (!mbar_wait(empty + s * 8, phase, abort_flag, p.status, kDevTimeoutGemmEmpty)) break;
                const uint32_t stage = base + s * stage_bytes, bar = full + s * 8, a_bytes = p.a_rows * kRowBytes;
                mbar_arrive_expect_tx(bar, tx);
                if constexpr (kMx) {
                    tma_load_2d_hint(stage, &w_map, bar, kb * kRowBytes, wtile * kTileN, stream_policy);
                    tma_load_2d_hint(stage + kWBytes, &a_map, bar, ((tile / p.tiles_per_group) * p.kb + kb) * kRowBytes, 0, keep_policy);
                } else if constexpr (KIND == Kind::kNv4) {
                    tma_load_2d_hint(stage, &w_map, bar, kb * kRowBytes, wtile * kTileN, stream_policy);
                    tma_load_2d_hint(stage + kWBytes, &a_map, bar, kb * kRowBytes, grp * M_PAD, keep_policy);
                    const uint32_t sf = stage + kWBytes + a_bytes;
                    tma_load_2d_hint(sf, &wsf_map, bar, 0, (wtile * p.kb + kb) * 4, stream_policy);
#pragma unroll
                    for (int b = 0; b < L::kBlocks; ++b)   // (a second block exists only where rows beyond 128 do: M_PAD = 256)
                        tma_load_2d_hint(sf + (1 + b) * kNvSfBytes, &asf_map, bar, 0, ((grp + b) * p.kb + kb) * 4, keep_policy);
                } else {
                    tma_load_2d_hint(stage, &w_map, bar, kb * (kRowBytes / 2), wtile * kTileN, stream_policy);
                    tma_load_2d_hint(stage + kWBytes, &a_map, bar, kb * (kRowBytes / 2), 0, keep_policy);
                }
                if (++s == S) s = 0, phase ^= 1u;
                if (++kb == p.kb) kb = 0, ++tile;
            }
        }
    } else if (warp == 1) {
        // ------------------------------------------------------------ MMAs
        if (elect_one()) {
            int s = 0;
            uint32_t phase = 0, seg = 0, img = 0, nv_set = 0;   // img: images taken so far
            int kb = kb0;
            const uint32_t sf_cols = tmem_base + L::kAccCols;
            bool alive = true;
            for (int n = 0; n < count && alive;) {
                const int seg_len = min(p.kb - kb, count - n);
                const uint32_t buf = kBuffers == 2 ? (seg & 1u) : 0u;
                if (seg >= static_cast<uint32_t>(kBuffers)) {   // the epilogue must have drained this buffer's previous segment
                    if (!mbar_wait(empty_tm + buf * 8, (seg / kBuffers - 1u) & 1u, abort_flag, p.status, kDevTimeoutGemmTmemEmpty)) break;
                    tc_fence_after();
                }
                const uint32_t d_buf = tmem_base + buf * (L::kAccs * M_PAD);
                for (int u = 0; u < seg_len; ++u) {
                    const int k = kb + u;
                    const uint32_t slot = img & (kImgSlots - 1);
                    const uint32_t img_addr = base + L::img_off(S, p.a_rows) + slot * L::kImgBytes;
                    const uint32_t set = (kMx ? img & 1u : nv_set) * (L::kSfwCols + L::kSfaCols);
                    const uint32_t sfw = sf_cols + set, sfa = sfw + L::kSfwCols;
                    if constexpr (kMx) {
                        if (u == 0 || (k & 3) == 0) {   // the first unit of a scale image
                            if (!mbar_wait(img_full + slot * 8, (img / kImgSlots) & 1u, abort_flag, p.status, kDevTimeoutGemmFull)) {
                                alive = false;
                                break;
                            }
                            tc_fence_after();
                            if (KIND == Kind::kMx8) tmem_cp_32x128b_warpx4(sfw, umma_smem_desc_noswz(img_addr, 16, 128));
#pragma unroll
                            for (int b = 0; b < L::kBlocks; ++b)
                                tmem_cp_32x128b_warpx4(sfa + b * 4, umma_smem_desc_noswz(img_addr + L::kImgW + b * kImgBlock, 16, 128));
                        }
                    }
                    if (!mbar_wait(full + s * 8, phase, abort_flag, p.status, kDevTimeoutGemmFull)) {
                        alive = false;
                        break;
                    }
                    tc_fence_after();
                    const uint32_t w_addr = base + s * stage_bytes, a_addr = w_addr + kWBytes;
                    if constexpr (KIND == Kind::kMx8W4)   // every unit has its own weight scales: four bytes per row
                        tmem_cp_32x128b_warpx4(sfw, umma_smem_desc_noswz(img_addr + (k & 3) * kImgBlock, 16, 128));
                    if constexpr (KIND == Kind::kNv4) {
                        const uint32_t sf = a_addr + p.a_rows * kRowBytes;
#pragma unroll
                        for (int i = 0; i < 4; ++i) {   // 32 rows x 16 bytes per K/64 step; 8-row groups 128 bytes apart
                            tmem_cp_32x128b_warpx4(sfw + i * 4, umma_smem_desc_noswz(sf + i * 512, 16, 128));
#pragma unroll
                            for (int b = 0; b < L::kBlocks; ++b)
                                tmem_cp_32x128b_warpx4(sfa + (i * L::kBlocks + b) * 4,
                                                       umma_smem_desc_noswz(sf + (1 + b) * kNvSfBytes + i * 512, 16, 128));
                        }
                    }
                    const uint32_t d = d_buf + (L::kAccs == 2 ? ((n + u) & 1) * M_PAD : 0);
                    const uint64_t w_desc = umma_smem_desc_sw128(w_addr), a_desc = umma_smem_desc_sw128(a_addr);
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const uint32_t acc = (u >= L::kAccs || i > 0) ? 1u : 0u;
                        if constexpr (kMx) {
                            // weights e4m3 (format 0) or e2m1 (5) x e4m3, ue8m0 scales (1)
                            const uint32_t idesc = umma_idesc_block_scaled(kTileN, p.a_rows, KIND == Kind::kMx8W4 ? 5 : 0, 0, 1,
                                                                           KIND == Kind::kMx8W4 ? i : (k & 3), k & 3);
                            umma_mxf8(d, w_desc + i * 2, a_desc + i * 2, idesc, sfw, sfa, acc);
                        } else if constexpr (KIND == Kind::kNv4) {
                            const uint32_t idesc = umma_idesc_block_scaled(kTileN, p.a_rows, 1, 1, 0, 0, 0);
                            umma_nvf4(d, w_desc + i * 2, a_desc + i * 2, idesc, sfw + i * 4, sfa + i * L::kBlocks * 4, acc);
                        } else {
                            umma_f16(d, w_desc + i * 2, a_desc + i * 2, umma_idesc(kTileN, p.a_rows, 1, 1), acc);
                        }
                    }
                    umma_commit(empty + s * 8);     // the stage's bytes are consumed once these retire
                    if (kMx && (u + 1 == seg_len || (k & 3) == 3)) {
                        umma_commit(img_empty + slot * 8);
                        ++img;
                    }
                    nv_set ^= 1u;
                    if (++s == S) s = 0, phase ^= 1u;
                }
                if (!alive) break;
                umma_commit(full_tm + buf * 8);     // the segment is complete
                n += seg_len;
                kb += seg_len;
                if (kb == p.kb) kb = 0;
                ++seg;
            }
        }
    } else if (warp < 4) {
        // ------------------------------------------------------------ scale images, one per (tile, four K blocks)
        if constexpr (kMx) {
            constexpr int kQ = (M_PAD + 31) / 32;      // activation rows of a lane: lane, lane + 32, ..
            const uint32_t me = warp - 2;
            int tile = tile0, kb = kb0, n = 0;
            auto advance = [&](int times) {
                for (; times > 0; --times) {
                    const int len = min(4 - (kb & 3), p.kb - kb);
                    n += len, kb += len;
                    if (kb == p.kb) kb = 0, ++tile;
                }
            };
            struct Raw {
                float4 a[kQ];
                float4 w;               // FP8 weights: the four K blocks' scales
                uint4 wsf[4];           // 4-bit weights: rows lane + 32 q, four words of four exponent bytes
            };
            // (through L2, the weights' scales too: this kernel may be resident while the one ahead still writes them, and the
            // read-only path may then serve lines that an earlier kernel of the chain left in L1)
            auto load = [&](Raw& r) {
                const int k0 = kb & ~3;
                const int col = (tile / p.tiles_per_group) * p.kb + k0;
#pragma unroll
                for (int q = 0; q < kQ; ++q) {
                    const int row = q * 32 + static_cast<int>(lane);
                    r.a[q] = make_float4(1.f, 1.f, 1.f, 1.f);      // rows beyond M: zeros times 2^0
                    if (row < p.M) {
                        const float* src = p.a_scales + static_cast<int64_t>(row) * p.scale_cols + col;
                        if (p.vec_scales) {
                            r.a[q] = __ldcg(reinterpret_cast<const float4*>(src));
                        } else {
                            r.a[q].x = __ldcg(src);
                            if (k0 + 1 < p.kb) r.a[q].y = __ldcg(src + 1);
                            if (k0 + 2 < p.kb) r.a[q].z = __ldcg(src + 2);
                            if (k0 + 3 < p.kb) r.a[q].w = __ldcg(src + 3);
                        }
                    }
                }
                if constexpr (KIND == Kind::kMx8) {
                    const float* src = p.w_scales + static_cast<int64_t>(tile) * p.kb + k0;
                    r.w.x = __ldcg(src);
                    r.w.y = k0 + 1 < p.kb ? __ldcg(src + 1) : 1.f;
                    r.w.z = k0 + 2 < p.kb ? __ldcg(src + 2) : 1.f;
                    r.w.w = k0 + 3 < p.kb ? __ldcg(src + 3) : 1.f;
                } else {
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        const int row = tile * kTileN + q * 32 + static_cast<int>(lane);
                        r.wsf[q] = make_uint4(0u, 0u, 0u, 0u);     // rows beyond N: zeros times 2^-127
                        if (row < p.N) {
                            const uint8_t* src = p.w_sf + static_cast<int64_t>(row) * p.sf_stride + k0 * 4;
                            if (p.vec_scales) {
                                r.wsf[q] = __ldcg(reinterpret_cast<const uint4*>(src));
                            } else {
                                const uint32_t* words = reinterpret_cast<const uint32_t*>(src);
                                r.wsf[q].x = __ldcg(words);
                                if (k0 + 1 < p.kb) r.wsf[q].y = __ldcg(words + 1);
                                if (k0 + 2 < p.kb) r.wsf[q].z = __ldcg(words + 2);
                                if (k0 + 3 < p.kb) r.wsf[q].w = __ldcg(words + 3);
                            }
                        }
                    }
                }
            };
            auto pack = [&](float4 v) {
                return exponent_byte(v.x, p.status) | exponent_byte(v.y, p.status) << 8 | exponent_byte(v.z, p.status) << 16 |
                       exponent_byte(v.w, p.status) << 24;
            };
            // Two images are in registers and each is refilled as soon as it is written out, four images ahead of the
            // one under way: a copy from one to the other would wait for the loads.
            Raw raw[2];
            uint32_t seq = me;                  // the image this warp writes next; (tile, kb, n) is the one it loads next
            int n_write[2];
            auto fill = [&](int h) {
                n_write[h] = n;
                if (n < count) load(raw[h]);
                advance(2);
            };
            auto write = [&](const Raw& now) -> bool {
                const uint32_t slot = seq & (kImgSlots - 1);
                if (!mbar_wait_lane0(img_empty + slot * 8, ((seq / kImgSlots) & 1u) ^ 1u, abort_flag, p.status, kDevTimeoutGemmEmpty))
                    return false;
                uint4* img = reinterpret_cast<uint4*>(base_ptr + L::img_off(S, p.a_rows) + slot * L::kImgBytes) + lane;
                if constexpr (KIND == Kind::kMx8) {
                    const uint32_t ew = pack(now.w);
                    img[0] = make_uint4(ew, ew, ew, ew);
                } else {
                    img[0] = make_uint4(now.wsf[0].x, now.wsf[1].x, now.wsf[2].x, now.wsf[3].x);
                    img[kImgBlock / 16] = make_uint4(now.wsf[0].y, now.wsf[1].y, now.wsf[2].y, now.wsf[3].y);
                    img[2 * kImgBlock / 16] = make_uint4(now.wsf[0].z, now.wsf[1].z, now.wsf[2].z, now.wsf[3].z);
                    img[3 * kImgBlock / 16] = make_uint4(now.wsf[0].w, now.wsf[1].w, now.wsf[2].w, now.wsf[3].w);
                }
#pragma unroll
                for (int b = 0; b < L::kBlocks; ++b) {
                    uint32_t word[4] = {0u, 0u, 0u, 0u};
#pragma unroll
                    for (int q = 0; q < 4; ++q)
                        if (b * 4 + q < kQ) word[q] = pack(now.a[b * 4 + q]);
                    img[(L::kImgW + b * kImgBlock) / 16] = make_uint4(word[0], word[1], word[2], word[3]);
                }
                fence_proxy_async_smem();       // the images are read by tcgen05.cp
                __syncwarp();
                if (lane == 0) mbar_arrive(img_full + slot * 8);
                seq += 2;
                return true;
            };
            advance(me);
            fill(0);
            fill(1);
            while (n_write[0] < count) {
                if (!write(raw[0])) break;
                fill(0);
                if (n_write[1] >= count || !write(raw[1])) break;
                fill(1);
            }
        }
    } else {
        // ------------------------------------------------------------ epilogue
        constexpr int kEpi = 32 * L::kEpiWarps, kCols = L::kCols;
        constexpr bool kEven = L::kEvenSlices;
        auto epi_sync = [] { asm volatile("bar.sync 1, %0;" ::"n"(kEpi) : "memory"); };
        const int et = static_cast<int>(threadIdx.x) - 128;
        const int row = et & 127, col0 = (et >> 7) * kCols;      // weight row inside the tile, first column
        const uint32_t lane_base = static_cast<uint32_t>((warp & 3) * 32) << 16;
        bool alive = true;
        int tile = tile0, kb = kb0;
        uint32_t seg = 0;
        constexpr int64_t slot_floats = static_cast<int64_t>(M_PAD) * kTileN;
        int grp = 0, seen_grp = -1;
        float scale = p.out_scale;
        uint32_t stored = 0xffffffffu;       // grouped rows without a token are padding: nobody reads them
        // sliced: who shares the first and the second tile of this range
        uint32_t held = 0;
        auto holders = [&](int i) -> Holders {
            if (!kEven) return unpack_holders(held, i);
            const int first = static_cast<int>(blockIdx.x) / p.sliced * p.sliced;
            return {first, first + p.sliced - 1};
        };
        // this CTA's slice of its first or second tile, once the partial sums of all are there
        auto slice = [&](int i) {
            const int of = kEven ? static_cast<int>(blockIdx.x) / p.sliced : tile0 + i;   // (not from tile0: it would take a register)
            if (et == 0 && alive) await_word(p.flags + of, [](int v) { return v == 0; }, abort_flag, p.status);
            epi_sync();
            alive = __all_sync(0xffffffffu, alive && !*abort_flag);
            if (alive) {
                const Holders h = holders(i);
                add_slice<KIND>(p.scratch, slot_floats, of, h, kEven ? h.first : start_slot(of), static_cast<int>(blockIdx.x) - h.first,
                                h.count(), et, kEpi, p.M, p.N, p.out_scale, p.c_is_fp32, p.c);
            }
        };
        for (int n = 0; n < count;) {
            // the segment [kb, kb_end) of `tile`
            const int seg_len = min(p.kb - kb, count - n);
            const bool from_zero = (kb == 0), to_end = (kb + seg_len == p.kb);
            const uint32_t buf = kBuffers == 2 ? (seg & 1u) : 0u;
            if constexpr (KIND == Kind::kNv4 && M_PAD == 16) {
                // a group's scale and row mask, once per group and before the wait: read per tile behind it, the two
                // dependent loads made the epilogue longer than a tile of eight units (w2 of the routed experts 266 -> 288 us)
                if (grouped) grp = tile / p.n_tiles;
                if (grouped && grp != seen_grp) {
                    seen_grp = grp;
                    scale = p.out_scale * __ldcg(p.expert_scale + __ldcg(p.group_expert + grp));
                    if (p.row_token) {
                        const int tok = lane < M_PAD ? __ldcg(p.row_token + grp * M_PAD + lane) : -1;
                        stored = __ballot_sync(0xffffffffu, tok >= 0);
                    }
                }
            }
            // The start of a tile whose K range goes on in the following CTAs (all resident: the grid is one CTA per SM): their
            // partials were finished first, so the flags are awaited (each by a thread of its own) and the first partial
            // is fetched while this segment's MMAs still run.
            const bool owner = !p.sliced && from_zero && !to_end;
            constexpr bool kAhead = kCols <= 32 || (M_PAD == 128 && KIND == Kind::kNv4);   // (what the registers hold without spills)
            float4 ahead[kAhead ? kCols / 4 : 1];
            int last = blockIdx.x;
            auto slot_of = [&](int c) {
                return reinterpret_cast<const float4*>(p.scratch + static_cast<int64_t>(c) * slot_floats) + col0 / 4 * kTileN + row;
            };
            if (!kEven && p.sliced) held |= holders_of(units, tile, p.kb, grid) << (16 * seg);
            if (owner) {
                last = cta_of(units, static_cast<uint32_t>(tile + 1) * static_cast<uint32_t>(p.kb) - 1u, grid);
                for (int c = blockIdx.x + 1 + et; c <= last && alive; c += kEpi)
                    await_word<200>(p.flags + c, [](int v) { return v != 0; }, abort_flag, p.status);
                epi_sync();
                alive = __all_sync(0xffffffffu, alive && !*abort_flag);
                if (kAhead && alive && col0 < p.M) {     // (the slot of a CTA has room for M_PAD columns)
#pragma unroll
                    for (int i = 0; i < kCols / 4; ++i) ahead[i] = __ldcg(slot_of(blockIdx.x + 1) + i * kTileN);
                }
            }
            if (alive) alive = mbar_wait_warp_fast(full_tm + buf * 8, (seg / kBuffers) & 1u, abort_flag, p.status, kDevTimeoutGemmTmemFull);
            float acc[kCols];
            if (alive) {
                tc_fence_after();
                const uint32_t t0 = tmem_base + lane_base + buf * (L::kAccs * M_PAD) + col0;
                uint32_t(&raw)[kCols] = reinterpret_cast<uint32_t(&)[kCols]>(acc);
                if constexpr (L::kAccs == 2) {
                    const uint32_t first = (n & 1) * M_PAD;      // a segment of one unit has only this sum
#pragma unroll
                    for (int c = 0; c < kCols; c += 16) {
                        uint32_t v0[16], v1[16];
                        tmem_ld_32x16(t0 + first + c, v0);
                        if (seg_len >= 2) tmem_ld_32x16(t0 + (M_PAD - first) + c, v1);
                        tmem_ld_wait();
#pragma unroll
                        for (int i = 0; i < 16; ++i) acc[c + i] = __uint_as_float(v0[i]) + (seg_len >= 2 ? __uint_as_float(v1[i]) : 0.f);
                    }
                } else {
#pragma unroll
                    for (int c = 0; c < kCols; c += 16) tmem_ld_32x16(t0 + c, reinterpret_cast<uint32_t(&)[16]>(raw[c]));
                    tmem_ld_wait();
                }
                tc_fence_before();
            } else {
#pragma unroll
                for (int i = 0; i < kCols; ++i) acc[i] = __int_as_float(0x7fffffff);
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(empty_tm + buf * 8);

            const int nrow0 = (tile - grp * p.n_tiles) * kTileN;
            if (p.sliced || !from_zero) {   // partial sums to this CTA's slot
                float4* slot = reinterpret_cast<float4*>(p.scratch + slot_index(p.sliced && !kEven, from_zero, tile) * slot_floats) + row;
#pragma unroll
                for (int c = 0; c < kCols; c += 4)
                    if (col0 + c < p.M) __stcg(slot + (col0 + c) / 4 * kTileN, make_float4(acc[c], acc[c + 1], acc[c + 2], acc[c + 3]));
                // The barrier orders all threads' stores before the one thread's release of the flag or counter behind it, which
                // covers them all: a fence of every thread's own in between held up the tail of short calls by 0.7 us.
                epi_sync();
            }
            if (p.sliced) {
                // The last arrival wraps the tile's counter back to zero, which is what the others wait for, once they have
                // nothing else to do.  No CTA arrives at a counter twice in a launch, the next launch's arrive after this one.
                const Holders h = holders(seg);
                if (M_PAD == 16 && p.last_adds) {
                    if (et == 0) *arrived_last = inc_acq_rel_gpu(p.flags + tile, h.count() - 1) == h.count() - 1;
                    epi_sync();
                    if (*arrived_last)
                        add_slice<KIND>(p.scratch, slot_floats, tile, h, start_slot(tile), 0, 1, et, kEpi, p.M, p.N, p.out_scale, p.c_is_fp32, p.c);
                    epi_sync();     // (before the word is written again)
                } else if (et == 0) {
                    inc_acq_rel_gpu(p.flags + tile, h.count() - 1);
                }
                if (kEven) slice(0);
            } else if (!from_zero) {
                if (et == 0) raise_flag(p.flags + blockIdx.x);
            } else {
                if (owner) {     // add the partials in CTA order
                    if (alive && col0 < p.M) {
                        for (int c = blockIdx.x + 1; c <= last; ++c) {
                            // (pieces of 32 columns, eight 16-byte loads in flight each: a condition per load would wait for
                            // every one by itself)
                            constexpr int kPiece = kCols < 32 ? kCols : 32;
#pragma unroll
                            for (int c0 = 0; c0 < kCols; c0 += kPiece)
                                if (col0 + c0 < p.M) {
                                    float4 v[kPiece / 4];
#pragma unroll
                                    for (int i = 0; i < kPiece / 4; ++i)
                                        v[i] = kAhead && c == static_cast<int>(blockIdx.x) + 1 ? ahead[c0 / 4 + i] : __ldcg(slot_of(c) + (c0 / 4 + i) * kTileN);
#pragma unroll
                                    for (int i = 0; i < kPiece / 4; ++i) {
                                        acc[c0 + 4 * i] += v[i].x, acc[c0 + 4 * i + 1] += v[i].y;
                                        acc[c0 + 4 * i + 2] += v[i].z, acc[c0 + 4 * i + 3] += v[i].w;
                                    }
                                }
                        }
                    }
                    epi_sync();
                    for (int c = blockIdx.x + 1 + et; c <= last; c += kEpi) lower_flag(p.flags + c);
                }
                const int nrow = nrow0 + row;
                // Rows of C that take 8-byte stores: the four lanes that hold four neighbouring weight rows exchange their
                // values so that each stores one activation row's four - a quarter of the store instructions.
                const bool wide = M_PAD > 16 && !(KIND == Kind::kBf16 && p.c_is_fp32) && (p.N & 3) == 0 &&
                                  (reinterpret_cast<uintptr_t>(p.c) & 7u) == 0;
                if (wide) {
                    if (alive) {
                        const float out = KIND == Kind::kNv4 ? p.out_scale : 1.f;
                        __nv_bfloat16* c = static_cast<__nv_bfloat16*>(p.c) + nrow0 + (row & ~3);
                        const bool in_n = nrow < p.N;    // (N is a multiple of four: the four lanes agree)
#pragma unroll
                        for (int i = 0; i < kCols; i += 4)
                            if (col0 + i < p.M) {
                                uint32_t rows01, rows23;
                                transpose4(to_bf16x2(acc[i] * out, acc[i + 1] * out), to_bf16x2(acc[i + 2] * out, acc[i + 3] * out),
                                           lane, rows01, rows23);
                                const int m = col0 + i + static_cast<int>(lane & 3);
                                if (m < p.M && in_n) *reinterpret_cast<uint2*>(c + static_cast<int64_t>(m) * p.N) = make_uint2(rows01, rows23);
                            }
                    }
                } else if (alive && nrow < p.N) {
                    const int64_t c_off = static_cast<int64_t>(grp) * M_PAD * p.N;
#pragma unroll
                    for (int i = 0; i < kCols; ++i)
                        if (col0 + i < p.M && (M_PAD > 16 || ((stored >> i) & 1u))) {
                            const int64_t at = c_off + static_cast<int64_t>(col0 + i) * p.N + nrow;
                            const float v = KIND == Kind::kNv4 ? acc[i] * scale : acc[i];
                            if (KIND == Kind::kBf16 && p.c_is_fp32) static_cast<float*>(p.c)[at] = v;
                            else static_cast<__nv_bfloat16*>(p.c)[at] = __float2bfloat16_rn(v);
                        }
                }
            }
            n += seg_len;
            kb += seg_len;
            if (kb == p.kb) kb = 0, ++tile;
            ++seg;
        }
        if (!kEven && p.sliced && !(M_PAD == 16 && p.last_adds)) {
#pragma unroll 1
            for (uint32_t i = 0; i < seg; ++i) slice(i);
        }
    }

    __syncthreads();
    if (*abort_flag) abort_drain_sleep();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem_base, L::kTmemCols);
    }
}

// Added in slices where every tile is cut into three ranges or more (and the slots suffice: one per CTA and one per tile).  Ranges that
// hold parts of two tiles take part in two additions, each behind that tile's last CTA: with 17 to 64 rows that pays from five
// ranges per tile on (FP8 4096 x 7168 at 64 rows, 148 ranges of 32 tiles: in slices 14.1 us, by the CTA with the tile's start 12.7; BF16
// 2624 x 7168, 102 ranges of 21: 14.0, 13.2), while at 128 rows the slices win from three on (the same two 18.0 / 18.4 and 17.6 / 19.0).
// The order of additions is the same.  (Either side at 17 to 64 rows of 4096 / 4608 / 5120 x 7168 and 4096 x 2048 / 4096, all formats: in slices
// 0.4 to 2.2 us longer.)
inline bool slice_wise(int grid, int n_tiles, int m_pad) {
    const int least = (m_pad == 32 || m_pad == 64) && grid % n_tiles != 0 ? 5 : 3;
    return grid >= least * n_tiles && grid + n_tiles <= kMaxGrid;
}
// Few activation rows: a sliced tile has one quad of sums per epilogue thread, which is one round of loads however few CTAs share
// them.  The CTA that arrives last at the tile's counter adds the whole tile, right there, and nobody has to wait for the
// others: FP8 2112 x 7168 at one row, plain calls, 9.0 -> 8.0 us; 128 to 4096 wide, 1 to 4 rows (general FP8 scales, with twice the threads, 8),
// 0.2 to 1.3 us.  With two quads the second round over up to sixteen partials costs more than the one wait of a CTA whose range is part of
// one tile (up to 1152 x 7168, 5 to 8 rows, 0.3 to 0.9 us), but less than the two waits of one that holds parts of two tiles
// (1280 to 4096 x 7168 0.3 to 0.9 us).
inline bool last_arrival_adds(int m, int threads, int grid, int n_tiles) {
    const int quads = (m + 3) / 4 * kTileN;
    return quads <= threads || (quads <= 2 * threads && grid % n_tiles != 0);
}
// Even slices: CTAs per tile, as many as the SMs hold when that is at least three (and every one gets a unit), else none.
inline int even_split(int n_tiles, int kb, int sms) {
    int split = sms / n_tiles;
    if (split > kb) split = kb;
    if (split > kMaxEvenSplit) split = kMaxEvenSplit;
    return split >= 3 ? split : 0;
}

template <Kind KIND, int M_PAD>
int launch(const CUtensorMap& w_map, const CUtensorMap& a_map, const CUtensorMap& wsf_map, const CUtensorMap& asf_map, Params& p,
           const DeviceInfo& dev, cudaStream_t stream) {
    using L = Layout<KIND, M_PAD>;
    int stages = p.group_expert ? kGroupedStages : kMaxStages;
    while (stages > 2 && L::total(stages, p.a_rows) > dev.smem_optin) --stages;
    if (L::total(stages, p.a_rows) > dev.smem_optin)
        return fail(WUDA_ERR_UNSUPPORTED, "device offers %d bytes of shared memory per block; the kernel needs more", dev.smem_optin);
    p.stages = stages;
    auto kernel = gemm_tc_kernel<KIND, M_PAD>;
    // (the same limit whatever the rows and stages: it is the kernel's, and another thread may set it before this launch)
    WUDA_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, dev.smem_optin));
    const int sms = gemm_sms(dev);
    // (grouped: the number of groups is only known on the device; one CTA per SM, idle ones return at once)
    int grid = p.group_expert ? sms : grid_of(static_cast<long long>(p.n_tiles) * p.kb, p.n_tiles, M_PAD, sms);
    if (L::kEvenSlices) {
        p.sliced = even_split(p.n_tiles, p.kb, sms);
        if (p.sliced) grid = p.n_tiles * p.sliced;
    } else {
        p.sliced = !p.group_expert && slice_wise(grid, p.n_tiles, M_PAD);
    }
    p.last_adds = last_arrival_adds(p.M, 32 * L::kEpiWarps, grid, p.n_tiles);
    WUDA_CUDA(launch_pdl(kernel, dim3(grid), dim3(L::kThreads), L::total(stages, p.a_rows), stream, w_map, a_map, wsf_map, asf_map, p));
    return WUDA_OK;
}

// The kernel for m activation rows.
template <Kind KIND>
int launch_for(int m, const CUtensorMap& w_map, const CUtensorMap& a_map, const CUtensorMap& wsf_map, const CUtensorMap& asf_map,
               Params& p, const DeviceInfo& dev, cudaStream_t stream) {
    if (m <= 16) return launch<KIND, 16>(w_map, a_map, wsf_map, asf_map, p, dev, stream);
    if (m <= 32) return launch<KIND, 32>(w_map, a_map, wsf_map, asf_map, p, dev, stream);
    if (m <= 64) return launch<KIND, 64>(w_map, a_map, wsf_map, asf_map, p, dev, stream);
    if constexpr (KIND != Kind::kBf16)      // (BF16 takes at most 128 rows)
        if (m > 128) return launch<KIND, 256>(w_map, a_map, wsf_map, asf_map, p, dev, stream);
    return launch<KIND, 128>(w_map, a_map, wsf_map, asf_map, p, dev, stream);
}

// Bytes of scratch a call with m rows wants: the flags and kMaxGrid partial-tile slots.
inline int64_t scratch_bytes(int m) {
    int m_pad = 16;
    while (m_pad < m) m_pad *= 2;
    return kFlagBytes + static_cast<int64_t>(kMaxGrid) * m_pad * kTileN * 4;
}
inline int rows_of(int m) { return (m + 15) / 16 * 16; }

}  // namespace gemmtc
}  // namespace wuda
