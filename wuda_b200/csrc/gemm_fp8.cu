// Block-scaled FP8 GEMM for decode-sized M on sm_100a:
//
//   C[M, N] (bf16) = A[M, K] (e4m3, fp32 scale per 1x128) x W[N, K]^T (e4m3, fp32 scale per 128x128)
//
// Numerics contract (dsv4_megakernel/origin/kernel.py:203-273, fp8_gemm_kernel): every
// 128-wide K block is accumulated in fp32 on its own and then added, multiplied by
// a_s[m, kb] * w_s[n / 128, kb], to a second fp32 accumulator (lines 246-250).  This is
// the generic form of the reference's wq_b / wo_b projections
// (dsv4_megakernel/megakernel/kernels/wq_b_fp8_gemm.cu:189-780, test/o_proj_csa.py:454-480),
// which use power-of-two UE8M0 scales; fp32 scales cannot ride the tensor core's
// block-scale path, so the promotion happens in registers.
//
// Design: decode GEMMs are bound by the weight stream (N*K bytes once from HBM), so
//  * swap-AB: the UMMA M dimension (128) is a tile of weight rows, the UMMA N dimension is the activation count rounded
//    up to 16; the activations (a few MB at most) are re-read from L2 for every weight tile (gemm_tc.cuh says why that
//    is cheap);
//  * the work split is gemm_tc.cuh's: stream-K, for few weight tiles with the partial sums added in slices;
//  * per unit: an elected thread fetches the weight tile (128 x 128 B) and the activation tile, another issues four
//    tcgen05.mma kind::f8f6f4 into a fresh TMEM stage, and an epilogue warpgroup adds the stage, times the unit's scales,
//    to its register accumulators.  The scales of a stage, already multiplied (a_s * w_s), are written beside it by a
//    warp that requested them four K blocks at a time, eight units earlier, and arrives on the stage's barrier: an
//    epilogue thread waits once per unit.  The two epilogue warpgroups take units alternately and their chains overlap; the
//    two accumulator sets are added when a tile's segment ends.  (Above 64 activation rows a thread cannot hold all
//    columns; the groups then split the columns and both take every unit.)
// Measured (as in gemm_tc.cuh, us; before = scales fetched by the epilogue threads behind two barriers per unit, resident
// activations for short K, partials added by one CTA per tile): 24576 x 7168 at 16 / 64 / 128 / 256 rows 38.3 -> 34.7,
// 47.1 -> 40.6, 66.1 -> 54.7, 131 -> 109 (two passes); 7168 x 16384 at 64 rows 32.9 -> 29.5; 2112 x 7168 at 1 / 64 rows
// 13.3 -> 12.3, 16.4 -> 11.0; 4096 x 7168 at 64 rows 17.6 -> 16.7.  The results are bit-identical to those of the earlier
// form: the order of the additions is the same.
// Every wait is bounded and reports through the status word; flags and counters end at zero all the same (gemm_tc.cuh).
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cstring>
#include <mutex>

#include "gemm_tc.cuh"
#include "host.h"
#include "ptx.cuh"

namespace wuda {
namespace gemm8 {

using gemmtc::await_word;
using gemmtc::cta_of;
using gemmtc::holders_of;
using gemmtc::inc_acq_rel_gpu;
using gemmtc::unpack_holders;
using gemmtc::kRowBytes;
using gemmtc::kTileN;
using gemmtc::kWBytes;
using gemmtc::ld_acquire_gpu;
using gemmtc::lower_flag;
using gemmtc::raise_flag;
using gemmtc::range_begin;
using gemmtc::slot_index;
using gemmtc::st_release_gpu;

constexpr int kFirstEpiWarp = 4;     // warp 0 copies, 1 issues MMAs, 2 prepares scales, 3 awaits partials, 4..11 are two epilogue warpgroups
constexpr int kEpiWarps = 8;
constexpr int kThreads = 32 * (kFirstEpiWarp + kEpiWarps);
// (more copies in flight cost DRAM efficiency: 24576 x 7168 at 16 rows 35.9 us with 6 stages, 37.3 with 10)
constexpr int kMaxStages = 6;

struct Params {
    const float* a_scales;     // [M, a_kb_total]
    const float* w_scales;     // [ceil(N/128), K/128]
    __nv_bfloat16* c;          // [M, N]
    float* scratch;            // partial-tile slots, fp32 [M_PAD / 4][128 weight rows][4 activation rows]: [grid], sliced also [n_tiles]
    int32_t* flags;            // one flag per CTA; sliced: one counter per weight tile; zero between calls
    int32_t* status;
    int M, N, K, kb;           // kb = K / 128
    int n_tiles;
    int a_rows;                // M rounded up to 16
    int stages;
    int sliced;                // a tile's partial sums are added by all of its CTAs, a slice each
    int last_adds;             // .. or by the one that completes the tile's counter
    int vec_scales;            // rows of a_scales can be read 16 bytes at a time
    // grouped form: weight tile t belongs to group t / group_tiles and reads the activations'
    // columns [group * K, (group + 1) * K); a_kb_total = K blocks in an activation row
    int group_tiles = 0;
    int a_kb_total = 0;
    // two-rank tensor parallelism (K split across two GPUs): peer exchange of fp32 tiles
    float* tp_my_inbox = nullptr;      // [2 sets][n_tiles][M_PAD][128] fp32 in THIS GPU's memory
    float* tp_peer_inbox = nullptr;    // the same buffer of the peer, mapped into this process
    int32_t* tp_my_flags = nullptr;    // [2 sets][n_tiles]: sequence number of the last tile received
    int32_t* tp_peer_flags = nullptr;
    int32_t* tp_ctrl = nullptr;        // this rank's control words: [0] last finished call, [1] CTAs done
    int tp_epoch = 0;                  // sequence number of this call (> 0, same on both ranks); 0: tp_ctrl[0] + 1
    unsigned long long tp_wait_ns = 0; // limit of one wait for the peer
};

template <int M_PAD>
struct Smem {
    static constexpr int kTmemStages = M_PAD <= 64 ? 8 : 4;
    static constexpr int kTmemCols = kTmemStages * M_PAD;
    // Up to M_PAD = 64 the two epilogue warpgroups take units alternately (all columns each) and add
    // their accumulators through a [M_PAD][128] fp32 buffer when a tile's segment ends; above that a
    // thread cannot hold M_PAD accumulators and the groups split the columns instead.
    static constexpr bool kAlternate = M_PAD <= 64;
    static constexpr int kCombineBytes = kAlternate ? M_PAD * kTileN * 4 : 0;
    static __host__ __device__ constexpr int stage_bytes(int a_rows) { return kWBytes + a_rows * kRowBytes; }
    // one row of scale products per TMEM stage
    static __host__ __device__ constexpr int scale_off(int stages, int a_rows) { return stages * stage_bytes(a_rows); }
    static __host__ __device__ constexpr int comb_off(int stages, int a_rows) { return scale_off(stages, a_rows) + kTmemStages * M_PAD * 4; }
    static __host__ __device__ constexpr int bar_off(int stages, int a_rows) { return comb_off(stages, a_rows) + kCombineBytes; }
    // barriers: full[6] empty[6] full_tm[8] empty_tm[8] partials
    static __host__ __device__ constexpr int misc_off(int stages, int a_rows) { return bar_off(stages, a_rows) + (2 * kMaxStages + 17) * 8; }
    static __host__ __device__ constexpr int total(int stages, int a_rows) { return misc_off(stages, a_rows) + 32 + 1024; }
};

__device__ __forceinline__ void epi_bar_sync() { asm volatile("bar.sync 1, 256;" ::: "memory"); }
__device__ __forceinline__ void st_release_sys(int32_t* p, int v) {
    asm volatile("st.release.sys.global.s32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ int ld_acquire_sys(const int32_t* p) {
    int v;
    asm volatile("ld.acquire.sys.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ float ld_volatile_f32(const float* p) {   // written by the peer GPU: bypass L1
    float v;
    asm volatile("ld.volatile.global.f32 %0, [%1];" : "=f"(v) : "l"(p) : "memory");
    return v;
}

template <int M_PAD>
__global__ void __launch_bounds__(kThreads, 1)
gemm_fp8_kernel(const __grid_constant__ CUtensorMap w_map, const __grid_constant__ CUtensorMap a_map,
                const Params p) {
    using L = Smem<M_PAD>;
    constexpr int kTS = L::kTmemStages;
    constexpr int kHalf = M_PAD / 2;                 // columns a warpgroup finishes
    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw_addr = smem_u32(smem_raw);
    const uint32_t base = (raw_addr + 1023u) & ~1023u;
    uint8_t* base_ptr = smem_raw + (base - raw_addr);
    const int S = p.stages;
    const uint32_t stage_bytes = L::stage_bytes(p.a_rows);
    const uint32_t bars = base + L::bar_off(S, p.a_rows);
    const uint32_t full = bars, empty = full + kMaxStages * 8, full_tm = empty + kMaxStages * 8, empty_tm = full_tm + 8 * 8, partials = empty_tm + 8 * 8;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(base_ptr + L::misc_off(S, p.a_rows));
    volatile int* abort_flag = reinterpret_cast<volatile int*>(base_ptr + L::misc_off(S, p.a_rows) + 4);
    volatile int* last_peer_slot = reinterpret_cast<volatile int*>(base_ptr + L::misc_off(S, p.a_rows) + 8);
    volatile int* arrived_last = reinterpret_cast<volatile int*>(base_ptr + L::misc_off(S, p.a_rows) + 12);
    float* products = reinterpret_cast<float*>(base_ptr + L::scale_off(S, p.a_rows));     // [kTS][M_PAD]: a_s * w_s
    float* comb = reinterpret_cast<float*>(base_ptr + L::comb_off(S, p.a_rows));
    constexpr bool kAlt = L::kAlternate;

    const int warp = __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x >> 5), 0);
    const uint32_t lane = lane_id();

    if (threadIdx.x == 0) {
        *abort_flag = 0;
        for (int i = 0; i < S; ++i) {
            mbar_init(full + i * 8, 1);
            mbar_init(empty + i * 8, 1);          // released by the UMMA commit
        }
        for (int i = 0; i < kTS; ++i) {
            mbar_init(full_tm + i * 8, 2);        // the MMAs have retired and the scale products are written
            mbar_init(empty_tm + i * 8, kAlt ? kEpiWarps / 2 : kEpiWarps);   // the warps that read a stage
        }
        mbar_init(partials, 1);
        fence_mbar_init();
    }
    if (warp == 1) {
        tmem_alloc(smem_u32(tmem_slot), L::kTmemCols);
        tmem_relinquish();
    }
    const uint32_t units = static_cast<uint32_t>(p.n_tiles) * static_cast<uint32_t>(p.kb);
    const uint32_t u0 = range_begin(units, blockIdx.x, gridDim.x);
    const int count = static_cast<int>(range_begin(units, blockIdx.x + 1, gridDim.x) - u0);
    const int tile0 = static_cast<int>(u0 / static_cast<uint32_t>(p.kb)), kb0 = static_cast<int>(u0) - tile0 * p.kb;
    // The last tile of a stream-K range may go on in the following CTAs (all resident: the grid is one CTA per SM).  If this
    // CTA holds its start, it adds their partials, of CTAs blockIdx.x + 1 .. last_peer, in CTA order.
    const uint32_t last_tile = (u0 + count - 1u) / static_cast<uint32_t>(p.kb);
    const bool shares = !p.sliced && last_tile * p.kb >= u0 && (last_tile + 1u) * p.kb > u0 + count;
    if (warp == 0 && elect_one()) {
        prefetch_tmap(&w_map);
        prefetch_tmap(&a_map);
        int tile = tile0, kb = kb0;
        for (int n = 0; n < count && n < S; ++n) {
            tma_prefetch_2d(&w_map, kb * kRowBytes, tile * kTileN);
            if (++kb == p.kb) kb = 0, ++tile;
        }
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    // all of the above ran while the kernel ahead was still finishing; its results are read from here on
    pdl_launch_dependents();
    pdl_wait();

    // two-rank form with the link's own numbering: this call's number is one more than the last
    // finished call's (the word is rewritten only after every CTA of this call has read it)
    const int tp_epoch = (p.tp_peer_inbox && p.tp_epoch == 0) ? ld_acquire_gpu(p.tp_ctrl) + 1 : p.tp_epoch;

    if (warp == 0) {
        // ------------------------------------------------------------ copies
        if (elect_one()) {
            const uint64_t stream_policy = policy_evict_first();
            const uint64_t keep_policy = policy_evict_last();
            int s = 0, tile = tile0, kb = kb0;
            uint32_t phase = 1;
            for (int n = 0; n < count; ++n) {
                const int a_x = kb * kRowBytes + (p.group_tiles ? (tile / p.group_tiles) * p.K : 0);
                if (!mbar_wait(empty + s * 8, phase, abort_flag, p.status, kDevTimeoutGemmEmpty)) break;
                const uint32_t stage = base + s * stage_bytes;
                mbar_arrive_expect_tx(full + s * 8, stage_bytes);
                tma_load_2d_hint(stage, &w_map, full + s * 8, kb * kRowBytes, tile * kTileN, stream_policy);
                tma_load_2d_hint(stage + kWBytes, &a_map, full + s * 8, a_x, 0, keep_policy);
                if (++s == S) s = 0, phase ^= 1u;
                if (++kb == p.kb) kb = 0, ++tile;
            }
        }
    } else if (warp == 1) {
        // ------------------------------------------------------------ MMAs
        if (elect_one()) {
            const uint32_t idesc = umma_idesc(kTileN, p.a_rows, 0, 0);
            int s = 0;
            uint32_t phase = 0;
            for (int n = 0; n < count; ++n) {
                const int ts = n % kTS;
                if (!mbar_wait(empty_tm + ts * 8, ((n / kTS) & 1) ^ 1, abort_flag, p.status, kDevTimeoutGemmTmemEmpty)) break;
                if (!mbar_wait(full + s * 8, phase, abort_flag, p.status, kDevTimeoutGemmFull)) break;
                tc_fence_after();
                const uint32_t w_addr = base + s * stage_bytes;
                const uint64_t w_desc = umma_smem_desc_sw128(w_addr), a_desc = umma_smem_desc_sw128(w_addr + kWBytes);
#pragma unroll
                for (int k = 0; k < 4; ++k)
                    umma_f8f6f4(tmem_base + ts * M_PAD, w_desc + k * 2, a_desc + k * 2, idesc, k > 0 ? 1u : 0u);
                umma_commit(full_tm + ts * 8);
                umma_commit(empty + s * 8);      // the stage's bytes are consumed once the UMMAs retire
                if (++s == S) s = 0, phase ^= 1u;
            }
        }
    } else if (warp == 2) {
        // ------------------------------------------------------------ scale products
        // In groups of four K blocks of a tile (aligned to four, cut at the ends of the range).  A lane holds the scales of
        // rows lane, lane + 32, ..; two groups are in registers, each refilled when it has been written out.  (One warp: it
        // sees every phase of the barriers it waits on.)  All through L2: gemm_tc.cuh says why.
        constexpr int kQ = (M_PAD + 31) / 32;
        int tile = tile0, kb = kb0, n = 0;
        struct Raw {
            float4 a[kQ], w;
            int n, k, len;          // first unit, its K block modulo four, units
        };
        auto group_len = [&] { return min(min(4 - (kb & 3), p.kb - kb), count - n); };
        auto fill = [&](Raw& r) {
            r.n = n, r.k = kb & 3, r.len = group_len();
            if (n < count) {
                const int k0 = kb & ~3, col = k0 + (p.group_tiles ? (tile / p.group_tiles) * p.kb : 0);
#pragma unroll
                for (int q = 0; q < kQ; ++q) {
                    const int row = q * 32 + static_cast<int>(lane);
                    r.a[q] = make_float4(0.f, 0.f, 0.f, 0.f);
                    if (row < p.M) {
                        const float* src = p.a_scales + static_cast<int64_t>(row) * p.a_kb_total + col;
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
                const float* src = p.w_scales + static_cast<int64_t>(tile) * p.kb + k0;
                r.w.x = __ldcg(src);
                r.w.y = k0 + 1 < p.kb ? __ldcg(src + 1) : 0.f;
                r.w.z = k0 + 2 < p.kb ? __ldcg(src + 2) : 0.f;
                r.w.w = k0 + 3 < p.kb ? __ldcg(src + 3) : 0.f;
                const int len = group_len();
                n += len, kb += len;
                if (kb == p.kb) kb = 0, ++tile;
            }
        };
        auto of = [](const float4& v, int i) { return i == 0 ? v.x : (i == 1 ? v.y : (i == 2 ? v.z : v.w)); };
        auto write = [&](const Raw& r) -> bool {
            for (int i = 0; i < r.len; ++i) {
                const int u = r.n + i, ts = u % kTS;
                const float w = of(r.w, r.k + i);
                float v[kQ];
#pragma unroll
                for (int q = 0; q < kQ; ++q) v[q] = __fmul_rn(of(r.a[q], r.k + i), w);
                if (!mbar_wait_warp_fast(empty_tm + ts * 8, ((u / kTS) & 1) ^ 1, abort_flag, p.status, kDevTimeoutGemmTmemEmpty))
                    return false;
#pragma unroll
                for (int q = 0; q < kQ; ++q)
                    if (q * 32 + static_cast<int>(lane) < M_PAD) products[ts * M_PAD + q * 32 + lane] = v[q];
                __syncwarp();
                if (lane == 0) mbar_arrive(full_tm + ts * 8);
            }
            return true;
        };
        Raw a, b;
        fill(a);
        fill(b);
        while (a.n < count) {
            if (!write(a)) break;
            fill(a);
            if (b.n >= count || !write(b)) break;
            fill(b);
        }
    } else if (warp == 3) {
        // ------------------------------------------------------------ the other CTAs' partials, awaited beside the stream
        // (each by a lane of its own; they are finished first)
        if (shares) {
            const int last_peer = cta_of(units, (last_tile + 1) * p.kb - 1, gridDim.x);
            for (int c = blockIdx.x + 1 + static_cast<int>(lane); c <= last_peer; c += 32)
                await_word<200>(p.flags + c, [](int v) { return v != 0; }, abort_flag, p.status);
            if (lane == 0) *last_peer_slot = last_peer;
            __syncwarp();
            if (lane == 0) mbar_arrive(partials);
        }
    } else if (warp >= kFirstEpiWarp) {
        // ------------------------------------------------------------ epilogue
        const int ew = warp - kFirstEpiWarp;
        const int grp = ew >> 2, half = grp;
        const int et = ew * 32 + static_cast<int>(lane);      // 0..255
        const int row_in_tile = (warp & 3) * 32 + static_cast<int>(lane);
        const uint32_t lane_base = static_cast<uint32_t>((warp & 3) * 32) << 16;
        // kAlt: this group takes the units with (n & 1) == grp and accumulates every column;
        // otherwise both groups take every unit and half of the columns each.
        constexpr int kCols = kAlt ? M_PAD : kHalf;
        const int col0 = kAlt ? 0 : half * kHalf;
        __align__(16) float acc[kCols];
#pragma unroll
        for (int i = 0; i < kCols; ++i) acc[i] = 0.f;
        bool alive = true;
        int tile = tile0, kb = kb0;
        int seg_kb0 = kb;                               // first K block of the running segment
        constexpr int64_t kSlotFloats = static_cast<int64_t>(M_PAD) * kTileN;
        int seg = 0;
        uint32_t held = 0;                              // sliced: who shares the first and the second tile of this range
        if (p.sliced) {
            held = holders_of(units, tile0, p.kb, gridDim.x);
            if (last_tile != static_cast<uint32_t>(tile0)) held |= holders_of(units, tile0 + 1, p.kb, gridDim.x) << 16;
        }

        // An aborting CTA keeps walking the loop (every wait then fails at once) so that all
        // 256 epilogue threads reach every named barrier; it only skips the arithmetic.
        for (int n = 0; n < count; ++n) {
            if (!kAlt || (n & 1) == grp) {
                const int ts = n % kTS;
                if (alive)
                    alive = mbar_wait_warp_fast(full_tm + ts * 8, (n / kTS) & 1, abort_flag, p.status, kDevTimeoutGemmTmemFull);
                if (alive) {
                    tc_fence_after();
                    const float* sc = products + ts * M_PAD + col0;
                    const uint32_t taddr = tmem_base + lane_base + ts * M_PAD + col0;
                    // acc[c] += v[c] * (a_s[c] * w_s): the products come as 16-byte shared-memory loads, the
                    // sums as packed fp32x2 operations (one instruction per two columns)
                    float2* acc2 = reinterpret_cast<float2*>(acc);
                    constexpr int kPiece = kCols < 32 ? 16 : 32;
                    uint32_t v[2][kPiece];
                    auto load = [&](int c, uint32_t (&dst)[kPiece]) {
                        if constexpr (kPiece == 32) tmem_ld_32x32(taddr + c, dst);
                        else tmem_ld_32x16(taddr + c, dst);
                    };
                    load(0, v[0]);
#pragma unroll
                    for (int c = 0; c < kCols; c += kPiece) {
                        tmem_ld_wait();
                        if (c + kPiece < kCols) load(c + kPiece, v[(c / kPiece + 1) & 1]);
                        const uint32_t* x = v[(c / kPiece) & 1];
                        const float4* s4 = reinterpret_cast<const float4*>(sc + c);
#pragma unroll
                        for (int i = 0; i < kPiece; i += 4) {
                            const float4 sv = s4[i >> 2];
                            acc2[(c + i) >> 1] = __ffma2_rn(make_float2(__uint_as_float(x[i]), __uint_as_float(x[i + 1])),
                                                            make_float2(sv.x, sv.y), acc2[(c + i) >> 1]);
                            acc2[((c + i) >> 1) + 1] = __ffma2_rn(make_float2(__uint_as_float(x[i + 2]), __uint_as_float(x[i + 3])),
                                                                  make_float2(sv.z, sv.w), acc2[((c + i) >> 1) + 1]);
                        }
                    }
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(empty_tm + ts * 8);
                }
            }

            // ---- end of a segment: the tile's K range ended, or this CTA's range did
            const bool seg_end = (kb + 1 == p.kb) || (n + 1 == count);
            if (seg_end) {
                auto poison = [&] {      // after a wait that ran out: whoever adds this to anything gets NaN
#pragma unroll
                    for (int i = 0; i < kCols; ++i) acc[i] = __int_as_float(0x7fffffff);
                };
                if (!alive) poison();
                if constexpr (kAlt) {
                    // Each group hands the other the columns that one finishes and adds what it gets
                    // to its own half; the sums land in acc[0, kHalf).  x + y == y + x, so the result
                    // does not depend on which group held which units.
                    // (constant register indices in both branches: the accumulators stay in registers)
                    if (half == 0) {
#pragma unroll
                        for (int i = 0; i < kHalf; ++i) comb[(kHalf + i) * kTileN + row_in_tile] = acc[kHalf + i];
                    } else {
#pragma unroll
                        for (int i = 0; i < kHalf; ++i) comb[i * kTileN + row_in_tile] = acc[i];
                    }
                    epi_bar_sync();
                    if (half == 0) {
#pragma unroll
                        for (int i = 0; i < kHalf; ++i) acc[i] = acc[i] + comb[i * kTileN + row_in_tile];
                    } else {
#pragma unroll
                        for (int i = 0; i < kHalf; ++i) acc[i] = acc[kHalf + i] + comb[(kHalf + i) * kTileN + row_in_tile];
                    }
                    epi_bar_sync();                      // the buffer is free for the next segment
                }
                const int c0 = half * kHalf;             // this thread finishes columns c0 .. c0 + kHalf - 1
                const int nrow = tile * kTileN + row_in_tile;
                const bool from_zero = (seg_kb0 == 0), to_end = (kb + 1 == p.kb);
                if (p.sliced || !from_zero) {
                    // partial sums to this CTA's slot, 16 bytes = four columns of a row
                    float4* slot = reinterpret_cast<float4*>(p.scratch + slot_index(p.sliced, from_zero, tile) * kSlotFloats) + row_in_tile;
#pragma unroll
                    for (int i = 0; i < kHalf; i += 4)
                        if (c0 + i < p.M) __stcg(slot + (c0 + i) / 4 * kTileN, make_float4(acc[i], acc[i + 1], acc[i + 2], acc[i + 3]));
                    epi_bar_sync();     // (the flag's release covers what the barrier orders before it: gemm_tc.cuh)
                }
                if (p.sliced) {
                    // (the last arrival wraps the tile's counter back to zero: gemm_tc.cuh)
                    const gemmtc::Holders h = unpack_holders(held, seg);
                    if (M_PAD == 16 && p.last_adds) {
                        if (et == 0) *arrived_last = inc_acq_rel_gpu(p.flags + tile, h.count() - 1) == h.count() - 1;
                        epi_bar_sync();
                        if (*arrived_last)
                            gemmtc::add_slice<gemmtc::Kind::kMx8>(p.scratch, kSlotFloats, tile, h, gemmtc::start_slot(tile), 0, 1, et, 32 * kEpiWarps,
                                                                  p.M, p.N, 1.f, 0, p.c);
                        epi_bar_sync();     // (before the word is written again)
                    } else if (et == 0) {
                        inc_acq_rel_gpu(p.flags + tile, h.count() - 1);
                    }
                } else if (!from_zero) {
                    if (et == 0) raise_flag(p.flags + blockIdx.x);
                } else {
                    if (!to_end) {
                        if (alive) alive = mbar_wait_warp_fast(partials, 0, abort_flag, p.status, kDevTimeoutPeerFlag);
                        alive = __all_sync(0xffffffffu, alive && !*abort_flag);
                        const int last = alive ? *last_peer_slot : cta_of(units, (last_tile + 1) * p.kb - 1, gridDim.x);
                        if (alive) {
                            // (the next partial's loads are in flight while one is added, where the registers hold two)
                            constexpr bool kTwo = kHalf <= 32;
                            constexpr int kPiece = kHalf < 32 ? kHalf : 32;
                            auto fetch = [&](int c, int i0, float4 (&v)[kPiece / 4]) {
                                const float4* peer = reinterpret_cast<const float4*>(p.scratch + static_cast<int64_t>(c) * kSlotFloats) + row_in_tile;
#pragma unroll
                                for (int i = 0; i < kPiece / 4; ++i) v[i] = __ldcg(peer + ((c0 + i0) / 4 + i) * kTileN);
                            };
#pragma unroll
                            for (int i0 = 0; i0 < kHalf; i0 += kPiece)
                                if (c0 + i0 < p.M) {
                                    float4 v[2][kPiece / 4];
                                    if (kTwo) fetch(blockIdx.x + 1, i0, v[0]);
                                    for (int c = blockIdx.x + 1; c <= last; c += 2) {
#pragma unroll
                                        for (int h = 0; h < 2; ++h) {
                                            if (c + h > last) break;
                                            if (!kTwo) fetch(c + h, i0, v[h]);
                                            else if (c + h < last) fetch(c + h + 1, i0, v[h ^ 1]);
#pragma unroll
                                            for (int i = 0; i < kPiece / 4; ++i) {
                                                acc[i0 + 4 * i] += v[h][i].x, acc[i0 + 4 * i + 1] += v[h][i].y;
                                                acc[i0 + 4 * i + 2] += v[h][i].z, acc[i0 + 4 * i + 3] += v[h][i].w;
                                            }
                                        }
                                    }
                                }
                        }
                        if (!alive) poison();
                        epi_bar_sync();
                        for (int c = blockIdx.x + 1 + et; c <= last; c += 32 * kEpiWarps) lower_flag(p.flags + c);   // free again
                    }
                    if (p.tp_peer_inbox) {
                        // Two-rank all-reduce fused into the epilogue: the finished fp32 tile goes
                        // straight into the peer GPU's inbox over NVLink (plain stores through the
                        // peer mapping, then a system-scope release of the tile's flag), and the
                        // peer's tile is awaited in this GPU's own inbox and added.  a + b == b + a
                        // in fp32, so both ranks hold bit-identical sums.  Inbox sets alternate
                        // with the call's sequence number: a rank can be one call ahead of its
                        // peer's reads, never two.
                        const int64_t set = static_cast<int64_t>(tp_epoch & 1) * p.n_tiles;
                        const int64_t tile_off = (set + tile) * (M_PAD * kTileN) + row_in_tile;
#pragma unroll
                        for (int i = 0; i < kHalf; ++i)
                            p.tp_peer_inbox[tile_off + (c0 + i) * kTileN] = acc[i];
                        __threadfence_system();
                        epi_bar_sync();
                        if (et == 0 && !*abort_flag) {
                            st_release_sys(p.tp_peer_flags + set + tile, tp_epoch);
                            const unsigned long long start = globaltimer_ns();
                            uint32_t spins = 0;
                            while (ld_acquire_sys(p.tp_my_flags + set + tile) != tp_epoch) {
                                if ((++spins & 63u) == 0u && (*abort_flag || globaltimer_ns() - start > p.tp_wait_ns)) {
                                    *abort_flag = 1;
                                    if (p.status) atomicCAS(p.status, 0, kDevTimeoutPeerFlag);
                                    break;
                                }
                                __nanosleep(100);
                            }
                        }
                        epi_bar_sync();
                        alive = __all_sync(0xffffffffu, alive && !*abort_flag);
                        if (alive) {
#pragma unroll
                            for (int i = 0; i < kHalf; ++i)
                                acc[i] += ld_volatile_f32(p.tp_my_inbox + tile_off + (c0 + i) * kTileN);
                        }
                    }
                    if (alive) {
                        if ((p.N & 3) == 0 && (reinterpret_cast<uintptr_t>(p.c) & 7u) == 0) {
                            // four lanes with neighbouring weight rows exchange, so that each stores 8 bytes of one activation row
                            __nv_bfloat16* c = p.c + tile * kTileN + (row_in_tile & ~3);
#pragma unroll
                            for (int i = 0; i < kHalf; i += 4)
                                if (c0 + i < p.M) {
                                    uint32_t rows01, rows23;
                                    gemmtc::transpose4(gemmtc::to_bf16x2(acc[i], acc[i + 1]), gemmtc::to_bf16x2(acc[i + 2], acc[i + 3]), lane,
                                                       rows01, rows23);
                                    const int m = c0 + i + static_cast<int>(lane & 3);
                                    if (m < p.M && nrow < p.N)
                                        *reinterpret_cast<uint2*>(c + static_cast<int64_t>(m) * p.N) = make_uint2(rows01, rows23);
                                }
                        } else if (nrow < p.N) {
#pragma unroll
                            for (int i = 0; i < kHalf; ++i)
                                if (c0 + i < p.M) p.c[static_cast<int64_t>(c0 + i) * p.N + nrow] = __float2bfloat16_rn(acc[i]);
                        }
                    }
                }
#pragma unroll
                for (int i = 0; i < kCols; ++i) acc[i] = 0.f;
                seg_kb0 = 0;
                ++seg;
            }
            if (++kb == p.kb) {
                kb = 0;
                ++tile;
            }
        }
        if (p.sliced && !(M_PAD == 16 && p.last_adds)) {
#pragma unroll 1
            for (int i = 0; i < seg; ++i) {
                if (et == 0 && alive) await_word(p.flags + tile0 + i, [](int v) { return v == 0; }, abort_flag, p.status);
                epi_bar_sync();
                alive = __all_sync(0xffffffffu, alive && !*abort_flag);
                if (alive)
                    gemmtc::add_slice<gemmtc::Kind::kMx8>(p.scratch, kSlotFloats, tile0 + i, unpack_holders(held, i), gemmtc::start_slot(tile0 + i),
                                                          static_cast<int>(blockIdx.x) - unpack_holders(held, i).first, unpack_holders(held, i).count(),
                                                          et, 32 * kEpiWarps, p.M, p.N, 1.f, 0, p.c);
            }
        }
    }

    __syncthreads();
    if (*abort_flag) abort_drain_sleep();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem_base, L::kTmemCols);
    }
    if (p.tp_peer_inbox && p.tp_epoch == 0 && threadIdx.x == 0) {
        // the last CTA to get here has seen every other CTA finish, hence read the old number
        __threadfence();
        if (atomicAdd(p.tp_ctrl + 1, 1) == static_cast<int>(gridDim.x) - 1) {
            p.tp_ctrl[1] = 0;
            st_release_gpu(p.tp_ctrl, tp_epoch);
        }
    }
}

template <int M_PAD>
static int launch(const CUtensorMap& w_map, const CUtensorMap& a_map, Params& p, const DeviceInfo& dev,
                  cudaStream_t stream) {
    using L = Smem<M_PAD>;
    int stages = kMaxStages;
    while (stages > 2 && L::total(stages, p.a_rows) > dev.smem_optin) --stages;
    const int smem = L::total(stages, p.a_rows);
    if (smem > dev.smem_optin)
        return fail(WUDA_ERR_UNSUPPORTED, "device offers %d bytes of shared memory per block; the kernel needs more",
                    dev.smem_optin);
    p.stages = stages;
    auto kernel = gemm_fp8_kernel<M_PAD>;
    WUDA_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, dev.smem_optin));
    const long long units = static_cast<long long>(p.n_tiles) * p.kb;
    const int sms = gemm_sms(dev);
    const int grid = gemmtc::grid_of(units, p.n_tiles, M_PAD, sms);
    p.sliced = !p.tp_peer_inbox && gemmtc::slice_wise(grid, p.n_tiles, M_PAD);     // (the two-rank form needs a finished tile in one CTA)
    // (Nine rows and more: not with 13 ranges per tile either, 1280 / 1408 x 7168 at 16 rows 10.5 / 9.2 us, in slices 8.8 / 9.0; nor with
    // short ranges, 4096 x 2048 0.5 us longer.)
    p.last_adds = gemmtc::last_arrival_adds(p.M, 32 * kEpiWarps, grid, p.n_tiles) && (p.M <= 8 || (grid < 13 * p.n_tiles && units >= 4ll * grid));
    WUDA_CUDA(launch_pdl(kernel, dim3(grid), dim3(kThreads), smem, stream, w_map, a_map, p));
    return WUDA_OK;
}

}  // namespace gemm8
}  // namespace wuda

// Scratch = flags or counters (the first kFlagBytes bytes), then kMaxGrid slots of one fp32 partial tile [M_PAD][128].
// The flags come first so that calls with different row counts, which size their slots differently, find them in the same
// place: one scratch buffer can then serve every GEMM of a stream without a slot of one call ever covering the flags of
// another.  All kinds share one layout.
using wuda::gemmtc::kFlagBytes;
using wuda::gemmtc::kMaxGrid;

extern "C" int64_t wuda_gemm_fp8_scratch_bytes(int m, int n) {
    if (m < 1 || n < 1 || m > 256) return -1;
    return wuda::gemmtc::scratch_bytes(m);
}

namespace {

// What every entry point of this file hands to the one set-up routine below.
struct GemmCall {
    const void* a = nullptr;
    const float* a_scales = nullptr;
    const void* w = nullptr;
    const float* w_scales = nullptr;
    void* c = nullptr;
    int m = 0, n = 0, k = 0;          // n = rows per group
    int groups = 1;
    float* slots = nullptr;           // [kMaxGrid][m_pad][128] fp32 partial tiles
    int32_t* flags = nullptr;         // [kMaxGrid], zero between calls
    int32_t* status = nullptr;
    cudaStream_t stream = nullptr;
    // two-rank form (inboxes == nullptr: none)
    void* my_inbox = nullptr;
    void* peer_inbox = nullptr;
    int epoch = 0;
    int peer_wait_ms = 0;
};

constexpr int64_t kTpFlagBytes = 4096;      // 2 sets x n_tiles tile flags, then the control words
constexpr int64_t kTpCtrlBytes = 64;        // last bytes of the flag block: {call sequence, CTAs done}

int64_t tp_bytes(int m, int n) {
    if (m < 1 || m > 256 || n < 1) return -1;
    int m_pad = 16;
    while (m_pad < m) m_pad *= 2;
    const int64_t n_tiles = (n + 127) / 128;
    if (2 * n_tiles * 4 > kTpFlagBytes - kTpCtrlBytes) return -1;
    return kTpFlagBytes + 2 * n_tiles * m_pad * 128 * 4;
}

// Parameter block, the two tensor maps and the launch for 1 <= m <= 128 (checked by the callers).
int gemm_fp8_setup_and_launch(const GemmCall& g) {
    using namespace wuda;
    using namespace wuda::gemm8;
    DeviceInfo dev;
    int st = current_device_info(&dev);
    if (st != WUDA_OK) return st;
    WUDA_REQUIRE(dev.num_sms <= kMaxGrid, "device has %d SMs; at most %d are supported", dev.num_sms, kMaxGrid);
    const int n_all = g.n * g.groups;
    int m_pad = 16;
    while (m_pad < g.m) m_pad *= 2;
    Params p;
    p.a_scales = g.a_scales;
    p.w_scales = g.w_scales;
    p.c = static_cast<__nv_bfloat16*>(g.c);
    p.status = g.status;
    p.M = g.m;
    p.N = n_all;
    p.K = g.k;
    p.kb = g.k / 128;
    p.n_tiles = (n_all + 127) / 128;
    p.group_tiles = g.groups > 1 ? g.n / 128 : 0;
    p.a_kb_total = g.groups * (g.k / 128);
    p.a_rows = gemmtc::rows_of(g.m);
    p.vec_scales = p.kb % 4 == 0 && aligned16(g.a_scales);
    p.sliced = 0;
    p.scratch = g.slots;
    p.flags = g.flags;
    p.stages = 0;
    if (g.peer_inbox) {
        p.tp_my_flags = static_cast<int32_t*>(g.my_inbox);
        p.tp_peer_flags = static_cast<int32_t*>(g.peer_inbox);
        p.tp_my_inbox = reinterpret_cast<float*>(static_cast<uint8_t*>(g.my_inbox) + kTpFlagBytes);
        p.tp_peer_inbox = reinterpret_cast<float*>(static_cast<uint8_t*>(g.peer_inbox) + kTpFlagBytes);
        p.tp_ctrl = reinterpret_cast<int32_t*>(static_cast<uint8_t*>(g.my_inbox) + kTpFlagBytes - kTpCtrlBytes);
        p.tp_epoch = g.epoch;
        p.tp_wait_ns = static_cast<unsigned long long>(g.peer_wait_ms) * 1000ull * 1000ull;
    }

    CUtensorMap w_map, a_map;
    {
        const uint64_t dims[2] = {static_cast<uint64_t>(g.k), static_cast<uint64_t>(n_all)};
        const uint64_t strides[1] = {static_cast<uint64_t>(g.k)};
        const uint32_t box[2] = {128u, 128u};
        st = encode_tensor_map(&w_map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, g.w, dims, strides, box,
                               CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B);
        if (st != WUDA_OK) return st;
    }
    {
        const uint64_t dims[2] = {static_cast<uint64_t>(g.k) * g.groups, static_cast<uint64_t>(g.m)};
        const uint64_t strides[1] = {static_cast<uint64_t>(g.k) * g.groups};
        const uint32_t box[2] = {128u, static_cast<uint32_t>(p.a_rows)};
        st = encode_tensor_map(&a_map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, g.a, dims, strides, box,
                               CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B);
        if (st != WUDA_OK) return st;
    }
    switch (m_pad) {
        case 16: return launch<16>(w_map, a_map, p, dev, g.stream);
        case 32: return launch<32>(w_map, a_map, p, dev, g.stream);
        case 64: return launch<64>(w_map, a_map, p, dev, g.stream);
        default: return launch<128>(w_map, a_map, p, dev, g.stream);
    }
}

// groups == 1: the plain GEMM.  groups > 1: `n` rows per group, group g multiplies the activations'
// columns [g * k, (g + 1) * k) by the weight rows [g * n, (g + 1) * n).
int gemm_fp8_entry(const void* a, const float* a_scales, const void* w, const float* w_scales, void* c_bf16,
                   int m, int n, int k, int groups, void* scratch, int64_t scratch_bytes,
                   int32_t* status_word, void* stream) {
    using namespace wuda;
    clear_error();
    WUDA_REQUIRE(groups >= 1, "groups must be >= 1 (got %d)", groups);
    WUDA_REQUIRE(groups == 1 || n % 128 == 0, "with groups the rows per group must be a multiple of 128 (got %d)", n);
    const int n_all = n * groups;
    WUDA_REQUIRE(m >= 0 && m <= 256, "m must be in [0, 256] (got %d)", m);
    WUDA_REQUIRE(n >= 1, "n must be >= 1 (got %d)", n);
    WUDA_REQUIRE(k >= 128 && k % 128 == 0, "k must be a positive multiple of 128 (got %d)", k);
    if (m == 0) return WUDA_OK;
    WUDA_REQUIRE(a && a_scales && w && w_scales && c_bf16 && scratch,
                 "a, a_scales, w, w_scales, c and scratch must not be NULL");
    WUDA_REQUIRE(aligned16(a) && aligned16(w), "a and w must be 16-byte aligned");
    WUDA_REQUIRE((reinterpret_cast<uintptr_t>(scratch) & 255u) == 0, "scratch must be 256-byte aligned");
    const int64_t need = wuda_gemm_fp8_scratch_bytes(m, n_all);
    WUDA_REQUIRE(scratch_bytes >= need, "scratch holds %lld bytes; %lld are needed (wuda_gemm_fp8_scratch_bytes)",
                 static_cast<long long>(scratch_bytes), static_cast<long long>(need));
    if (m > 128) {
        // Above 128 rows a warpgroup's 128 accumulator columns no longer fit the register file;
        // two passes of <= 128 rows (the weights stream twice) are faster than one that spills.
        int st2 = gemm_fp8_entry(a, a_scales, w, w_scales, c_bf16, 128, n, k, groups, scratch, scratch_bytes, status_word,
                                 stream);
        if (st2 != WUDA_OK) return st2;
        return gemm_fp8_entry(static_cast<const uint8_t*>(a) + static_cast<int64_t>(128) * k * groups,
                              a_scales + static_cast<int64_t>(128) * (k / 128) * groups, w, w_scales,
                              static_cast<__nv_bfloat16*>(c_bf16) + static_cast<int64_t>(128) * n_all, m - 128, n, k,
                              groups, scratch, scratch_bytes, status_word, stream);
    }
    GemmCall g;
    g.a = a, g.a_scales = a_scales, g.w = w, g.w_scales = w_scales, g.c = c_bf16;
    g.m = m, g.n = n, g.k = k, g.groups = groups;
    g.flags = gemm_flags(scratch);
    g.slots = reinterpret_cast<float*>(static_cast<uint8_t*>(scratch) + kFlagBytes);
    g.status = status_word;
    g.stream = static_cast<cudaStream_t>(stream);
    return gemm_fp8_setup_and_launch(g);
}

}  // namespace

extern "C" int wuda_gemm_fp8_blockscaled(const void* a, const float* a_scales, const void* w, const float* w_scales,
                                         void* c_bf16, int m, int n, int k, void* scratch, int64_t scratch_bytes,
                                         int32_t* status_word, void* stream) {
    return gemm_fp8_entry(a, a_scales, w, w_scales, c_bf16, m, n, k, 1, scratch, scratch_bytes, status_word, stream);
}

extern "C" int wuda_gemm_fp8_grouped(const void* a, const float* a_scales, const void* w, const float* w_scales,
                                     void* c_bf16, int m, int n_per_group, int k, int groups, void* scratch,
                                     int64_t scratch_bytes, int32_t* status_word, void* stream) {
    return gemm_fp8_entry(a, a_scales, w, w_scales, c_bf16, m, n_per_group, k, groups, scratch, scratch_bytes,
                          status_word, stream);
}

// ---------------------------------------------------------------------------------------------
// Allocation-free entry point.
//
// Some hosts must never see a device allocation from a library they call: a serving process
// that carved up all device memory at start-up and hands it out through its own pool (a stray
// cudaMalloc can fail there, or fragment what is left), and latency-critical loops in which
// cudaMalloc / cudaFree would synchronise the whole device and stall every other stream.  The
// regular entry point leaves the scratch to the caller; this one needs no scratch argument at
// all: the partial-tile slots and flags of the stream-K fix-up live in a fixed array inside the
// library's device image.  The price is a limit on m (kNoAllocMaxM) and kNoAllocScratchBytes of
// device memory held by every GPU that loads the library, until the process exits.
//
// The array is shared by every call on a device and keeps what the last call left in it.  The
// partial tiles are always written before they are read, so only the flags have to start at
// zero; the kernel resets each flag after use, and the entry point clears all of them again
// before every launch in case an earlier call ended abnormally.  Two calls that overlap on the
// GPU (different streams) would race on the slots: calls through this entry point must be
// ordered one after another on the device.  The flags sit at the start of the array, so calls with
// different m (different slot sizes) share it without moving them.
constexpr int kNoAllocMaxM = 64;
constexpr int64_t kNoAllocSlotBytes = static_cast<int64_t>(kMaxGrid) * kNoAllocMaxM * 128 * 4;
constexpr int64_t kNoAllocScratchBytes = kFlagBytes + kNoAllocSlotBytes;   // 6,292,480 bytes

static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocScratchBytes];

// The array's name is only a handle in host code; the device address comes from
// cudaGetSymbolAddress, asked once per device with that device current.
static int noalloc_scratch_address(int device, void** out) {
    static std::mutex mu;
    static void* cached[64] = {};
    if (device < 0 || device >= 64) return wuda::fail(WUDA_ERR_UNSUPPORTED, "device ordinal %d out of range", device);
    std::lock_guard<std::mutex> lock(mu);
    if (!cached[device]) {
        void* ptr = nullptr;
        cudaError_t err = cudaGetSymbolAddress(&ptr, g_noalloc_scratch);
        if (err != cudaSuccess || !ptr) {
            cudaGetLastError();
            return wuda::fail(WUDA_ERR_CUDA, "cudaGetSymbolAddress(no-alloc scratch) failed: %s", cudaGetErrorString(err));
        }
        cached[device] = ptr;
    }
    *out = cached[device];
    return WUDA_OK;
}

extern "C" int wuda_gemm_fp8_blockscaled_noalloc(const void* a, const float* a_scales, const void* w,
                                                 const float* w_scales, void* c_bf16, int m, int n, int k,
                                                 int32_t* status_word, void* stream) {
    using namespace wuda;
    clear_error();
    WUDA_REQUIRE(m >= 0, "m must be >= 0 (got %d)", m);
    if (m > kNoAllocMaxM)
        return fail(WUDA_ERR_UNSUPPORTED,
                    "the allocation-free entry point handles m <= %d (got %d): its built-in scratch is %lld bytes; "
                    "use wuda_gemm_fp8_blockscaled with caller-provided scratch for larger m",
                    kNoAllocMaxM, m, static_cast<long long>(kNoAllocScratchBytes));
    WUDA_REQUIRE(n >= 1, "n must be >= 1 (got %d)", n);
    WUDA_REQUIRE(k >= 128 && k % 128 == 0, "k must be a positive multiple of 128 (got %d)", k);
    if (m == 0) return WUDA_OK;
    WUDA_REQUIRE(a && a_scales && w && w_scales && c_bf16, "a, a_scales, w, w_scales and c must not be NULL");
    WUDA_REQUIRE(aligned16(a) && aligned16(w), "a and w must be 16-byte aligned");

    DeviceInfo dev;
    int st = current_device_info(&dev);
    if (st != WUDA_OK) return st;
    void* scratch = nullptr;
    st = noalloc_scratch_address(dev.device, &scratch);   // first call on a device: symbol lookup
    if (st != WUDA_OK) return st;

    GemmCall g;
    g.a = a, g.a_scales = a_scales, g.w = w, g.w_scales = w_scales, g.c = c_bf16;
    g.m = m, g.n = n, g.k = k;
    g.flags = static_cast<int32_t*>(scratch);
    g.slots = reinterpret_cast<float*>(static_cast<uint8_t*>(scratch) + kFlagBytes);
    g.status = status_word;
    g.stream = static_cast<cudaStream_t>(stream);
    // the flags must start at zero whatever the previous call left behind
    WUDA_CUDA(cudaMemsetAsync(g.flags, 0, kMaxGrid * sizeof(int32_t), g.stream));
    return gemm_fp8_setup_and_launch(g);
}

// ---------------------------------------------------------------------------------------------
// Two-rank tensor-parallel form: the K dimension is split across two GPUs (row-parallel
// linear, dsv4_megakernel/origin/model.py:166-180: y = x_r W_r^T summed over ranks in fp32,
// then cast; the reference's megakernel only fabricates this sum,
// dsv4_megakernel/megakernel/test/test_e2e_decode.py:186-194).  Each rank runs the same GEMM on
// its K slice; the all-reduce happens tile by tile inside the epilogue through peer memory.
//
// The exchange buffer of a rank ("inbox") is ordinary device memory made visible to the peer
// process with CUDA IPC.  Layout: a 4 KB flag block (2 sets x n_tiles int32 tile flags; its last
// 64 bytes hold the link's own call sequence number and a count of finished CTAs), then
// 2 sets x n_tiles x [M_PAD][128] fp32 tiles.
//
// Call sequence numbers.  A tile's flag carries the number of the call that delivered it, so both
// ranks must number their calls alike.  epoch >= 1: the host numbers them (1, 2, 3, .. on both
// ranks).  epoch == 0: the link numbers them itself - every CTA reads the last finished number from
// the control words and the last CTA to finish stores the new one - so the same launch can be
// replayed from a CUDA graph.  A link uses one of the two forms for its whole life.
extern "C" int64_t wuda_tp2_inbox_bytes(int m, int n) { return tp_bytes(m, n); }

extern "C" int wuda_tp2_alloc(int64_t bytes, void** local_base, unsigned char* ipc_handle_64) {
    using namespace wuda;
    clear_error();
    WUDA_REQUIRE(bytes > 0 && local_base && ipc_handle_64, "bytes must be > 0 and the outputs must not be NULL");
    void* ptr = nullptr;
    WUDA_CUDA(cudaMalloc(&ptr, static_cast<size_t>(bytes)));
    cudaError_t err = cudaMemset(ptr, 0, static_cast<size_t>(bytes));
    cudaIpcMemHandle_t h;
    if (err == cudaSuccess) err = cudaIpcGetMemHandle(&h, ptr);
    if (err != cudaSuccess) {
        cudaFree(ptr);
        cudaGetLastError();
        return fail(WUDA_ERR_CUDA, "preparing the exchange buffer failed: %s", cudaGetErrorString(err));
    }
    static_assert(sizeof(cudaIpcMemHandle_t) == 64, "IPC handle is 64 bytes");
    memcpy(ipc_handle_64, &h, 64);
    *local_base = ptr;
    return WUDA_OK;
}

extern "C" int wuda_tp2_open(const unsigned char* ipc_handle_64, void** peer_base) {
    using namespace wuda;
    clear_error();
    WUDA_REQUIRE(ipc_handle_64 && peer_base, "handle and output must not be NULL");
    cudaIpcMemHandle_t h;
    memcpy(&h, ipc_handle_64, 64);
    WUDA_CUDA(cudaIpcOpenMemHandle(peer_base, h, cudaIpcMemLazyEnablePeerAccess));
    return WUDA_OK;
}

extern "C" int wuda_tp2_close(void* peer_base) {
    using namespace wuda;
    clear_error();
    if (peer_base) WUDA_CUDA(cudaIpcCloseMemHandle(peer_base));
    return WUDA_OK;
}

extern "C" int wuda_tp2_free(void* local_base) {
    using namespace wuda;
    clear_error();
    if (local_base) WUDA_CUDA(cudaFree(local_base));
    return WUDA_OK;
}

extern "C" int wuda_gemm_fp8_blockscaled_tp2(const void* a, const float* a_scales, const void* w,
                                             const float* w_scales, void* c_bf16, int m, int n, int k_local,
                                             void* scratch, int64_t scratch_bytes, void* my_inbox, void* peer_inbox,
                                             int epoch, int peer_wait_ms, int32_t* status_word, void* stream) {
    using namespace wuda;
    clear_error();
    // one pass only: a second pass of rows would need a second exchange under its own sequence number
    WUDA_REQUIRE(m >= 1 && m <= 128, "m must be in [1, 128] (got %d); split larger batches into calls of <= 128 rows", m);
    WUDA_REQUIRE(n >= 1, "n must be >= 1 (got %d)", n);
    WUDA_REQUIRE(k_local >= 128 && k_local % 128 == 0, "k_local must be a positive multiple of 128 (got %d)", k_local);
    WUDA_REQUIRE(a && a_scales && w && w_scales && c_bf16 && scratch && my_inbox && peer_inbox,
                 "a, a_scales, w, w_scales, c, scratch and both inboxes must not be NULL");
    WUDA_REQUIRE(epoch >= 0, "epoch must be >= 1 and grow by one per call on both ranks, or 0 for the link's own "
                 "numbering (got %d)", epoch);
    WUDA_REQUIRE(peer_wait_ms >= 1 && peer_wait_ms <= 10000, "peer_wait_ms must be in [1, 10000] (got %d)", peer_wait_ms);
    WUDA_REQUIRE(aligned16(a) && aligned16(w), "a and w must be 16-byte aligned");
    WUDA_REQUIRE((reinterpret_cast<uintptr_t>(scratch) & 255u) == 0, "scratch must be 256-byte aligned");
    const int64_t need = wuda_gemm_fp8_scratch_bytes(m, n);
    WUDA_REQUIRE(scratch_bytes >= need, "scratch holds %lld bytes; %lld are needed (wuda_gemm_fp8_scratch_bytes)",
                 static_cast<long long>(scratch_bytes), static_cast<long long>(need));
    WUDA_REQUIRE(tp_bytes(m, n) > 0, "n is too large for the exchange buffer's flag block");
    GemmCall g;
    g.a = a, g.a_scales = a_scales, g.w = w, g.w_scales = w_scales, g.c = c_bf16;
    g.m = m, g.n = n, g.k = k_local;
    g.flags = gemm_flags(scratch);
    g.slots = reinterpret_cast<float*>(static_cast<uint8_t*>(scratch) + kFlagBytes);
    g.status = status_word;
    g.stream = static_cast<cudaStream_t>(stream);
    g.my_inbox = my_inbox, g.peer_inbox = peer_inbox, g.epoch = epoch, g.peer_wait_ms = peer_wait_ms;
    return gemm_fp8_setup_and_launch(g);
}
