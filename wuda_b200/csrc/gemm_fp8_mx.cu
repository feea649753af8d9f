// Block-scaled FP8 GEMM whose scales are powers of two, with the scales applied INSIDE the tensor core:
//
//   C[M, N] (bf16) = sum over 128-wide K blocks of (a[m, kb] * a_scale[m, kb]) . (w[n, kb] * w_scale[n/128, kb])
//
// Same operands and layouts as wuda_gemm_fp8_blockscaled (e4m3, fp32 scales: 1x128 for the activations,
// 128x128 for the weights; origin/kernel.py:203-273), restricted to scales that are exact powers of two -
// which is what the reference's checkpoints and quantisers produce (UE8M0 scales:
// dsv4_megakernel/megakernel/kernels/wq_b_fp8_gemm.cu:139-183 writes them, include/cluster_mma_fp8.cuh:144-301
// consumes them through block-scaled MMAs).  Then tcgen05.mma kind::mxf8f6f4.block_scale (one UE8M0 scale per
// 32 K-elements and operand row, read from tensor memory) multiplies by 2^(e_a - 127) * 2^(e_w - 127) on the way
// into the accumulator, a weight tile accumulates over its whole K range in TMEM, and the CUDA-core promotion of
// every K block - what bounds the general kernel from 64 rows up - is gone.  The epilogue runs once per tile
// segment.
//
// The kernel is gemm_tc.cuh's.  A unit (128 x 128 bytes) is four MMAs of K = 32; the scale of a K block is one of the four
// bytes of a 32-bit scale column, four K blocks to a column (4-bit weights: the four bytes of a weight row's column
// are the four 32-wide scales of one K block, so every unit has its own weight image).
// A scale that is not a power of two is truncated to one and reported (WUDA_DEV_SCALE_NOT_POW2); a zero scale
// reads as 2^-127.
// Measured (as in gemm_tc.cuh, us; before = scale images built unit by unit by the fetching warps, two accumulators,
// passes of 128 rows, partials added by one CTA per tile):
//   24576 x 7168 at 64 rows 44.4 -> 38.6; 7168 x 16384 at 256 rows 78.6 -> 51.0; 73728 x 1536 at 64 rows (the q
//   projection; before with the activations resident in shared memory) 29.6 -> 28.7; 4096 x 7168 at 64 rows 20.5 -> 18.4;
//   4-bit weights: 24576 x 7168 at 64 rows 37.6 -> 30.7, 7168 x 16384 at 200 rows 75.9 -> 44.4
#include "gemm_tc.cuh"

namespace wuda {
namespace gemm8mx {

using namespace gemmtc;

// 4-bit weights (W4): two to a byte ([N, K/2], low nibble first), with one exponent byte per row and 32 K-elements
// (origin/kernel.py:441-536, fp4_gemm).  The tensor core reads 4-bit operands of this kind from shared memory in the
// padded form - 16 values in 8 bytes, then 8 bytes of nothing - which is what a tensor map of type 16U4_ALIGN16B makes
// of the packed rows: a unit's weight tile still fills 16 KB of the stage but is 8 KB of global memory, and the
// barrier counts those 8 KB.

// One pass over the weights.  groups = 1 is the plain GEMM.  w_sf != NULL: 4-bit weights (plain form only).
static int run(const void* a, const float* a_scales, const void* w, const float* w_scales, const uint8_t* w_sf, void* c_bf16, int m,
               int n_per_group, int k, int groups, void* scratch, int64_t scratch_bytes, int32_t* status_word, void* stream) {
    const int n = n_per_group * groups;
    const bool w4 = w_sf != nullptr;
    WUDA_REQUIRE(aligned16(a) && aligned16(w), "a and w must be 16-byte aligned");
    WUDA_REQUIRE(!w4 || ((reinterpret_cast<uintptr_t>(w) & 31u) == 0 && (reinterpret_cast<uintptr_t>(w_sf) & 3u) == 0),
                 "packed 4-bit weights must be 32-byte aligned and their scale bytes 4-byte aligned");
    WUDA_REQUIRE((reinterpret_cast<uintptr_t>(scratch) & 255u) == 0, "scratch must be 256-byte aligned");
    const int64_t need = wuda_gemm_fp8_scratch_bytes(m, n);
    WUDA_REQUIRE(scratch_bytes >= need, "scratch holds %lld bytes; %lld are needed (wuda_gemm_fp8_scratch_bytes)",
                 static_cast<long long>(scratch_bytes), static_cast<long long>(need));
    DeviceInfo dev;
    int st = current_device_info(&dev);
    if (st != WUDA_OK) return st;
    WUDA_REQUIRE(dev.num_sms <= kMaxGrid, "device has %d SMs; at most %d are supported", dev.num_sms, kMaxGrid);
    Params p = {};
    p.c = c_bf16;
    p.a_scales = a_scales;
    p.w_scales = w_scales;
    p.w_sf = w_sf;
    p.sf_stride = k / 32;
    p.status = status_word;
    p.M = m;
    p.N = n;
    p.kb = k / 128;
    p.n_tiles = (n + 127) / 128;
    p.a_rows = rows_of(m);
    p.tiles_per_group = groups > 1 ? n_per_group / 128 : p.n_tiles;
    p.scale_cols = groups * p.kb;
    p.vec_scales = p.kb % 4 == 0 && aligned16(a_scales) && (!w4 || aligned16(w_sf));
    p.scratch = reinterpret_cast<float*>(static_cast<uint8_t*>(scratch) + kFlagBytes);
    p.flags = gemm_flags(scratch);

    CUtensorMap w_map, a_map;
    {
        // 4-bit weights: dimensions and box in elements, the row stride in bytes; shared memory gets the padded form
        const uint64_t dims[2] = {static_cast<uint64_t>(k), static_cast<uint64_t>(n)};
        const uint64_t strides[1] = {static_cast<uint64_t>(w4 ? k / 2 : k)};
        const uint32_t box[2] = {128u, 128u};
        st = encode_tensor_map(&w_map, w4 ? CU_TENSOR_MAP_DATA_TYPE_16U4_ALIGN16B : CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, w, dims, strides,
                               box, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B);
        if (st != WUDA_OK) return st;
    }
    {
        const uint64_t row = static_cast<uint64_t>(k) * groups;
        const uint64_t dims[2] = {row, static_cast<uint64_t>(m)};
        const uint64_t strides[1] = {row};
        const uint32_t box[2] = {128u, static_cast<uint32_t>(p.a_rows)};
        st = encode_tensor_map(&a_map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, a, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B,
                               CU_TENSOR_MAP_L2_PROMOTION_L2_128B);
        if (st != WUDA_OK) return st;
    }
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    return w4 ? launch_for<Kind::kMx8W4>(m, w_map, a_map, w_map, a_map, p, dev, s)
              : launch_for<Kind::kMx8>(m, w_map, a_map, w_map, a_map, p, dev, s);
}

// Rows of a pass: all of them if the scratch has room for their partial sums, else passes of 128.
static int rows_per_pass(int m, int n, int64_t scratch_bytes) {
    return m <= 128 || scratch_bytes >= wuda_gemm_fp8_scratch_bytes(m, n) ? m : 128;
}

}  // namespace gemm8mx
}  // namespace wuda

extern "C" int wuda_gemm_fp8_grouped_pow2(const void* a, const float* a_scales, const void* w, const float* w_scales, void* c_bf16,
                                          int m, int n_per_group, int k, int groups, void* scratch, int64_t scratch_bytes,
                                          int32_t* status_word, void* stream) {
    using namespace wuda;
    clear_error();
    WUDA_REQUIRE(m >= 0 && m <= 256, "m must be in [0, 256] (got %d)", m);
    WUDA_REQUIRE(groups >= 1 && n_per_group >= 1, "groups and n_per_group must be >= 1");
    WUDA_REQUIRE(groups == 1 || n_per_group % 128 == 0, "n_per_group must be a multiple of 128 when there are several groups (got %d)",
                 n_per_group);
    WUDA_REQUIRE(k >= 128 && k % 128 == 0, "k must be a positive multiple of 128 (got %d)", k);
    if (m == 0) return WUDA_OK;
    WUDA_REQUIRE(a && a_scales && w && w_scales && c_bf16 && scratch, "a, a_scales, w, w_scales, c and scratch must not be NULL");
    const int64_t n = static_cast<int64_t>(n_per_group) * groups;
    const int64_t row = static_cast<int64_t>(k) * groups;
    const int pass = gemm8mx::rows_per_pass(m, static_cast<int>(n), scratch_bytes);
    for (int m0 = 0; m0 < m; m0 += pass) {
        const int rows = m - m0 < pass ? m - m0 : pass;
        const int st = gemm8mx::run(static_cast<const uint8_t*>(a) + m0 * row, a_scales + m0 * (row / 128), w, w_scales, nullptr,
                                    static_cast<__nv_bfloat16*>(c_bf16) + m0 * n, rows, n_per_group, k, groups, scratch, scratch_bytes,
                                    status_word, stream);
        if (st != WUDA_OK) return st;
    }
    return WUDA_OK;
}

extern "C" int wuda_gemm_fp8_blockscaled_pow2(const void* a, const float* a_scales, const void* w, const float* w_scales, void* c_bf16,
                                              int m, int n, int k, void* scratch, int64_t scratch_bytes, int32_t* status_word,
                                              void* stream) {
    return wuda_gemm_fp8_grouped_pow2(a, a_scales, w, w_scales, c_bf16, m, n, k, 1, scratch, scratch_bytes, status_word, stream);
}

// FP8 activations x 4-bit weights (origin/kernel.py:441-536, fp4_gemm): a e4m3 [m, k] with one power-of-two fp32 scale per
// row and 128 K-elements; w e2m1 [n, k/2] bytes, the element of the lower K index in the low nibble (torch.float4_e2m1fn_x2),
// with one exponent byte (float8_e8m0fnu) per row and 32 K-elements, [n, k/32]; c bf16 [m, n].
extern "C" int wuda_gemm_fp8_fp4_pow2(const void* a, const float* a_scales, const void* w_packed, const void* w_sf, void* c_bf16,
                                      int m, int n, int k, void* scratch, int64_t scratch_bytes, int32_t* status_word,
                                      void* stream) {
    using namespace wuda;
    clear_error();
    WUDA_REQUIRE(m >= 0 && m <= 256, "m must be in [0, 256] (got %d)", m);
    WUDA_REQUIRE(n >= 1, "n must be >= 1 (got %d)", n);
    WUDA_REQUIRE(k >= 128 && k % 128 == 0, "k must be a positive multiple of 128 (got %d)", k);
    if (m == 0) return WUDA_OK;
    WUDA_REQUIRE(a && a_scales && w_packed && w_sf && c_bf16 && scratch, "a, a_scales, w_packed, w_sf, c and scratch must not be NULL");
    const int pass = gemm8mx::rows_per_pass(m, n, scratch_bytes);
    for (int m0 = 0; m0 < m; m0 += pass) {
        const int rows = m - m0 < pass ? m - m0 : pass;
        const int st = gemm8mx::run(static_cast<const uint8_t*>(a) + static_cast<int64_t>(m0) * k, a_scales + static_cast<int64_t>(m0) * (k / 128),
                                    w_packed, nullptr, static_cast<const uint8_t*>(w_sf),
                                    static_cast<__nv_bfloat16*>(c_bf16) + static_cast<int64_t>(m0) * n, rows, n, k, 1, scratch,
                                    scratch_bytes, status_word, stream);
        if (st != WUDA_OK) return st;
    }
    return WUDA_OK;
}
