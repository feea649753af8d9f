// NVFP4 block-scaled GEMM for decode-sized M on sm_100a:
//
//   C[M, N] (bf16) = gs_a * gs_w * sum_k (e2m1 a[m,k] * ue4m3 a_sf[m, k/16]) * (e2m1 w[n,k] * ue4m3 w_sf[n, k/16])
//
// Operands are packed 4-bit e2m1 (two per byte, low nibble first; value table and rounding as in
// dsv4_megakernel/origin/convert.py:11-14 and megakernel/test/test_mqa_logits_fp4.py:69-115), with one
// ue4m3 scale per 16 elements along K and one fp32 scale per tensor.  The reference has no NVFP4
// GEMM (its FP4 path, origin/kernel.py:441-536, is W4A8 with 1x32 e8m0 scales); this is the form the
// benchmark configuration names.
//
// The kernel is gemm_tc.cuh's: tcgen05.mma kind::mxf4nvf4.block_scale.scale_vec::4X (K = 64 per instruction, four to a
// unit of 256 K-elements) reads the block scales from TMEM, where tcgen05.cp puts them from the unit's own copy; the
// epilogue multiplies by gs_a * gs_w.
//
// Scale layout in global memory ("packed"): per 128 rows x 256 K one 2 KB block
// [4 K/64 steps][32 = row % 32][4 = row / 32][4 scales of the step], blocks ordered [row tile][K/256].
// It is the image tcgen05.cp.32x128b.warpx4 expects, so a unit's scales are one contiguous copy.
// Measured (as in gemm_tc.cuh, us; before = four fetching and two issuing warps, passes of 128 rows): 24576 x 7168 at
// 8 rows 24.1 -> 21.3, at 128 rows 34.9 -> 28.7, at 200 rows 66.8 -> 36.9; 7168 x 16384 at 64 rows 23.6 -> 19.3; routed
// experts of 64 tokens (grouped) 884 -> 877 per block
//
// Grouped form (routed experts): row group g (16 activation rows) belongs to expert group_expert[g]; flat tile
// T = g * n_tiles + tile of the expert's N rows.  The number of groups is read on the device, so nothing is
// synchronised with the host between routing and the GEMM.
#include "gemm_tc.cuh"

extern "C" int64_t wuda_gemm_nvfp4_scratch_bytes(int m, int n) {
    if (m < 1 || n < 1 || m > 256) return -1;
    return wuda::gemmtc::scratch_bytes(m);
}

extern "C" int wuda_gemm_nvfp4(const void* a, const void* a_sf_packed, float a_global_scale, const void* w,
                               const void* w_sf_packed, float w_global_scale, void* c_bf16, int m, int n, int k,
                               void* scratch, int64_t scratch_bytes, int32_t* status_word, void* stream) {
    using namespace wuda;
    using namespace wuda::gemmtc;
    clear_error();
    WUDA_REQUIRE(m >= 0 && m <= 256, "m must be in [0, 256] (got %d)", m);
    WUDA_REQUIRE(n >= 1, "n must be >= 1 (got %d)", n);
    WUDA_REQUIRE(k >= 256 && k % 256 == 0, "k must be a positive multiple of 256 (got %d)", k);
    if (m == 0) return WUDA_OK;
    WUDA_REQUIRE(a && a_sf_packed && w && w_sf_packed && c_bf16 && scratch,
                 "a, a_sf_packed, w, w_sf_packed, c and scratch must not be NULL");
    if (m > 128 && scratch_bytes < wuda_gemm_nvfp4_scratch_bytes(m, n)) {
        // No room for the partial sums of all rows: two passes over the weights, one per 128-row tile of the
        // activations and of their packed scales ([row tile][k / 256][2048 bytes]).
        int st2 = wuda_gemm_nvfp4(a, a_sf_packed, a_global_scale, w, w_sf_packed, w_global_scale, c_bf16, 128, n, k, scratch,
                                  scratch_bytes, status_word, stream);
        if (st2 != WUDA_OK) return st2;
        return wuda_gemm_nvfp4(static_cast<const uint8_t*>(a) + static_cast<int64_t>(128) * (k / 2),
                               static_cast<const uint8_t*>(a_sf_packed) + static_cast<int64_t>(k / 256) * 2048, a_global_scale,
                               w, w_sf_packed, w_global_scale,
                               static_cast<__nv_bfloat16*>(c_bf16) + static_cast<int64_t>(128) * n, m - 128, n, k, scratch,
                               scratch_bytes, status_word, stream);
    }
    WUDA_REQUIRE(aligned16(a) && aligned16(w) && aligned16(a_sf_packed) && aligned16(w_sf_packed),
                 "operands and packed scales must be 16-byte aligned");
    WUDA_REQUIRE((reinterpret_cast<uintptr_t>(scratch) & 255u) == 0, "scratch must be 256-byte aligned");
    const int64_t need = wuda_gemm_nvfp4_scratch_bytes(m, n);
    WUDA_REQUIRE(scratch_bytes >= need, "scratch holds %lld bytes; %lld are needed (wuda_gemm_nvfp4_scratch_bytes)",
                 static_cast<long long>(scratch_bytes), static_cast<long long>(need));

    DeviceInfo dev;
    int st = current_device_info(&dev);
    if (st != WUDA_OK) return st;
    WUDA_REQUIRE(dev.num_sms <= kMaxGrid, "device has %d SMs; at most %d are supported", dev.num_sms, kMaxGrid);

    Params p = {};
    p.c = c_bf16;
    p.status = status_word;
    p.out_scale = a_global_scale * w_global_scale;
    p.M = m;
    p.N = n;
    p.kb = k / 256;
    p.n_tiles = (n + 127) / 128;
    p.a_rows = rows_of(m);
    p.scratch = reinterpret_cast<float*>(static_cast<uint8_t*>(scratch) + kFlagBytes);
    p.flags = gemm_flags(scratch);

    CUtensorMap w_map, a_map, wsf_map, asf_map;
    const uint64_t row_bytes = static_cast<uint64_t>(k) / 2;
    {
        const uint64_t dims[2] = {row_bytes, static_cast<uint64_t>(n)};
        const uint64_t strides[1] = {row_bytes};
        const uint32_t box[2] = {128u, 128u};
        st = encode_tensor_map(&w_map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, w, dims, strides, box,
                               CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B);
        if (st != WUDA_OK) return st;
    }
    {
        const uint64_t dims[2] = {row_bytes, static_cast<uint64_t>(m)};
        const uint64_t strides[1] = {row_bytes};
        const uint32_t box[2] = {128u, static_cast<uint32_t>(p.a_rows)};
        st = encode_tensor_map(&a_map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, a, dims, strides, box,
                               CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B);
        if (st != WUDA_OK) return st;
    }
    {   // packed scales as rows of 512 bytes (one K/64 step of 128 rows); a unit's block is 4 rows
        const uint64_t dims[2] = {128ull, static_cast<uint64_t>(p.n_tiles) * p.kb * 4};
        const uint64_t strides[1] = {512ull};
        const uint32_t box[2] = {128u, 4u};
        st = encode_tensor_map(&wsf_map, CU_TENSOR_MAP_DATA_TYPE_UINT32, 2, w_sf_packed, dims, strides, box,
                               CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_NONE);
        if (st != WUDA_OK) return st;
    }
    {
        const uint64_t dims[2] = {128ull, static_cast<uint64_t>((m + 127) / 128) * p.kb * 4};
        const uint64_t strides[1] = {512ull};
        const uint32_t box[2] = {128u, 4u};
        st = encode_tensor_map(&asf_map, CU_TENSOR_MAP_DATA_TYPE_UINT32, 2, a_sf_packed, dims, strides, box,
                               CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_NONE);
        if (st != WUDA_OK) return st;
    }
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    return launch_for<Kind::kNv4>(m, w_map, a_map, wsf_map, asf_map, p, dev, s);
}

// Grouped form for the routed experts: activations [max_groups * 16, k] quantised per group (see
// moe.cu), expert weights stacked [experts * n, k / 2] with their packed scales stacked per expert.
extern "C" int wuda_gemm_nvfp4_grouped(const void* a, const void* a_sf_packed, float a_global_scale, const void* w,
                                       const void* w_sf_packed, const float* w_global_scales,
                                       const int32_t* group_expert, const int32_t* num_groups, const int32_t* row_token,
                                       void* c_bf16, int max_groups, int experts, int n, int k, void* scratch, int64_t scratch_bytes,
                                       int32_t* status_word, void* stream) {
    using namespace wuda;
    using namespace wuda::gemmtc;
    clear_error();
    WUDA_REQUIRE(max_groups >= 1 && experts >= 1, "max_groups and experts must be >= 1");
    WUDA_REQUIRE(n >= 128 && n % 128 == 0, "n (rows per expert) must be a positive multiple of 128 (got %d)", n);
    WUDA_REQUIRE(k >= 256 && k % 256 == 0, "k must be a positive multiple of 256 (got %d)", k);
    WUDA_REQUIRE(a && a_sf_packed && w && w_sf_packed && w_global_scales && group_expert && num_groups && c_bf16 && scratch,
                 "no array may be NULL");
    WUDA_REQUIRE(aligned16(a) && aligned16(w) && aligned16(a_sf_packed) && aligned16(w_sf_packed),
                 "operands and packed scales must be 16-byte aligned");
    WUDA_REQUIRE((reinterpret_cast<uintptr_t>(scratch) & 255u) == 0, "scratch must be 256-byte aligned");
    const int64_t need = wuda_gemm_nvfp4_scratch_bytes(16, n);
    WUDA_REQUIRE(scratch_bytes >= need, "scratch holds %lld bytes; %lld are needed (wuda_gemm_nvfp4_scratch_bytes(16, n))",
                 static_cast<long long>(scratch_bytes), static_cast<long long>(need));
    DeviceInfo dev;
    int st = current_device_info(&dev);
    if (st != WUDA_OK) return st;
    WUDA_REQUIRE(dev.num_sms <= kMaxGrid, "device has %d SMs; at most %d are supported", dev.num_sms, kMaxGrid);

    constexpr int m_pad = 16;
    Params p = {};
    p.c = c_bf16;
    p.status = status_word;
    p.out_scale = a_global_scale;
    p.M = m_pad;
    p.N = n;
    p.kb = k / 256;
    p.n_tiles = n / 128;
    p.a_rows = m_pad;
    p.scratch = reinterpret_cast<float*>(static_cast<uint8_t*>(scratch) + kFlagBytes);
    p.flags = gemm_flags(scratch);
    p.group_expert = group_expert;
    p.num_groups = num_groups;
    p.row_token = row_token;
    p.expert_scale = w_global_scales;

    CUtensorMap w_map, a_map, wsf_map, asf_map;
    const uint64_t row_bytes = static_cast<uint64_t>(k) / 2;
    {
        const uint64_t dims[2] = {row_bytes, static_cast<uint64_t>(experts) * n};
        const uint64_t strides[1] = {row_bytes};
        const uint32_t box[2] = {128u, 128u};
        st = encode_tensor_map(&w_map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, w, dims, strides, box,
                               CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B);
        if (st != WUDA_OK) return st;
    }
    {
        const uint64_t dims[2] = {row_bytes, static_cast<uint64_t>(max_groups) * m_pad};
        const uint64_t strides[1] = {row_bytes};
        const uint32_t box[2] = {128u, static_cast<uint32_t>(p.a_rows)};
        st = encode_tensor_map(&a_map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, a, dims, strides, box,
                               CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B);
        if (st != WUDA_OK) return st;
    }
    {
        const uint64_t dims[2] = {128ull, static_cast<uint64_t>(experts) * p.n_tiles * p.kb * 4};
        const uint64_t strides[1] = {512ull};
        const uint32_t box[2] = {128u, 4u};
        st = encode_tensor_map(&wsf_map, CU_TENSOR_MAP_DATA_TYPE_UINT32, 2, w_sf_packed, dims, strides, box,
                               CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_NONE);
        if (st != WUDA_OK) return st;
    }
    {
        const uint64_t dims[2] = {128ull, static_cast<uint64_t>(max_groups) * p.kb * 4};
        const uint64_t strides[1] = {512ull};
        const uint32_t box[2] = {128u, 4u};
        st = encode_tensor_map(&asf_map, CU_TENSOR_MAP_DATA_TYPE_UINT32, 2, a_sf_packed, dims, strides, box,
                               CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_NONE);
        if (st != WUDA_OK) return st;
    }
    return launch<Kind::kNv4, m_pad>(w_map, a_map, wsf_map, asf_map, p, dev, static_cast<cudaStream_t>(stream));
}
