// BF16 GEMM for decode-sized M on sm_100a:
//
//   C[M, N] (bf16 or fp32) = A[M, K] (bf16) x W[N, K]^T (bf16), fp32 accumulation
//
// It carries the projections the reference keeps in BF16 because their outputs feed fp32 state:
// the BF16 segment of the front mixed GEMM (dsv4_megakernel/megakernel/kernels/
// front_mixed_gemm_csa_swapab.cu:10-258, segment layout include/front_mixed_gemm.cuh:390-425) and
// the origin's plain `linear` (origin/model.py:108-120).
//
// The kernel is gemm_tc.cuh's: a unit is 128 weight rows x 64 K-elements, four tcgen05.mma kind::f16 (K = 16); nothing is
// rescaled between K blocks.
// Measured (as in gemm_tc.cuh, us; before = four fetching and two issuing warps, partials added by one CTA per tile):
// 7168 x 16384 at 64 rows 50.3 -> 46.7, 4096 x 7168 at 100 rows 27.7 -> 23.0, 256 x 7168 at 64 rows (the router) 16.4 -> 10.3.
#include "gemm_tc.cuh"

extern "C" int64_t wuda_gemm_bf16_scratch_bytes(int m, int n) {
    if (m < 1 || n < 1 || m > 128) return -1;
    return wuda::gemmtc::scratch_bytes(m);
}

extern "C" int wuda_gemm_bf16(const void* a_bf16, const void* w_bf16, void* c, int c_is_fp32, int m, int n, int k,
                              void* scratch, int64_t scratch_bytes, int32_t* status_word, void* stream) {
    using namespace wuda;
    using namespace wuda::gemmtc;
    clear_error();
    WUDA_REQUIRE(m >= 0 && m <= 128, "m must be in [0, 128] (got %d)", m);
    WUDA_REQUIRE(n >= 1, "n must be >= 1 (got %d)", n);
    WUDA_REQUIRE(k >= 64 && k % 64 == 0, "k must be a positive multiple of 64 (got %d)", k);
    if (m == 0) return WUDA_OK;
    WUDA_REQUIRE(a_bf16 && w_bf16 && c && scratch, "a, w, c and scratch must not be NULL");
    WUDA_REQUIRE(aligned16(a_bf16) && aligned16(w_bf16), "a and w must be 16-byte aligned");
    WUDA_REQUIRE((reinterpret_cast<uintptr_t>(scratch) & 255u) == 0, "scratch must be 256-byte aligned");
    const int64_t need = wuda_gemm_bf16_scratch_bytes(m, n);
    WUDA_REQUIRE(scratch_bytes >= need, "scratch holds %lld bytes; %lld are needed (wuda_gemm_bf16_scratch_bytes)",
                 static_cast<long long>(scratch_bytes), static_cast<long long>(need));

    DeviceInfo dev;
    int st = current_device_info(&dev);
    if (st != WUDA_OK) return st;
    WUDA_REQUIRE(dev.num_sms <= kMaxGrid, "device has %d SMs; at most %d are supported", dev.num_sms, kMaxGrid);

    Params p = {};
    p.c = c;
    p.c_is_fp32 = c_is_fp32 != 0;
    p.status = status_word;
    p.M = m;
    p.N = n;
    p.kb = k / 64;
    p.n_tiles = (n + 127) / 128;
    p.a_rows = rows_of(m);
    p.scratch = reinterpret_cast<float*>(static_cast<uint8_t*>(scratch) + kFlagBytes);
    p.flags = gemm_flags(scratch);

    CUtensorMap w_map, a_map;
    {
        const uint64_t dims[2] = {static_cast<uint64_t>(k), static_cast<uint64_t>(n)};
        const uint64_t strides[1] = {static_cast<uint64_t>(k) * 2};
        const uint32_t box[2] = {64u, 128u};
        st = encode_tensor_map(&w_map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, w_bf16, dims, strides, box,
                               CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B);
        if (st != WUDA_OK) return st;
    }
    {
        const uint64_t dims[2] = {static_cast<uint64_t>(k), static_cast<uint64_t>(m)};
        const uint64_t strides[1] = {static_cast<uint64_t>(k) * 2};
        const uint32_t box[2] = {64u, static_cast<uint32_t>(p.a_rows)};
        st = encode_tensor_map(&a_map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, a_bf16, dims, strides, box,
                               CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B);
        if (st != WUDA_OK) return st;
    }
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    return launch_for<Kind::kBf16>(m, w_map, a_map, w_map, a_map, p, dev, s);
}
