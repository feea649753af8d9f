// Host-side helpers shared by the entry points: status codes and the per-thread error
// message, argument checks, and TMA tensor-map encoding through the driver entry point
// (resolved at run time, so the library has no link-time dependency on libcuda and
// loads on a machine without a GPU).
#pragma once
#include <cstdarg>
#include <cstdint>
#include <cuda.h>
#include <cuda_runtime.h>

#include "../../include/wuda_b200.h"

namespace wuda {

int fail(int status, const char* fmt, ...);
void clear_error();

#define WUDA_REQUIRE(cond, ...)                                         \
    do {                                                                \
        if (!(cond)) return ::wuda::fail(WUDA_ERR_INVALID_ARGUMENT, __VA_ARGS__); \
    } while (0)

#define WUDA_CUDA(expr)                                                                   \
    do {                                                                                  \
        cudaError_t err__ = (expr);                                                       \
        if (err__ != cudaSuccess)                                                         \
            return ::wuda::fail(WUDA_ERR_CUDA, "%s failed: %s", #expr, cudaGetErrorString(err__)); \
    } while (0)

inline bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

// Device properties cached per device (SM count, opt-in shared memory).
struct DeviceInfo {
    int device = -1;
    int num_sms = 0;
    int smem_optin = 0;
    int cc_major = 0;
};
int current_device_info(DeviceInfo* out);
// SMs the GEMM launches of the calling thread may cover: all of the device's, or fewer after wuda_gemm_sm_limit
int gemm_sms(const DeviceInfo& dev);
// How many CTAs they take (their waits for one another count on all of them being there at the same time):
namespace gemmtc {
// Ranges that share a weight tile at most (adding partial sums costs as much as streaming M_PAD / 64 units of weights, so wide
// tiles are cut into fewer).
constexpr int max_split(int m_pad) { return m_pad <= 16 ? 16 : (m_pad == 32 ? 12 : (m_pad == 64 ? 8 : 6)); }
inline int grid_of(long long units, int n_tiles, int m_pad, int sms) {
    int grid = units < sms ? static_cast<int>(units) : sms;
    if (static_cast<long long>(n_tiles) * max_split(m_pad) < grid) grid = n_tiles * max_split(m_pad);
    return grid;
}
}  // namespace gemmtc
// Where those launches find their flags: at the front of the scratch, or where wuda_gemm_flags said
int32_t* gemm_flags(void* scratch);

// wuda_csa_decode_step whose w64, window rows and state rings a launch of the caller's produces: `produce` enqueues it on the
// stream it is given, beside the q norm and projection, which do not need them.
int csa_decode_step(const wuda_csa_weights* w, const wuda_csa_caches* c, const wuda_csa_step* s, const wuda_csa_workspace* ws, int m,
                    void* stream, int (*produce)(void* context, void* stream), void* context);

// wuda_mhc_pre; with act_quant its FP8 output is what wuda_rmsnorm_quant_fp8 makes of `normed` with power-of-two scales (the two
// differ in where the smallest scale lies, and for infinities and NaN).
int mhc_pre_as(bool act_quant, const void* hidden_states, const float* weight, const float* base, const float* scale,
               const void* attn_norm_gamma, float hc_eps, float rms_eps, float norm_eps, float* pre, float* post, float* comb,
               void* collapsed_bf16, void* normed_bf16, void* x_fp8, float* x_scales, void* workspace, int64_t workspace_bytes, int m,
               int hidden, void* stream);

// wuda_moe_gather_quant_nvfp4 beside a GEMM of reserved_sms CTAs (0: none) on another stream, which it leaves their SMs.
int moe_gather_beside(int reserved_sms, const void* x_bf16, const int32_t* pair_row, void* a_fp4, void* a_sf_packed, float global_scale,
                      int tokens, int topk, int k, void* stream);

// rank-`rank` tiled tensor map. dims/box are innermost-first; strides_bytes has rank-1
// entries (stride of dims 1..rank-1). Returns a wuda_status.
int encode_tensor_map(CUtensorMap* map, CUtensorMapDataType dtype, int rank, const void* base,
                      const uint64_t* dims, const uint64_t* strides_bytes, const uint32_t* box,
                      CUtensorMapSwizzle swizzle, CUtensorMapL2promotion promo);

// ---- programmatic dependent launch.  Every kernel of the library but two (moe_route.cu and the SwiGLU of
// norm_rope_quant.cu say why) is launched with the attribute
// that lets it start while the kernel before it in the stream is still running; it then runs its
// prologue (barrier set-up, TMEM allocation, descriptor prefetch) and stops at pdl_wait() until
// the earlier kernel has completed and its writes are visible, before its first access to global memory.
// pdl_launch_dependents() is called at the start, so the next kernel gets the same head start.
template <typename... KArgs, typename... Args>
inline cudaError_t launch_pdl(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream,
                              Args&&... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...);
}

#ifdef __CUDACC__
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
// Asks L2 for the line at p: a hint that reads nothing into the SM, so it may go out before pdl_wait().
__device__ __forceinline__ void prefetch_l2(const void* p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }
__device__ __forceinline__ void pdl_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
#endif

}  // namespace wuda
