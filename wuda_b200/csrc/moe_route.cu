// MoE router: from a token's fp32 expert logits to its top-k experts and routing weights.
//   score  = softmax(logits) | sigmoid(logits) | sqrt(softplus(logits))
//   select = the k largest of score + bias (the bias steers the choice only), ties to the lower expert
//   weight = score[selected], divided by their sum unless softmax, times route_scale
// After the origin's Gate.forward (dsv4_megakernel/origin/model.py:563-584); the logits themselves are
// the bf16 x fp32 -> fp32 projection `linear(x.float(), weight.float())`, which wuda_gemm_bf16 produces
// with fp32 output.  One warp per token: a lane holds experts lane, lane + 32, ..; k rounds of a
// warp arg-max pick the experts in descending order.  A chain of latencies, so a round is two warp reductions in
// hardware (the largest key, then the lowest expert that has it) instead of ten shuffles and their compares, and a lane
// holds no more than the 8 scores of 256 experts where that is all there are: 64 tokens, 256
// experts, top-8: 8.5 -> 5.6 us in a profiler's list (cold, launch included).
#include "host.h"

namespace wuda {
namespace route {

constexpr int kMaxPerLane = 16;   // up to 512 experts (8 of them where 256 are enough)
constexpr int kWarpsPerCta = 4;

struct Params {
    const float* logits;   // [tokens, experts]
    const float* bias;     // [experts] or nullptr
    float* weights;        // [tokens, k]
    int32_t* indices;      // [tokens, k]
    int tokens, experts, k, score_func;
    float route_scale;
};

// Orders as the floats do (no NaN, no -0): larger value, larger key; never 0.
__device__ __forceinline__ uint32_t ordered_key(float v) {
    const uint32_t b = __float_as_uint(v);
    return b ^ (b >> 31 ? 0xffffffffu : 0x80000000u);
}

template <int kPerLane>
__global__ void __launch_bounds__(32 * kWarpsPerCta) moe_route_kernel(Params p) {
    pdl_launch_dependents();
    pdl_wait();   // nothing of global memory is touched before the kernel ahead has finished
    const int lane = threadIdx.x & 31;
    const int t = blockIdx.x * kWarpsPerCta + (threadIdx.x >> 5);
    if (t >= p.tokens) return;                         // whole warps
    const float* row = p.logits + static_cast<int64_t>(t) * p.experts;
    float score[kPerLane], pick[kPerLane];
    float mx = -INFINITY;
#pragma unroll
    for (int j = 0; j < kPerLane; ++j) {
        const int e = lane + 32 * j;
        score[j] = e < p.experts ? row[e] : -INFINITY;
        mx = fmaxf(mx, score[j]);
    }
    if (p.score_func == 0) {                           // softmax over all experts
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        float sum = 0.f;
#pragma unroll
        for (int j = 0; j < kPerLane; ++j) {
            score[j] = lane + 32 * j < p.experts ? expf(score[j] - mx) : 0.f;
            sum += score[j];
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
#pragma unroll
        for (int j = 0; j < kPerLane; ++j) score[j] = __fdiv_rn(score[j], sum);
    } else {
#pragma unroll
        for (int j = 0; j < kPerLane; ++j) {
            const float x = score[j];
            if (p.score_func == 1) {
                score[j] = __fdiv_rn(1.0f, 1.0f + expf(-x));
            } else {                                    // sqrt(softplus(x)), softplus as log1p(exp(x)) with the usual cut
                const float sp = x > 20.f ? x : log1pf(expf(x));
                score[j] = __fsqrt_rn(sp);
            }
        }
    }
#pragma unroll
    for (int j = 0; j < kPerLane; ++j) {
        const int e = lane + 32 * j;
        pick[j] = e < p.experts ? (p.bias ? score[j] + __ldg(p.bias + e) : score[j]) : -INFINITY;
    }
    float wsum = 0.f, mine = 0.f;                      // lane r keeps the r-th selected weight
    int mine_e = 0;
    for (int r = 0; r < p.k; ++r) {
        float best = -INFINITY;
        int best_e = 0x7fffffff, best_j = 0;
#pragma unroll
        for (int j = 0; j < kPerLane; ++j)
            if (pick[j] > best) {                       // strict: the lower expert wins inside a lane
                best = pick[j];
                best_e = lane + 32 * j;
                best_j = j;
            }
        // (a lane without a candidate has key 0; adding zero makes one key of the two zeros)
        const uint32_t key = best > -INFINITY ? ordered_key(best + 0.0f) : 0u;
        const uint32_t top = __reduce_max_sync(0xffffffffu, key);
        const int e = static_cast<int>(__reduce_min_sync(0xffffffffu, key == top ? static_cast<uint32_t>(best_e) : 0x7fffffffu));
        const bool owner = e == best_e && best > -INFINITY;
        float s = 0.f;
        if (owner) {
#pragma unroll
            for (int j = 0; j < kPerLane; ++j)
                if (j == best_j) {
                    s = score[j];
                    pick[j] = -INFINITY;
                }
        }
        s = __shfl_sync(0xffffffffu, s, e & 31);
        wsum += s;
        if (lane == r) {
            mine = s;
            mine_e = e;
        }
    }
    if (lane < p.k) {
        float w = p.score_func == 0 ? mine : __fdiv_rn(mine, wsum);
        p.weights[static_cast<int64_t>(t) * p.k + lane] = w * p.route_scale;
        p.indices[static_cast<int64_t>(t) * p.k + lane] = mine_e;
    }
}

}  // namespace route
}  // namespace wuda

extern "C" int wuda_moe_route(const float* logits, const float* bias, float* weights, int32_t* indices, int tokens,
                              int experts, int k, int score_func, float route_scale, void* stream) {
    using namespace wuda;
    using namespace wuda::route;
    clear_error();
    WUDA_REQUIRE(tokens >= 0, "tokens must be >= 0 (got %d)", tokens);
    WUDA_REQUIRE(experts >= 1 && experts <= 32 * kMaxPerLane, "experts must be in [1, %d] (got %d)", 32 * kMaxPerLane,
                 experts);
    WUDA_REQUIRE(k >= 1 && k <= 32 && k <= experts, "k must be in [1, min(32, experts)] (got %d)", k);
    WUDA_REQUIRE(score_func >= 0 && score_func <= 2, "score_func must be 0 (softmax), 1 (sigmoid) or 2 (sqrt softplus)");
    if (tokens == 0) return WUDA_OK;
    WUDA_REQUIRE(logits && weights && indices, "logits, weights and indices must not be NULL");
    Params p;
    p.logits = logits;
    p.bias = bias;
    p.weights = weights;
    p.indices = indices;
    p.tokens = tokens;
    p.experts = experts;
    p.k = k;
    p.score_func = score_func;
    p.route_scale = route_scale;
    // An ordinary launch, not a programmatic one: nothing of the chain behind this kernel (dispatch, gather) then waits on the
    // SMs before the router projection is through, and the shared expert's GEMMs, which a layer runs on a second stream
    // meanwhile, find them free (with the same of the SwiGLU quantisation and a smaller grid of the gather, a layer at batch
    // 64 / 128: 1186 -> 1160 / 1475 -> 1444 us).  In one stream, too, the block it belongs to is shorter: router, shared and 64 routed experts
    // of 2048, 1 / 16 / 64 / 128 tokens: early 81.8 / 248.2 / 301.3 / 440.0 us, ordinary 80.9 / 246.4 / 300.1 / 439.0, although the projection and this kernel
    // by themselves are 0.6 / 0.2 / 0.2 / 0 us faster early.
    const auto kernel = experts <= 256 ? moe_route_kernel<8> : moe_route_kernel<kMaxPerLane>;
    kernel<<<dim3((tokens + kWarpsPerCta - 1) / kWarpsPerCta), dim3(32 * kWarpsPerCta), 0, static_cast<cudaStream_t>(stream)>>>(p);
    WUDA_CUDA(cudaGetLastError());
    return WUDA_OK;
}
