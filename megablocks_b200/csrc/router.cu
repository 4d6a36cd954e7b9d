// Router selection kernels for sm_100a: softmax -> top-k -> optional p-norm
// normalisation in one pass over the logits, and the matching backward.
//
// Reference semantics (megablocks/layers/router.py:87-106): scores are the
// softmax of the logits rounded to the logits' dtype; the k largest *rounded*
// scores are selected (ties go to the lowest expert id); weights are optionally
// divided by their p-norm (p = 1 or 2).  One warp owns one token; with at most
// 1024 experts a lane holds at most 32 scores in registers; the kernels are compiled for 1, 2, 4,
// 8, 16 and 32 scores per lane and the launch picks the smallest that covers the expert count, so
// a 64-expert router does not walk 32 mostly empty slots per loop.
#include "common.cuh"

namespace mb {

namespace {

constexpr int kMaxPerLane = kRouterMaxExperts / 32;
constexpr int kMaxTopK = kRouterMaxTopK;

// A token with a NaN or +inf logit has NaN scores.  They are selected like the largest ones, so every
// token gets top_k distinct ids of [0, experts) (scores lie in [0, 1], taken ones count as -1), and its
// weights are NaN: an overflow is seen in the loss and not read as an address.
__device__ __forceinline__ float selection_key(float score) { return score != score ? INFINITY : score; }
__device__ __forceinline__ float selected_score(float key) { return key == INFINITY ? NAN : key; }

// Score of a selected id in the backward kernels; an id of no expert has none.
template <typename T>
__device__ __forceinline__ float score_of(const T* scores, int e, int num_experts) {
  return static_cast<unsigned>(e) < static_cast<unsigned>(num_experts) ? to_float(scores[e]) : NAN;
}

template <typename T, int PL>
__global__ void __launch_bounds__(128)
router_topk_fwd_kernel(const T* __restrict__ logits, int64_t tokens, int num_experts, int top_k, float norm_p,
                       T* __restrict__ scores, T* __restrict__ weights, int64_t* __restrict__ experts) {
  const int lane = threadIdx.x & 31;
  const int64_t t = int64_t(blockIdx.x) * 4 + (threadIdx.x >> 5);
  if (t >= tokens) return;
  const T* row = logits + t * num_experts;
  float v[PL];
  float vmax = -INFINITY;
#pragma unroll
  for (int j = 0; j < PL; ++j) {
    const int e = lane + j * 32;
    v[j] = e < num_experts ? to_float(row[e]) : -INFINITY;
    vmax = fmaxf(vmax, v[j]);
  }
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) vmax = fmaxf(vmax, __shfl_xor_sync(0xffffffffu, vmax, d));
  float sum = 0.f;
#pragma unroll
  for (int j = 0; j < PL; ++j) {
    const int e = lane + j * 32;
    v[j] = e < num_experts ? __expf(v[j] - vmax) : 0.f;
    sum += v[j];
  }
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, d);
  const float inv = 1.f / sum;
  T* srow = scores + t * num_experts;
#pragma unroll
  for (int j = 0; j < PL; ++j) {
    const int e = lane + j * 32;
    if (e < num_experts) {
      const T r = from_float<T>(v[j] * inv);
      srow[e] = r;
      v[j] = selection_key(to_float(r));          // selection runs on the rounded scores
    } else {
      v[j] = -1.f;
    }
  }
  float chosen_w[kMaxTopK];
  int chosen_e[kMaxTopK];
  for (int s = 0; s < top_k; ++s) {
    float best = -2.f;
    int best_e = 0x7fffffff;
#pragma unroll
    for (int j = 0; j < PL; ++j) {
      const int e = lane + j * 32;
      if (v[j] > best) { best = v[j]; best_e = e; }   // ascending e within a lane: first wins ties
    }
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) {
      const float ob = __shfl_xor_sync(0xffffffffu, best, d);
      const int oe = __shfl_xor_sync(0xffffffffu, best_e, d);
      if (ob > best || (ob == best && oe < best_e)) { best = ob; best_e = oe; }
    }
    chosen_w[s] = selected_score(best);
    chosen_e[s] = best_e;
    if ((best_e & 31) == lane) {
#pragma unroll
      for (int j = 0; j < PL; ++j)
        if (j == (best_e >> 5)) v[j] = -1.f;
    }
  }
  if (lane == 0) {
    float norm = 1.f;
    if (norm_p > 0.f) {
      float acc = 0.f;
      for (int s = 0; s < top_k; ++s) acc += (norm_p == 1.f) ? fabsf(chosen_w[s]) : chosen_w[s] * chosen_w[s];
      norm = (norm_p == 1.f) ? acc : sqrtf(acc);
      norm = to_float(from_float<T>(norm));   // the norm is itself a tensor of dtype T
    }
    for (int s = 0; s < top_k; ++s) {
      weights[t * top_k + s] = from_float<T>(norm_p > 0.f ? chosen_w[s] / norm : chosen_w[s]);
      experts[t * top_k + s] = chosen_e[s];
    }
  }
}

// The same for expert counts that are LANES x VEC (VEC = 16 bytes of logits, LANES a power of two up to
// 32): LANES lanes share a token and each holds VEC consecutive experts, so a row is one 16-byte access
// per lane, the shuffle trees are log2(LANES) deep and a warp works on 32 / LANES tokens at once.  Bound
// by issue and shuffle latency, not by the 4 bytes an expert moves: with a warp per token the 64-expert
// fp16 router took 23.5 us forward and 24.9 us backward for 65536 tokens (17 MB each way).
template <typename T, int VEC>
struct alignas(16) RouterVec {
  T v[VEC];
};

template <typename T, int LANES>
__global__ void __launch_bounds__(256)
router_topk_fwd_vec_kernel(const T* __restrict__ logits, int64_t tokens, int top_k, float norm_p,
                           T* __restrict__ scores, T* __restrict__ weights, int64_t* __restrict__ experts) {
  constexpr int VEC = 16 / sizeof(T);
  constexpr int E = LANES * VEC;
  const int l = threadIdx.x % LANES;
  const int64_t tok = (int64_t(blockIdx.x) * 256 + threadIdx.x) / LANES;
  const bool live = tok < tokens;                 // idle groups stay for the shuffles
  const int64_t t = live ? tok : tokens - 1;
  RouterVec<T, VEC> raw;
  *reinterpret_cast<uint4*>(&raw) = *reinterpret_cast<const uint4*>(logits + t * E + l * VEC);
  float v[VEC];
  float vmax = -INFINITY;
#pragma unroll
  for (int j = 0; j < VEC; ++j) {
    v[j] = to_float(raw.v[j]);
    vmax = fmaxf(vmax, v[j]);
  }
#pragma unroll
  for (int d = LANES / 2; d > 0; d >>= 1) vmax = fmaxf(vmax, __shfl_xor_sync(0xffffffffu, vmax, d));
  float sum = 0.f;
#pragma unroll
  for (int j = 0; j < VEC; ++j) {
    v[j] = __expf(v[j] - vmax);
    sum += v[j];
  }
#pragma unroll
  for (int d = LANES / 2; d > 0; d >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, d);
  const float inv = 1.f / sum;
#pragma unroll
  for (int j = 0; j < VEC; ++j) {
    raw.v[j] = from_float<T>(v[j] * inv);
    v[j] = selection_key(to_float(raw.v[j]));     // selection runs on the rounded scores
  }
  if (live) *reinterpret_cast<uint4*>(scores + t * E + l * VEC) = *reinterpret_cast<const uint4*>(&raw);
  float chosen[kMaxTopK];
  float norm = 0.f;
#pragma unroll
  for (int s = 0; s < kMaxTopK; ++s) {
    if (s >= top_k) break;
    float best = -2.f;
    int best_e = 0x7fffffff;
#pragma unroll
    for (int j = 0; j < VEC; ++j)
      if (v[j] > best) { best = v[j]; best_e = l * VEC + j; }      // ascending: first wins ties
#pragma unroll
    for (int d = LANES / 2; d > 0; d >>= 1) {
      const float ob = __shfl_xor_sync(0xffffffffu, best, d);
      const int oe = __shfl_xor_sync(0xffffffffu, best_e, d);
      if (ob > best || (ob == best && oe < best_e)) { best = ob; best_e = oe; }
    }
    chosen[s] = selected_score(best);
    norm += norm_p == 1.f ? fabsf(chosen[s]) : chosen[s] * chosen[s];
#pragma unroll
    for (int j = 0; j < VEC; ++j)
      if (best_e == l * VEC + j) v[j] = -1.f;
    if (live && l == 0) experts[t * top_k + s] = best_e;
  }
  if (live && l == 0) {
    norm = norm_p == 1.f ? norm : sqrtf(norm);
    norm = to_float(from_float<T>(norm));         // the norm is itself a tensor of dtype T
#pragma unroll
    for (int s = 0; s < kMaxTopK; ++s) {
      if (s >= top_k) break;
      weights[t * top_k + s] = from_float<T>(norm_p > 0.f ? chosen[s] / norm : chosen[s]);
    }
  }
}

template <typename T, int LANES>
__global__ void __launch_bounds__(256)
router_topk_bwd_vec_kernel(const T* __restrict__ scores, const int64_t* __restrict__ experts,
                           const T* __restrict__ dscores, const T* __restrict__ dweights, int64_t tokens, int top_k,
                           float norm_p, T* __restrict__ dlogits) {
  constexpr int VEC = 16 / sizeof(T);
  constexpr int E = LANES * VEC;
  const int l = threadIdx.x % LANES;
  const int64_t tok = (int64_t(blockIdx.x) * 256 + threadIdx.x) / LANES;
  const bool live = tok < tokens;
  const int64_t t = live ? tok : tokens - 1;
  RouterVec<T, VEC> sv, gv;
  *reinterpret_cast<uint4*>(&sv) = *reinterpret_cast<const uint4*>(scores + t * E + l * VEC);
  *reinterpret_cast<uint4*>(&gv) = *reinterpret_cast<const uint4*>(dscores + t * E + l * VEC);
  // Gradient with respect to the k selected (pre-normalisation) scores.
  float dsel[kMaxTopK], raw[kMaxTopK];
  int sel[kMaxTopK];
  float norm_acc = 0.f, dot = 0.f;
#pragma unroll
  for (int s = 0; s < kMaxTopK; ++s) {
    if (s >= top_k) break;
    sel[s] = static_cast<int>(experts[t * top_k + s]);
    raw[s] = score_of(scores + t * E, sel[s], E);
    dsel[s] = to_float(dweights[t * top_k + s]);
    norm_acc += (norm_p == 1.f) ? fabsf(raw[s]) : raw[s] * raw[s];
    dot += dsel[s] * raw[s];
  }
  if (norm_p > 0.f) {
    const float norm = (norm_p == 1.f) ? norm_acc : sqrtf(norm_acc);
#pragma unroll
    for (int s = 0; s < kMaxTopK; ++s) {
      if (s >= top_k) break;
      const float dnorm = (norm_p == 1.f) ? (raw[s] >= 0.f ? 1.f : -1.f) : raw[s] / norm;
      dsel[s] = dsel[s] / norm - dot * dnorm / (norm * norm);
    }
  }
  float g[VEC];
  float inner = 0.f;
#pragma unroll
  for (int j = 0; j < VEC; ++j) {
    g[j] = to_float(gv.v[j]);
#pragma unroll
    for (int s = 0; s < kMaxTopK; ++s) {
      if (s >= top_k) break;
      if (sel[s] == l * VEC + j) g[j] += dsel[s];
    }
    inner += g[j] * to_float(sv.v[j]);
  }
#pragma unroll
  for (int d = LANES / 2; d > 0; d >>= 1) inner += __shfl_xor_sync(0xffffffffu, inner, d);
#pragma unroll
  for (int j = 0; j < VEC; ++j) gv.v[j] = from_float<T>(to_float(sv.v[j]) * (g[j] - inner));
  if (live) *reinterpret_cast<uint4*>(dlogits + t * E + l * VEC) = *reinterpret_cast<const uint4*>(&gv);
}

// Lanes per token of the vector kernels, 0 when the expert count or an address does not fit them.
template <typename T>
int router_vec_lanes(int num_experts, const void* a, const void* b, const void* c) {
  constexpr int VEC = 16 / sizeof(T);
  const uintptr_t any = reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(b) | reinterpret_cast<uintptr_t>(c);
  if (any % 16 != 0 || num_experts % VEC != 0) return 0;
  const int lanes = num_experts / VEC;
  return lanes <= 32 && (lanes & (lanes - 1)) == 0 ? lanes : 0;
}

#define MB_ROUTER_LANES(lanes, CALL) \
  switch (lanes) {                   \
    case 1: CALL(1); break;          \
    case 2: CALL(2); break;          \
    case 4: CALL(4); break;          \
    case 8: CALL(8); break;          \
    case 16: CALL(16); break;        \
    default: CALL(32); break;        \
  }

// dlogits = s * (g - <g, s>) with g = dscores + scatter(top-k weight grads).
template <typename T, int PL>
__global__ void __launch_bounds__(128)
router_topk_bwd_kernel(const T* __restrict__ scores, const int64_t* __restrict__ experts,
                       const T* __restrict__ dscores, const T* __restrict__ dweights, int64_t tokens,
                       int num_experts, int top_k, float norm_p, T* __restrict__ dlogits) {
  const int lane = threadIdx.x & 31;
  const int64_t t = int64_t(blockIdx.x) * 4 + (threadIdx.x >> 5);
  if (t >= tokens) return;
  const T* srow = scores + t * num_experts;
  const T* grow = dscores + t * num_experts;
  // Gradient with respect to the k selected (pre-normalisation) scores.
  float dsel[kMaxTopK];
  int sel[kMaxTopK];
  float raw[kMaxTopK];
  float norm_acc = 0.f, dot = 0.f;
  for (int s = 0; s < top_k; ++s) {
    sel[s] = static_cast<int>(experts[t * top_k + s]);
    raw[s] = score_of(srow, sel[s], num_experts);
    dsel[s] = to_float(dweights[t * top_k + s]);
    norm_acc += (norm_p == 1.f) ? fabsf(raw[s]) : raw[s] * raw[s];
    dot += dsel[s] * raw[s];
  }
  if (norm_p > 0.f) {
    const float norm = (norm_p == 1.f) ? norm_acc : sqrtf(norm_acc);
    for (int s = 0; s < top_k; ++s) {
      const float dnorm = (norm_p == 1.f) ? (raw[s] >= 0.f ? 1.f : -1.f) : raw[s] / norm;
      dsel[s] = dsel[s] / norm - dot * dnorm / (norm * norm);
    }
  }
  float g[PL];
  float inner = 0.f;
#pragma unroll
  for (int j = 0; j < PL; ++j) {
    const int e = lane + j * 32;
    float gv = 0.f;
    if (e < num_experts) {
      gv = to_float(grow[e]);
      for (int s = 0; s < top_k; ++s)
        if (sel[s] == e) gv += dsel[s];
      inner += gv * to_float(srow[e]);
    }
    g[j] = gv;
  }
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) inner += __shfl_xor_sync(0xffffffffu, inner, d);
  T* drow = dlogits + t * num_experts;
#pragma unroll
  for (int j = 0; j < PL; ++j) {
    const int e = lane + j * 32;
    if (e < num_experts) drow[e] = from_float<T>(to_float(srow[e]) * (g[j] - inner));
  }
}

}  // namespace

cudaError_t router_topk_fwd(DType type, const void* logits, int64_t tokens, int num_experts, int top_k,
                            float norm_p, void* scores, void* weights, int64_t* experts, cudaStream_t stream) {
  if (num_experts > 32 * kMaxPerLane || top_k < 1 || top_k > kMaxTopK || top_k > num_experts)
    return cudaErrorInvalidValue;
  if (tokens == 0) return cudaSuccess;
#define MB_ROUTER_FWD(PL)                                                                            \
  router_topk_fwd_kernel<T, PL><<<ceil_div(tokens, 4), 128, 0, stream>>>(                            \
      static_cast<const T*>(logits), tokens, num_experts, top_k, norm_p, static_cast<T*>(scores),    \
      static_cast<T*>(weights), experts)
#define MB_ROUTER_FWD_VEC(LANES)                                                                     \
  router_topk_fwd_vec_kernel<T, LANES><<<ceil_div(tokens, 256 / LANES), 256, 0, stream>>>(            \
      static_cast<const T*>(logits), tokens, top_k, norm_p, static_cast<T*>(scores), static_cast<T*>(weights), experts)
  MB_SWITCH_FLOAT(type, T, {
    const int lanes = router_vec_lanes<T>(num_experts, logits, scores, nullptr);
    if (lanes > 0) {
      MB_ROUTER_LANES(lanes, MB_ROUTER_FWD_VEC)
      return cudaGetLastError();
    }
    if (num_experts <= 32) MB_ROUTER_FWD(1);
    else if (num_experts <= 64) MB_ROUTER_FWD(2);
    else if (num_experts <= 128) MB_ROUTER_FWD(4);
    else if (num_experts <= 256) MB_ROUTER_FWD(8);
    else if (num_experts <= 512) MB_ROUTER_FWD(16);
    else MB_ROUTER_FWD(32);
  })
#undef MB_ROUTER_FWD
#undef MB_ROUTER_FWD_VEC
  return cudaGetLastError();
}

cudaError_t router_topk_bwd(DType type, const void* scores, const int64_t* experts, const void* dscores,
                            const void* dweights, int64_t tokens, int num_experts, int top_k, float norm_p,
                            void* dlogits, cudaStream_t stream) {
  if (tokens == 0) return cudaSuccess;
  if (num_experts > 32 * kMaxPerLane) return cudaErrorInvalidValue;
#define MB_ROUTER_BWD(PL)                                                                                          \
  router_topk_bwd_kernel<T, PL><<<ceil_div(tokens, 4), 128, 0, stream>>>(                                          \
      static_cast<const T*>(scores), experts, static_cast<const T*>(dscores), static_cast<const T*>(dweights),     \
      tokens, num_experts, top_k, norm_p, static_cast<T*>(dlogits))
#define MB_ROUTER_BWD_VEC(LANES)                                                                                   \
  router_topk_bwd_vec_kernel<T, LANES><<<ceil_div(tokens, 256 / LANES), 256, 0, stream>>>(                          \
      static_cast<const T*>(scores), experts, static_cast<const T*>(dscores), static_cast<const T*>(dweights),     \
      tokens, top_k, norm_p, static_cast<T*>(dlogits))
  MB_SWITCH_FLOAT(type, T, {
    const int lanes = router_vec_lanes<T>(num_experts, scores, dscores, dlogits);
    if (lanes > 0 && top_k <= kMaxTopK) {
      MB_ROUTER_LANES(lanes, MB_ROUTER_BWD_VEC)
      return cudaGetLastError();
    }
    if (num_experts <= 32) MB_ROUTER_BWD(1);
    else if (num_experts <= 64) MB_ROUTER_BWD(2);
    else if (num_experts <= 128) MB_ROUTER_BWD(4);
    else if (num_experts <= 256) MB_ROUTER_BWD(8);
    else if (num_experts <= 512) MB_ROUTER_BWD(16);
    else MB_ROUTER_BWD(32);
  })
#undef MB_ROUTER_BWD
#undef MB_ROUTER_BWD_VEC
  return cudaGetLastError();
}

}  // namespace mb
