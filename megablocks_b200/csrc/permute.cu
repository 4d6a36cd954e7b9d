// Row permutation kernels for sm_100a: token order <-> expert order.
//
// Functional counterparts in the reference are the Triton row-copy kernels
// (megablocks/backend/kernels.py:34-518).  The kernels here are destination
// driven: every output row is written exactly once by one warp (payload rows,
// pad rows and rows past the last bin alike), so no output is ever pre-zeroed,
// and the reduction over the top-k copies of a token happens in registers in
// token order - deterministic, no atomics, no [tokens, k, h] staging buffer.
// Rows move as 16-byte vectors whenever the row size allows it.
#include <type_traits>

#include "common.cuh"

namespace mb {

namespace {

constexpr int kWarpsPerCta = 4;

template <typename T, int VEC>
struct Pack {
  T v[VEC];
};

template <typename T, int VEC>
__device__ __forceinline__ Pack<T, VEC> load_pack(const T* p) {
  Pack<T, VEC> out;
  if constexpr (VEC * sizeof(T) == 16) {
    *reinterpret_cast<uint4*>(out.v) = *reinterpret_cast<const uint4*>(p);
  } else {
#pragma unroll
    for (int i = 0; i < VEC; ++i) out.v[i] = p[i];
  }
  return out;
}

template <typename T, int VEC>
__device__ __forceinline__ void store_pack(T* p, const Pack<T, VEC>& in) {
  if constexpr (VEC * sizeof(T) == 16) {
    *reinterpret_cast<uint4*>(p) = *reinterpret_cast<const uint4*>(in.v);
  } else {
#pragma unroll
    for (int i = 0; i < VEC; ++i) p[i] = in.v[i];
  }
}

// Copy held by row r of the expert-ordered buffer, or -1 for a pad row: e = group of r in padded_bins or
// (BINNED) r / capacity, off = r - first row of the group, indices[start(e) + off] if off < count(e).
template <bool BINNED>
__device__ __forceinline__ int copy_of_row(int64_t r, const int* __restrict__ indices, const int* __restrict__ bins,
                                           const int* __restrict__ padded_bins, int num_bins, int capacity) {
  const int row = static_cast<int>(r);
  int e, pstart = 0;
  if constexpr (BINNED) {
    e = row / capacity;
    pstart = e * capacity;
  } else {
    e = upper_bound_i32(padded_bins, num_bins, row);
    if (e > 0 && e < num_bins) pstart = __ldg(padded_bins + e - 1);
  }
  // The loads do not wait for one another.
  const bool real = e < num_bins;
  const int start = real && e > 0 ? __ldg(bins + e - 1) : 0;
  const int end = real ? __ldg(bins + e) : 0;
  const int off = row - pstart;
  return off < end - start ? __ldg(indices + start + off) : -1;
}

// out[r] = x[copy / top_k] (* weight[copy]) for every row r of the expert-ordered buffer, zero for pad rows.
template <typename T, int VEC, bool BINNED>
__global__ void __launch_bounds__(kWarpsPerCta * 32)
gather_rows_kernel(const T* __restrict__ x, const int* __restrict__ indices, const T* __restrict__ weights,
                   const int* __restrict__ bins, const int* __restrict__ padded_bins, int num_bins, int capacity,
                   int top_k, int64_t out_rows, int cols, T* __restrict__ out) {
  const int lane = threadIdx.x & 31;
  const int64_t r = int64_t(blockIdx.x) * kWarpsPerCta + (threadIdx.x >> 5);
  if (r >= out_rows) return;
  int src_token = -1;
  float scale = 1.f;
  const int copy = copy_of_row<BINNED>(r, indices, bins, padded_bins, num_bins, capacity);
  if (copy >= 0) {
    src_token = copy / top_k;
    if (weights != nullptr) scale = to_float(weights[copy]);
  }
  T* dst = out + r * cols;
  if (src_token < 0) {
    Pack<T, VEC> z;
#pragma unroll
    for (int i = 0; i < VEC; ++i) z.v[i] = from_float<T>(0.f);
    for (int c = lane * VEC; c < cols; c += 32 * VEC) store_pack<T, VEC>(dst + c, z);
    return;
  }
  const T* src = x + int64_t(src_token) * cols;
  if (weights == nullptr) {
    // Four vector loads in flight per lane before the first store.
    for (int c0 = lane * VEC; c0 < cols; c0 += 4 * 32 * VEC) {
      Pack<T, VEC> p[4];
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (c0 + j * 32 * VEC < cols) p[j] = load_pack<T, VEC>(src + c0 + j * 32 * VEC);
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (c0 + j * 32 * VEC < cols) store_pack<T, VEC>(dst + c0 + j * 32 * VEC, p[j]);
    }
  } else {
    for (int c = lane * VEC; c < cols; c += 32 * VEC) {
      Pack<T, VEC> p = load_pack<T, VEC>(src + c);
#pragma unroll
      for (int i = 0; i < VEC; ++i) p.v[i] = from_float<T>(to_float(p.v[i]) * scale);
      store_pack<T, VEC>(dst + c, p);
    }
  }
}

// inverse[copy] = row of that copy in the expert-ordered buffer (or -1 when dropped).
// capacity < 0: padded layout (row = padded_start(e) + off); capacity >= 0: binned
// layout (row = e * capacity + off, dropped when off >= capacity).
__global__ void inverse_map_kernel(const int* __restrict__ indices, const int* __restrict__ bins,
                                   const int* __restrict__ padded_bins, int num_bins, int n, int capacity,
                                   int* __restrict__ inverse) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int e = upper_bound_i32(bins, num_bins, i);
  if (e >= num_bins) {            // a position past the last bin: its copy belongs to no expert
    inverse[__ldg(indices + i)] = -1;
    return;
  }
  const int off = i - (e ? __ldg(bins + e - 1) : 0);
  int row;
  if (capacity < 0) row = (e ? __ldg(padded_bins + e - 1) : 0) + off;
  else row = off < capacity ? e * capacity + off : -1;
  inverse[__ldg(indices + i)] = row;
}

// out[t] = sum_s weight[t*k+s] * x[inverse[t*k+s]] [+ bias]  (fp32 accumulate, one rounding).
// Bound by memory: k rows read, one written per token.  Rows are cut into slices while there are too few
// tokens to fill the SMs; a warp takes CHUNKS pieces of 32 lanes x 16 bytes of COPIES copies at a time.
//   COPIES = 0 (top-1): a plain loop over the slice at full occupancy is at the bandwidth (32768 x 768 bf16
//   in 14.4 us, 100 MB); four pieces in flight per lane cost it 96 registers and twice the time.
//   COPIES = 1: many tokens.  Full occupancy (64 warps an SM, 32 registers) hides the latency, and more in
//   flight costs it: 32768 tokens x 768, two copies, takes 32 us with this plain loop, 36 at 40 registers, 34.6
//   with two copies in flight, 40 with two pieces of two.
//   COPIES = 2: few tokens, bound by latency.  With the search of the rows, whole rows and one load at a time
//   against slices, top-2: 16 x 4096 12.9 us | 4.3, 2047 x 4096 15.4 | 10.7.
// The layer's output bias rides along here (BIAS): as an elementwise add of its own it read and wrote the
// whole output again with a broadcast operand that the library does not vectorise (56 us for 32768 x 768
// bf16, 80 us for 65536 x 512 fp16).
template <typename T, int VEC, int CHUNKS, int COPIES, bool BIAS>
__global__ void __launch_bounds__(kWarpsPerCta * 32, COPIES <= 1 ? 64 / kWarpsPerCta : 0)
combine_rows_kernel(const T* __restrict__ x, const int* __restrict__ inverse, const T* __restrict__ weights,
                    const T* __restrict__ bias, int top_k, int64_t tokens, int cols, int slice_cols,
                    T* __restrict__ out) {
  const int lane = threadIdx.x & 31;
  const int64_t t = int64_t(blockIdx.x) * kWarpsPerCta + (threadIdx.x >> 5);
  if (t >= tokens) return;
  const int begin = blockIdx.y * slice_cols;
  const int end = min(cols, begin + slice_cols);
  T* dst = out + t * cols;
  if constexpr (COPIES == 0) {
    const int row = __ldg(inverse + t);
    const float w = (weights != nullptr) ? to_float(weights[t]) : 1.f;
    for (int c = begin + lane * VEC; c < end; c += 32 * VEC) {
      Pack<T, VEC> p;
      if (row >= 0) {
        p = load_pack<T, VEC>(x + int64_t(row) * cols + c);
        if (!BIAS && weights != nullptr) {
#pragma unroll
          for (int i = 0; i < VEC; ++i) p.v[i] = from_float<T>(to_float(p.v[i]) * w);
        }
      } else {
#pragma unroll
        for (int i = 0; i < VEC; ++i) p.v[i] = from_float<T>(0.f);
      }
      if constexpr (BIAS) {
        const Pack<T, VEC> b = load_pack<T, VEC>(bias + c);
#pragma unroll
        for (int i = 0; i < VEC; ++i)
          p.v[i] = from_float<T>((row >= 0 ? to_float(p.v[i]) * w : 0.f) + to_float(b.v[i]));
      }
      store_pack<T, VEC>(dst + c, p);
    }
  } else if constexpr (COPIES == 1) {
    for (int c = begin + lane * VEC; c < end; c += 32 * VEC) {
      float acc[VEC];
#pragma unroll
      for (int i = 0; i < VEC; ++i) acc[i] = 0.f;
      for (int s = 0; s < top_k; ++s) {
        const int64_t copy = t * top_k + s;
        const int row = __ldg(inverse + copy);
        if (row < 0) continue;
        const float w = (weights != nullptr) ? to_float(weights[copy]) : 1.f;
        const Pack<T, VEC> p = load_pack<T, VEC>(x + int64_t(row) * cols + c);
        // Each product is rounded to T before the sum, as when the k scaled copies are first stored and
        // then added.
#pragma unroll
        for (int i = 0; i < VEC; ++i) acc[i] += to_float(from_float<T>(to_float(p.v[i]) * w));
      }
      if constexpr (BIAS) {
        const Pack<T, VEC> b = load_pack<T, VEC>(bias + c);
#pragma unroll
        for (int i = 0; i < VEC; ++i) acc[i] += to_float(b.v[i]);
      }
      Pack<T, VEC> o;
#pragma unroll
      for (int i = 0; i < VEC; ++i) o.v[i] = from_float<T>(acc[i]);
      store_pack<T, VEC>(dst + c, o);
    }
  } else {
    for (int c0 = begin + lane * VEC; c0 < end; c0 += CHUNKS * 32 * VEC) {
      float acc[CHUNKS][VEC];
#pragma unroll
      for (int j = 0; j < CHUNKS; ++j)
#pragma unroll
        for (int i = 0; i < VEC; ++i) acc[j][i] = 0.f;
      for (int s = 0; s < top_k; s += COPIES) {
        int row[COPIES];
        float w[COPIES];
        Pack<T, VEC> p[COPIES][CHUNKS];
#pragma unroll
        for (int u = 0; u < COPIES; ++u) {
          const int64_t copy = t * top_k + s + u;
          row[u] = s + u < top_k ? __ldg(inverse + copy) : -1;
          w[u] = (weights != nullptr && s + u < top_k) ? to_float(weights[copy]) : 1.f;
        }
#pragma unroll
        for (int u = 0; u < COPIES; ++u)
#pragma unroll
          for (int j = 0; j < CHUNKS; ++j) {
            const int c = c0 + j * 32 * VEC;
            if (row[u] >= 0 && c < end) p[u][j] = load_pack<T, VEC>(x + int64_t(row[u]) * cols + c);
          }
#pragma unroll
        for (int u = 0; u < COPIES; ++u)
#pragma unroll
          for (int j = 0; j < CHUNKS; ++j) {
            if (row[u] < 0 || c0 + j * 32 * VEC >= end) continue;
#pragma unroll
            for (int i = 0; i < VEC; ++i) acc[j][i] += to_float(from_float<T>(to_float(p[u][j].v[i]) * w[u]));
          }
      }
#pragma unroll
      for (int j = 0; j < CHUNKS; ++j) {
        const int c = c0 + j * 32 * VEC;
        if (c >= end) break;
        if constexpr (BIAS) {
          const Pack<T, VEC> b = load_pack<T, VEC>(bias + c);
#pragma unroll
          for (int i = 0; i < VEC; ++i) acc[j][i] += to_float(b.v[i]);
        }
        Pack<T, VEC> o;
#pragma unroll
        for (int i = 0; i < VEC; ++i) o.v[i] = from_float<T>(acc[j][i]);
        store_pack<T, VEC>(dst + c, o);
      }
    }
  }
}

// wgrad[copy] = <x[row(copy)], grad[copy / top_k]>, one warp per copy.  VEC > 1: both rows are read
// in 16-byte pieces (rows of a multiple of 16 bytes at 16-byte aligned bases).
template <typename T, int VEC>
__global__ void __launch_bounds__(kWarpsPerCta * 32)
wgrad_kernel(const T* __restrict__ x, const T* __restrict__ grad, const int* __restrict__ inverse, int top_k,
             int64_t copies, int cols, T* __restrict__ wgrad) {
  const int lane = threadIdx.x & 31;
  const int64_t copy = int64_t(blockIdx.x) * kWarpsPerCta + (threadIdx.x >> 5);
  if (copy >= copies) return;
  const int row = __ldg(inverse + copy);
  float acc = 0.f;
  if (row >= 0) {
    const T* a = x + int64_t(row) * cols;
    const T* b = grad + (copy / top_k) * cols;
    if constexpr (VEC > 1) {
      float acc2 = 0.f;
      for (int c = lane * VEC; c < cols; c += 32 * VEC) {
        const Pack<T, VEC> pa = load_pack<T, VEC>(a + c), pb = load_pack<T, VEC>(b + c);
#pragma unroll
        for (int k = 0; k < VEC; k += 2) {
          acc = fmaf(to_float(pa.v[k]), to_float(pb.v[k]), acc);
          acc2 = fmaf(to_float(pa.v[k + 1]), to_float(pb.v[k + 1]), acc2);
        }
      }
      acc += acc2;
    } else {
      for (int c = lane; c < cols; c += 32) acc += to_float(a[c]) * to_float(b[c]);
    }
  }
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, d);
  if (lane == 0) wgrad[copy] = from_float<T>(acc);
}

// Backward of the weighted un-permutation in one pass over the expert-ordered rows: for row r with
// copy c of token t, dx[r] = weight[c] * grad[t] and dweight[c] = <x[r], grad[t]>; pad rows of dx are
// zero.  Bound by memory: as two kernels (the gather above and wgrad_kernel) grad is read twice and an
// inverse index map is built in between.  One warp per row, two 16-byte loads of each operand in
// flight per lane.  dweight entries of copies without a row are cleared by the launcher.
template <typename T, int VEC, bool BINNED>
__global__ void __launch_bounds__(kWarpsPerCta * 32)
scatter_bwd_kernel(const T* __restrict__ x, const T* __restrict__ grad, const int* __restrict__ indices,
                   const T* __restrict__ weights, const int* __restrict__ bins, const int* __restrict__ padded_bins,
                   int num_bins, int capacity, int top_k, int64_t out_rows, int cols, T* __restrict__ dx,
                   T* __restrict__ dweights) {
  const int lane = threadIdx.x & 31;
  const int64_t r = int64_t(blockIdx.x) * kWarpsPerCta + (threadIdx.x >> 5);
  if (r >= out_rows) return;
  const int copy = copy_of_row<BINNED>(r, indices, bins, padded_bins, num_bins, capacity);
  T* dst = dx + r * cols;
  if (copy < 0) {
    Pack<T, VEC> z;
#pragma unroll
    for (int i = 0; i < VEC; ++i) z.v[i] = from_float<T>(0.f);
    for (int c = lane * VEC; c < cols; c += 32 * VEC) store_pack<T, VEC>(dst + c, z);
    return;
  }
  const float w = to_float(weights[copy]);
  const T* g = grad + int64_t(copy / top_k) * cols;
  const T* row = x + r * cols;
  float acc[2] = {0.f, 0.f};
  for (int c0 = lane * VEC; c0 < cols; c0 += 2 * 32 * VEC) {
    Pack<T, VEC> pg[2], px[2];
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const int c = c0 + j * 32 * VEC;
      if (c < cols) {
        pg[j] = load_pack<T, VEC>(g + c);
        px[j] = load_pack<T, VEC>(row + c);
      }
    }
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const int c = c0 + j * 32 * VEC;
      if (c < cols) {
#pragma unroll
        for (int i = 0; i < VEC; ++i) {
          const float gv = to_float(pg[j].v[i]);
          acc[j] = fmaf(to_float(px[j].v[i]), gv, acc[j]);
          pg[j].v[i] = from_float<T>(gv * w);
        }
        store_pack<T, VEC>(dst + c, pg[j]);
      }
    }
  }
  float dot = acc[0] + acc[1];
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, d);
  if (lane == 0) dweights[copy] = from_float<T>(dot);
}

template <typename T>
int vec_width(int64_t cols, const void* a, const void* b) {
  constexpr int full = 16 / sizeof(T);
  const bool aligned = (reinterpret_cast<uintptr_t>(a) % 16 == 0) && (reinterpret_cast<uintptr_t>(b) % 16 == 0);
  return (aligned && cols % full == 0) ? full : 1;
}

}  // namespace

cudaError_t gather_rows(DType type, const void* x, const int* indices, const void* weights, const int* bins,
                        const int* padded_bins, int num_bins, int capacity, int top_k, int64_t out_rows, int cols,
                        void* out, cudaStream_t stream) {
  const int grid = ceil_div(out_rows, kWarpsPerCta);
  MB_SWITCH_FLOAT(type, T, {
    constexpr int kFull = 16 / sizeof(T);
    auto run = [&](auto kernel) {
      kernel<<<grid, kWarpsPerCta * 32, 0, stream>>>(static_cast<const T*>(x), indices, static_cast<const T*>(weights),
                                                     bins, padded_bins, num_bins, capacity, top_k, out_rows, cols,
                                                     static_cast<T*>(out));
    };
    const bool wide = vec_width<T>(cols, x, out) > 1;
    if (capacity >= 0) {
      if (wide) run(gather_rows_kernel<T, kFull, true>);
      else run(gather_rows_kernel<T, 1, true>);
    } else {
      if (wide) run(gather_rows_kernel<T, kFull, false>);
      else run(gather_rows_kernel<T, 1, false>);
    }
  })
  return cudaGetLastError();
}

cudaError_t inverse_map(const int* indices, const int* bins, const int* padded_bins, int num_bins, int n,
                        int capacity, int* inverse, cudaStream_t stream) {
  inverse_map_kernel<<<ceil_div(n, 256), 256, 0, stream>>>(indices, bins, padded_bins, num_bins, n, capacity,
                                                          inverse);
  return cudaGetLastError();
}

cudaError_t combine_rows(DType type, const void* x, const int* inverse, const void* weights, const void* bias,
                         int top_k, int64_t tokens, int cols, int sms, void* out, cudaStream_t stream) {
  if (tokens == 0 || cols == 0) return cudaSuccess;
  MB_SWITCH_FLOAT(type, T, {
    constexpr int kFull = 16 / sizeof(T);
    const bool wide = vec_width<T>(cols, x, out) > 1 && reinterpret_cast<uintptr_t>(bias) % 16 == 0;
    const bool single = top_k == 1;
    // Warps for all SMs (64 on each) come from the tokens or, while those are too few, from slices of the
    // rows.  One copy at a time where the tokens alone (nearly) fill the SMs, or half of them with rows of one
    // piece, which have no slices; else two, and two pieces of each where a row has more than four.  9000 tokens
    // (0.95 of the warps) x 4096, three copies: 1.2 times as long with two; 6000: 1.0; 2047: 0.7.
    const int piece = 32 * (wide ? kFull : 1);
    const int pieces = ceil_div(cols, piece);
    const int64_t warps = int64_t(sms) * 64;
    const bool full = tokens >= warps * 3 / 4 || (pieces == 1 && tokens >= warps / 2);
    const int chunks = !single && !full && pieces > 4 ? 2 : 1;
    const int steps = ceil_div(pieces, chunks);
    const int64_t wanted = (warps + tokens - 1) / tokens;
    int per_slice = ceil_div(steps, wanted < steps ? static_cast<int>(wanted) : steps);
    per_slice = max(per_slice, ceil_div(steps, 65535));       // the grid's limit
    const dim3 grid(ceil_div(tokens, kWarpsPerCta), ceil_div(steps, per_slice));
    auto run = [&](auto kernel) {
      kernel<<<grid, kWarpsPerCta * 32, 0, stream>>>(
          static_cast<const T*>(x), inverse, static_cast<const T*>(weights), static_cast<const T*>(bias), top_k, tokens,
          cols, per_slice * chunks * piece, static_cast<T*>(out));
    };
    auto pick = [&](auto vec, auto with_bias) {
      constexpr int V = decltype(vec)::value;
      constexpr bool B = decltype(with_bias)::value;
      if (single) run(combine_rows_kernel<T, V, 1, 0, B>);
      else if (full) run(combine_rows_kernel<T, V, 1, 1, B>);
      else if (chunks == 2) run(combine_rows_kernel<T, V, 2, 2, B>);
      else run(combine_rows_kernel<T, V, 1, 2, B>);
    };
    auto pick_bias = [&](auto vec) {
      if (bias != nullptr) pick(vec, std::true_type{});
      else pick(vec, std::false_type{});
    };
    if (wide) pick_bias(std::integral_constant<int, kFull>{});
    else pick_bias(std::integral_constant<int, 1>{});
  })
  return cudaGetLastError();
}

cudaError_t scatter_bwd(DType type, const void* x, const void* grad, const int* indices, const void* weights,
                        const int* bins, const int* padded_bins, int num_bins, int capacity, int top_k, int64_t copies,
                        int64_t out_rows, int cols, void* dx, void* dweights, cudaStream_t stream) {
  MB_SWITCH_FLOAT(type, T, {
    constexpr int kFull = 16 / sizeof(T);
    const cudaError_t rc = cudaMemsetAsync(dweights, 0, size_t(copies) * sizeof(T), stream);
    if (rc != cudaSuccess) return rc;
    const int grid = ceil_div(out_rows, kWarpsPerCta);
    auto run = [&](auto kernel) {
      kernel<<<grid, kWarpsPerCta * 32, 0, stream>>>(
          static_cast<const T*>(x), static_cast<const T*>(grad), indices, static_cast<const T*>(weights), bins,
          padded_bins, num_bins, capacity, top_k, out_rows, cols, static_cast<T*>(dx), static_cast<T*>(dweights));
    };
    const bool wide = vec_width<T>(cols, x, grad) > 1 && reinterpret_cast<uintptr_t>(dx) % 16 == 0;
    if (capacity >= 0) {
      if (wide) run(scatter_bwd_kernel<T, kFull, true>);
      else run(scatter_bwd_kernel<T, 1, true>);
    } else {
      if (wide) run(scatter_bwd_kernel<T, kFull, false>);
      else run(scatter_bwd_kernel<T, 1, false>);
    }
  })
  return cudaGetLastError();
}

cudaError_t scatter_wgrad(DType type, const void* x, const void* grad, const int* inverse, int top_k,
                          int64_t copies, int cols, void* wgrad, cudaStream_t stream) {
  MB_SWITCH_FLOAT(type, T, {
    constexpr int kFull = 16 / sizeof(T);
    if (vec_width<T>(cols, x, grad) > 1) {
      wgrad_kernel<T, kFull><<<ceil_div(copies, kWarpsPerCta), kWarpsPerCta * 32, 0, stream>>>(
          static_cast<const T*>(x), static_cast<const T*>(grad), inverse, top_k, copies, cols,
          static_cast<T*>(wgrad));
    } else {
      wgrad_kernel<T, 1><<<ceil_div(copies, kWarpsPerCta), kWarpsPerCta * 32, 0, stream>>>(
          static_cast<const T*>(x), static_cast<const T*>(grad), inverse, top_k, copies, cols,
          static_cast<T*>(wgrad));
    }
  })
  return cudaGetLastError();
}

}  // namespace mb
