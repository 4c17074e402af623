// Layer norm (weight, no bias) of a sublayer's output, added to a 32-bit residual stream: one CTA per token row.
// The row comes from the split-K partial sums of the linear before it, from an embedding table, or from fp32 rows picked
// by index (final norm of the rows whose logits are wanted); mean and variance are taken over the exact fp32 row in two
// passes (variance = mean of squared deviations).
#include "common.cuh"

namespace b200 {
namespace outnorm {

constexpr int kThreads = 256;
constexpr int kMaxWidth = 16384;  // the row is kept in shared memory
constexpr int kMaxVecWidth = 8192;  // multiples of 4 up to here stay in registers (the widths that real models have)

template <int THREADS = kThreads>
__device__ __forceinline__ float block_sum(float v, float* red) {
  v = warp_sum(v);
  __syncthreads();  // `red` may still be read from the previous call
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  float s = 0.f;
#pragma unroll
  for (int i = 0; i < THREADS / 32; ++i) s += red[i];
  return s;
}

template <typename T>
__device__ __forceinline__ float4 load4(const T* p);
template <>
__device__ __forceinline__ float4 load4<float>(const float* p) {
  return *reinterpret_cast<const float4*>(p);
}
template <>
__device__ __forceinline__ float4 load4<__nv_bfloat16>(const __nv_bfloat16* p) {
  const uint2 v = *reinterpret_cast<const uint2*>(p);
  return make_float4(bf16_lo(v.x), bf16_hi(v.x), bf16_lo(v.y), bf16_hi(v.y));
}
__device__ __forceinline__ void store4(float* p, float4 v) { *reinterpret_cast<float4*>(p) = v; }
__device__ __forceinline__ void store4(__nv_bfloat16* p, float4 v) {
  *reinterpret_cast<uint2*>(p) = make_uint2(pack_bf16x2(v.x, v.y), pack_bf16x2(v.z, v.w));
}

// Source row of output row `row` that does not come from partial sums; returns false for an index out of range (zeros).
__device__ __forceinline__ bool source_row(const b200_out_norm_args& a, int row, int64_t& src) {
  if (a.table != nullptr) {
    src = a.ids[row];
    return src >= 0 && src < a.table_rows;
  }
  src = a.row_index ? a.row_index[row] : row;
  return src >= 0 && src < a.source_rows;
}

// width % 4 == 0 and width <= SLOTS * THREADS * 4: the row lives in registers.  Bound by latency with few rows, by bytes in flight with many.  What the sums do
// not need is read before them (kEarly), the weight before the kernel in front has ended, the residual row together with the sublayer's: behind two block sums
// each was one more trip to memory.  One row of 2048 and eight splits 3.6 -> 2.3 us, 64 of 4096 6.3 -> 3.9, 6208 of 2048 58.9 -> 37.0 us (floor 26.8).  It costs
// registers, so CTAs (8192 rows of 8192 240 -> 390 us): with several rows on an SM only short ones do it.
template <typename T, int SLOTS, int THREADS, bool kEarly, int CTAS>
__global__ void __launch_bounds__(THREADS, CTAS)
out_norm_vec_kernel(b200_out_norm_args a) {
  __shared__ float red[THREADS / 32];
  pdl_launch_dependents();
  const int tid = threadIdx.x;
  const int row = blockIdx.x;
  const int W = a.width;
  const T* gamma = static_cast<const T*>(a.gamma);
  constexpr int kEarlySlots = kEarly ? SLOTS : 1;
  float4 v[SLOTS], early_g[kEarlySlots], early_h[kEarlySlots];
  if constexpr (kEarly) {
#pragma unroll
    for (int i = 0; i < SLOTS; ++i) {
      const int c = (i * THREADS + tid) * 4;
      if (c < W) early_g[i] = load4(gamma + c);
    }
  }
  pdl_wait();
  float* hidden = a.hidden + static_cast<int64_t>(row) * W;
  if constexpr (kEarly) {
#pragma unroll
    for (int i = 0; i < SLOTS; ++i) {
      const int c = (i * THREADS + tid) * 4;
      if (a.accumulate && c < W) early_h[i] = *reinterpret_cast<const float4*>(hidden + c);
    }
  }
  float sum = 0.f;
  if (a.partials != nullptr) {
    const float* base = a.partials + static_cast<int64_t>(row) * W;
    const int64_t stride = static_cast<int64_t>(a.rows) * W;
#pragma unroll
    for (int i = 0; i < SLOTS; ++i) {
      const int c = (i * THREADS + tid) * 4;
      float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
      if (c < W) {
#pragma unroll 4
        for (int s = 0; s < a.num_splits; ++s) {
          const float4 t = __ldcg(reinterpret_cast<const float4*>(base + s * stride + c));
          acc.x += t.x;
          acc.y += t.y;
          acc.z += t.z;
          acc.w += t.w;
        }
      }
      v[i] = acc;
    }
  } else {
    int64_t src;
    const bool ok = source_row(a, row, src);
#pragma unroll
    for (int i = 0; i < SLOTS; ++i) {
      const int c = (i * THREADS + tid) * 4;
      v[i] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (c < W && ok)
        v[i] = a.table ? load4(static_cast<const T*>(a.table) + src * W + c) : load4(a.rows_in + src * W + c);
    }
  }
#pragma unroll
  for (int i = 0; i < SLOTS; ++i) sum += v[i].x + v[i].y + v[i].z + v[i].w;
  const float mean = block_sum<THREADS>(sum, red) / W;
  float sq = 0.f;
#pragma unroll
  for (int i = 0; i < SLOTS; ++i) {
    const int c = (i * THREADS + tid) * 4;
    if (c < W) {
      v[i].x -= mean;
      v[i].y -= mean;
      v[i].z -= mean;
      v[i].w -= mean;
      sq += v[i].x * v[i].x + v[i].y * v[i].y + v[i].z * v[i].z + v[i].w * v[i].w;
    }
  }
  const float inv = 1.f / sqrtf(block_sum<THREADS>(sq, red) / W + a.eps);
#pragma unroll
  for (int i = 0; i < SLOTS; ++i) {
    const int c = (i * THREADS + tid) * 4;
    if (c < W) {
      const float4 g = kEarly ? early_g[i % kEarlySlots] : load4(gamma + c);
      float4 o = make_float4(v[i].x * inv * g.x, v[i].y * inv * g.y, v[i].z * inv * g.z, v[i].w * inv * g.w);
      if (a.hidden != nullptr) {
        if (a.accumulate) {
          const float4 p = kEarly ? early_h[i % kEarlySlots] : *reinterpret_cast<const float4*>(hidden + c);
          o = make_float4(p.x + o.x, p.y + o.y, p.z + o.z, p.w + o.w);
        }
        store4(hidden + c, o);
      }
      if (a.y != nullptr) store4(static_cast<T*>(a.y) + static_cast<int64_t>(row) * W + c, o);
    }
  }
}

// Any width up to kMaxWidth: the row is kept in shared memory.
template <typename T>
__global__ void __launch_bounds__(kThreads)
out_norm_any_kernel(b200_out_norm_args a) {
  extern __shared__ float row_smem[];
  __shared__ float red[kThreads / 32];
  pdl_launch_dependents();
  pdl_wait();
  const int tid = threadIdx.x;
  const int row = blockIdx.x;
  const int W = a.width;
  const T* gamma = static_cast<const T*>(a.gamma);
  int64_t src = 0;
  const bool ok = a.partials != nullptr || source_row(a, row, src);
  float sum = 0.f;
  for (int c = tid; c < W; c += kThreads) {
    float v = 0.f;
    if (a.partials != nullptr) {
      for (int s = 0; s < a.num_splits; ++s) v += a.partials[(static_cast<int64_t>(s) * a.rows + row) * W + c];
    } else if (ok) {
      v = a.table ? simt::to_f32(static_cast<const T*>(a.table)[src * W + c]) : a.rows_in[src * W + c];
    }
    row_smem[c] = v;
    sum += v;
  }
  const float mean = block_sum(sum, red) / W;
  float sq = 0.f;
  for (int c = tid; c < W; c += kThreads) {
    const float d = row_smem[c] - mean;
    sq += d * d;
  }
  const float inv = 1.f / sqrtf(block_sum(sq, red) / W + a.eps);
  for (int c = tid; c < W; c += kThreads) {
    float o = (row_smem[c] - mean) * inv * simt::to_f32(gamma[c]);
    if (a.hidden != nullptr) {
      float* h = a.hidden + static_cast<int64_t>(row) * W + c;
      if (a.accumulate) o += *h;
      *h = o;
    }
    if (a.y != nullptr) simt::store_as(static_cast<T*>(a.y) + static_cast<int64_t>(row) * W + c, o);
  }
}

template <typename T, int SLOTS, int THREADS, bool kEarly, int CTAS>
static int launch_vec(const b200_out_norm_args& a, cudaStream_t s) {
  return launch_pdl(out_norm_vec_kernel<T, SLOTS, THREADS, kEarly, CTAS>, dim3(a.rows), dim3(THREADS), 0, s, a);
}
template <typename T>
static int launch(const b200_out_norm_args& a, cudaStream_t s) {
  const bool aligned = a.width % 4 == 0 && a.width <= kMaxVecWidth && aligned16(a.partials) && aligned16(a.table) && aligned16(a.rows_in) &&
                       aligned16(a.gamma) && aligned16(a.hidden) && aligned16(a.y);
  if (aligned) {
    const int slots = (a.width + 2047) / 2048, sms = sm_count();
    if (a.width <= 1024) return launch_vec<T, 1, 256, true, 4>(a, s);
    if (slots == 1) return a.rows <= 2 * sms ? launch_vec<T, 1, 512, true, 2>(a, s) : launch_vec<T, 2, 256, true, 4>(a, s);
    // Longer rows: one on each SM; up to 3072 columns (three vectors for each of 256 threads) four; else two, or three if there are more rows than that.
    // One CTA of 1024 threads a row up to 296 rows, and 512 or 256 threads with more, had been slower there than 256 for every row (us with 1, 4 splits, that
    // first / 1024 and so on / now): 200 rows of 3072 4.3, 4.9 / 5.1, 5.9 / 3.9, 4.3; 296 of 4096 5.3, 6.1 / 5.9, 6.9 / 3.5, 4.6; 600 of 8192 13.3, 28.3 / 13.7, 32.3 /
    // 11.5, 25.3; 1200 of 4096 11.9, 22.8 / 11.9, 25.8 / 9.7, 20.6.
    if (a.rows <= sms) return slots == 2 ? launch_vec<T, 2, 512, true, 1>(a, s) : slots == 3 ? launch_vec<T, 3, 512, true, 1>(a, s) : launch_vec<T, 4, 512, true, 1>(a, s);
    if (a.width <= 3072) return launch_vec<T, 3, 256, false, 4>(a, s);
    if (a.rows <= 2 * sms) return slots == 2 ? launch_vec<T, 2, 512, true, 2>(a, s) : slots == 3 ? launch_vec<T, 3, 512, false, 2>(a, s) : launch_vec<T, 4, 512, false, 2>(a, s);
    return slots == 2 ? launch_vec<T, 2, 512, false, 3>(a, s) : slots == 3 ? launch_vec<T, 3, 512, false, 3>(a, s) : launch_vec<T, 4, 512, false, 3>(a, s);
  }
  static std::atomic<uint64_t> done{0};
  if (ensure_dynamic_smem(out_norm_any_kernel<T>, kMaxWidth * 4, done) != B200_OK) return B200_ERR_LAUNCH;
  return launch_pdl(out_norm_any_kernel<T>, dim3(a.rows), dim3(kThreads), static_cast<size_t>(a.width) * 4, s, a);
}

}  // namespace outnorm
}  // namespace b200

extern "C" {

int b200_out_norm(const b200_out_norm_args* a, b200_stream_t stream) {
  using namespace b200;
  if (!a || a->rows <= 0 || a->width <= 0 || a->width > outnorm::kMaxWidth || !a->gamma || (!a->hidden && !a->y))
    return B200_ERR_INVALID_ARGUMENT;
  const int sources = (a->partials != nullptr) + (a->table != nullptr) + (a->rows_in != nullptr);
  if (sources != 1 || (a->partials && a->num_splits < 1) || (a->table && (!a->ids || a->table_rows <= 0)) ||
      (a->rows_in && a->source_rows <= 0) || (a->accumulate && !a->hidden))
    return B200_ERR_INVALID_ARGUMENT;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  if (a->dtype == B200_DTYPE_BF16) return outnorm::launch<__nv_bfloat16>(*a, s);
  if (a->dtype == B200_DTYPE_F32) return outnorm::launch<float>(*a, s);
  return B200_ERR_INVALID_ARGUMENT;
}

}  // extern "C"
