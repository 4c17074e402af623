// Generalized delta rule: a linear recurrence per head over a [key channel] x [value channel] fp32 state.
//
//   S <- diag(w) S - (a u)(u^T S) + k v^T        o = S^T r
//
// The value channels (columns of S) do not talk to each other, so a column's state values live in the registers of NI lanes
// (I key channels each) and a token costs one fused pass: d = u . s, s = w s - (a u) d + k v, o = r . s.  The state is stored
// [head][value channel][key channel].  Everything is fp32 from the loads on, two key channels per instruction (fma.f32x2); only
// the linears' outputs (r, k, v, x_a, x_g, x_w1 / z) arrive in `dtype`.
//
//   delta_decode_kernel  one token per row; bound by reading and writing the state once.  A warp takes a (row, head) by itself (few of them: two or four warps),
//                        two columns per lane group at a time with the next two on their way; the CTA's warps - rows of one
//                        head - share W_w2's rows in shared memory.  The product with W_w2, the decay, the unit key, the head
//                        norm and the output gate are part of it.
//   delta_block_scan_kernel  rows of any length, heads of 33 to 128: one CTA per (row, head, 64 columns) walks the row's tokens four at a time.  Compute warps
//                        hold two columns on four lanes (a vector is read from shared memory once for both); other warps prepare blocks of
//                        four tokens (decays, unit key, removal vector, their products with one another) meanwhile.
//   delta_scan_kernel    the same a token at a time, a column on two lanes, for the other sizes
//   delta_finish_kernel  head norm + weight + output gate behind the scan (a head's columns may be spread over CTAs there).
#include "common.cuh"

namespace b200 {
namespace delta {

constexpr int kScanTokens = 16;  // tokens prepared at a time

__device__ __forceinline__ float sigmoid(float x) { return 1.f / (1.f + expf(-x)); }

// The same without a branch, so that several are under way together: the fast reciprocal and one Newton-Raphson step, r (2 - y r), which is as close as the
// division (6e-8).  Below e^-80 it stays there.
__device__ __forceinline__ float sigmoid_in_line(float x) {
  const float y = 1.f + expf(-x > 80.f ? 80.f : -x), r = __fdividef(1.f, y);
  return fmaf(r, fmaf(-y, r, 1.f), r);
}

// For output gates: fp32 arithmetic with the fast exponential and division (about 1e-6 relative).
__device__ __forceinline__ float gate_sigmoid(float x) { return __fdividef(1.f, 1.f + __expf(-x)); }

template <int NI, int STRIDE = 1>
__device__ __forceinline__ float lane_sum(float v) {  // over the NI lanes of a column, STRIDE lanes apart
#pragma unroll
  for (int o = NI / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o * STRIDE);
  return v;
}

// Two fp32 values in one 64-bit register.
using f32x2 = unsigned long long;
__device__ __forceinline__ f32x2 pack2(float lo, float hi) {
  f32x2 v;
  asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(lo), "f"(hi));
  return v;
}
__device__ __forceinline__ float sum2(f32x2 v) {
  float lo, hi;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
  return lo + hi;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
  f32x2 d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
  f32x2 d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
  f32x2 d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ void unpack2(f32x2 v, float& lo, float& hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v)); }

// Lane `ni` of the NI lanes of a column owns key channels (q * NI + ni) * 4 + e, q = 0 .. I / 4 - 1, e = 0 .. 3: 16-byte
// pieces, neighbouring lanes adjacent.
template <int NI, int I>
__device__ __forceinline__ void load_column(const float* col, int dim, int ni, bool full, f32x2 (&s)[I / 2]) {
#pragma unroll
  for (int q = 0; q < I / 4; ++q) {
    const int i = (q * NI + ni) * 4;
    if (full) {
      const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(col + i);
      s[q * 2] = v.x;
      s[q * 2 + 1] = v.y;
    } else {
      float x[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) x[e] = i + e < dim ? col[i + e] : 0.f;
      s[q * 2] = pack2(x[0], x[1]);
      s[q * 2 + 1] = pack2(x[2], x[3]);
    }
  }
}
template <int NI, int I>
__device__ __forceinline__ void store_column(float* col, int dim, int ni, bool full, const f32x2 (&s)[I / 2]) {
#pragma unroll
  for (int q = 0; q < I / 4; ++q) {
    const int i = (q * NI + ni) * 4;
    if (full) {
      *reinterpret_cast<ulonglong2*>(col + i) = make_ulonglong2(s[q * 2], s[q * 2 + 1]);
    } else {
      float x[4];
      asm("mov.b64 {%0, %1}, %2;" : "=f"(x[0]), "=f"(x[1]) : "l"(s[q * 2]));
      asm("mov.b64 {%0, %1}, %2;" : "=f"(x[2]), "=f"(x[3]) : "l"(s[q * 2 + 1]));
#pragma unroll
      for (int e = 0; e < 4; ++e)
        if (i + e < dim) col[i + e] = x[e];
    }
  }
}

struct TokenVectors {  // shared-memory vectors of one token, each [DIM]
  const float *r, *w, *k, *u, *au;
};
__device__ __forceinline__ ulonglong2 piece(const float* p) { return *reinterpret_cast<const ulonglong2*>(p); }

// One token on N columns: `o` gets this lane's part of each column's output (the caller sums it over the NI lanes).  The
// vectors are read once for all columns.
template <int NI, int I, int N, int STRIDE = 1>
__device__ __forceinline__ void step(f32x2 (&s)[N][I / 2], const TokenVectors& tv, const float (&v)[N], int ni, float (&o)[N]) {
  f32x2 nd[N], acc[N][2];
#pragma unroll
  for (int n = 0; n < N; ++n) acc[n][0] = acc[n][1] = 0ull;
#pragma unroll
  for (int q = 0; q < I / 4; ++q) {
    const ulonglong2 u = piece(tv.u + (q * NI + ni) * 4);
#pragma unroll
    for (int n = 0; n < N; ++n) {
      acc[n][0] = fma2(u.x, s[n][q * 2], acc[n][0]);
      acc[n][1] = fma2(u.y, s[n][q * 2 + 1], acc[n][1]);
    }
  }
#pragma unroll
  for (int n = 0; n < N; ++n) {
    const float d = -lane_sum<NI, STRIDE>(sum2(acc[n][0]) + sum2(acc[n][1]));
    nd[n] = pack2(d, d);
    acc[n][0] = acc[n][1] = 0ull;
  }
  f32x2 vv[N];
#pragma unroll
  for (int n = 0; n < N; ++n) vv[n] = pack2(v[n], v[n]);
#pragma unroll
  for (int q = 0; q < I / 4; ++q) {
    const int i = (q * NI + ni) * 4;
    const ulonglong2 w = piece(tv.w + i), k = piece(tv.k + i), au = piece(tv.au + i), r = piece(tv.r + i);
#pragma unroll
    for (int n = 0; n < N; ++n) {
      f32x2& x = s[n][q * 2];
      f32x2& y = s[n][q * 2 + 1];
      x = fma2(au.x, nd[n], fma2(w.x, x, mul2(k.x, vv[n])));
      y = fma2(au.y, nd[n], fma2(w.y, y, mul2(k.y, vv[n])));
      acc[n][0] = fma2(r.x, x, acc[n][0]);
      acc[n][1] = fma2(r.y, y, acc[n][1]);
    }
  }
#pragma unroll
  for (int n = 0; n < N; ++n) o[n] = sum2(acc[n][0]) + sum2(acc[n][1]);
}

// ---------------------------------------------------------------------------------------------------------------
// Decode
// ---------------------------------------------------------------------------------------------------------------
template <int DIM>
struct DecodeShape {
  static constexpr int kI = 16;
  static constexpr int NI = DIM / kI;
  static constexpr int kGroups = 32 / NI;  // columns side by side in a warp
  static constexpr int kCols = 2;          // columns per lane group and pass
  static constexpr int kPasses = DIM / (kGroups * kCols);
  static constexpr int kWarps = DIM <= 64 ? 8 : 4;
  static constexpr int kElems = DIM / 32;  // vector entries per lane
};

// 16 bytes of W_w2 times 16 / sizeof(T) entries of tanh(x_w1).
__device__ __forceinline__ float dot16(const __nv_bfloat16* w, const float* l, float z) {
  const uint4 x = *reinterpret_cast<const uint4*>(w);
  const float4 a = *reinterpret_cast<const float4*>(l), b = *reinterpret_cast<const float4*>(l + 4);
  z = fmaf(bf16_lo(x.x), a.x, z);
  z = fmaf(bf16_hi(x.x), a.y, z);
  z = fmaf(bf16_lo(x.y), a.z, z);
  z = fmaf(bf16_hi(x.y), a.w, z);
  z = fmaf(bf16_lo(x.z), b.x, z);
  z = fmaf(bf16_hi(x.z), b.y, z);
  z = fmaf(bf16_lo(x.w), b.z, z);
  return fmaf(bf16_hi(x.w), b.w, z);
}
__device__ __forceinline__ float dot16(const float* w, const float* l, float z) {
  const float4 x = *reinterpret_cast<const float4*>(w), a = *reinterpret_cast<const float4*>(l);
  return fmaf(x.w, a.w, fmaf(x.z, a.z, fmaf(x.y, a.y, fmaf(x.x, a.x, z))));
}

// Shared memory: per warp six vectors [DIM] and tanh(x_w1) [rank, rounded up]; then W_w2's rows of the head.
// PARTS warps share a (row, head): each takes every PARTS-th pass over the columns, and all prepare the token.
template <typename T, int DIM, int PARTS>
__global__ void __launch_bounds__(DecodeShape<DIM>::kWarps * 32, DIM <= 64 ? 1 : 2)
delta_decode_kernel(b200_delta_args a, int w2_stride) {
  using D = DecodeShape<DIM>;
  constexpr int NI = D::NI, I = D::kI, N = D::kCols, EL = D::kElems, VEC = 16 / sizeof(T);
  extern __shared__ __align__(16) float dyn[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  constexpr int kPasses = D::kPasses / PARTS;  // of a warp
  static_assert(D::kPasses % PARTS == 0 && (kPasses == 1 || kPasses % 2 == 0), "");
  const int head = blockIdx.x, dim = a.dim, row = blockIdx.y * (D::kWarps / PARTS) + warp / PARTS, part = warp % PARTS;
  __shared__ float part_sq[D::kWarps];
  const bool full = dim == DIM;
  const int rank_pad = (a.rank + 3) / 4 * 4;
  float* vec = dyn + warp * (6 * DIM);  // r, w, k, u, a u, v (later o)
  float* lora = dyn + D::kWarps * 6 * DIM + warp * rank_pad;
  T* w2_s = reinterpret_cast<T*>(dyn + D::kWarps * (6 * DIM + rank_pad));
  pdl_launch_dependents();
  const int in = row < a.num_rows ? a.state_in[row] : -1, out = row < a.num_rows ? a.state_out[row] : -1;
  const T* w2 = static_cast<const T*>(a.w2) + static_cast<int64_t>(head) * dim * a.rank;
  if (w2_stride > 0) {  // whole 16-byte pieces, straight to shared memory
    const int per_row = a.rank / VEC;
    for (int i = tid; i < dim * per_row; i += D::kWarps * 32) {
      const int r = i / per_row, c = i - r * per_row;
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(w2_s + r * w2_stride + c * VEC)),
                   "l"(w2 + static_cast<int64_t>(r) * a.rank + c * VEC)
                   : "memory");
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  const bool has_in = static_cast<unsigned>(in) < static_cast<unsigned>(a.state_slots);
  const bool live = static_cast<unsigned>(out) < static_cast<unsigned>(a.state_slots);
  const int64_t head_elems = static_cast<int64_t>(dim) * dim;
  const int ni = lane % NI, group = lane / NI;
  const float* src = a.state + (static_cast<int64_t>(has_in ? in : 0) * a.heads + head) * head_elems;
  float* dst_state = a.state + (static_cast<int64_t>(live ? out : 0) * a.heads + head) * head_elems;
  auto fetch = [&](f32x2 (&s)[N][I / 2], int pass) {
#pragma unroll
    for (int n = 0; n < N; ++n) {
      const int j = (pass * N + n) * D::kGroups + group;
      if (has_in && live && j < dim) {
        load_column<NI, I>(src + j * dim, dim, ni, full, s[n]);
      } else {
#pragma unroll
        for (int e = 0; e < I / 2; ++e) s[n][e] = 0ull;
      }
    }
  };
  // The state was written by an earlier step (steps are separated by copies on the stream): fetch it before the wait.
  f32x2 cur[N][I / 2], ahead[N][I / 2];
  fetch(cur, part);
  float bias_w[EL], bias_a[EL], norm[EL];
#pragma unroll
  for (int e = 0; e < EL; ++e) {
    const int i = head * dim + min(lane + e * 32, dim - 1);
    bias_w[e] = simt::to_f32(static_cast<const T*>(a.decay_bias)[i]);
    bias_a[e] = simt::to_f32(static_cast<const T*>(a.removal_bias)[i]);
    norm[e] = simt::to_f32(static_cast<const T*>(a.norm_weight)[i]);
  }
  pdl_wait();
  const int64_t hd = static_cast<int64_t>(a.heads) * dim;
  const T* p = static_cast<const T*>(a.proj) + static_cast<int64_t>(min(row, a.num_rows - 1)) * a.proj_ld;
  T xr[EL], xk[EL], xa[EL], xg[EL], xv[EL], xl[4];
#pragma unroll
  for (int e = 0; e < 4; ++e) xl[e] = p[a.off_w1 + min(lane + e * 32, a.rank - 1)];
#pragma unroll
  for (int e = 0; e < EL; ++e) {  // clamped addresses: no branches, all loads in flight together
    const int i = head * dim + min(lane + e * 32, dim - 1);
    xr[e] = p[a.off_r + i];
    xk[e] = p[a.off_k + i];
    xv[e] = p[a.off_v + i];
    xa[e] = p[a.off_a + i];
    xg[e] = p[a.off_g + i];
  }
  if (kPasses > 1) fetch(ahead, part + PARTS);
#pragma unroll
  for (int e = 0; e < 4; ++e)
    if (lane + e * 32 < a.rank) lora[lane + e * 32] = tanhf(simt::to_f32(xl[e]));
  for (int r = lane + 128; r < a.rank; r += 32) lora[r] = tanhf(simt::to_f32(p[a.off_w1 + r]));
  float k[EL], ksq = 0.f;
#pragma unroll
  for (int e = 0; e < EL; ++e) {
    k[e] = lane + e * 32 < dim ? simt::to_f32(xk[e]) : 0.f;
    ksq += k[e] * k[e];
  }
  const float unit = 1.f / sqrtf(warp_sum(ksq) + a.unit_eps);
  if (w2_stride > 0) asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();  // W_w2's rows (and, within the warp, lora)
  // z = W_w2 tanh(x_w1): a lane per key channel
  float z[EL];
#pragma unroll
  for (int e = 0; e < EL; ++e) z[e] = 0.f;
  if (w2_stride > 0) {
#pragma unroll 2
    for (int r = 0; r < a.rank; r += VEC)
#pragma unroll
      for (int e = 0; e < EL; ++e) z[e] = dot16(w2_s + min(lane + e * 32, dim - 1) * w2_stride + r, lora + r, z[e]);
  } else {
    for (int r = 0; r < a.rank; ++r)
#pragma unroll
      for (int e = 0; e < EL; ++e)
        z[e] = fmaf(simt::to_f32(w2[static_cast<int64_t>(min(lane + e * 32, dim - 1)) * a.rank + r]), lora[r], z[e]);
  }
#pragma unroll
  for (int e = 0; e < EL; ++e) {
    const int i = lane + e * 32;
    const bool ok = i < dim;
    const float u = k[e] * unit;
    vec[i] = ok ? simt::to_f32(xr[e]) : 0.f;
    vec[DIM + i] = ok ? expf(-a.decay_scale * sigmoid(z[e] + bias_w[e])) : 0.f;
    vec[2 * DIM + i] = k[e];
    vec[3 * DIM + i] = u;
    vec[4 * DIM + i] = u * sigmoid(simt::to_f32(xa[e]) + bias_a[e]);
    vec[5 * DIM + i] = simt::to_f32(xv[e]);
  }
  __syncwarp();
  if (row >= a.num_rows) return;
  const TokenVectors tv{vec, vec + DIM, vec + 2 * DIM, vec + 3 * DIM, vec + 4 * DIM};
  float osq = 0.f;
  auto run = [&](f32x2 (&s)[N][I / 2], int pass) {
    float v[N], o[N];
#pragma unroll
    for (int n = 0; n < N; ++n) v[n] = vec[5 * DIM + (pass * N + n) * D::kGroups + group];
    step<NI, I, N>(s, tv, v, ni, o);
#pragma unroll
    for (int n = 0; n < N; ++n) {
      const int j = (pass * N + n) * D::kGroups + group;
      o[n] = lane_sum<NI>(o[n]);
      if (j < dim) {
        if (live) store_column<NI, I>(dst_state + j * dim, dim, ni, full, s[n]);
        if (ni == 0) {
          vec[5 * DIM + j] = o[n];  // (only this lane group has read the value there)
          osq += o[n] * o[n];
        }
      }
    }
  };
  if constexpr (kPasses == 1) {
    run(cur, part);
  } else {
#pragma unroll 1
    for (int k = 0; k < kPasses; k += 2) {
      run(cur, part + k * PARTS);
      if (k + 2 < kPasses) fetch(cur, part + (k + 2) * PARTS);
      run(ahead, part + (k + 1) * PARTS);
      if (k + 3 < kPasses) fetch(ahead, part + (k + 3) * PARTS);
    }
  }
  osq = warp_sum(osq);
  if constexpr (PARTS > 1) {
    if (lane == 0) part_sq[warp] = osq;
    asm volatile("bar.sync %0, %1;" ::"r"(1 + warp / PARTS), "r"(32 * PARTS) : "memory");  // the warps of the row
    osq = 0.f;
#pragma unroll
    for (int k = 0; k < PARTS; ++k) osq += part_sq[warp - part + k];
  }
  const float inv = 1.f / sqrtf(osq / dim + a.eps);
  __syncwarp();
  T* dst = static_cast<T*>(a.out) + row * hd + head * dim;
#pragma unroll
  for (int e = 0; e < EL; ++e) {
    const int i = lane + e * 32;
    if (e % PARTS != part) continue;
    const int owner = i / (D::kGroups * N) % PARTS;  // the warp that had the column
    if (i < dim) simt::store_as(dst + i, live ? vec[(owner - part) * 6 * DIM + 5 * DIM + i] * inv * norm[e] * gate_sigmoid(simt::to_f32(xg[e])) : 0.f);
  }
}

// ---------------------------------------------------------------------------------------------------------------
// Scan
// ---------------------------------------------------------------------------------------------------------------
// The k-th longest row.  A row's tokens are one chain, so the longest rows end last: their CTAs start first and get an SM of their own, the shortest
// rows share what is left.  (Warp-collective; more than 32 rows are taken as they come.  A row whose tokens end before they start counts as an empty one:
// any row is in front of the lanes that have none.)
__device__ __forceinline__ int longest_first(const int32_t* cu_tokens, int rows, int k) {
  if (rows > 32) return k;
  const int lane = threadIdx.x & 31, len = lane < rows ? max(cu_tokens[lane + 1] - cu_tokens[lane], 0) : -1;
  int rank = 0;
#pragma unroll
  for (int j = 0; j < 32; ++j) {
    const int other = __shfl_sync(0xffffffffu, len, j);
    rank += other > len || (other == len && j < lane);
  }
  return __ffs(__ballot_sync(0xffffffffu, rank == k)) - 1;
}

template <int DIM, int COLS, int LANES>
struct ScanShape {  // COLS columns per CTA, LANES lanes for each
  static constexpr int I = DIM / LANES;
  static constexpr int NI = LANES;  // 32 / NI apart: neighbouring lanes read one address
  static constexpr int kStride = 32 / NI;
  static constexpr int kComputeThreads = COLS * NI;
  static constexpr int kComputeWarps = kComputeThreads / 32;
  static constexpr int kPrepWarps = kComputeWarps < 2 ? 2 : kComputeWarps;
  static constexpr int kThreads = kComputeThreads + kPrepWarps * 32;
  static constexpr int kTokPerWarp = kScanTokens / kPrepWarps;  // tokens one warp prepares
  static constexpr int kBatch = kTokPerWarp < 4 ? kTokPerWarp : 4;  // of which this many at a time
  static constexpr int kElems = DIM / 32;                       // key channels per lane while preparing
  static_assert(kComputeThreads % 32 == 0 && kScanTokens % kPrepWarps == 0 && kTokPerWarp % kBatch == 0 && DIM % 32 == 0, "");
  static constexpr int kBufFloats = kScanTokens * (5 * DIM + COLS);
  static constexpr int kSmemBytes = 2 * kBufFloats * 4;
};

template <typename T, int DIM, int COLS, int LANES>
__global__ void __launch_bounds__(ScanShape<DIM, COLS, LANES>::kThreads)
delta_scan_kernel(b200_delta_args a) {
  using Sh = ScanShape<DIM, COLS, LANES>;
  constexpr int NI = Sh::NI, I = Sh::I, EL = Sh::kElems, VL = (COLS + 31) / 32;
  extern __shared__ __align__(16) float smem[];
  const int tid = threadIdx.x, lane = tid & 31;
  const int dim = a.dim;
  const int col_blocks = (dim + COLS - 1) / COLS;
  const int head = blockIdx.x / col_blocks, cb = blockIdx.x - head * col_blocks;
  const int row = longest_first(a.cu_tokens, a.num_rows, blockIdx.y);
  pdl_launch_dependents();
  const int t_begin = a.cu_tokens[row], n_tok = min(a.cu_tokens[row + 1], a.num_tokens) - t_begin;
  pdl_wait();
  if (n_tok <= 0) return;
  const int64_t hd = static_cast<int64_t>(a.heads) * dim;
  const int chunks = (n_tok + kScanTokens - 1) / kScanTokens;

  if (tid >= Sh::kComputeThreads) {
    // ------------------------------- preparing warps -------------------------------
    const int warp = (tid - Sh::kComputeThreads) >> 5;
    const T* proj = static_cast<const T*>(a.proj);
    const T* zin = static_cast<const T*>(a.z);
    float bias_w[EL], bias_a[EL];
#pragma unroll
    for (int e = 0; e < EL; ++e) {
      const int i = head * dim + min(lane + e * 32, dim - 1);
      bias_w[e] = simt::to_f32(static_cast<const T*>(a.decay_bias)[i]);
      bias_a[e] = simt::to_f32(static_cast<const T*>(a.removal_bias)[i]);
    }
    for (int c = 0; c < chunks; ++c) {
      float* buf = smem + (c & 1) * Sh::kBufFloats;
#pragma unroll 1
      for (int q0 = 0; q0 < Sh::kTokPerWarp; q0 += Sh::kBatch) {
        // addresses are clamped, so that the loads need no branches and are all in flight together
        T xr[Sh::kBatch][EL], xk[Sh::kBatch][EL], xa[Sh::kBatch][EL], xz[Sh::kBatch][EL], xv[Sh::kBatch][VL];
#pragma unroll
        for (int q = 0; q < Sh::kBatch; ++q) {
          const int64_t t = t_begin + min(c * kScanTokens + warp * Sh::kTokPerWarp + q0 + q, n_tok - 1);
          const T* p = proj + t * a.proj_ld + head * dim;
          const T* z = zin + t * hd + head * dim;
#pragma unroll
          for (int e = 0; e < EL; ++e) {
            const int i = min(lane + e * 32, dim - 1);
            xr[q][e] = p[a.off_r + i];
            xk[q][e] = p[a.off_k + i];
            xa[q][e] = p[a.off_a + i];
            xz[q][e] = z[i];
          }
#pragma unroll
          for (int e = 0; e < VL; ++e) xv[q][e] = p[a.off_v + min(cb * COLS + lane + e * 32, dim - 1)];
        }
#pragma unroll
        for (int q = 0; q < Sh::kBatch; ++q) {
          const int tt = warp * Sh::kTokPerWarp + q0 + q;
          float ksq = 0.f, k[EL];
#pragma unroll
          for (int e = 0; e < EL; ++e) {
            k[e] = lane + e * 32 < dim ? simt::to_f32(xk[q][e]) : 0.f;
            ksq += k[e] * k[e];
          }
          const float unit = 1.f / sqrtf(warp_sum(ksq) + a.unit_eps);
#pragma unroll
          for (int e = 0; e < EL; ++e) {
            const int i = lane + e * 32;
            float* b = buf + tt * 5 * DIM + i;
            const float u = k[e] * unit;
            b[0] = i < dim ? simt::to_f32(xr[q][e]) : 0.f;
            b[DIM] = i < dim ? expf(-a.decay_scale * sigmoid(simt::to_f32(xz[q][e]) + bias_w[e])) : 0.f;
            b[2 * DIM] = k[e];
            b[3 * DIM] = u;
            b[4 * DIM] = u * sigmoid(simt::to_f32(xa[q][e]) + bias_a[e]);
          }
#pragma unroll
          for (int e = 0; e < VL; ++e)
            if (lane + e * 32 < COLS) buf[kScanTokens * 5 * DIM + tt * COLS + lane + e * 32] = simt::to_f32(xv[q][e]);
        }
      }
      __syncthreads();  // chunk c is ready, chunk c - 1 has been read: its buffer is free
    }
    __syncthreads();
    return;
  }

  // --------------------------------- compute warps ---------------------------------
  const bool full = dim == DIM;
  const int in = a.state_in[row], out = a.state_out[row];
  const int64_t head_elems = static_cast<int64_t>(dim) * dim;
  constexpr int ST = Sh::kStride;
  const int ni = lane / ST, group = (tid >> 5) * ST + lane % ST, col = cb * COLS + group;  // this thread's column
  f32x2 s[1][I / 2];
  if (static_cast<unsigned>(in) < static_cast<unsigned>(a.state_slots) && col < dim) {
    load_column<NI, I>(a.state + (static_cast<int64_t>(in) * a.heads + head) * head_elems + static_cast<int64_t>(col) * dim, dim, ni, full, s[0]);
  } else {
#pragma unroll
    for (int e = 0; e < I / 2; ++e) s[0][e] = 0ull;
  }
  float* o_dst = a.o_f32 + static_cast<int64_t>(t_begin) * hd + head * dim + col;
  __syncthreads();  // chunk 0 is ready
  for (int c = 0; c < chunks; ++c) {
    const float* buf = smem + (c & 1) * Sh::kBufFloats;
    const float* values = buf + kScanTokens * 5 * DIM + group;
    const int cnt = min(kScanTokens, n_tok - c * kScanTokens);
#pragma unroll 1  // (256 channels fill the registers, 32 have nothing to hide)
    for (int tt = 0; tt < cnt; ++tt) {
      const float* v0 = buf + tt * 5 * DIM;
      const TokenVectors tv{v0, v0 + DIM, v0 + 2 * DIM, v0 + 3 * DIM, v0 + 4 * DIM};
      const float v[1] = {values[tt * COLS]};
      float o[1];
      step<NI, I, 1, ST>(s, tv, v, ni, o);
      const float sum = lane_sum<NI, ST>(o[0]);
      if (ni == 0 && col < dim) *o_dst = sum;
      o_dst += hd;
    }
    __syncthreads();  // chunk c has been read, chunk c + 1 is ready
  }
  if (static_cast<unsigned>(out) < static_cast<unsigned>(a.state_slots) && col < dim)
    store_column<NI, I>(a.state + (static_cast<int64_t>(out) * a.heads + head) * head_elems + static_cast<int64_t>(col) * dim, dim, ni, full, s[0]);
}

// ---------------------------------------------------------------------------------------------------------------
// Scan, four tokens at a time
// ---------------------------------------------------------------------------------------------------------------
// With S the state in front of four tokens and w[a..b] the product of their decays, what token j removes and reads is
//
//   d_j = (u_j w[0..j-1]) . S + sum_(s<j)  (u_j . k_s w[s+1..j-1]) v_s - (u_j . a_s u_s w[s+1..j-1]) d_s
//   o_j = (r_j w[0..j]) . S   + sum_(s<=j) (r_j . k_s w[s+1..j]) v_s   - (r_j . a_s u_s w[s+1..j]) d_s
//   S  <- w[0..3] S + sum_s (k_s w[s+1..3]) v_s - (a_s u_s w[s+1..3]) d_s
//
// so one pass over a column's registers gives all eight dot products with S and one more all four updates: one lane sum in the chain for four tokens instead
// of four.  Decays are only ever multiplied, never divided by, so nothing grows however small they are.
// A row is a chain of tokens; what bounds one is what its SM can do for a token.  2048 tokens, 32 heads of 64: 506 us a token at a time, 372 now; the compute
// warps alone take 297 (84 16-byte reads of shared memory and 272 packed multiply-adds for each block and warp), the preparing ones 250 (mostly the exponentials;
// with a branch in the sigmoids' divisions 338).  Products of 16 tokens on mma.sync in three bf16 terms need as many instructions to prepare: 388 to 403 us.
constexpr int kBlockTokens = 4;
// Of a block, in floats: u w[0..j-1], r w[0..j], k w[s+1..3], a u w[s+1..3] of its tokens and w[0..3], each [DIM]; the values [4][COLS]; the products of the
// tokens with one another, four matrices [4][4] (j, s): u.k, u.au (zero where s >= j), r.k, r.au (zero where s > j).
template <int DIM, int COLS, int BLOCKS>
struct BlockShape {
  static constexpr int kU = 0, kR = 4 * DIM, kK = 8 * DIM, kB = 12 * DIM, kW = 16 * DIM, kV = 17 * DIM, kPairs = kV + 4 * COLS;
  static constexpr int kFloats = kPairs + 64;
  static constexpr int NI = 4, N = 2, I = DIM / NI, kStride = 32 / NI;
  static constexpr int kGroups = COLS / N, kComputeThreads = kGroups * NI, kComputeWarps = kComputeThreads / 32;
  static constexpr int kTokens = BLOCKS * kBlockTokens, kBlocks = BLOCKS, kPrepWarps = kBlocks, kThreads = kComputeThreads + kPrepWarps * 32;
  static constexpr int kElems = DIM / 32, kValues = COLS / 32;
  static constexpr int kSmemBytes = 2 * kBlocks * kFloats * 4;
  static_assert(COLS % 32 == 0 && DIM % 32 == 0 && kFloats % 4 == 0, "");
};

// Sums of N values over the warp, that of value i in lane i (and N, 2 N, ... further on).
template <int N>
__device__ __forceinline__ float transposed_sum(float (&v)[N], int lane) {
#pragma unroll
  for (int o = N / 2; o > 0; o >>= 1)
#pragma unroll
    for (int i = 0; i < o; ++i) {
      const bool high = lane & o;
      const float give = high ? v[i] : v[i + o], keep = high ? v[i + o] : v[i];
      v[i] = keep + __shfl_xor_sync(0xffffffffu, give, o);
    }
#pragma unroll
  for (int o = N; o < 32; o <<= 1) v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
  return v[0];
}

// o += a b where `p`, one predicated multiply-add.  (Selected operands make a block 2 % longer, 2048 tokens x 32 heads of 64 371 -> 381 us; branches 25 %.)
__device__ __forceinline__ void add_if(bool p, float& o, float a, float b) {
  asm("{ .reg .pred p; setp.ne.s32 p, %3, 0; @p fma.rn.f32 %0, %1, %2, %0; }" : "+f"(o) : "f"(a), "f"(b), "r"(static_cast<int>(p)));
}

template <typename T, int DIM, int COLS, int BLOCKS>
__global__ void __launch_bounds__(BlockShape<DIM, COLS, BLOCKS>::kThreads)
delta_block_scan_kernel(b200_delta_args a) {
  using Sh = BlockShape<DIM, COLS, BLOCKS>;
  constexpr int NI = Sh::NI, I = Sh::I, N = Sh::N, EL = Sh::kElems, VL = Sh::kValues, J = kBlockTokens;
  extern __shared__ __align__(16) float smem[];
  const int tid = threadIdx.x, lane = tid & 31;
  const int dim = a.dim;
  const int col_blocks = (dim + COLS - 1) / COLS;
  const int head = blockIdx.x / col_blocks, cb = blockIdx.x - head * col_blocks;
  const int row = longest_first(a.cu_tokens, a.num_rows, blockIdx.y);
  pdl_launch_dependents();
  const int t_begin = a.cu_tokens[row], n_tok = min(a.cu_tokens[row + 1], a.num_tokens) - t_begin;
  pdl_wait();
  if (n_tok <= 0) return;
  const int64_t hd = static_cast<int64_t>(a.heads) * dim;
  const int chunks = (n_tok + Sh::kTokens - 1) / Sh::kTokens;

  if (tid >= Sh::kComputeThreads) {
    // ------------------------------- preparing warps: a block each -------------------------------
    const int warp = (tid - Sh::kComputeThreads) >> 5;
    const T* proj = static_cast<const T*>(a.proj) + head * dim;
    const T* zin = static_cast<const T*>(a.z) + head * dim;
    float bias_w[EL], bias_a[EL];
    int at[EL], col[VL];  // clamped, so that the loads need no branches and are all in flight together
#pragma unroll
    for (int e = 0; e < EL; ++e) {
      at[e] = min(lane + e * 32, dim - 1);
      bias_w[e] = simt::to_f32(static_cast<const T*>(a.decay_bias)[head * dim + at[e]]);
      bias_a[e] = simt::to_f32(static_cast<const T*>(a.removal_bias)[head * dim + at[e]]);
    }
#pragma unroll
    for (int e = 0; e < VL; ++e) col[e] = min(cb * COLS + lane + e * 32, dim - 1);
    // Where this lane's product of two tokens goes: (j, s) of s < j first u.k, then u.au, of s <= j then r.k, then r.au.
    int place = 0;
    {
      int i = 0;
#pragma unroll
      for (int m = 0; m < 4; ++m)
#pragma unroll
        for (int j = 0; j < J; ++j)
#pragma unroll
          for (int s = 0; s < J; ++s)
            if (m < 2 ? s < j : s <= j) {
              if (i == lane) place = (m * J + j) * J + s;
              ++i;
            }
    }
    for (int i = lane; i < 2 * 64; i += 32) smem[((i / 64) * Sh::kBlocks + warp) * Sh::kFloats + Sh::kPairs + i % 64] = 0.f;
    __syncwarp();
    T xr[J][EL], xk[J][EL], xa[J][EL], xz[J][EL], xv[J][VL];
    auto fetch = [&](int c) {
#pragma unroll
      for (int q = 0; q < J; ++q) {
        const int64_t t = t_begin + min(c * Sh::kTokens + warp * J + q, n_tok - 1);
        const T* p = proj + t * a.proj_ld;
        const T* z = zin + t * hd;
#pragma unroll
        for (int e = 0; e < EL; ++e) {
          xr[q][e] = p[a.off_r + at[e]];
          xk[q][e] = p[a.off_k + at[e]];
          xa[q][e] = p[a.off_a + at[e]];
          xz[q][e] = z[at[e]];
        }
#pragma unroll
        for (int e = 0; e < VL; ++e) xv[q][e] = p[a.off_v + col[e]];
      }
    };
    fetch(0);
    for (int c = 0; c < chunks; ++c) {
      float* buf = smem + ((c & 1) * Sh::kBlocks + warp) * Sh::kFloats + lane;
      float r[J][EL], w[J][EL], k[J][EL], u[J][EL], au[J][EL], sums[J];
#pragma unroll
      for (int q = 0; q < J; ++q) {
        const bool live = c * Sh::kTokens + warp * J + q < n_tok;  // (past the end: nothing is written, nothing decays)
        float ksq = 0.f;
#pragma unroll
        for (int e = 0; e < EL; ++e) {
          const bool ok = live && lane + e * 32 < dim;
          k[q][e] = ok ? simt::to_f32(xk[q][e]) : 0.f;
          r[q][e] = ok ? simt::to_f32(xr[q][e]) : 0.f;
          ksq += k[q][e] * k[q][e];
        }
        sums[q] = warp_sum(ksq);
#pragma unroll
        for (int e = 0; e < EL; ++e) {
          w[q][e] = live ? expf(-a.decay_scale * sigmoid_in_line(simt::to_f32(xz[q][e]) + bias_w[e])) : 1.f;
          au[q][e] = sigmoid_in_line(simt::to_f32(xa[q][e]) + bias_a[e]);
        }
#pragma unroll
        for (int e = 0; e < VL; ++e) buf[Sh::kV + q * COLS + e * 32] = live ? simt::to_f32(xv[q][e]) : 0.f;
      }
      if (c + 1 < chunks) fetch(c + 1);
      // One root and one division for the four tokens, a lane each.
      const float root = 1.f / sqrtf((lane & 2 ? lane & 1 ? sums[3] : sums[2] : lane & 1 ? sums[1] : sums[0]) + a.unit_eps);
#pragma unroll
      for (int q = 0; q < J; ++q) {
        const bool live = c * Sh::kTokens + warp * J + q < n_tok;  // (past the end: zeros whatever the root of unit_eps is)
        const float unit = __shfl_sync(0xffffffffu, root, q);
#pragma unroll
        for (int e = 0; e < EL; ++e) {
          u[q][e] = live ? k[q][e] * unit : 0.f;
          au[q][e] = live ? au[q][e] * u[q][e] : 0.f;
        }
      }
      float pairs[32];
      {
        // k and a u of token s on their way through the decays behind it
        float kk[J][EL], bb[J][EL];
#pragma unroll
        for (int s = 0; s < J; ++s)
#pragma unroll
          for (int e = 0; e < EL; ++e) {
            kk[s][e] = k[s][e];
            bb[s][e] = au[s][e];
          }
#pragma unroll
        for (int j = 0; j < J; ++j)
#pragma unroll
          for (int s = 0; s <= j; ++s) {
            float uk = 0.f, ub = 0.f, rk = 0.f, rb = 0.f;
#pragma unroll
            for (int e = 0; e < EL; ++e) {
              if (s < j) {
                uk = fmaf(u[j][e], kk[s][e], uk);
                ub = fmaf(u[j][e], bb[s][e], ub);
                kk[s][e] *= w[j][e];
                bb[s][e] *= w[j][e];
              }
              rk = fmaf(r[j][e], kk[s][e], rk);
              rb = fmaf(r[j][e], bb[s][e], rb);
            }
            if (s < j) {
              pairs[j * (j - 1) / 2 + s] = uk;
              pairs[6 + j * (j - 1) / 2 + s] = ub;
            }
            pairs[12 + j * (j + 1) / 2 + s] = rk;
            pairs[22 + j * (j + 1) / 2 + s] = rb;
          }
#pragma unroll
        for (int s = 0; s < J; ++s)
#pragma unroll
          for (int e = 0; e < EL; ++e) {
            buf[Sh::kK + s * DIM + e * 32] = kk[s][e];
            buf[Sh::kB + s * DIM + e * 32] = bb[s][e];
          }
      }
#pragma unroll
      for (int e = 0; e < EL; ++e) {
        float p = w[0][e];
        buf[Sh::kU + e * 32] = u[0][e];
        buf[Sh::kR + e * 32] = r[0][e] * p;
#pragma unroll
        for (int j = 1; j < J; ++j) {
          buf[Sh::kU + j * DIM + e * 32] = u[j][e] * p;
          p *= w[j][e];
          buf[Sh::kR + j * DIM + e * 32] = r[j][e] * p;
        }
        buf[Sh::kW + e * 32] = p;
      }
      const float sum = transposed_sum<32>(pairs, lane);
      buf[Sh::kPairs - lane + place] = sum;
      __syncthreads();  // chunk c is ready, chunk c - 1 has been read: its buffer is free
    }
    __syncthreads();
    return;
  }

  // --------------------------------- compute warps ---------------------------------
  const bool full = dim == DIM;
  const int in = a.state_in[row], out = a.state_out[row];
  const int64_t head_elems = static_cast<int64_t>(dim) * dim;
  constexpr int ST = Sh::kStride;
  const int ni = lane / ST, group = (tid >> 5) * ST + lane % ST;  // this thread's columns: cb * COLS + n * kGroups + group
  f32x2 s[N][I / 2];
#pragma unroll
  for (int n = 0; n < N; ++n) {
    const int j = cb * COLS + n * Sh::kGroups + group;
    if (static_cast<unsigned>(in) < static_cast<unsigned>(a.state_slots) && j < dim) {
      load_column<NI, I>(a.state + (static_cast<int64_t>(in) * a.heads + head) * head_elems + static_cast<int64_t>(j) * dim, dim, ni, full, s[n]);
    } else {
#pragma unroll
      for (int e = 0; e < I / 2; ++e) s[n][e] = 0ull;
    }
  }
  float* o_dst = a.o_f32 + (static_cast<int64_t>(t_begin) + ni) * hd + head * dim + cb * COLS + group;  // this lane's token of every block
  __syncthreads();  // chunk 0 is ready
  for (int c = 0; c < chunks; ++c) {
    const int left = n_tok - c * Sh::kTokens, blocks = min(Sh::kBlocks, (left + J - 1) / J);
#pragma unroll 2
    for (int b = 0; b < blocks; ++b) {
      const float* buf = smem + ((c & 1) * Sh::kBlocks + b) * Sh::kFloats;
      f32x2 du[J][N], dr[J][N];
#pragma unroll
      for (int j = 0; j < J; ++j)
#pragma unroll
        for (int n = 0; n < N; ++n) du[j][n] = dr[j][n] = 0ull;
#pragma unroll
      for (int q = 0; q < I / 4; ++q) {
        const int i = (q * NI + ni) * 4;
#pragma unroll
        for (int j = 0; j < J; ++j) {
          const ulonglong2 u = piece(buf + Sh::kU + j * DIM + i);
#pragma unroll
          for (int n = 0; n < N; ++n) du[j][n] = fma2(u.y, s[n][q * 2 + 1], fma2(u.x, s[n][q * 2], du[j][n]));
        }
#pragma unroll
        for (int j = 0; j < J; ++j) {
          const ulonglong2 r = piece(buf + Sh::kR + j * DIM + i);
#pragma unroll
          for (int n = 0; n < N; ++n) dr[j][n] = fma2(r.y, s[n][q * 2 + 1], fma2(r.x, s[n][q * 2], dr[j][n]));
        }
      }
      float v[J][N], d[J][N];
#pragma unroll
      for (int j = 0; j < J; ++j)
#pragma unroll
        for (int n = 0; n < N; ++n) {
          v[j][n] = buf[Sh::kV + j * COLS + n * Sh::kGroups + group];
          d[j][n] = lane_sum<NI, ST>(sum2(du[j][n]));
        }
      const float* pairs = buf + Sh::kPairs;
#pragma unroll
      for (int j = 1; j < J; ++j) {
        const float4 uk = *reinterpret_cast<const float4*>(pairs + j * J), ub = *reinterpret_cast<const float4*>(pairs + 16 + j * J);
        const float k[3] = {uk.x, uk.y, uk.z}, g[3] = {ub.x, ub.y, ub.z};
#pragma unroll
        for (int n = 0; n < N; ++n)
#pragma unroll
          for (int t = 0; t < j; ++t) d[j][n] = fmaf(-g[t], d[t][n], fmaf(k[t], v[t][n], d[j][n]));
      }
      f32x2 vv[J][N], nd[J][N];
#pragma unroll
      for (int j = 0; j < J; ++j)
#pragma unroll
        for (int n = 0; n < N; ++n) {
          vv[j][n] = pack2(v[j][n], v[j][n]);
          nd[j][n] = pack2(-d[j][n], -d[j][n]);
        }
#pragma unroll
      for (int q = 0; q < I / 4; ++q) {
        const int i = (q * NI + ni) * 4;
        const ulonglong2 w = piece(buf + Sh::kW + i);
#pragma unroll
        for (int n = 0; n < N; ++n) {
          s[n][q * 2] = mul2(w.x, s[n][q * 2]);
          s[n][q * 2 + 1] = mul2(w.y, s[n][q * 2 + 1]);
        }
#pragma unroll
        for (int j = 0; j < J; ++j) {
          const ulonglong2 k = piece(buf + Sh::kK + j * DIM + i), g = piece(buf + Sh::kB + j * DIM + i);
#pragma unroll
          for (int n = 0; n < N; ++n) {
            s[n][q * 2] = fma2(g.x, nd[j][n], fma2(k.x, vv[j][n], s[n][q * 2]));
            s[n][q * 2 + 1] = fma2(g.y, nd[j][n], fma2(k.y, vv[j][n], s[n][q * 2 + 1]));
          }
        }
      }
      // Token ni's output: its four partial sums from the lanes of the column, and what the block's tokens up to it wrote.
      const float4 rk = *reinterpret_cast<const float4*>(pairs + 32 + ni * J), rb = *reinterpret_cast<const float4*>(pairs + 48 + ni * J);
#pragma unroll
      for (int n = 0; n < N; ++n) {
        float p[J];
#pragma unroll
        for (int j = 0; j < J; ++j) p[j] = sum2(dr[j][n]);
        const bool high = ni & 2, odd = ni & 1;
        const float a0 = (high ? p[2] : p[0]) + __shfl_xor_sync(0xffffffffu, high ? p[0] : p[2], 2 * ST);
        const float a1 = (high ? p[3] : p[1]) + __shfl_xor_sync(0xffffffffu, high ? p[1] : p[3], 2 * ST);
        float o = (odd ? a1 : a0) + __shfl_xor_sync(0xffffffffu, odd ? a0 : a1, ST);
        // (Later tokens' coefficients are zeros, but their values need not be numbers: they are left out.)
        add_if(ni >= 3, o, rk.w, v[3][n]);
        add_if(ni >= 2, o, rk.z, v[2][n]);
        add_if(ni >= 1, o, rk.y, v[1][n]);
        o = fmaf(rk.x, v[0][n], o);
        add_if(ni >= 3, o, -rb.w, d[3][n]);
        add_if(ni >= 2, o, -rb.z, d[2][n]);
        add_if(ni >= 1, o, -rb.y, d[1][n]);
        o = fmaf(-rb.x, d[0][n], o);
        if (b * J + ni < left && cb * COLS + n * Sh::kGroups + group < dim) o_dst[n * Sh::kGroups] = o;
      }
      o_dst += J * hd;
    }
    __syncthreads();  // chunk c has been read, chunk c + 1 is ready
  }
#pragma unroll
  for (int n = 0; n < N; ++n) {
    const int j = cb * COLS + n * Sh::kGroups + group;
    if (static_cast<unsigned>(out) < static_cast<unsigned>(a.state_slots) && j < dim)
      store_column<NI, I>(a.state + (static_cast<int64_t>(out) * a.heads + head) * head_elems + static_cast<int64_t>(j) * dim, dim, ni, full, s[n]);
  }
}

// kFinishUnits (token, head) units in turn with all their loads in flight: LPH lanes of four channels each, in vectors, or a warp, channels 32 apart: in registers
// (LPH < 0, up to 128 of them) or (LPH == 0) not.  Bound by the bytes in flight: 6208 tokens x 32 heads of 64 55 us with a warp and single channels for each, 20 in vectors
// (floor 15); 6000 x 32 heads of 66, which are no vectors, 60 us in registers, 87 in the loop; 8 heads of 256 54 in a kernel of its own, 74 behind the registers' code.
constexpr int kFinishUnits = 4;
template <typename T, int LPH>
__global__ void __launch_bounds__(256, LPH > 0 ? 4 : 1)
delta_finish_kernel(b200_delta_args a) {
  pdl_launch_dependents();
  pdl_wait();
  const int dim = a.dim;
  const uint32_t total = static_cast<uint32_t>(a.num_tokens) * a.heads, heads = a.heads;  // (the launch checks that it fits)
  const T* proj = static_cast<const T*>(a.proj);
  const T* weight = static_cast<const T*>(a.norm_weight);
  T* out = static_cast<T*>(a.out);
  if constexpr (LPH > 0) {
    constexpr int kGroups = 256 / LPH;
    const int lane = threadIdx.x % LPH, i = min(lane * 4, dim - 4);
    const uint32_t first = blockIdx.x * kGroups * kFinishUnits + threadIdx.x / LPH;  // then kGroups apart
    float v[kFinishUnits][4], g[kFinishUnits][4], w[kFinishUnits][4];
#pragma unroll
    for (int k = 0; k < kFinishUnits; ++k) {
      const uint32_t unit = min(first + k * kGroups, total - 1), t = unit / heads;
      const int at = static_cast<int>(unit - t * heads) * dim;
      conv::load<float, 4>(a.o_f32 + static_cast<int64_t>(unit) * dim + i, v[k]);
      conv::load<T, 4>(proj + t * a.proj_ld + a.off_g + at + i, g[k]);
      conv::load<T, 4>(weight + at + i, w[k]);
    }
#pragma unroll
    for (int k = 0; k < kFinishUnits; ++k) {
      float sq = lane * 4 < dim ? v[k][0] * v[k][0] + v[k][1] * v[k][1] + v[k][2] * v[k][2] + v[k][3] * v[k][3] : 0.f;
#pragma unroll
      for (int o = LPH / 2; o > 0; o >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, o);
      const uint32_t unit = first + k * kGroups;
      const float inv = 1.f / sqrtf(sq / dim + a.eps);
      float y[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) y[e] = v[k][e] * inv * w[k][e] * gate_sigmoid(g[k][e]);
      if (lane * 4 < dim && unit < total) conv::store<T, 4>(out + static_cast<int64_t>(unit) * dim + i, y);
    }
    return;
  }
  const int lane = threadIdx.x & 31;
  const uint32_t first = (blockIdx.x * 8 + (threadIdx.x >> 5)) * kFinishUnits;
  if constexpr (LPH < 0) {  // heads in registers
    float v[kFinishUnits][4], w[kFinishUnits][4];
    T g[kFinishUnits][4];
#pragma unroll
    for (int k = 0; k < kFinishUnits; ++k) {
      const uint32_t unit = min(first + k, total - 1), t = unit / heads;
      const int at = static_cast<int>(unit - t * heads) * dim;
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        if (e * 32 >= dim) break;
        const int i = min(lane + e * 32, dim - 1);
        v[k][e] = a.o_f32[static_cast<int64_t>(unit) * dim + i];
        g[k][e] = proj[t * a.proj_ld + a.off_g + at + i];
        w[k][e] = simt::to_f32(weight[at + i]);
      }
    }
#pragma unroll
    for (int k = 0; k < kFinishUnits; ++k) {
      float sq = 0.f;
#pragma unroll
      for (int e = 0; e < 4; ++e) sq += lane + e * 32 < dim ? v[k][e] * v[k][e] : 0.f;
      const float inv = 1.f / sqrtf(warp_sum(sq) / dim + a.eps);
#pragma unroll
      for (int e = 0; e < 4; ++e)
        if (lane + e * 32 < dim && first + k < total)
          simt::store_as(out + static_cast<int64_t>(first + k) * dim + lane + e * 32,
                         v[k][e] * inv * w[k][e] * gate_sigmoid(simt::to_f32(g[k][e])));
    }
    return;
  }
  for (int k = 0; k < kFinishUnits; ++k) {
    const int64_t unit = first + k;
    if (unit >= total) return;
    const int64_t t = unit / heads;
    const int at = static_cast<int>(unit - t * heads) * dim;
    const float* o = a.o_f32 + unit * dim;
    float sq = 0.f;
    for (int i = lane; i < dim; i += 32) sq += o[i] * o[i];
    const float inv = 1.f / sqrtf(warp_sum(sq) / dim + a.eps);
    for (int i = lane; i < dim; i += 32)
      simt::store_as(out + unit * dim + i, o[i] * inv * simt::to_f32(weight[at + i]) *
                                               sigmoid(simt::to_f32(proj[t * a.proj_ld + a.off_g + at + i])));
  }
}

template <typename T>
__global__ void __launch_bounds__(256)
delta_lora_kernel(b200_delta_args a) {
  pdl_launch_dependents();
  pdl_wait();
  const int64_t i = static_cast<int64_t>(blockIdx.x) * 256 + threadIdx.x;
  if (i >= static_cast<int64_t>(a.num_tokens) * a.rank) return;
  const int64_t t = i / a.rank;
  simt::store_as(static_cast<T*>(a.lora) + i, tanhf(simt::to_f32(static_cast<const T*>(a.proj)[t * a.proj_ld + a.off_w1 + (i - t * a.rank)])));
}

// ---------------------------------------------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------------------------------------------
static bool valid_common(const b200_delta_args* a) {
  return a && a->proj && a->num_tokens > 0 && a->heads > 0 && a->heads <= 65535 && a->dim > 0 && a->dim <= 256 &&
         (a->dtype == B200_DTYPE_BF16 || a->dtype == B200_DTYPE_F32);
}
static bool valid_state(const b200_delta_args* a) {
  return a->state && a->state_in && a->state_out && a->state_slots > 0 && aligned16(a->state) && a->decay_bias && a->removal_bias;
}

template <typename T, int DIM>
static int launch_decode(const b200_delta_args& a, cudaStream_t s) {
  using D = DecodeShape<DIM>;
  const int vec = 16 / static_cast<int>(sizeof(T));
  int w2_stride = a.rank + vec;  // rows an odd number of 16-byte pieces apart where rank is a multiple of 2 * vec
  size_t bytes = static_cast<size_t>(D::kWarps) * (6 * DIM + (a.rank + 3) / 4 * 4) * 4;
  const size_t w2_bytes = static_cast<size_t>(a.dim) * w2_stride * sizeof(T);
  if (a.rank % vec == 0 && aligned16(a.w2) && w2_bytes <= 72 * 1024)
    bytes += w2_bytes;
  else
    w2_stride = 0;  // read where it is used
  if (bytes > 200 * 1024) return B200_ERR_INVALID_ARGUMENT;
  auto go = [&](auto parts) {
    constexpr int PARTS = decltype(parts)::value, kRows = D::kWarps / PARTS;
    static std::atomic<uint64_t> done{0};
    if (ensure_dynamic_smem(delta_decode_kernel<T, DIM, PARTS>, 200 * 1024, done) != B200_OK) return static_cast<int>(B200_ERR_LAUNCH);
    return launch_pdl(delta_decode_kernel<T, DIM, PARTS>, dim3(a.heads, (a.num_rows + kRows - 1) / kRows), dim3(D::kWarps * 32), bytes, s, a, w2_stride);
  };
  if constexpr (D::kPasses >= 4) {
    const int64_t tasks = static_cast<int64_t>(a.heads) * a.num_rows;
    // (Of 256 channels two CTAs of two rows fit an SM: four tasks, with rows that only fill a CTA up.)
    const int64_t in_twos = DIM > 128 ? static_cast<int64_t>(a.heads) * (a.num_rows + a.num_rows % 2) : tasks;
    // Four warps for each of few tasks, two up to four tasks an SM; with more each of them has enough on its way, and the token would be prepared several times.
    // us, one / two / four: 32 heads of 64, one row 4.8 / 3.7 / 3.3, 8 rows 7.2 / 4.8 / 4.2, 16 rows 7.3 / 5.1 / 8.1, 32 rows 9.3 / 12.3 / 18.5; 16 heads of 128, one row 12.3 /
    // 7.8 / 5.9, 64 rows 27 / 30 / 37; two rows x 4 heads of 256 43.5 / 25.6 / 15.2, 37 rows x 16, whose CTAs of two rows are eight too many for a wave, 76.6 / 81.5 (of 96 channels 20.1 / 18.7).
    if (tasks <= 2 * sm_count()) return go(std::integral_constant<int, 4>{});
    if (in_twos <= 4 * sm_count()) return go(std::integral_constant<int, 2>{});
  }
  return go(std::integral_constant<int, 1>{});
}
template <typename T>
static int decode_by_dim(const b200_delta_args& a, cudaStream_t s) {
  if (a.dim <= 32) return launch_decode<T, 32>(a, s);
  if (a.dim <= 64) return launch_decode<T, 64>(a, s);
  if (a.dim <= 128) return launch_decode<T, 128>(a, s);
  return launch_decode<T, 256>(a, s);
}
template <typename T, int DIM, int COLS, int LANES>
static int launch_scan(const b200_delta_args& a, cudaStream_t s) {
  using Sh = ScanShape<DIM, COLS, LANES>;
  static std::atomic<uint64_t> done{0};
  if (ensure_dynamic_smem(delta_scan_kernel<T, DIM, COLS, LANES>, Sh::kSmemBytes, done) != B200_OK) return B200_ERR_LAUNCH;
  const int col_blocks = (a.dim + COLS - 1) / COLS;
  // Not a programmatic launch: CTAs that arrive while the previous kernel still holds most SMs would pile up on the others,
  // and a CTA stays where it is for the length of a prompt.
  delta_scan_kernel<T, DIM, COLS, LANES><<<dim3(a.heads * col_blocks, a.num_rows), Sh::kThreads, Sh::kSmemBytes, s>>>(a);
  return launch_status();
}
template <typename T, int DIM, int COLS, int BLOCKS>
static int launch_block_scan(const b200_delta_args& a, cudaStream_t s) {
  using Sh = BlockShape<DIM, COLS, BLOCKS>;
  static std::atomic<uint64_t> done{0};
  if (ensure_dynamic_smem(delta_block_scan_kernel<T, DIM, COLS, BLOCKS>, Sh::kSmemBytes, done) != B200_OK) return B200_ERR_LAUNCH;
  const int col_blocks = (a.dim + COLS - 1) / COLS;
  delta_block_scan_kernel<T, DIM, COLS, BLOCKS><<<dim3(a.heads * col_blocks, a.num_rows), Sh::kThreads, Sh::kSmemBytes, s>>>(a);  // (not programmatic: see launch_scan)
  return launch_status();
}
template <typename T, int DIM>
static int block_scan_by_size(const b200_delta_args& a, cudaStream_t s) {
  // Eight preparing warps, and one CTA on an SM, while a CTA's own pace counts: rows of 128 tokens and more on average and, with heads of up to 64, CTAs for
  // little more than two rounds of the SMs.  Else four, and two CTAs of up to 64 (which takes 128 registers a thread: with 130 rows of one token 41 -> 57).  us, eight / four: heads of 64, 160 CTAs 378 / 481, 256 of 400 tokens and less
  // 102 / 110, 320 583 / 615, 384 682 / 647, 512 841 / 764; rows of 64 tokens 33.8 / 29.8.  Heads of 128: 256 CTAs 791 / 961, 2048 1340 / 1497; rows of 16 40 / 34.
  const int64_t ctas = static_cast<int64_t>(a.num_rows) * a.heads;
  if (a.num_tokens / 128 >= a.num_rows && (DIM > 64 || 4 * ctas <= 9 * sm_count())) return launch_block_scan<T, DIM, 64, 8>(a, s);
  return launch_block_scan<T, DIM, 64, 4>(a, s);
}
template <typename T>
static int scan_by_dim(const b200_delta_args& a, cudaStream_t s) {
  // Blocks of four tokens against one token at a time: 6208 tokens in 5 rows x 32 heads of 64 378 us, 581; 8 rows x 64 heads 764, 872; 16 heads of 128, 5448
  // tokens in 4 rows 711, 918; 64 rows x 32 heads of one token 42, 42.  256 channels do not fit the registers four times, 32 are not worth the preparation.
  if (a.dim <= 32) return launch_scan<T, 32, 32, 2>(a, s);
  if (a.dim <= 64) return block_scan_by_size<T, 64>(a, s);
  if (a.dim <= 128) return block_scan_by_size<T, 128>(a, s);
  return launch_scan<T, 256, 32, 2>(a, s);
}

}  // namespace delta
}  // namespace b200

extern "C" {

int b200_delta_decode(const b200_delta_args* a, b200_stream_t stream) {
  using namespace b200;
  if (!delta::valid_common(a) || !delta::valid_state(a) || !a->w2 || !a->norm_weight || !a->out || a->rank <= 0 || a->rank > 4096 ||
      a->num_rows != a->num_tokens || a->num_rows > 65535)
    return B200_ERR_INVALID_ARGUMENT;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  return a->dtype == B200_DTYPE_F32 ? delta::decode_by_dim<float>(*a, s) : delta::decode_by_dim<__nv_bfloat16>(*a, s);
}

int b200_delta_lora(const b200_delta_args* a, b200_stream_t stream) {
  using namespace b200;
  if (!delta::valid_common(a) || !a->lora || a->rank <= 0) return B200_ERR_INVALID_ARGUMENT;
  const unsigned blocks = static_cast<unsigned>((static_cast<int64_t>(a->num_tokens) * a->rank + 255) / 256);
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  if (a->dtype == B200_DTYPE_F32) return launch_pdl(delta::delta_lora_kernel<float>, dim3(blocks), dim3(256), 0, s, *a);
  return launch_pdl(delta::delta_lora_kernel<__nv_bfloat16>, dim3(blocks), dim3(256), 0, s, *a);
}

int b200_delta_scan(const b200_delta_args* a, b200_stream_t stream) {
  using namespace b200;
  if (!delta::valid_common(a) || !delta::valid_state(a) || !a->z || !a->o_f32 || !a->cu_tokens || a->num_rows < 0 || a->num_rows > 65535)
    return B200_ERR_INVALID_ARGUMENT;
  if (a->num_rows == 0) return B200_OK;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  return a->dtype == B200_DTYPE_F32 ? delta::scan_by_dim<float>(*a, s) : delta::scan_by_dim<__nv_bfloat16>(*a, s);
}

int b200_delta_finish(const b200_delta_args* a, b200_stream_t stream) {
  using namespace b200;
  if (!delta::valid_common(a) || !a->o_f32 || !a->norm_weight || !a->out || static_cast<int64_t>(a->num_tokens) * a->heads > (1u << 30))
    return B200_ERR_INVALID_ARGUMENT;
  const bool vec = a->dim % 4 == 0 && a->dim <= 128 && a->proj_ld % 4 == 0 && a->off_g % 4 == 0 && aligned16(a->proj) && aligned16(a->o_f32) && aligned16(a->norm_weight) &&
                   aligned16(a->out);
  const int lanes = !vec ? 0 : a->dim <= 64 ? 16 : 32, per_block = (lanes ? 256 / lanes : 8) * delta::kFinishUnits;
  const dim3 grid(static_cast<unsigned>((static_cast<int64_t>(a->num_tokens) * a->heads + per_block - 1) / per_block));
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  auto go = [&](auto zero) {
    using T = decltype(zero);
    if (lanes == 16) return launch_pdl(delta::delta_finish_kernel<T, 16>, grid, dim3(256), 0, s, *a);
    if (lanes == 32) return launch_pdl(delta::delta_finish_kernel<T, 32>, grid, dim3(256), 0, s, *a);
    if (a->dim <= 128) return launch_pdl(delta::delta_finish_kernel<T, -1>, grid, dim3(256), 0, s, *a);
    return launch_pdl(delta::delta_finish_kernel<T, 0>, grid, dim3(256), 0, s, *a);
  };
  return a->dtype == B200_DTYPE_F32 ? go(0.f) : go(__nv_bfloat16{});
}

}  // extern "C"
