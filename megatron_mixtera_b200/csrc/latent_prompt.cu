// Latent attention of prompts on expanded keys and values (b200_latent_prompt_attention) on tcgen05: the structure of attention_prompt.cu - 256 queries
// of one row and head as two blocks of 128 that take turns between the tensor core and the softmax, S, P (hi + lo bf16 terms) and O in tensor
// memory - over contiguous key rows.  A key is a head's `dim` expanded entries and the `rot_dim` rotated ones that all heads share, staged as up to three
// tiles of 64 columns, of the two arrays by a tensor map each.
//
// The queries of a 192-column key take 96 KB of shared memory and two key tiles as much; values then have one stage (32 KB) instead of two.  The mma.sync
// kernel it stands beside (latent_prompt_kernel) takes 64 queries per CTA; it keeps the steps whose CTAs of 256 would leave most SMs idle, and short rows.
//
// Measured, 128 + 64 entries per key, 128 per value: 6208 tokens in 5 rows x 16 heads 489 -> 188 us, 2048 tokens of one row 262 -> 75 us, 3264 in 3 rows x 32
// heads 413 -> 157 us; 896 tokens in 8 rows (128 CTAs) 25.5 -> 22.7 us, the line below which the other kernel stays.
#include "common.cuh"

namespace b200 {
namespace latent {
namespace prompt {

using attn::prompt::add2;
using attn::prompt::arrived32;
using attn::prompt::exp2_fast;
using attn::prompt::fma2;
using attn::prompt::kKeys;
using attn::prompt::kLazy;
using attn::prompt::kSoftmaxWarps;
using attn::prompt::kThreadsPrompt;
using attn::prompt::kTransposeB;
using attn::prompt::load32;
using attn::prompt::pack2;
using attn::prompt::umma_f16_ts;
using attn::prompt::unpack2;

constexpr int kQueries = 256;

template <int KS, int VS>
struct Config {  // tiles of 64 columns of a key, of a value
  static constexpr int kSub = 128 * 128;
  static constexpr int kQ = KS * kSub, kK = KS * kSub, kV = VS * kSub;
  static constexpr int kKStages = 2, kVStages = KS + VS >= 5 ? 1 : 2;
  static constexpr int kOffK = 2 * kQ, kOffV = kOffK + kKStages * kK, kBarriers = kOffV + kVStages * kV;
  static constexpr int kSmemBytes = kBarriers + 256 + 1024;
  static_assert(kSmemBytes <= 227 * 1024, "");
};

template <int KS, int VS>
__global__ void __launch_bounds__(kThreadsPrompt, 1)
latent_prompt_umma_kernel(const __grid_constant__ CUtensorMap map_kv, const __grid_constant__ CUtensorMap map_rows, const __grid_constant__ b200_latent_args a) {
  using C = Config<KS, VS>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* k_full = reinterpret_cast<uint64_t*>(smem + C::kBarriers);
  uint64_t* k_empty = k_full + 2;
  uint64_t* v_full = k_empty + 2;
  uint64_t* v_empty = v_full + 2;
  uint64_t* q_full = v_empty + 2;  // per block from here on
  uint64_t* s_full = q_full + 2;
  uint64_t* p_full = s_full + 2;
  uint64_t* o_full = p_full + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(o_full + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int row = blockIdx.y, head = blockIdx.z;
  const int t_begin = a.cu_tokens[row], n_tok = a.cu_tokens[row + 1] - t_begin;
  const int q0 = (gridDim.x - 1 - blockIdx.x) * kQueries;  // the blocks with the most keys start first
  const int e_begin = a.cu_keys[row], key_begin = a.key_start[row];
  if (q0 >= n_tok) {
    pdl_wait();
    return;
  }
  const int n_q = min(kQueries, n_tok - q0);
  const int pos0 = key_begin + (a.cu_keys[row + 1] - e_begin) - n_tok + q0;  // position of query q0: the newest keys are the row's tokens
  const int start = max(window_start(pos0, a.window), key_begin), end = pos0 + n_q;
  const int n = (end - start + kKeys - 1) / kKeys;  // at least 1: a query sees itself
  const bool two = n_q > 128;                       // whether the second block has queries

  if (tid == 0) {
    for (int s = 0; s < 2; ++s) {
      mbar_init(&k_full[s], 1);
      mbar_init(&k_empty[s], 1);
      mbar_init(&v_full[s], 1);
      mbar_init(&v_empty[s], 1);
      mbar_init(&q_full[s], kSoftmaxWarps / 2);
      mbar_init(&s_full[s], 1);
      mbar_init(&p_full[s], kSoftmaxWarps / 2);
      mbar_init(&o_full[s], 1);
    }
    *abort_flag = 0;
    fence_barrier_init();
    prefetch_tensormap(&map_kv);
    prefetch_tensormap(&map_rows);
  }
  if (warp == kSoftmaxWarps) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish_alloc_permit();
  }
  tcgen05_fence_before_sync();
  __syncthreads();
  tcgen05_fence_after_sync();
  const uint32_t tmem = *tmem_slot;
  pdl_launch_dependents();  // (behind the allocation: a successor's CTA must not hold tensor memory we wait for)
  pdl_wait();

  if (warp == kSoftmaxWarps) {
    if (lane == 0) {
      const int dim_tiles = (a.dim + 63) / 64;
      for (int i = 0; i < n; ++i) {
        const int r = e_begin + start + i * kKeys - key_begin;
        const int ks = i % C::kKStages, vs = i % C::kVStages;
        uint8_t* kd = smem + C::kOffK + ks * C::kK;
        uint8_t* vd = smem + C::kOffV + vs * C::kV;
        mbar_wait_bounded(&k_empty[ks], ((i / C::kKStages) & 1) ^ 1, abort_flag, kStatusAttnTimeout);
        mbar_arrive_expect_tx(&k_full[ks], C::kK);
#pragma unroll
        for (int s = 0; s < KS; ++s) {
          if (s < dim_tiles)
            tma_load_2d(kd + s * C::kSub, &map_kv, &k_full[ks], head * a.dim + s * 64, r);
          else
            tma_load_2d(kd + s * C::kSub, &map_rows, &k_full[ks], a.kv_pad + (s - dim_tiles) * 64, r);
        }
        mbar_wait_bounded(&v_empty[vs], ((i / C::kVStages) & 1) ^ 1, abort_flag, kStatusAttnTimeout);
        mbar_arrive_expect_tx(&v_full[vs], C::kV);
#pragma unroll
        for (int s = 0; s < VS; ++s) tma_load_2d(vd + s * C::kSub, &map_kv, &v_full[vs], a.heads * a.dim + head * a.vdim + s * 64, r);
      }
    }
  } else if (warp == kSoftmaxWarps + 1) {
    constexpr uint32_t idesc_s = umma_idesc_bf16(128, kKeys), idesc_o = umma_idesc_bf16(128, VS * 64) | kTransposeB;
    auto scores = [&](int b, int stage) {  // S_b = Q_b K^T
      if (lane == 0) {
        const uint64_t q = umma_desc_k_major_sw128(smem_u32(smem + b * C::kQ));
        const uint64_t k = umma_desc_k_major_sw128(smem_u32(smem + C::kOffK + stage * C::kK));
#pragma unroll
        for (int ks = 0; ks < KS * 4; ++ks) {
          const int at = (ks >> 2) * (C::kSub >> 4) + (ks & 3) * 2;
          umma_f16(tmem + b * kKeys, q + at, k + at, idesc_s, ks > 0);
        }
        umma_commit(&s_full[b]);
      }
    };
    mbar_wait_bounded(&q_full[0], 0, abort_flag, kStatusAttnTimeout);
    if (two) mbar_wait_bounded(&q_full[1], 0, abort_flag, kStatusAttnTimeout);
    mbar_wait_bounded(&k_full[0], 0, abort_flag, kStatusAttnTimeout);
    tcgen05_fence_after_sync();
    scores(0, 0);
    if (two) scores(1, 0);
    if (lane == 0) umma_commit(&k_empty[0]);
    for (int i = 0; i < n; ++i) {
      const int vs = i % C::kVStages, k_next = (i + 1) % C::kKStages;
      mbar_wait_bounded(&v_full[vs], (i / C::kVStages) & 1, abort_flag, kStatusAttnTimeout);
      uint8_t* v_tile = smem + C::kOffV + vs * C::kV;
      if (i == n - 1) {  // rows behind the newest key may hold anything
        const int valid = min(end - (start + i * kKeys), kKeys);
        for (int s = 0; s < VS; ++s)
          for (int v = valid * 8 + lane; v < kKeys * 8; v += 32) *reinterpret_cast<uint4*>(v_tile + s * C::kSub + v * 16) = make_uint4(0, 0, 0, 0);
        fence_proxy_async_smem();
        __syncwarp();
      }
#pragma unroll
      for (int b = 0; b < 2; ++b) {
        if (b == 1 && !two) continue;
        mbar_wait_bounded(&p_full[b], i & 1, abort_flag, kStatusAttnTimeout);
        tcgen05_fence_after_sync();
        if (lane == 0) {  // O_b += (P_hi + P_lo) V
          const uint64_t v = umma_desc_mn_major_sw128(smem_u32(v_tile), C::kSub);
          const uint32_t o = tmem + 2 * kKeys + b * 128, probs = tmem + b * kKeys;
#pragma unroll
          for (int ks = 0; ks < kKeys / 16; ++ks) {
            const uint32_t hi = probs + (ks >> 1) * 32 + (ks & 1) * 8;
            umma_f16_ts(o, hi, v + ks * 128, idesc_o, i > 0 || ks > 0);
            umma_f16_ts(o, hi + 16, v + ks * 128, idesc_o, 1);
          }
        }
        if (i + 1 < n) {
          mbar_wait_bounded(&k_full[k_next], ((i + 1) / C::kKStages) & 1, abort_flag, kStatusAttnTimeout);
          tcgen05_fence_after_sync();
          scores(b, k_next);
        } else if (lane == 0) {
          umma_commit(&o_full[b]);
        }
      }
      if (lane == 0) {
        umma_commit(&v_empty[vs]);
        if (i + 1 < n) umma_commit(&k_empty[k_next]);
      }
      __syncwarp();
    }
  } else if ((warp >> 2) == 0 || two) {
    // ---------------- softmax: thread = query ----------------
    const int b = warp >> 2, rho = tid & 127, qi = b * 128 + rho;
    const uint32_t lanes = static_cast<uint32_t>((warp & 3) * 32) << 16;
    const uint32_t s_addr = tmem + lanes + b * kKeys, o_addr = tmem + lanes + 2 * kKeys + b * 128;
    const bool live = qi < n_q;
    const int64_t t = t_begin + q0 + qi;
    const int last = live ? pos0 + qi : 0x7fffffff, oldest = live ? window_start(pos0 + qi, a.window) : 0;  // (idle rows take the plain path)
    {
      uint8_t* q_row = smem + b * C::kQ + rho * 128;
      const __nv_bfloat16* q = a.q != nullptr ? static_cast<const __nv_bfloat16*>(a.q) + t * a.q_ld : static_cast<const __nv_bfloat16*>(a.proj) + t * a.proj_ld;
      q += head * (a.dim + a.rot_dim);
      const __nv_bfloat16* qr = static_cast<const __nv_bfloat16*>(a.q_full) + (t * a.heads + head) * a.q_stride + a.q_rot_at;
      const int dim_pieces = (a.dim + 63) / 64 * 8, rot_w = a.row_width - a.kv_pad;
#pragma unroll 4
      for (int c = 0; c < KS * 8; ++c) {
        uint4 v = make_uint4(0, 0, 0, 0);
        if (live) {
          if (c < dim_pieces) {
            if (c * 8 < a.dim) v = *reinterpret_cast<const uint4*>(q + c * 8);
          } else if ((c - dim_pieces) * 8 < rot_w) {
            v = *reinterpret_cast<const uint4*>(qr + (c - dim_pieces) * 8);
          }
        }
        *reinterpret_cast<uint4*>(q_row + (c >> 3) * C::kSub + (((c & 7) ^ (rho & 7)) << 4)) = v;
      }
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(&q_full[b]);
    }
    const float factor = a.scale * kLog2e;
    float top = -INFINITY, sum = 0.f;
    for (int i = 0; i < n; ++i) {
      const int key0 = start + i * kKeys;
      mbar_wait_bounded(&s_full[b], i & 1, abort_flag, kStatusAttnTimeout);
      tcgen05_fence_after_sync();
      __syncwarp();
      if (!__all_sync(0xffffffffu, !live || (key0 >= oldest && key0 + kKeys - 1 <= last))) {  // masks: written back over the products
#pragma unroll 1
        for (int c0 = 0; c0 < kKeys; c0 += 32) {
          float w[32];
          load32(s_addr + c0, w);
          tmem_ld_wait();
          arrived32(w);
#pragma unroll
          for (int c = 0; c < 32; ++c) {
            const int key = key0 + c0 + c;
            if (key < oldest || key > last) w[c] = -INFINITY;
          }
          tmem_st_32x32b_x16(s_addr + c0, *reinterpret_cast<const uint32_t(*)[16]>(reinterpret_cast<uint32_t*>(w)));
          tmem_st_32x32b_x16(s_addr + c0 + 16, *reinterpret_cast<const uint32_t(*)[16]>(reinterpret_cast<uint32_t*>(w) + 16));
        }
        tmem_st_wait();
      }
      float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
      for (int c0 = 0; c0 < kKeys; c0 += 64) {
        float v[64];
        load32(s_addr + c0, v);
        load32(s_addr + c0 + 32, v + 32);
        tmem_ld_wait();
        arrived32(v);
        arrived32(v + 32);
#pragma unroll
        for (int c = 0; c < 64; ++c) mx[c & 3] = fmaxf(mx[c & 3], v[c]);
      }
      const float seen = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])) * factor;
      const bool grow = seen > top + kLazy;  // (top starts at -inf)
      if (__any_sync(0xffffffffu, grow)) {
        const float next = fmaxf(top, seen);
        const float alpha = next == -INFINITY ? 1.f : exp2_fast(top - next);
        top = next;
        sum *= alpha;
        if (i > 0) {
#pragma unroll 1
          for (int c = 0; c < VS * 64; c += 16) {
            uint32_t o[16];
            tmem_ld_32x32b_x16(o_addr + c, o);
            tmem_ld_wait();
#pragma unroll
            for (int k = 0; k < 16; ++k) o[k] = __float_as_uint(__uint_as_float(o[k]) * alpha);
            tmem_st_32x32b_x16(o_addr + c, o);
          }
        }
      }
      const float use = top == -INFINITY ? 0.f : top;
      const uint64_t f2 = pack2(factor, factor), m2 = pack2(-use, -use), minus = pack2(-1.f, -1.f);
      uint64_t sums[2] = {pack2(0.f, 0.f), pack2(0.f, 0.f)};
      float v[2][32];
      load32(s_addr, v[0]);
#pragma unroll
      for (int c0 = 0; c0 < kKeys; c0 += 32) {
        float* now = v[(c0 >> 5) & 1];
        uint32_t hi[16], lo[16];
        tmem_ld_wait();
        arrived32(now);
        if (c0 + 32 < kKeys) load32(s_addr + c0 + 32, v[((c0 >> 5) & 1) ^ 1]);
#pragma unroll
        for (int k = 0; k < 16; ++k) {
          float x, y, rx, ry;
          unpack2(fma2(pack2(now[2 * k], now[2 * k + 1]), f2, m2), x, y);
          x = exp2_fast(x);
          y = exp2_fast(y);
          const uint64_t xy = pack2(x, y);
          sums[k & 1] = add2(sums[k & 1], xy);
          hi[k] = pack_bf16x2(x, y);
          unpack2(fma2(pack2(bf16_lo(hi[k]), bf16_hi(hi[k])), minus, xy), rx, ry);
          lo[k] = pack_bf16x2(rx, ry);
        }
        tmem_st_32x32b_x16(s_addr + c0, hi);
        tmem_st_32x32b_x16(s_addr + c0 + 16, lo);
      }
      float s0, s1, s2, s3;
      unpack2(sums[0], s0, s1);
      unpack2(sums[1], s2, s3);
      sum += (s0 + s1) + (s2 + s3);
      tmem_st_wait();
      tcgen05_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(&p_full[b]);
    }

    mbar_wait_bounded(&o_full[b], 0, abort_flag, kStatusAttnTimeout);
    tcgen05_fence_after_sync();
    __syncwarp();
    sum += sink_weight(a, head, top);
    const float inv = live ? (a.value_gates ? 1.f : gate_of<__nv_bfloat16>(a, t, head)) / sum : 0.f;
    __nv_bfloat16* dst = static_cast<__nv_bfloat16*>(a.out) + (t * a.heads + head) * a.vdim;
    const __nv_bfloat16* gates = static_cast<const __nv_bfloat16*>(a.proj) + t * a.proj_ld + a.gate_offset + head * a.vdim;
#pragma unroll 1
    for (int c0 = 0; c0 < VS * 64; c0 += 32) {
      float o[32];
      __syncwarp();
      load32(o_addr + c0, o);
      tmem_ld_wait();
      arrived32(o);
      if (!live) continue;
#pragma unroll
      for (int k = 0; k < 32; k += 8) {
        if (c0 + k >= a.vdim) continue;
        uint32_t w[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          float x = o[k + 2 * j] * inv, y = o[k + 2 * j + 1] * inv;
          if (a.value_gates) {  // one per channel (4-byte loads: even columns)
            const uint32_t g = *reinterpret_cast<const uint32_t*>(gates + c0 + k + 2 * j);
            x = __fdividef(x, 1.f + __expf(-bf16_lo(g)));
            y = __fdividef(y, 1.f + __expf(-bf16_hi(g)));
          }
          w[j] = pack_bf16x2(x, y);
        }
        if ((reinterpret_cast<uintptr_t>(dst) & 15) == 0) {
          *reinterpret_cast<uint4*>(dst + c0 + k) = make_uint4(w[0], w[1], w[2], w[3]);
        } else {
#pragma unroll
          for (int j = 0; j < 4; ++j) *reinterpret_cast<uint32_t*>(dst + c0 + k + 2 * j) = w[j];
        }
      }
    }
  }

  tcgen05_fence_before_sync();
  __syncthreads();
  if (warp == kSoftmaxWarps) tmem_dealloc(tmem, 512);
}

// Whether this kernel takes the call: 64-column tiles that hold a key and a value, and enough CTAs of 256 queries for the SMs.  It masks and takes maxima
// in front of the scale, which therefore has to be positive: the other kernel has any.
// Rows of up to 64 tokens are one CTA in either kernel, on an SM that holds one here and two or three there (16 heads, 64 rows of 64 tokens 82 us here, 47
// there); from about 100 on a row saves CTAs here (64 of 100: 95 and 109).  A long row among short ones saves ~0.023 us a head for each 64 x 64 products,
// a short row costs ~0.03 us a head (32 heads, 64 rows that continue with a token beside 4 of 300: 206 us here, 151 there; beside one of 2048: 361, 565).
static bool applicable(const b200_latent_args& a) {
  const int64_t longest = a.max_row_tokens;
  if (longest <= 64 || (a.num_tokens < 64ll * a.num_rows && longest * longest < 12000ll * a.num_rows)) return false;
  const int key_tiles = (a.dim + 63) / 64 + (a.rot_dim + 63) / 64;
  const int64_t ctas = static_cast<int64_t>((a.max_row_tokens + kQueries - 1) / kQueries) * a.num_rows * a.heads;
  return a.scale > 0.f && key_tiles <= 3 && a.vdim <= 128 && a.num_keys > 0 && a.row_width % 8 == 0 && a.kv_pad % 8 == 0 && a.num_tokens >= kQueries &&
         ctas * 2 >= sm_count() && aligned16(a.q_full);
}

template <int KS, int VS>
static int launch(const b200_latent_args& a, cudaStream_t s) {
  using C = Config<KS, VS>;
  const uint64_t ld = static_cast<uint64_t>(a.heads) * (a.dim + a.vdim);
  const uint64_t kd[2] = {ld, static_cast<uint64_t>(a.num_keys)}, rd[2] = {static_cast<uint64_t>(a.row_width), static_cast<uint64_t>(a.num_keys)};
  const uint64_t ks[1] = {ld * 2}, rs[1] = {static_cast<uint64_t>(a.row_width) * 2};
  const uint32_t box[2] = {64, 128};
  const CUtensorMap* mk = get_tensor_map(a.key_values, 2, kd, ks, box, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B);
  const CUtensorMap* mr = get_tensor_map(a.key_rows, 2, rd, rs, box, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B);
  if (!mk || !mr) return B200_ERR_DRIVER;
  static std::atomic<uint64_t> done{0};
  if (ensure_dynamic_smem(latent_prompt_umma_kernel<KS, VS>, C::kSmemBytes, done) != B200_OK) return B200_ERR_LAUNCH;
  const dim3 grid((a.max_row_tokens + kQueries - 1) / kQueries, a.num_rows, a.heads);
  return launch_pdl(latent_prompt_umma_kernel<KS, VS>, grid, dim3(kThreadsPrompt), C::kSmemBytes, s, *mk, *mr, a);
}

static int launch_by_size(const b200_latent_args& a, cudaStream_t s) {
  const int key_tiles = (a.dim + 63) / 64 + (a.rot_dim + 63) / 64;
  if (a.vdim <= 64) return key_tiles <= 1 ? launch<1, 1>(a, s) : key_tiles == 2 ? launch<2, 1>(a, s) : launch<3, 1>(a, s);
  return key_tiles <= 1 ? launch<1, 2>(a, s) : key_tiles == 2 ? launch<2, 2>(a, s) : launch<3, 2>(a, s);
}

}  // namespace prompt
}  // namespace latent
}  // namespace b200
