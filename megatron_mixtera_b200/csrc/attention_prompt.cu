// Prompt attention on tcgen05: the work units of paged_prefill_kernel (attention.cu, same arguments and results), four at a time.
//
// paged_prefill_kernel gives a CTA one unit of 64 (token, head) rows and computes with mma.sync: 0.10 of the tensor peak, bound by the issue of
// its products.  Here a CTA takes four consecutive units, 256 rows, as two blocks of 128 that take turns: while one block's rows go through the softmax,
// the tensor core computes the other's S = Q K^T and O += P V.  Products run as 128 x 128 tiles with every accumulator in tensor memory:
//
//   columns   0 - 255   S of both blocks [128 rows][128 keys] fp32; a row's thread overwrites its S with P, split into hi + lo bf16 terms
//                       (of every 32 columns, 16 + 16), which the second product reads as A operand from tensor memory
//   columns 256 - 511   O of both blocks [128 rows][DV] fp32
//
//   warps 0-3, 4-7      softmax of block 0, 1: one row per thread (no shuffles); queries in, outputs out
//   warp 8, lane 0      TMA: key and value tiles of 128 tokens as two boxes of 64 (a box never straddles a chunk), two stages each
//   warp 9              UMMA issuer; clears value rows behind the newest key (a product with a zero weight must not meet a NaN)
//
// Measured (32 query heads of 128 in 8 groups, bf16): 4 prompts of 2048 tokens 727 -> 255 us, 4096 + 3000 + 2000 + 2500 tokens 1467 -> 461 us; 64 heads, one
// prompt of 8192: 5096 -> 1340 us, 821 TFLOP/s counting two products per (query, key, head).  Bound by the chain product -> softmax -> product, of which two
// blocks hide most; a CTA's queries and first tiles are not overlapped with the one before it on the SM.
//
// Three products of 128 x 128 x 128 per tile and block (one for S, two for P's terms) take 1536 clocks, a block's softmax about as many.  O is rescaled only
// when a row's maximum has grown by more than 2^8 since the last time: P and the row sums stay relative to the maximum in use, in fp32 until the
// split, so the result is the same within rounding.  (Two blocks in turn and the lazy maximum are steps of a published method, FlashAttention-4; the maximum in
// use moves for all rows of a warp when one of them grows, so a row's last bits may depend on its neighbours'.)  Units of several requests in one CTA are taken
// request by request (a "run"), the other rows idle.
#include "common.cuh"

namespace b200 {
namespace attn {
namespace prompt {

constexpr int kSoftmaxWarps = 8, kThreadsPrompt = (kSoftmaxWarps + 2) * 32;
constexpr int kKeys = 128;         // keys per tile: two pool tiles of kTile
constexpr int kRingStages = 2;
constexpr int kUnitsPerCta = kUnitsPerGroup;
constexpr float kLazy = 8.f;       // log2 of how far a maximum may grow before O is rescaled
constexpr uint32_t kTransposeB = 1u << 16;  // instruction descriptor: B is MN-major

template <int DK, int DV>
struct Config {
  static constexpr int kSubK = DK / 64, kSubV = DV / 64;  // 128-byte swizzle rows hold 64 bf16 values
  static constexpr int kSub = 128 * 128;                  // [128 rows][64 dims]
  static constexpr int kQ = kSubK * kSub;                 // one block's queries
  static constexpr int kK = kSubK * kSub, kV = kSubV * kSub;
  static constexpr int kOffK = 2 * kQ, kOffV = kOffK + kRingStages * kK;
  static constexpr int kBarriers = kOffV + kRingStages * kV;
  static constexpr int kSmemBytes = kBarriers + 256 + 1024;
};

__device__ __forceinline__ void umma_f16_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "setp.ne.b32 p, %4, 0;\n"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n"
      "}\n" ::"r"(tmem_d),
      "r"(tmem_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ uint64_t pack2(float a, float b) {
  uint64_t v;
  asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(a), "f"(b));
  return v;
}
__device__ __forceinline__ void unpack2(uint64_t v, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ float exp2_fast(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

__device__ __forceinline__ void load32(uint32_t taddr, float* v) { tmem_ld_32x32b_x32(taddr, *reinterpret_cast<uint32_t(*)[32]>(v)); }

// The values of a load that has been waited for: keeps the compiler from using them any earlier.
__device__ __forceinline__ void arrived32(float* v) {
#pragma unroll
  for (int i = 0; i < 32; i += 8)
    asm volatile("" : "+f"(v[i]), "+f"(v[i + 1]), "+f"(v[i + 2]), "+f"(v[i + 3]), "+f"(v[i + 4]), "+f"(v[i + 5]), "+f"(v[i + 6]), "+f"(v[i + 7]));
}

// The units of one request among a CTA's four, and the keys they see.
struct Run {
  int row = 0, mask = 0;        // block-table row; units that belong to it
  int base = 0, kept = 0, blocks = 0, max_kv = 0;
  __device__ __forceinline__ int block_key(int b) const { return b < kept ? b * kTile : base + (b - kept) * kTile; }
  __device__ __forceinline__ int tiles() const { return (blocks + 1) >> 1; }
  __device__ __forceinline__ bool active(int block) const { return (mask >> (2 * block) & 3) != 0; }
};

template <int DK, int DV, int FORM>
__global__ void __launch_bounds__(kThreadsPrompt, 1)
paged_prompt_kernel(const __grid_constant__ CUtensorMap map_k, const __grid_constant__ CUtensorMap map_v, const __grid_constant__ Params p,
                    const int32_t* __restrict__ units, int num_units, int all) {
  using C = Config<DK, DV>;
  constexpr bool SEPARATE = FORM != kFused, EXTRA = FORM == kExtra;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* k_full = reinterpret_cast<uint64_t*>(smem + C::kBarriers);
  uint64_t* k_empty = k_full + kRingStages;
  uint64_t* v_full = k_empty + kRingStages;
  uint64_t* v_empty = v_full + kRingStages;
  uint64_t* q_full = v_empty + kRingStages;  // per block from here on
  uint64_t* s_full = q_full + 2;
  uint64_t* p_full = s_full + 2;
  uint64_t* o_full = p_full + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(o_full + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int h = blockIdx.x % p.nkv;
  // the last units of a request see the most keys: they start first
  const int first_unit = ((num_units + kUnitsPerCta - 1) / kUnitsPerCta - 1 - static_cast<int>(blockIdx.x / p.nkv)) * kUnitsPerCta;
  if (!all && !prompt_group<DV>(p, units, num_units, first_unit)) {  // paged_prefill_kernel's, or padding
    if (blockIdx.x == 0) pdl_wait();                                 // (a kernel never ends before its predecessor)
    return;
  }
  const int G = p.G;

  if (tid == 0) {
    for (int s = 0; s < kRingStages; ++s) {
      mbar_init(&k_full[s], 1);
      mbar_init(&k_empty[s], 1);
      mbar_init(&v_full[s], 1);
      mbar_init(&v_empty[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&q_full[b], kSoftmaxWarps / 2);
      mbar_init(&s_full[b], 1);
      mbar_init(&p_full[b], kSoftmaxWarps / 2);
      mbar_init(&o_full[b], 1);
    }
    *abort_flag = 0;
    fence_barrier_init();
    prefetch_tensormap(&map_k);
    prefetch_tensormap(&map_v);
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
  pdl_wait();  // queries, pool and lengths are earlier kernels' output

  int left = 0;  // units to do
#pragma unroll
  for (int u = 0; u < kUnitsPerCta; ++u) left |= (unit_entry(p, units, num_units, first_unit + u).z > 0) << u;
  auto unit_at = [&](int u) { return *reinterpret_cast<const int4*>(units + 4 * static_cast<int64_t>(first_unit + u)); };
  // The next run (warp-collective; every warp finds the same ones).
  auto next_run = [&](Run& r) {
    const int lead = __ffs(left) - 1;
    r.mask = 0;
    r.row = unit_at(lead).x;
    int max_kv = 0, min_kv = 0x7fffffff;
    for (int u = lead; u < kUnitsPerCta; ++u) {
      if ((left >> u & 1) == 0) continue;
      const int4 e = unit_at(u);
      if (e.x == r.row) {
        r.mask |= 1 << u;
        for (int j = lane; j < e.z; j += 32) {
          const int kv = p.kv_len[e.y + j];
          max_kv = max(max_kv, kv);
          min_kv = min(min_kv, kv);
        }
      }
    }
    max_kv = __reduce_max_sync(0xffffffffu, max_kv);
    min_kv = __reduce_min_sync(0xffffffffu, min_kv);
    left &= ~r.mask;
    r.max_kv = max_kv;
    r.base = SEPARATE ? first_tile_key(p, min_kv) : 0;
    r.kept = EXTRA ? kept_tiles(p, r.base) : 0;
    r.blocks = r.kept + (max_kv - r.base + kTile - 1) / kTile;
  };

  if (warp == kSoftmaxWarps) {
    // ---------------- key and value tiles ----------------
    int it = 0;
    while (left) {
      Run r;
      next_run(r);
      const int32_t* bt_row = p.block_table + static_cast<int64_t>(r.row) * p.max_chunks;
      if (lane == 0) {
        for (int i = 0; i < r.tiles(); ++i, ++it) {
          const int s = it % kRingStages;
          const uint32_t free_phase = ((it / kRingStages) & 1) ^ 1;
          const int halves = min(2, r.blocks - 2 * i);
          int tok_row[2] = {0, 0};
          for (int b = 0; b < halves; ++b) {
            const int key = r.block_key(2 * i + b), c = key / p.chunk;
            tok_row[b] = bt_row[c] * p.chunk + (key - c * p.chunk);
          }
          uint8_t* kdst = smem + C::kOffK + s * C::kK;
          uint8_t* vdst = smem + C::kOffV + s * C::kV;
          mbar_wait_bounded(&k_empty[s], free_phase, abort_flag, kStatusAttnTimeout);
          mbar_arrive_expect_tx(&k_full[s], halves * (C::kK / 2));
          for (int b = 0; b < halves; ++b)
#pragma unroll
            for (int sub = 0; sub < C::kSubK; ++sub)
              tma_load_3d(kdst + sub * C::kSub + b * (C::kSub / 2), &map_k, &k_full[s], sub * 64, h, tok_row[b]);
          mbar_wait_bounded(&v_empty[s], free_phase, abort_flag, kStatusAttnTimeout);
          mbar_arrive_expect_tx(&v_full[s], halves * (C::kV / 2));
          for (int b = 0; b < halves; ++b)
#pragma unroll
            for (int sub = 0; sub < C::kSubV; ++sub)
              tma_load_3d(vdst + sub * C::kSub + b * (C::kSub / 2), &map_v, &v_full[s], sub * 64, EXTRA ? h >> p.kshift : h, tok_row[b]);
        }
      }
      it = __shfl_sync(0xffffffffu, it, 0);
    }
  } else if (warp == kSoftmaxWarps + 1) {
    // ---------------- products ----------------
    constexpr uint32_t idesc_s = umma_idesc_bf16(128, kKeys), idesc_o = umma_idesc_bf16(128, DV) | kTransposeB;
    int it = 0, q_phase[2] = {0, 0}, p_phase[2] = {0, 0};
    auto scores = [&](int b, int stage) {  // S_b = Q_b K^T
      if (lane == 0) {
        const uint64_t q = umma_desc_k_major_sw128(smem_u32(smem + b * C::kQ));
        const uint64_t k = umma_desc_k_major_sw128(smem_u32(smem + C::kOffK + stage * C::kK));
#pragma unroll
        for (int ks = 0; ks < DK / 16; ++ks) {
          const int at = (ks >> 2) * (C::kSub >> 4) + (ks & 3) * 2;
          umma_f16(tmem + b * kKeys, q + at, k + at, idesc_s, ks > 0);
        }
        umma_commit(&s_full[b]);
      }
    };
    while (left) {
      Run r;
      next_run(r);
      const int n = r.tiles();
      if (n == 0) continue;
#pragma unroll
      for (int b = 0; b < 2; ++b)
        if (r.active(b)) {
          mbar_wait_bounded(&q_full[b], q_phase[b] & 1, abort_flag, kStatusAttnTimeout);
          ++q_phase[b];
        }
      mbar_wait_bounded(&k_full[it % kRingStages], (it / kRingStages) & 1, abort_flag, kStatusAttnTimeout);
      tcgen05_fence_after_sync();
#pragma unroll
      for (int b = 0; b < 2; ++b)
        if (r.active(b)) scores(b, it % kRingStages);
      if (lane == 0) umma_commit(&k_empty[it % kRingStages]);
      for (int i = 0; i < n; ++i, ++it) {
        const int s = it % kRingStages, s_next = (it + 1) % kRingStages;
        mbar_wait_bounded(&v_full[s], (it / kRingStages) & 1, abort_flag, kStatusAttnTimeout);
        uint8_t* v_tile = smem + C::kOffV + s * C::kV;
        if (i == n - 1) {  // rows behind the newest key (or of a missing second half) hold anything
          const int key1 = 2 * i + 1 < r.blocks ? r.block_key(2 * i + 1) : 0x3fffffff;
          for (int half = 0; half < 2; ++half) {
            const int key = half == 0 ? r.block_key(2 * i) : key1;
            const int valid = min(max(r.max_kv - key, 0), kTile);
            for (int sub = 0; sub < C::kSubV; ++sub)
              for (int v = valid * 8 + lane; v < kTile * 8; v += 32)
                *reinterpret_cast<uint4*>(v_tile + sub * C::kSub + half * (C::kSub / 2) + v * 16) = make_uint4(0, 0, 0, 0);
          }
          fence_proxy_async_smem();
          __syncwarp();
        }
#pragma unroll
        for (int b = 0; b < 2; ++b) {
          if (!r.active(b)) continue;
          mbar_wait_bounded(&p_full[b], p_phase[b] & 1, abort_flag, kStatusAttnTimeout);
          ++p_phase[b];
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
            mbar_wait_bounded(&k_full[s_next], ((it + 1) / kRingStages) & 1, abort_flag, kStatusAttnTimeout);
            tcgen05_fence_after_sync();
            scores(b, s_next);
          } else if (lane == 0) {
            umma_commit(&o_full[b]);
          }
        }
        if (lane == 0) {
          umma_commit(&v_empty[s]);
          if (i + 1 < n) umma_commit(&k_empty[s_next]);
        }
        __syncwarp();
      }
    }
  } else {
    // ---------------- softmax: thread = row ----------------
    const int b = warp >> 2;                 // block
    const int rho = tid & 127;               // row of the block
    const int unit = 2 * b + (rho >> 6), j = (rho & 63) / G, g = (rho & 63) - j * G;
    const uint32_t lanes = static_cast<uint32_t>((warp & 3) * 32) << 16;
    const uint32_t s_addr = tmem + lanes + b * kKeys, o_addr = tmem + lanes + 2 * kKeys + b * 128;
    int s_phase = 0, o_phase = 0;
    int my_tok = -1;
    if (left >> unit & 1) {
      const int4 e = unit_at(unit);
      if (j < e.z) my_tok = e.y + j;
    }
    const int head = query_head<FORM>(p, h, g < G ? g : 0);
    const float scale_log2 = p.scale_log2;
    while (left) {
      Run r;
      next_run(r);
      if (!r.active(b)) continue;
      const int n = r.tiles();
      const int tok = (r.mask >> unit & 1) ? my_tok : -1;
      // (idle rows see everything: they take the plain path and are never stored)
      const int kv = tok >= 0 ? p.kv_len[tok] : 0x7fffffff;
      const int first = SEPARATE && tok >= 0 ? first_key(p, kv) : 0;
      float top = -INFINITY, sum = 0.f;
      if (n > 0) {
        // ---- queries: this row, rotated where the form asks for it ----
        uint8_t* q_row = smem + b * C::kQ + rho * 128;
        auto put = [&](int c, uint4 v) {  // dims [8 c, 8 c + 8)
          *reinterpret_cast<uint4*>(q_row + (c >> 3) * C::kSub + (((c & 7) ^ (rho & 7)) << 4)) = v;
        };
        if (tok < 0) {
#pragma unroll
          for (int c = 0; c < DK / 8; ++c) put(c, make_uint4(0, 0, 0, 0));
        } else {
          const __nv_bfloat16* q = p.qkv + tok * p.q_token + query_offset<FORM>(p, h, g);
          const bool vec = (reinterpret_cast<uintptr_t>(q) & 15) == 0;
          auto get = [&](int c) {
            if (vec) return *reinterpret_cast<const uint4*>(q + c * 8);
            const uint32_t* w = reinterpret_cast<const uint32_t*>(q + c * 8);
            return make_uint4(w[0], w[1], w[2], w[3]);
          };
          if (SEPARATE || p.cos == nullptr) {
#pragma unroll
            for (int c = 0; c < DK / 8; ++c) put(c, !SEPARATE || c * 8 < p.dk ? get(c) : make_uint4(0, 0, 0, 0));
          } else {
            const int64_t at = p.pos_q[tok] * (DK / 2);
#pragma unroll
            for (int c = 0; c < DK / 16; ++c) {
              const uint4 lo4 = get(c), hi4 = get(c + DK / 16);
              const uint32_t* c2 = reinterpret_cast<const uint32_t*>(p.cos + at + c * 8);
              const uint32_t* s2 = reinterpret_cast<const uint32_t*>(p.sin + at + c * 8);
              const uint32_t lo[4] = {lo4.x, lo4.y, lo4.z, lo4.w}, hi[4] = {hi4.x, hi4.y, hi4.z, hi4.w};
              uint32_t out_lo[4], out_hi[4];
#pragma unroll
              for (int k = 0; k < 4; ++k) {
                float a1 = bf16_lo(lo[k]), b1 = bf16_hi(lo[k]), a2 = bf16_lo(hi[k]), b2 = bf16_hi(hi[k]);
                rope_pair(a1, a2, bf16_lo(c2[k]), bf16_lo(s2[k]), a1, a2);
                rope_pair(b1, b2, bf16_hi(c2[k]), bf16_hi(s2[k]), b1, b2);
                out_lo[k] = pack_bf16x2(a1, b1);
                out_hi[k] = pack_bf16x2(a2, b2);
              }
              put(c, make_uint4(out_lo[0], out_lo[1], out_lo[2], out_lo[3]));
              put(c + DK / 16, make_uint4(out_hi[0], out_hi[1], out_hi[2], out_hi[3]));
            }
          }
        }
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) mbar_arrive(&q_full[b]);
      }
      const float* bias = EXTRA && p.bias != nullptr ? p.bias + static_cast<int64_t>(head) * p.bias_len : nullptr;
      const float far_bias = bias != nullptr ? __ldg(bias + p.bias_len - 1) * kLog2e : 0.f;

      for (int i = 0; i < n; ++i) {
        const int key0 = r.block_key(2 * i), key1 = 2 * i + 1 < r.blocks ? r.block_key(2 * i + 1) : 0x3fffffff;
        mbar_wait_bounded(&s_full[b], s_phase & 1, abort_flag, kStatusAttnTimeout);
        ++s_phase;
        tcgen05_fence_after_sync();
        // ---- scores in the log2 domain are v * factor ----
        float factor = scale_log2;
        bool in_sight = key0 >= first && key1 >= first && key0 + kTile <= kv && key1 + kTile <= kv;
        if (EXTRA && bias != nullptr) in_sight = in_sight && max(key0, key1) + kTile <= kv - p.bias_len + 1;
        const bool plain = __all_sync(0xffffffffu, in_sight || tok < 0);
        if (!plain || (EXTRA && (p.cap_out > 0.f || bias != nullptr))) {  // masks, caps and biases: written back over the products
          if (EXTRA) factor = 1.f;
#pragma unroll 1
          for (int c0 = 0; c0 < kKeys; c0 += 32) {
            float w[32];
            load32(s_addr + c0, w);
            tmem_ld_wait();
            arrived32(w);
            const int key = (c0 < kTile ? key0 : key1 - kTile) + c0;
            if (EXTRA && plain) {
#pragma unroll
              for (int c = 0; c < 32; ++c) w[c] = (p.cap_out > 0.f ? capped(p, w[c]) : w[c] * scale_log2) + far_bias;
            } else {
#pragma unroll
              for (int c = 0; c < 32; ++c) {
                if (EXTRA) w[c] = extra_score(p, w[c], bias, kv - 1 - (key + c));
                if (key + c >= kv || (SEPARATE && key + c < first && !(EXTRA && key + c < p.keep_first))) w[c] = -INFINITY;
              }
            }
            tmem_st_32x32b_x16(s_addr + c0, *reinterpret_cast<const uint32_t(*)[16]>(reinterpret_cast<uint32_t*>(w)));
            tmem_st_32x32b_x16(s_addr + c0 + 16, *reinterpret_cast<const uint32_t(*)[16]>(reinterpret_cast<uint32_t*>(w) + 16));
          }
          tmem_st_wait();
        }
        float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};  // (four chains; the factor is positive)
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
        // ---- the maximum in use ----
        const bool grow = seen > top + kLazy;  // (top starts at -inf)
        if (__any_sync(0xffffffffu, grow)) {
          const float next = fmaxf(top, seen);
          const float alpha = next == -INFINITY ? 1.f : exp2_fast(top - next);
          top = next;
          sum *= alpha;
          if (i > 0) {
#pragma unroll 1
            for (int c = 0; c < DV; c += 16) {
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
        // ---- P = 2^(v factor - use) as hi + lo terms: of every 32 columns of S, 16 and 16 ----
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
          if (c0 + 32 < kKeys) load32(s_addr + c0 + 32, v[((c0 >> 5) & 1) ^ 1]);  // under this chunk's exponentials
#pragma unroll
          for (int k = 0; k < 16; ++k) {
            float a, e;
            unpack2(fma2(pack2(now[2 * k], now[2 * k + 1]), f2, m2), a, e);
            a = exp2_fast(a);
            e = exp2_fast(e);
            const uint64_t pe = pack2(a, e);
            sums[k & 1] = add2(sums[k & 1], pe);
            hi[k] = pack_bf16x2(a, e);
            float ra, re;
            unpack2(fma2(pack2(bf16_lo(hi[k]), bf16_hi(hi[k])), minus, pe), ra, re);
            lo[k] = pack_bf16x2(ra, re);
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

      // ---- normalise and store ----
      if (n > 0) {
        mbar_wait_bounded(&o_full[b], o_phase & 1, abort_flag, kStatusAttnTimeout);
        ++o_phase;
        tcgen05_fence_after_sync();
      }
      float top_scale = 1.f;
      if (EXTRA && p.sinks != nullptr) {
        const float sink = p.sinks[head] * kLog2e, most = fmaxf(top, sink);
        top_scale = exp2f(top - most);
        sum = sum * top_scale + exp2f(sink - most);
      }
      float inv = sum > 0.f ? 1.f / sum : 0.f;  // a token that sees no key gets zeros, as flash-attn does
      if (EXTRA && tok >= 0) inv *= top_scale * (p.diff ? p.out_scale : output_factor(p, tok, head));
#pragma unroll 1
      for (int c0 = 0; c0 < DV; c0 += 32) {
        float o[32];
        __syncwarp();
        if (n > 0) {
          load32(o_addr + c0, o);
          tmem_ld_wait();
          arrived32(o);
        }
        if (tok < 0 || (c0 >= p.dv && !(EXTRA && p.diff))) continue;
        if (n == 0) {
#pragma unroll
          for (int k = 0; k < 32; ++k) o[k] = 0.f;
        }
        if (EXTRA && p.diff) {
          float4* o32 = reinterpret_cast<float4*>(p.ws_o + (static_cast<int64_t>(tok) * p.nq + head) * DV + c0);
#pragma unroll
          for (int k = 0; k < 8; ++k) o32[k] = make_float4(o[4 * k] * inv, o[4 * k + 1] * inv, o[4 * k + 2] * inv, o[4 * k + 3] * inv);
          continue;
        }
        const int count = min(32, p.dv - c0);
        if (EXTRA && p.value_gates) {
          const uint32_t* gates = reinterpret_cast<const uint32_t*>(p.gate + tok * p.gate_ld + head * p.dv + c0);
#pragma unroll
          for (int k = 0; k < 16; ++k) {
            if (2 * k >= count) continue;
            const uint32_t gt = gates[k];
            o[2 * k] = __fdividef(o[2 * k], 1.f + __expf(-bf16_lo(gt)));
            o[2 * k + 1] = __fdividef(o[2 * k + 1], 1.f + __expf(-bf16_hi(gt)));
          }
        }
        __nv_bfloat16* dst = p.out + tok * p.out_ld + head * p.dv + c0;
        const bool vec = (reinterpret_cast<uintptr_t>(dst) & 15) == 0;
#pragma unroll
        for (int k = 0; k < 32; k += 8) {
          if (k >= count) continue;
          uint32_t w[4];
#pragma unroll
          for (int q = 0; q < 4; ++q) w[q] = pack_bf16x2(o[k + 2 * q] * inv, o[k + 2 * q + 1] * inv);
          if (vec && k + 8 <= count) {
            *reinterpret_cast<uint4*>(dst + k) = make_uint4(w[0], w[1], w[2], w[3]);
          } else {
#pragma unroll
            for (int q = 0; q < 4; ++q)
              if (k + 2 * q < count) *reinterpret_cast<uint32_t*>(dst + k + 2 * q) = w[q];
          }
        }
      }
    }
  }

  tcgen05_fence_before_sync();
  __syncthreads();
  if (warp == kSoftmaxWarps) tmem_dealloc(tmem, 512);
}

// Whether four units per CTA leave enough CTAs for the SMs: one for every second SM, of the units that the tokens fill.  (A prompt of 300 tokens, 40 CTAs
// here and 152 there: 17.5 us with either; 8 prompts of 300, 304 CTAs: 44 us here, 60 us with one unit per CTA.)  With keys and values of 64 columns the
// other kernel takes half as long: there only lists come here whose units are 97 % full, so few of them a request's last (8 prompts of 300 over 16 heads
// 27 us here, 21 there; 4 of 2048 113 and 201).
template <int DK, int DV>
static bool preferred(const Params& p, const int32_t* units, int num_units, int mix) {
  const int qb = 64 / p.G, filled = std::min(num_units, (p.T + qb - 1) / qb);
  if (mix == kShortRequests || (DK == 64 && DV == 64 && (num_units - filled) * 32 > num_units)) return false;
  return aligned16(units) && static_cast<int64_t>((filled + kUnitsPerCta - 1) / kUnitsPerCta) * p.nkv * 2 >= sm_count();
}

template <int DK, int DV, int FORM>
static int launch(const Params& p, const CUtensorMap* mk, const CUtensorMap* mv, const int32_t* units, int num_units, bool all,
                  cudaStream_t stream) {
  using C = Config<DK, DV>;
  static std::atomic<uint64_t> smem_attr_done{0};
  if (ensure_dynamic_smem(paged_prompt_kernel<DK, DV, FORM>, C::kSmemBytes, smem_attr_done) != B200_OK) return B200_ERR_LAUNCH;
  const int64_t ctas = static_cast<int64_t>((num_units + kUnitsPerCta - 1) / kUnitsPerCta) * p.nkv;
  if (ctas > 0x7fffffff) return B200_ERR_INVALID_ARGUMENT;
  return launch_pdl(paged_prompt_kernel<DK, DV, FORM>, dim3(static_cast<unsigned>(ctas)), dim3(kThreadsPrompt), C::kSmemBytes, stream, *mk, *mv, p,
                    units, num_units, all ? 1 : 0);
}

}  // namespace prompt
}  // namespace attn
}  // namespace b200
