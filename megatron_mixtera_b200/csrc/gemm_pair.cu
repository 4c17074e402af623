// y[M, N] = x[M, K] * w[N, K]^T for many tokens (prompts): bf16 operands, or E4M3 with one E8M0 scale per 32 elements.
//
// The weight-streaming kernels (gemm_bf16.cu, gemm_mxfp8.cu) give a CTA one 128-feature x 256-token tile: 48 KB per K block through the L2 -> SM path
// for 128 x 256 outputs, one tile's epilogue after its products, two stages of copies in flight where a K block is 128 bytes wide.  With thousands of
// tokens that path and the epilogue bound them, not HBM.  Here a PAIR of CTAs on two SMs owns 256 tokens x 256 features (tcgen05.mma.cta_group::2,
// M = 256, N = 256): each CTA stages its 128 tokens and its 128 weight rows, 32 KB per K block for the same 128 x 256 outputs, and walks over tiles
// (persistent) so that the next tile's copies and, with bf16, its products run under the epilogue.
//
//   warps 0-7           epilogue: TMEM lane = token, so a thread holds consecutive features of one token and stores them from registers
//   warp 8, lane 0      producer of its CTA; all copies complete on the LEADER's (cluster rank 0) full barrier
//   warp 9, lane 0      leader only: the pair's MMAs; commits go to both CTAs' barriers
//
// Measured, before -> after (burst; the power cap takes 10 % off both in long runs): bf16, 7700 tokens, 28672 x 4096: 1145 -> 1400 TFLOP/s, 4096 x 14336:
// 1220 -> 1370; MXFP8, 13000 tokens, 28672 x 4096 with SwiGLU and quantisation: 1430 -> 2110, 4096 x 14336: 1410 -> 2100.  What bounds them now: with scales the
// copies of ~34 KB per K block and the read-out of the one accumulator; bf16 stops short of the power cap (cuBLAS reaches 1590 in the same burst).
//
// Experts' products (moe.cu) are the same kernel over a device-built list of (expert, first row, rows <= 256) entries, the shared expert's tiles in front.
//
// bf16 accumulators are double-buffered (2 x 256 columns = all of tensor memory); with scales there is one accumulator beside the scale slots, and
// the eight epilogue warps read it out before they compute.  Tiles are walked in groups of token blocks, features outermost within a group and backwards in
// every other one, so that what the pairs work on at a time stays in L2.
#include "common.cuh"
#include "quant.cuh"

namespace b200 {
namespace gemm {
namespace pair {

constexpr int kEpilogueWarps = 8;
constexpr int kThreadsPair = (kEpilogueWarps + 2) * 32;
constexpr int kTile = 256;      // tokens, and features, of a pair's tile

// Features as they are; [64 gate | 64 up] rows; [16 gate | 16 up] rows (experts); rank 0 holds gate rows, rank 1 the matching up rows.
enum Form { kPlain, kGated64, kGated16, kGatedHalves };

template <bool MX>
struct Config {
  static constexpr int kStageX = 128 * 128, kStageW = 128 * 128;  // bytes: 128 rows of 128 bytes (64 bf16 or 128 E4M3)
  static constexpr int kOffSfX = kStageX + kStageW;
  static constexpr int kOffSfW = kOffSfX + 512;
  static constexpr int kTx = MX ? kOffSfW + 2 * 512 : kOffSfX;
  static constexpr int kStageBytes = (kTx + 1023) / 1024 * 1024;
  static constexpr int kStages = 6;
  static constexpr int kBuffers = MX ? 1 : 2;
  static constexpr int kSfCols = 12;  // scale columns of a stage: 4 of the tokens, 8 of the features
  static constexpr int kSmemBytes = kStages * kStageBytes + 1024 + 256;
  static constexpr int kTmemCols = 512;
  static_assert(!MX || kTile + kStages * kSfCols <= kTmemCols, "one accumulator and the scale slots");
};

struct Args {
  Params p;         // experts: sizes of one expert's problem (N: weight rows per expert)
  uint8_t* q_out;   // kGatedHalves: E4M3 [M][F] and its scales instead of y
  uint8_t* sf_out;
  int k_tiles;      // K / 128 (scaled operands)
  int m_tiles, n_tiles, tiles;
  int group_m;      // token blocks of a group of tiles
  // Experts: tokens sorted by expert, a device-built list of (expert, first row, rows <= 256) entries instead of m_tiles.  A second problem (a shared
  // expert: all tokens, weights and sizes of its own) may come in front of it.
  Params shared;
  const int4* list;
  const int32_t* list_length;
  int list_capacity, experts, shared_n_tiles, shared_tiles;
};

// One 256 x 256 tile of work.
struct Unit {
  const Params* p;
  int m0, m_end, nt, w_row;  // first token row and the end of the rows it may write, feature block, first weight row
  bool shared;
};

__device__ __forceinline__ void umma_f16_pair(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "setp.ne.b32 p, %4, 0;\n"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n"
      "}\n" ::"r"(tmem_d),
      "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void umma_mxf8_pair(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc, uint32_t tmem_sfa,
                                               uint32_t tmem_sfb, uint32_t accumulate) {
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "setp.ne.b32 p, %4, 0;\n"
      "tcgen05.mma.cta_group::2.kind::mxf8f6f4.block_scale [%0], %1, %2, %3, [%5], [%6], p;\n"
      "}\n" ::"r"(tmem_d),
      "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate), "r"(tmem_sfa), "r"(tmem_sfb)
      : "memory");
}
// Scale tile -> tensor memory, in both CTAs of the pair: each copies from its own shared memory.
__device__ __forceinline__ void tmem_cp_32x128b_warpx4_pair(uint32_t taddr, uint64_t smem_desc) {
  asm volatile("tcgen05.cp.cta_group::2.32x128b.warpx4 [%0], %1;" ::"r"(taddr), "l"(smem_desc) : "memory");
}

// 16 consecutive bf16 outputs (32 bytes, one sector) of a token.
__device__ __forceinline__ void store16(__nv_bfloat16* dst, const float* v, int count, bool vec) {
  if (vec) {
    uint32_t w[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) w[i] = pack_bf16x2(v[2 * i], v[2 * i + 1]);
    *reinterpret_cast<uint4*>(dst) = make_uint4(w[0], w[1], w[2], w[3]);
    *reinterpret_cast<uint4*>(dst + 8) = make_uint4(w[4], w[5], w[6], w[7]);
  } else {
#pragma unroll
    for (int i = 0; i < 16; ++i)
      if (i < count) dst[i] = __float2bfloat16_rn(v[i]);
  }
}

// silu(g) u with the rounding points of the unfused path: both products, silu and the result in bf16.
__device__ __forceinline__ float swiglu_rounded(uint32_t g_bits, uint32_t u_bits) {
  const float g = bf16_round(__uint_as_float(g_bits)), u = bf16_round(__uint_as_float(u_bits));
  return bf16_round(bf16_round(g / (1.f + expf(-g))) * u);
}

template <bool MX, int FORM, bool EXPERTS>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kThreadsPair, 1)
gemm_pair_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x,
                 const __grid_constant__ CUtensorMap map_sfw, const __grid_constant__ CUtensorMap map_sfx, const __grid_constant__ Args a) {
  using C = Config<MX>;
  extern __shared__ uint8_t smem_raw[];
  // (the dynamic shared memory of both CTAs starts at the same offset: the pair's MMA and the remote arrives rely on that)
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + C::kStages * C::kStageBytes);  // used in the leader only
  uint64_t* empty_bar = full_bar + C::kStages;
  uint64_t* acc_full = empty_bar + C::kStages;
  uint64_t* acc_empty = acc_full + 2;                                                    // used in the leader only
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t rank = cluster_cta_rank();  // 0 = leader
  const int first = blockIdx.x >> 1, stride = gridDim.x >> 1;
  constexpr int kProducerWarp = kEpilogueWarps, kMmaWarp = kEpilogueWarps + 1;

  if (tid == 0) {
    for (int s = 0; s < C::kStages; ++s) {
      mbar_init(&full_bar[s], 1);   // the leader's producer (it expects the bytes of both CTAs)
      mbar_init(&empty_bar[s], 1);  // the MMA commit
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&acc_full[b], 1);                       // the MMA commit
      mbar_init(&acc_empty[b], 2 * kEpilogueWarps);     // the epilogue warps of both CTAs
    }
    *abort_flag = 0;
    fence_barrier_init();
    prefetch_tensormap(&map_w);
    prefetch_tensormap(&map_x);
  }
  if (warp == kProducerWarp) {
    tmem_alloc_pair(tmem_slot, C::kTmemCols);
    tmem_relinquish_alloc_permit_pair();
  }
  tcgen05_fence_before_sync();
  __syncthreads();
  cluster_barrier();  // both CTAs' barriers are initialised and both allocations made before anything crosses over
  tcgen05_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  pdl_launch_dependents();

  pdl_wait();  // operands (and the list of experts' tiles) are earlier kernels' output, and y may still be read by them
  const int tiles = EXPERTS ? a.shared_tiles + min(*a.list_length, a.list_capacity) * a.n_tiles : a.tiles;
  // tile number -> unit; false for an entry that no kernel of ours writes (every role leaves it out)
  auto unit_of = [&](int tile, Unit& u) {
    u.p = &a.p;
    u.shared = false;
    if constexpr (EXPERTS) {
      if (tile < a.shared_tiles) {
        u.p = &a.shared;
        u.shared = true;
        u.m0 = tile / a.shared_n_tiles * kTile;
        u.nt = tile % a.shared_n_tiles;
        u.m_end = a.shared.M;
        u.w_row = u.nt * kTile;
        return true;
      }
      const int4 e = a.list[(tile - a.shared_tiles) / a.n_tiles];
      u.nt = (tile - a.shared_tiles) % a.n_tiles;
      u.m0 = e.y;
      u.m_end = min(e.y + min(e.z, kTile), a.p.M);
      u.w_row = e.x * a.p.N + u.nt * kTile;
      return static_cast<unsigned>(e.x) < static_cast<unsigned>(a.experts) && e.y >= 0 && e.z > 0;
    } else {
      const int per_group = a.group_m * a.n_tiles;
      const int group = tile / per_group, in = tile - group * per_group;
      const int rows = min(a.group_m, a.m_tiles - group * a.group_m);
      u.nt = in / rows;
      u.m0 = (group * a.group_m + (in - u.nt * rows)) * kTile;
      if (group & 1) u.nt = a.n_tiles - 1 - u.nt;
      u.m_end = a.p.M;
      u.w_row = u.nt * kTile;
      return true;
    }
  };

  if (warp == kProducerWarp) {
    if (lane == 0) {
      const uint32_t leader_full0 = cluster_addr_of(&full_bar[0], 0);  // (barriers are 8 bytes apart)
      int it = 0;
      for (int tile = first; tile < tiles; tile += stride) {
        Unit u;
        if (!unit_of(tile, u)) continue;
        const int m0 = u.m0 + static_cast<int>(rank) * 128, num_kb = u.p->num_k_blocks;
        // scaled operands: this CTA's weight tile (128 rows), and the two whose scales both CTAs need
        const int tile0 = FORM == kGatedHalves ? u.nt : 2 * u.nt;
        const int tile1 = FORM == kGatedHalves ? u.nt + a.n_tiles : 2 * u.nt + 1;
        const int w_tile = rank == 0 ? tile0 : tile1;
        const CUtensorMap* mx_ = EXPERTS && u.shared ? &map_sfx : &map_x;  // (without scales those maps are the second problem's)
        const CUtensorMap* mw = EXPERTS && u.shared ? &map_sfw : &map_w;
        for (int kb = 0; kb < num_kb; ++kb, ++it) {
          const int s = it % C::kStages;
          mbar_wait_bounded(&empty_bar[s], ((it / C::kStages) & 1) ^ 1, abort_flag, kStatusGemmTimeout);
          if (rank == 0) mbar_arrive_expect_tx(&full_bar[s], 2 * C::kTx);
          uint8_t* stage = smem + s * C::kStageBytes;
          const uint32_t full = leader_full0 + 8 * s;
          if constexpr (MX) {
            tma_load_2d_pair(stage, &map_x, full, kb * 128, m0);
            tma_load_2d_pair(stage + C::kStageX, &map_w, full, 0, (w_tile * a.k_tiles + kb) * 128);  // packed tile
            tma_load_2d_pair(stage + C::kOffSfX, &map_sfx, full, 0, (m0 >> 7) * a.k_tiles + kb);
            tma_load_2d_pair(stage + C::kOffSfW, &map_sfw, full, 0, tile0 * a.k_tiles + kb);
            tma_load_2d_pair(stage + C::kOffSfW + 512, &map_sfw, full, 0, tile1 * a.k_tiles + kb);
          } else {
            tma_load_2d_pair(stage, mx_, full, kb * 64, m0);
            tma_load_2d_pair(stage + C::kStageX, mw, full, kb * 64, u.w_row + static_cast<int>(rank) * 128);
          }
        }
      }
    }
  } else if (warp == kMmaWarp) {
    if (lane == 0 && rank == 0) {
      // ------- UMMA issuer (leader): D[token, feature] = X[token, k] * W[feature, k]^T, 256 x 256 per pair -------
      int it = 0, n = 0;
      for (int tile = first; tile < tiles; tile += stride) {
        Unit u;
        if (!unit_of(tile, u)) continue;
        const int num_kb = u.p->num_k_blocks;
        const int b = n % C::kBuffers;
        mbar_wait_bounded(&acc_empty[b], ((n / C::kBuffers) & 1) ^ 1, abort_flag, kStatusGemmTimeout);
        const uint32_t acc = tmem_base + b * kTile;
        for (int kb = 0; kb < num_kb; ++kb, ++it) {
          const int s = it % C::kStages;
          mbar_wait_bounded(&full_bar[s], (it / C::kStages) & 1, abort_flag, kStatusGemmTimeout);
          tcgen05_fence_after_sync();
          const uint32_t stage_addr = smem_u32(smem + s * C::kStageBytes);
          const uint64_t x_desc = umma_desc_k_major_sw128(stage_addr);
          const uint64_t w_desc = umma_desc_k_major_sw128(stage_addr + C::kStageX);
          if constexpr (MX) {
            const uint32_t sfx = tmem_base + kTile + s * C::kSfCols, sfw = sfx + 4;
            tmem_cp_32x128b_warpx4_pair(sfx, umma_desc_sf_tile(stage_addr + C::kOffSfX));
            tmem_cp_32x128b_warpx4_pair(sfw, umma_desc_sf_tile(stage_addr + C::kOffSfW));
            tmem_cp_32x128b_warpx4_pair(sfw + 4, umma_desc_sf_tile(stage_addr + C::kOffSfW + 512));
#pragma unroll
            for (int k = 0; k < 4; ++k)
              umma_mxf8_pair(acc, x_desc + 2 * k, w_desc + 2 * k, umma_idesc_mxf8(256, 256, k, k), sfx, sfw, (kb > 0 || k > 0) ? 1u : 0u);
          } else {
#pragma unroll
            for (int k = 0; k < 4; ++k)
              umma_f16_pair(acc, x_desc + 2 * k, w_desc + 2 * k, umma_idesc_bf16(256, 256), (kb > 0 || k > 0) ? 1u : 0u);
          }
          umma_commit_both(&empty_bar[s]);
        }
        umma_commit_both(&acc_full[b]);
        ++n;
      }
    }
  } else {
    // ---------------- epilogue: lane quadrant = warp % 4, 128 of the 256 columns per warp ----------------
    const int quad = warp & 3, half = warp >> 2;
    const uint32_t leader_acc_empty0 = cluster_addr_of(&acc_empty[0], 0);
    int n = 0;
    for (int tile = first; tile < tiles; tile += stride) {
      Unit u;
      if (!unit_of(tile, u)) continue;
      const Params& p = *u.p;
      const int nt = u.nt;
      const int b = n % C::kBuffers;
      const int m = u.m0 + static_cast<int>(rank) * 128 + quad * 32 + lane;  // this thread's token
      const bool m_ok = m < u.m_end;
      mbar_wait_bounded(&acc_full[b], (n / C::kBuffers) & 1, abort_flag, kStatusGemmTimeout);
      ++n;
      tcgen05_fence_after_sync();
      const uint32_t acc = tmem_base + (static_cast<uint32_t>(quad * 32) << 16) + b * kTile;
      auto release = [&] {
        tcgen05_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive_cluster(leader_acc_empty0 + 8 * b);
      };
      if constexpr (FORM == kPlain) {
        constexpr int kChunk = MX ? 128 : 64;  // (a single accumulator is read out as a whole before anything else)
        const int n0 = nt * kTile + half * 128;
        const uint32_t from = acc + half * 128;
        const bool vec = (p.ldy & 7) == 0 && (reinterpret_cast<uintptr_t>(p.y) & 15) == 0;
        const bool vec_f = (p.N & 3) == 0;
#pragma unroll 1
        for (int c0 = 0; c0 < 128; c0 += kChunk) {
          uint32_t r[kChunk];
          __syncwarp();  // (rows past the last token have left the loop's body early)
#pragma unroll
          for (int j = 0; j < kChunk; j += 32) tmem_ld_32x32b_x32(from + c0 + j, *reinterpret_cast<uint32_t(*)[32]>(r + j));
          tmem_ld_wait();
          if (c0 + kChunk == 128) release();
          if (!m_ok) continue;
          if (p.keep_partials) {
            float* dst = p.partials + static_cast<int64_t>(m) * p.N + n0 + c0;
#pragma unroll
            for (int j = 0; j < kChunk; j += 4) {
              const int left = p.N - (n0 + c0 + j);
              if (left >= 4 && vec_f) {
                __stcg(reinterpret_cast<float4*>(dst + j), make_float4(__uint_as_float(r[j]), __uint_as_float(r[j + 1]), __uint_as_float(r[j + 2]),
                                                                       __uint_as_float(r[j + 3])));
              } else {
#pragma unroll
                for (int k = 0; k < 4; ++k)
                  if (k < left) __stcg(dst + j + k, __uint_as_float(r[j + k]));
              }
            }
            continue;
          }
          __nv_bfloat16* dst = p.y + static_cast<int64_t>(m) * p.ldy + n0 + c0;
#pragma unroll
          for (int j = 0; j < kChunk; j += 16) {
            const int left = p.N - (n0 + c0 + j);
            float v[16];
#pragma unroll
            for (int k = 0; k < 16; ++k) {
              v[k] = __uint_as_float(r[j + k]);
              // bias is added to the bf16-rounded product, as `matmul(x, w.t()) + bias` does
              if (p.bias != nullptr && k < left) v[k] = bf16_round(v[k]) + __bfloat162float(p.bias[n0 + c0 + j + k]);
              v[k] = apply_act(v[k], p.act);
            }
            if (left > 0) store16(dst + j, v, left, vec && left >= 16);
          }
        }
      } else if constexpr (FORM == kGated16) {
        // columns [16 gate | 16 up] in turn: this warp's 128 columns give 64 outputs
        const int o0 = nt * 128 + half * 64;
        const uint32_t from = acc + half * 128;
        const bool vec = (p.ldy & 7) == 0 && (reinterpret_cast<uintptr_t>(p.y) & 15) == 0;
        const float scale = p.row_scale != nullptr && m_ok ? p.row_scale[m] : 1.f;
#pragma unroll 1
        for (int c0 = 0; c0 < 128; c0 += 32) {
          uint32_t r[32];
          __syncwarp();
          tmem_ld_32x32b_x32(from + c0, r);
          tmem_ld_wait();
          if (c0 == 96) release();
          if (!m_ok || o0 + c0 / 2 >= (p.N >> 1)) continue;
          float v[16];
#pragma unroll
          for (int k = 0; k < 16; ++k) {
            const float gt = __uint_as_float(r[k]) * scale, up = __uint_as_float(r[16 + k]) * scale;
            v[k] = p.gated == kGatedPlain ? __fdividef(gt, 1.f + __expf(-gt)) * up : clamped_glu_fast(gt, up, p.glu_limit, p.glu_alpha);
          }
          store16(p.y + static_cast<int64_t>(m) * p.ldy + o0 + c0 / 2, v, 16, vec);
        }
      } else if constexpr (FORM == kGated64) {
        // columns [64 gate | 64 up] twice: this warp's 128 columns give 64 outputs
        const int o0 = nt * 128 + half * 64;  // first output column
        const uint32_t from = acc + half * 128;
        const bool vec = (p.ldy & 7) == 0 && (reinterpret_cast<uintptr_t>(p.y) & 15) == 0;
#pragma unroll 1
        for (int c0 = 0; c0 < 64; c0 += 32) {
          uint32_t g[32], u[32];
          __syncwarp();
          tmem_ld_32x32b_x32(from + c0, g);
          tmem_ld_32x32b_x32(from + 64 + c0, u);
          tmem_ld_wait();
          if (c0 == 32) release();
          if (!m_ok || o0 + c0 >= (p.N >> 1)) continue;
          __nv_bfloat16* dst = p.y + static_cast<int64_t>(m) * p.ldy + o0 + c0;
#pragma unroll
          for (int j = 0; j < 32; j += 16) {
            float v[16];
#pragma unroll
            for (int k = 0; k < 16; ++k) v[k] = swiglu_rounded(g[j + k], u[j + k]);
            store16(dst + j, v, 16, vec);
          }
        }
      } else {
        // columns [128 gate | 128 up]: this warp finishes 64 of the 128 features, two scale blocks of 32
        const int f0 = nt * 128 + half * 64;
        const int F = p.N >> 1;
        const bool vec = (p.ldy & 7) == 0 && (reinterpret_cast<uintptr_t>(p.y) & 15) == 0;
        uint32_t g[64], u[64];
        __syncwarp();
#pragma unroll
        for (int j = 0; j < 64; j += 32) {
          tmem_ld_32x32b_x32(acc + half * 64 + j, *reinterpret_cast<uint32_t(*)[32]>(g + j));
          tmem_ld_32x32b_x32(acc + 128 + half * 64 + j, *reinterpret_cast<uint32_t(*)[32]>(u + j));
        }
        tmem_ld_wait();
        release();
        if (!m_ok) continue;
#pragma unroll
        for (int c0 = 0; c0 < 64; c0 += 32) {
          float v[32];
          float amax = 0.f;
#pragma unroll
          for (int j = 0; j < 32; ++j) {
            v[j] = swiglu_rounded(g[c0 + j], u[c0 + j]);
            amax = fmaxf(amax, fabsf(v[j]));
          }
          const int col = f0 + c0;
          if (a.q_out != nullptr) {
            const uint32_t e = mx::e8m0_scale_byte(amax);
            const float inv = scalbnf(1.0f, 127 - static_cast<int>(e));
            uint32_t w[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              const uint32_t lo = __nv_cvt_float2_to_fp8x2(make_float2(v[4 * j] * inv, v[4 * j + 1] * inv), __NV_SATFINITE, __NV_E4M3);
              const uint32_t hi = __nv_cvt_float2_to_fp8x2(make_float2(v[4 * j + 2] * inv, v[4 * j + 3] * inv), __NV_SATFINITE, __NV_E4M3);
              w[j] = lo | (hi << 16);
            }
            uint4* dst = reinterpret_cast<uint4*>(a.q_out + static_cast<int64_t>(m) * F + col);
            dst[0] = make_uint4(w[0], w[1], w[2], w[3]);
            dst[1] = make_uint4(w[4], w[5], w[6], w[7]);
            a.sf_out[mx::sf_offset(m, col >> 5, F / 128)] = static_cast<uint8_t>(e);
          } else {
            __nv_bfloat16* dst = p.y + static_cast<int64_t>(m) * p.ldy + col;
            store16(dst, v, 16, vec);
            store16(dst + 16, v + 16, 16, vec);
          }
        }
      }
    }
  }

  // Neither CTA may leave (or free tensor memory) while the other's MMA, copies or arrives can still reach it.
  tcgen05_fence_before_sync();
  __syncthreads();
  cluster_barrier();
  if (warp == kProducerWarp) tmem_dealloc_pair(tmem_base, C::kTmemCols);
}

// Whether the pairs' tiles are the better split: at least one tile for every pair of SMs, of more rows than one block of the streaming kernels' tokens.  (64
// tiles, 1024 tokens x 4096 x 4096: 48.8 us here, 44.2 us with K split over the streaming kernel's CTAs.)
static int64_t tiles_of(int M, int N) { return static_cast<int64_t>((M + kTile - 1) / kTile) * ((N + kTile - 1) / kTile); }
static bool enough(int M, int N, int fewest) { return M > fewest && tiles_of(M, N) >= sm_count() / 2; }

// A pair's tile costs ~8 us more than its products do here (start, operands only behind the wait, the last epilogue), the streaming kernel's two CTAs for the
// same outputs ~4.  Up to two waves of pairs (148 tiles) that is made up for by about 370 000 tiles x K: K 512 20 us against 13, 1024 23.5 and 18.4, 2048 31.5 and
// 28.8, 4096 50.5 and 49-58 (75 tiles 47.8, 112 51.9), 8192 1.04-1.11 x as fast.  From three waves on by K 1280 (1.04-1.16 x; 1024: 0.87-1.03 x, 1.04-1.13 x from
// 444 tiles on; 512: 0.70-0.86 x).  256 x 128256 x 8192: 489 us on the streaming kernel, 417 here.
static bool preferred_bf16(int M, int N, int K) {
  if (!enough(M, N, 128)) return false;
  const int64_t tiles = tiles_of(M, N);
  return tiles <= sm_count() ? tiles * K >= 368640 : K >= (tiles >= 3 * sm_count() ? 1024 : 1280);
}
// SwiGLU in the epilogue, which the streaming kernel does not overlap: 1.1-2.0 x as fast at any K.
static bool preferred_swiglu(int M, int N) { return enough(M, N, 128); }
// Scales double what a byte of operands is worth: up to 148 tiles from K 1024 on (1.03-1.6 x as fast; 512: 0.91-0.94 x), else from 512 on (0.98-1.17 x; 256: 0.88-0.99 x).
// Up to 256 rows the streaming kernel reads a weight once as well.
static bool preferred_mxfp8(int M, int N, int K) { return enough(M, N, 256) && K >= (tiles_of(M, N) <= sm_count() ? 1024 : 512); }
// The streaming kernel's CTAs take 128 x 128 gate and up rows: one wave of them is faster than two of pairs (1100 x 4096 x 4096, 144 CTAs or 80 tiles: 27.5 and 39.6 us).
static bool preferred_mxfp8_swiglu(int M, int F, int K) {
  const bool one_wave = static_cast<int64_t>((M + 127) / 128) * (F / 128) <= sm_count() && tiles_of(M, 2 * F) > sm_count() / 2;
  return preferred_mxfp8(M, 2 * F, K) && !one_wave;
}

template <bool MX, int FORM, bool EXPERTS = false>
static int launch(Args& a, const CUtensorMap* mw, const CUtensorMap* mx_, const CUtensorMap* msw, const CUtensorMap* msx, cudaStream_t stream) {
  using C = Config<MX>;
  a.n_tiles = (a.p.N + kTile - 1) / kTile;
  if (!EXPERTS) {
    a.m_tiles = (a.p.M + kTile - 1) / kTile;
    a.tiles = a.m_tiles * a.n_tiles;
    // The weights are read once for each group, so long groups, while their tokens stay in L2 beside the weights in use: 16 blocks of up to 8 KB a token.  In
    // long runs at the power cap, us with 8 and 16 blocks, features always forwards: 7700 x 28672 x 4096 1420, 1397, x 14336 -> 4096 722, 732; MXFP8 15500 x 28672 x
    // 4096 1830, 1804, x 14336 -> 4096 893, 902.  Every other group backwards: 0 to 1.2 % less.  (A group's size at run time costs a tile of a short K: MXFP8 1.7 % with K 512, 0.8 %
    // up to 2048.)
    a.group_m = static_cast<int64_t>(a.p.K) * (MX ? 1 : 2) <= 8192 ? 16 : 8;
  }
  static std::atomic<uint64_t> smem_attr_done{0};
  if (ensure_dynamic_smem(gemm_pair_kernel<MX, FORM, EXPERTS>, C::kSmemBytes, smem_attr_done) != B200_OK) return B200_ERR_LAUNCH;
  const int pairs = min(sm_count() / 2, a.tiles);
  return launch_pdl(gemm_pair_kernel<MX, FORM, EXPERTS>, dim3(2 * pairs), dim3(kThreadsPair), C::kSmemBytes, stream, *mw, *mx_, *msw, *msx, a);
}

static Params params(void* y, int64_t ldy, const void* bias, int M, int N, int K, int k_block, int act, float* partials) {
  Params p;
  p.bias = static_cast<const __nv_bfloat16*>(bias);
  p.y = static_cast<__nv_bfloat16*>(y);
  p.partials = partials;
  p.ldy = ldy;
  p.M = M;
  p.N = N;
  p.K = K;
  p.num_k_blocks = (K + k_block - 1) / k_block;
  p.k_blocks_per_split = p.num_k_blocks;
  p.num_splits = 1;
  p.keep_partials = partials != nullptr;
  p.gated = 0;
  p.act = act;
  return p;
}

// bf16; `partials`: the fp32 product [M][N] instead of y.
static int launch_bf16(const void* x, int64_t ldx, const void* w, const void* bias, void* y, int64_t ldy, int M, int N, int K, cudaStream_t stream,
                       float* partials, bool gated, int act) {
  const uint64_t wd[2] = {static_cast<uint64_t>(K), static_cast<uint64_t>(N)}, xd[2] = {static_cast<uint64_t>(K), static_cast<uint64_t>(M)};
  const uint64_t ws[1] = {static_cast<uint64_t>(K) * 2}, xs[1] = {static_cast<uint64_t>(ldx) * 2};
  const uint32_t box[2] = {64, 128};
  const CUtensorMap* mw = get_tensor_map(w, 2, wd, ws, box, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B);
  const CUtensorMap* mx_ = get_tensor_map(x, 2, xd, xs, box, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B);
  if (!mw || !mx_) return B200_ERR_DRIVER;
  Args a = {};
  a.p = params(y, ldy, bias, M, N, K, 64, act, partials);
  return gated ? launch<false, kGated64>(a, mw, mx_, mw, mx_, stream) : launch<false, kPlain>(a, mw, mx_, mw, mx_, stream);
}

// E4M3 with E8M0 scales; `halves`: w is [gate ; up] (N = 2 F rows), the output silu(gate) up as E4M3 + scales (q_out, sf_out) or bf16 (y).
static int launch_mxfp8(const void* xq, const void* x_sf, const void* wq, const void* w_sf, const void* bias, void* y, int64_t ldy, int M, int N, int K,
                        cudaStream_t stream, float* partials, bool halves, void* q_out, void* sf_out) {
  const int k_tiles = K / 128, w_tiles = (N + 127) / 128, x_tiles = (M + 127) / 128;
  const uint64_t wd[2] = {128, static_cast<uint64_t>(w_tiles) * k_tiles * 128}, xd[2] = {static_cast<uint64_t>(K), static_cast<uint64_t>(M)};
  const uint64_t ws[1] = {128}, xs[1] = {static_cast<uint64_t>(K)};
  const uint32_t box[2] = {128, 128};
  const CUtensorMap* mw = get_tensor_map(wq, 2, wd, ws, box, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_DATA_TYPE_UINT8);
  const CUtensorMap* mx_ = get_tensor_map(xq, 2, xd, xs, box, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_DATA_TYPE_UINT8);
  // a scale tile is a row of 512 bytes = 128 words
  const uint64_t swd[2] = {128, static_cast<uint64_t>(w_tiles) * k_tiles}, sxd[2] = {128, static_cast<uint64_t>(x_tiles) * k_tiles};
  const uint64_t ss[1] = {512};
  const uint32_t sbox[2] = {128, 1};
  const CUtensorMap* msw = get_tensor_map(w_sf, 2, swd, ss, sbox, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_DATA_TYPE_INT32);
  const CUtensorMap* msx = get_tensor_map(x_sf, 2, sxd, ss, sbox, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_DATA_TYPE_INT32);
  if (!mw || !mx_ || !msw || !msx) return B200_ERR_DRIVER;
  Args a = {};
  a.p = params(y, ldy, bias, M, N, K, 128, B200_ACT_NONE, partials);
  a.k_tiles = k_tiles;
  a.q_out = static_cast<uint8_t*>(q_out);
  a.sf_out = static_cast<uint8_t*>(sf_out);
  return halves ? launch<true, kGatedHalves>(a, mw, mx_, msw, msx, stream) : launch<true, kPlain>(a, mw, mx_, msw, msx, stream);
}

// Experts' products (and the shared expert's, where there is one) over a list of 256-row entries.
static int launch_experts(const GroupedProblem& routed, const GroupedProblem& shared, const GroupedParams& gp, cudaStream_t stream) {
  auto maps = [&](const GroupedProblem& g, const Params& p, const CUtensorMap*& mw, const CUtensorMap*& mx_) {
    const uint64_t wd[2] = {static_cast<uint64_t>(p.K), static_cast<uint64_t>(p.N) * g.experts}, xd[2] = {static_cast<uint64_t>(p.K), static_cast<uint64_t>(p.M)};
    const uint64_t ws[1] = {static_cast<uint64_t>(p.K) * 2}, xs[1] = {static_cast<uint64_t>(g.ldx) * 2};
    const uint32_t box[2] = {64, 128};
    mw = get_tensor_map(g.w, 2, wd, ws, box, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B);
    mx_ = get_tensor_map(g.x, 2, xd, xs, box, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B);
    return mw && mx_;
  };
  const CUtensorMap *mw, *mx_;
  if (!maps(routed, gp.routed, mw, mx_)) return B200_ERR_DRIVER;
  const CUtensorMap *mws = mw, *mxs = mx_;
  Args a = {};
  a.p = gp.routed;
  a.shared_n_tiles = 1;
  if (shared.x != nullptr) {
    if (!maps(shared, gp.shared, mws, mxs)) return B200_ERR_DRIVER;
    a.shared = gp.shared;
    a.shared_n_tiles = (gp.shared.N + kTile - 1) / kTile;
    a.shared_tiles = a.shared_n_tiles * ((gp.shared.M + kTile - 1) / kTile);
  }
  for (Params* p : {&a.p, &a.shared}) {
    p->num_k_blocks = (p->K + 63) / 64;
    p->num_splits = 1;
    p->keep_partials = 0;
    p->partials = nullptr;
    p->bias = nullptr;
  }
  a.list = gp.tiles;
  a.list_length = gp.num_tiles;
  a.list_capacity = gp.max_tiles;
  a.experts = gp.experts;
  const int64_t most = a.shared_tiles + static_cast<int64_t>(gp.max_tiles) * ((gp.routed.N + kTile - 1) / kTile);
  if (most > 0x7fffffff) return B200_ERR_INVALID_ARGUMENT;
  a.tiles = static_cast<int>(most);
  return gp.routed.gated != 0 ? launch<false, kGated16, true>(a, mw, mx_, mws, mxs, stream) : launch<false, kPlain, true>(a, mw, mx_, mws, mxs, stream);
}

}  // namespace pair
}  // namespace gemm
}  // namespace b200
