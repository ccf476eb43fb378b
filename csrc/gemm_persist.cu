// bf16 GEMM for more than a few hundred tokens on pairs of SMs: tcgen05.mma with cta_group::2, persistent over the output tiles.
//
//     out[t, f] = sum_k X[t, k] W[f, k]  (+ sum_r X2[t, r] W2[f, r])  (+ residual[t, f])
//
// Orientation: tokens on lanes.  A pair of CTAs owns a tile of 256 tokens by bn features; each CTA holds 128 tokens of X and bn / 2 features of
// W per 64-wide k block, the tensor cores of both SMs read both halves of W, and each CTA's tensor memory receives its 128 tokens x bn
// features.  A lane's registers are then consecutive features of one token: the epilogue packs them (gate and up rows of an
// interleaved SwiGLU weight lie side by side) and stores 16 bytes at a time.
//
// What bounds it, and why this split: the tensor pipe for tiles of 256 features (0.52 us for 128 of the reduction at 1965 MHz, measured 0.6 to 0.8:
// all SMs at once draw the clock down), the operands' way from L2 for narrower ones (114 GB/s per SM, 0.35 us at 64 features).  gemm_fl_kernel (gemm_tcgen05.cu) has one tile per
// CTA: start-up, first loads and an epilogue that stages single bf16 values stand before and behind every main loop (24 us at K = 2048),
// and its 256 x 256 tiles leave a last wave of up to one sixth empty.  Here a CTA keeps two accumulators, so the epilogue of a tile runs under the
// main loop of the next, the pipeline never drains between tiles, and a tile is half as long (two SMs work on it) at the same operand
// bytes per product.  us, gemm_fl_kernel / this / cuBLAS on the same operands (plain, SwiGLU or residual as the layers use them):
//   tokens          4096 x 2048          12288 x 2048 SwiGLU    2048 x 2048 + residual   2048 x 6144 + residual
//   504          13.3 / 10.6 / 8.8        26.2 / 24.7 / 19.8       11.6 / 9.3 / 6.8        20.3 / 20.4 / 14.3
//   1504         22.4 / 21.9 / 19.0       62.2 / 53.4 / 50.9       17.4 / 14.8 / 11.0      38.0 / 31.4 / 26.6
//   3072         44.8 / 36.3 / 35.8        122 / 104 / 102         25.3 / 22.9 / 18.9      61.8 / 60.2 / 50.5
//   15696         201 / 172 / 171          672 / 533 / 505          139 / 97 / 90          372 / 269 / 254
// A stage holds 128 of the reduction, two blocks of 64 that one copy per operand brings: a step of the producer's and of the issuer's loop takes
// about 500 cycles whatever it carries (waits, branches, the election of a lane), and with blocks of 64 that stood above the tensor pipe (15696
// tokens, 2048 x 2048: 102 us; 264 tokens 15.6 us, now 8.9).
//
// Warp roles in each CTA: warp 0 = TMA producer (both CTAs signal the first CTA's barrier), warp 1 = tensor-memory owner and, in the first CTA of
// the pair, MMA issuer, warps 2..9 = epilogue (warp w reads tensor-memory lanes 32 * (w % 4) .. + 31).  An epilogue warp stages its own 32 tokens
// x 64 weight rows and stores them with its own TMA store, so the epilogue warps never wait for one another.
#include <cuda.h>

#include "attn_common.cuh"
#include "common.cuh"
#include "gemm_maps.cuh"

namespace tahb {

struct PersistParams {
  int M, F_out;              // tokens, output features
  int kb_main, kb_ext;       // blocks of 64 of the reduction: of the product and of its K-extension
  int bn;                    // weight rows of a tile, a multiple of 64
  int stages, stage_bytes, b_bytes;
  int tiles_m, tiles_n, group;
  int a_mn, b_mn;            // operand stored [reduction, token] / [reduction, feature] (the backward products)
  const __nv_bfloat16* residual;
  long long ldr;
  float act_up, act_low;     // xIELU
  int* status;
  const uint32_t* wait_flag; // rows of X that peers deliver, see gemm_tcgen05.cu
  const uint32_t* wait_target;
  int wait_world;
  unsigned long long wait_limit_ns;
};

constexpr int PERSIST_STAGE_SPACE = 192 * 1024;       // of operand stages
constexpr int PERSIST_STG = 4096;                     // an epilogue warp's staging buffer: 32 tokens x 64 features
constexpr int PERSIST_THREADS = 320;
constexpr int PERSIST_SMEM = PERSIST_STAGE_SPACE + 8 * PERSIST_STG + 1024 /*alignment*/ + 512 /*barriers*/;
constexpr int PERSIST_MAX_STAGES = 4;
// Where a product waits for weights that are being gathered, its CTAs may hold all SMs before those of shard_gather_push_kernel have theirs: one of 256 threads
// of 32 registers fits beside (320 threads of up to 159), and its 8 bytes of shared memory do; every CTA costs 1 KB more.
static_assert(PERSIST_SMEM + 1024 + 128 + 1024 <= 228 * 1024, "the gather's CTAs fit beside");
constexpr int PERSIST_A = 32768;                      // a CTA's 128 tokens x 128 of the reduction

// ---- the cta_group::2 forms ------------------------------------------------------------------
__device__ __forceinline__ void tmem_alloc_pair(uint32_t* smem_result, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(smem_result)), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tmem_relinquish_pair() { asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_dealloc_pair(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void umma_bf16_pair(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(tmem_d), "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
      : "memory");
}
// arrives at this CTA's barrier, or at this barrier of both CTAs, once the products issued so far have completed
__device__ __forceinline__ void umma_commit_own(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void umma_commit_pair(uint64_t* bar, uint32_t bar_peer) {
  umma_commit_own(bar);
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar_peer) : "memory");
}
// a copy into this CTA's shared memory that reports to a barrier of either CTA of the pair (no multicast)
__device__ __forceinline__ void tma_load_2d_pair(void* smem_dst, const void* tmap, int x, int y, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
      ::"r"(smem_u32(smem_dst)), "l"(reinterpret_cast<uint64_t>(tmap)), "r"(bar), "r"(x), "r"(y)
      : "memory");
}
__device__ __forceinline__ void tma_load_3d_pair(void* smem_dst, const void* tmap, int x, int y, int z, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
      ::"r"(smem_u32(smem_dst)), "l"(reinterpret_cast<uint64_t>(tmap)), "r"(bar), "r"(x), "r"(y), "r"(z)
      : "memory");
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
// groups of p.group token tiles by all feature tiles: the tiles that run at once share few rows of X and W, which stay in L2
__device__ __forceinline__ void persist_tile(const PersistParams& p, int tile, int& tm, int& tn) {
  const int width = p.group * p.tiles_n, g = tile / width, first = g * p.group, rows = min(p.group, p.tiles_m - first), r = tile - g * width;
  tm = first + r % rows;
  tn = r / rows;
}

// The residual of this lane's token, features f0 .. f0 + 63, zeros where the matrix ends (whole pieces of 8 features)
__device__ __forceinline__ void persist_residual(const PersistParams& p, int t, int f0, uint4 (&r)[8]) {
  const uint4* src = reinterpret_cast<const uint4*>(p.residual + (size_t)min(t, p.M - 1) * p.ldr + f0);
  const int n = (p.F_out - f0) / 8;
#pragma unroll
  for (int i = 0; i < 8; ++i) r[i] = i < n ? __ldcs(src + i) : make_uint4(0u, 0u, 0u, 0u);
}

template <int MODE>
__device__ __forceinline__ float persist_act(const PersistParams& p, float a) {
  const float z = bf16_round(a);
  if constexpr (MODE == 3) return 0.5f * z * (1.0f + erff(z * 0.70710678118654752f));
  const float neg = p.act_low * (ex2_approx(z * 1.4426950408889634f) - 1.0f - z);
  return fmaf(0.5f, z, z > 0.f ? p.act_up * z * z : neg);
}

// 64 weight rows' worth of this lane's token into the warp's staging buffer: 64 output features (row of 128 bytes, 128-byte swizzle) or 32 of a
// SwiGLU (64 bytes, 64-byte swizzle); `acc`: the first tensor-memory column
template <int MODE>
__device__ __forceinline__ void persist_chunk(const PersistParams& p, uint32_t acc, uint8_t* stg, int lane, const uint4 (&res)[8]) {
  if constexpr (MODE >= 2) {
    // activations piece by piece: unrolled over the chunk their code is fetched for longer than it runs (256 tokens, 12288 x 2048 SwiGLU)
    constexpr int PIECES = MODE == 2 ? 4 : 8;
#pragma unroll 1
    for (int c = 0; c < PIECES; ++c) {
      float a[16];
      if constexpr (MODE == 2) tmem_ld16(acc + c * 16, a);
      else tmem_ld8(acc + c * 8, a);
      tmem_ld_wait();
      uint4 pk;
      __nv_bfloat162* o = reinterpret_cast<__nv_bfloat162*>(&pk);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        if constexpr (MODE == 2) {
          const float* v = a + j * 4;
          o[j] = __floats2bfloat162_rn(bf16_round(silu(bf16_round(v[0]))) * bf16_round(v[1]), bf16_round(silu(bf16_round(v[2]))) * bf16_round(v[3]));
        } else {
          o[j] = __floats2bfloat162_rn(persist_act<MODE>(p, a[2 * j]), persist_act<MODE>(p, a[2 * j + 1]));
        }
      }
      if constexpr (MODE == 2) *reinterpret_cast<uint4*>(stg + lane * 64 + ((c ^ ((lane >> 1) & 3)) << 4)) = pk;
      else *reinterpret_cast<uint4*>(stg + lane * 128 + ((c ^ (lane & 7)) << 4)) = pk;
    }
  } else {
    float a[64];
    tmem_ld32(acc, a);
    tmem_ld32(acc + 32, a + 32);
    tmem_ld_wait();
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      uint4 pk;
      __nv_bfloat162* o = reinterpret_cast<__nv_bfloat162*>(&pk);
      const __nv_bfloat162* r = reinterpret_cast<const __nv_bfloat162*>(&res[c]);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        if constexpr (MODE == 1) {
          const float2 f = __bfloat1622float2(r[j]);
          o[j] = __floats2bfloat162_rn(bf16_round(a[c * 8 + 2 * j]) + f.x, bf16_round(a[c * 8 + 2 * j + 1]) + f.y);
        } else {
          o[j] = __floats2bfloat162_rn(a[c * 8 + 2 * j], a[c * 8 + 2 * j + 1]);
        }
      }
      *reinterpret_cast<uint4*>(stg + lane * 128 + ((c ^ (lane & 7)) << 4)) = pk;
    }
  }
}

// MODE: 0 plain, 1 residual, 2 SwiGLU of interleaved rows, 3 GELU, 4 xIELU
template <int MODE>
__global__ void __launch_bounds__(PERSIST_THREADS, 1) __cluster_dims__(2, 1, 1)
gemm_persist_kernel(const __grid_constant__ CUtensorMap tm_x, const __grid_constant__ CUtensorMap tm_w, const __grid_constant__ CUtensorMap tm_x2,
                    const __grid_constant__ CUtensorMap tm_w2, const __grid_constant__ CUtensorMap tm_out, const __grid_constant__ PersistParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* staging = smem + PERSIST_STAGE_SPACE;                             // [8 epilogue warps]
  uint64_t* full = reinterpret_cast<uint64_t*>(staging + 8 * PERSIST_STG);   // [stages], used in the first CTA
  uint64_t* empty = full + PERSIST_MAX_STAGES;                               // [stages]
  uint64_t* acc_full = empty + PERSIST_MAX_STAGES;                           // [2]
  uint64_t* acc_empty = acc_full + 2;                                        // [2], used in the first CTA: 8 epilogue warps of 2 CTAs
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  uint64_t* last = reinterpret_cast<uint64_t*>(tmem_slot + 2);               // products in flight when the issuer gives up

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = (int)cluster_ctarank();
  int n_tiles = p.tiles_m * p.tiles_n;
  const int first = blockIdx.x >> 1, step = gridDim.x >> 1;

  if (threadIdx.x == 0) {
    for (int s = 0; s < p.stages; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&acc_full[b], 1);
      mbar_init(&acc_empty[b], 16);
    }
    mbar_init(last, 1);
    *abort_flag = 0;
    mbar_fence_init();
    prefetch_tensormap(&tm_x);
    prefetch_tensormap(&tm_w);
  }
  if (warp == 1) {
    tmem_alloc_pair(tmem_slot, 512);
    tmem_relinquish_pair();
  }
  tc_fence_before();
  __syncwarp();
  cluster_sync_all();           // both CTAs' barriers exist before either one's copies or products report to them
  tc_fence_after();
  pdl_wait();
  const uint32_t tmem_base = *tmem_slot;
  if (p.wait_world > 0) {
    // Both CTAs wait for the peers' rows in front of everything, and skip all tiles if one of them does not see them come.
    if (threadIdx.x == 0 && !wait_peer_rows(p.wait_flag, p.wait_target, p.wait_world, p.status, p.wait_limit_ns)) {
      *abort_flag = 1;
      st_dsmem_u32(dsmem_addr(smem_u32(const_cast<int*>(abort_flag)), rank ^ 1), 1);
    }
    cluster_sync_all();
    asm volatile("fence.proxy.async.global;" ::: "memory");   // the TMA loads below see the landed rows
    if (*abort_flag) n_tiles = 0;
  }

  if (warp == 0) {
    // ---------------- TMA producer ----------------
    const uint32_t full0 = dsmem_addr(smem_u32(full), 0);
    int s = 0;
    uint32_t ph = 1;
    bool going = true;
    int issued = 0;
    for (int tile = first; tile < n_tiles && going; tile += step) {
      int tm, tn;
      persist_tile(p, tile, tm, tn);
      const int t0 = tm * 256 + rank * 128, f0 = tn * p.bn + rank * (p.bn / 2);
      auto blocks = [&](const CUtensorMap* ma, const CUtensorMap* mb, int n) {
        for (int g = 0; g < n; g += 2) {
          if (!mbar_wait_tight(&empty[s], ph, abort_flag, p.status, STATUS_TIMEOUT_STAGE_EMPTY)) {
            going = false;
            break;
          }
          if (elect_one()) {
            uint8_t* st = smem + s * p.stage_bytes;
            const uint32_t bar = full0 + s * 8;
            if (rank == 0) mbar_expect_tx(&full[s], 2 * p.stage_bytes);
            if (p.a_mn) {
              tma_load_2d_pair(st, ma, t0, g * 64, bar);
              tma_load_2d_pair(st + 16384, ma, t0 + 64, g * 64, bar);
            } else {
              tma_load_3d_pair(st, ma, 0, t0, g, bar);
            }
            if (p.b_mn) {
              tma_load_2d_pair(st + PERSIST_A, mb, f0, g * 64, bar);
              if (p.b_bytes > 16384) tma_load_2d_pair(st + PERSIST_A + 16384, mb, f0 + 64, g * 64, bar);
            } else {
              tma_load_3d_pair(st + PERSIST_A, mb, 0, f0, g, bar);
            }
          }
          ++issued;
          if (++s == p.stages) { s = 0; ph ^= 1; }
        }
      };
      blocks(&tm_x, &tm_w, p.kb_main);
      if (p.kb_ext > 0 && going) blocks(&tm_x2, &tm_w2, p.kb_ext);
    }
    __syncwarp();
    // Given up: the first CTA, whose barriers both CTAs' copies report to, stays until they have landed (bounded); the other one leaves with it.
    if (*abort_flag && rank == 0)
      for (int j = issued > p.stages ? issued - p.stages : 0; j < issued; ++j) mbar_drain(&full[j % p.stages], (j / p.stages) & 1);
    pdl_launch_dependents();
  } else if (warp == 1) {
    // ---------------- MMA issuer (first CTA of the pair) ----------------
    // The whole warp walks the loop and one elected lane issues: what a single lane of a diverged warp issues is wrapped in a loop over
    // the active lanes, and costs several times as much.
    if (rank == 0) {
      const uint32_t idesc = umma_idesc_bf16(256, p.bn) | (p.a_mn ? (1u << 15) : 0u) | (p.b_mn ? (1u << 16) : 0u);
      const uint32_t a_step = (p.a_mn ? 2048u : 32u) >> 4, b_step = (p.b_mn ? 2048u : 32u) >> 4;
      // from the first to the second block of 64 of a stage
      const uint32_t a_next = (p.a_mn ? 8192u : 16384u) >> 4, b_next = (p.b_mn ? 8192u : p.b_bytes / 2) >> 4;
      const uint32_t a_addr = smem_u32(smem), b_addr = a_addr + PERSIST_A, stage16 = p.stage_bytes >> 4;
      const uint64_t da0 = p.a_mn ? umma_desc_mn_sw128(a_addr, 16384) : umma_desc_sw128(a_addr);
      const uint64_t db0 = p.b_mn ? umma_desc_mn_sw128(b_addr, 16384) : umma_desc_sw128(b_addr);
      const uint32_t empty_peer = dsmem_addr(smem_u32(empty), 1), acc_full_peer = dsmem_addr(smem_u32(acc_full), 1);
      int s = 0;
      uint32_t ph = 0;
      int n = 0;
      bool going = true;
      for (int tile = first; tile < n_tiles; tile += step, ++n) {
        const int buf = n & 1;
        if (!mbar_wait_tight(&acc_empty[buf], ((n >> 1) & 1) ^ 1, abort_flag, p.status, STATUS_TIMEOUT_ACCUM)) {
          going = false;
          break;
        }
        tc_fence_after();
        const uint32_t d = tmem_base + buf * 256;
        uint32_t acc = 0u;
        auto blocks = [&](int n_blocks) {
          for (int g = 0; g < n_blocks; g += 2) {
            if (!mbar_wait_tight(&full[s], ph, abort_flag, p.status, STATUS_TIMEOUT_TMA_FULL)) {
              going = false;
              break;
            }
            tc_fence_after();
            if (elect_one()) {
              uint64_t da = da0 + (uint64_t)(s * stage16), db = db0 + (uint64_t)(s * stage16);
#pragma unroll
              for (int k = 0; k < 4; ++k) umma_bf16_pair(d, da + (uint64_t)(k * a_step), db + (uint64_t)(k * b_step), idesc, k > 0 ? 1u : acc);
              if (g + 1 < n_blocks) {
                da += a_next;
                db += b_next;
#pragma unroll
                for (int k = 0; k < 4; ++k) umma_bf16_pair(d, da + (uint64_t)(k * a_step), db + (uint64_t)(k * b_step), idesc, 1u);
              }
              umma_commit_pair(&empty[s], empty_peer + s * 8);
            }
            acc = 1u;
            if (++s == p.stages) { s = 0; ph ^= 1; }
          }
        };
        blocks(p.kb_main);
        if (p.kb_ext > 0 && going) blocks(p.kb_ext);
        if (!going) break;
        if (elect_one()) umma_commit_pair(&acc_full[buf], acc_full_peer + buf * 8);
      }
      if (!going) {
        if (elect_one()) umma_commit_own(last);
        mbar_drain(last, 0);
      }
    }
    __syncwarp();
  } else {
    // ---------------- epilogue: two warps per lane quarter with alternate chunks ----------------
    const int q = warp & 3, half = (warp - 2) >> 2;
    uint8_t* stg = staging + (warp - 2) * PERSIST_STG;
    const uint32_t lanes = tmem_base + (static_cast<uint32_t>(q * 32) << 16);
    const uint32_t acc_empty0 = dsmem_addr(smem_u32(acc_empty), 0);
    constexpr int CH = MODE == 2 ? 32 : 64;          // output features of a chunk
    const int out_bn = MODE == 2 ? p.bn / 2 : p.bn;
    int n = 0;
    uint4 res[8];
    for (int tile = first; tile < n_tiles; tile += step, ++n) {
      int tm, tn;
      persist_tile(p, tile, tm, tn);
      const int t0 = tm * 256 + rank * 128 + q * 32, o0 = tn * out_bn;
      const int chunks = t0 < p.M ? (min(out_bn, p.F_out - o0) + CH - 1) / CH : 0;
      if constexpr (MODE == 1) {
        if (half < chunks) persist_residual(p, t0 + lane, o0 + half * 64, res);       // under the main loop
      }
      const int buf = n & 1;
      if (!mbar_wait_tight(&acc_full[buf], (n >> 1) & 1, abort_flag, p.status, STATUS_TIMEOUT_ACCUM)) break;
      tc_fence_after();
#pragma unroll 1
      for (int c = half; c < chunks; c += 2) {
        if (lane == 0) tma_store_wait_read();          // the buffer's last store has read it
        __syncwarp();
        persist_chunk<MODE>(p, lanes + buf * 256 + c * 64, stg, lane, res);
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) {
          tma_store_2d(&tm_out, stg, o0 + c * CH, t0);
          tma_store_commit();
        }
        if constexpr (MODE == 1) {
          if (c + 2 < chunks) persist_residual(p, t0 + lane, o0 + (c + 2) * 64, res);
        }
        __syncwarp();
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(acc_empty0 + buf * 8);
      __syncwarp();
    }
    if (lane == 0) tma_store_wait_read();
    __syncwarp();
    tc_fence_before();
  }
  cluster_sync_all();             // neither CTA leaves while the other's copies, products or arrivals can still reach it
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc_pair(tmem_base, 512);
  }
}

template <int MODE>
static int launch_persist(const CUtensorMap& mx, const CUtensorMap& mw, const CUtensorMap& mx2, const CUtensorMap& mw2, const CUtensorMap& mo,
                          const PersistParams& p, int pairs, cudaStream_t stream) {
  auto kern = gemm_persist_kernel<MODE>;
  static bool configured = false;
  if (!configured) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, PERSIST_SMEM) != cudaSuccess) return -10;
    configured = true;
  }
  return launch_chain(kern, dim3(2 * pairs), dim3(PERSIST_THREADS), PERSIST_SMEM, stream, mx, mw, mx2, mw2, mo, p) == cudaSuccess ? 0 : -12;
}

}  // namespace tahb

using namespace tahb;

// out[M, F'] = op(X) op(W)^T (+ X2 W2^T) (+ residual), F' = F or, with act 2, F / 2.  F counts weight rows.  x_t: X is stored [K, M]; w_t: W is
// stored [K, F]; K (the reduction) is a multiple of 64 unless both are transposed (then its tail reads as zeros).  act: 0 none, 1 GELU, 2 SwiGLU of
// interleaved rows, 3 xIELU, without a residual but for 0.  bn: weight rows of a tile, a multiple of 64 up to 256.  Every
// operand, out and residual lie on 16-byte boundaries with row pitches that are multiples of 8 elements.  wait_*: see tahb_gemm_tp.
extern "C" int tahb_gemm_persist(const void* W, const void* X, void* out, const void* residual, const void* W2, const void* X2, int M, int F,
                                 int K, int R, long long ldw, long long ldx, long long ldo, long long ldr, long long ldw2, long long ldx2,
                                 int act, float act_up, float act_low, int x_t, int w_t, int bn, int* status, cudaStream_t stream,
                                 const void* wait_flag, const void* wait_target, int wait_world) {
  if (M <= 0 || F <= 0) return 0;
  const int Kp = (K + 63) / 64 * 64;
  if (K <= 0 || R % 64 || (Kp != K && !(x_t && w_t))) return -20;
  if (act < 0 || act > 3 || (act && (residual != nullptr || x_t || w_t))) return -29;
  if (R > 0 && (x_t || w_t)) return -27;
  if (bn < 64 || bn > 256 || bn % 64) return -22;
  if (act == 2 && F % 2) return -29;
  PersistParams p;
  p.b_mn = w_t != 0;
  p.a_mn = x_t != 0;
  p.b_bytes = p.b_mn ? (bn / 2 + 63) / 64 * 16384 : bn / 2 * 256;
  CUtensorMap mx, mw, mx2, mw2, mo;
  int rc;
  if ((rc = x_t ? make_map_mn_two(&mx, X, K, M, ldx) : make_map_two(&mx, X, M, K, ldx, 128))) return rc;
  if ((rc = w_t ? make_map_mn_two(&mw, W, K, F, ldw) : make_map_two(&mw, W, F, K, ldw, bn / 2))) return rc;
  mx2 = mx;
  mw2 = mw;
  if (R > 0) {
    if ((rc = make_map_two(&mx2, X2, M, R, ldx2, 128))) return rc;
    if ((rc = make_map_two(&mw2, W2, F, R, ldw2, bn / 2))) return rc;
  }
  p.F_out = act == 2 ? F / 2 : F;
  // output pieces: 32 tokens x 64 features, or 32 features
  if ((rc = act == 2 ? make_map_half(&mo, out, M, p.F_out, ldo, 32) : make_map(&mo, out, M, p.F_out, ldo, 32, true))) return rc;
  if (residual != nullptr && ((reinterpret_cast<uintptr_t>(residual) & 15) || (ldr & 7) || (F & 7))) return -2;
  p.M = M;
  p.kb_main = Kp / 64;
  p.kb_ext = R / 64;
  p.bn = bn;
  p.stage_bytes = PERSIST_A + p.b_bytes;
  p.stages = PERSIST_STAGE_SPACE / p.stage_bytes;
  if (p.stages > PERSIST_MAX_STAGES) p.stages = PERSIST_MAX_STAGES;
  p.tiles_m = (M + 255) / 256;
  p.tiles_n = (F + bn - 1) / bn;
  p.group = 8;
  p.act_up = act_up;
  p.act_low = act_low;
  p.residual = reinterpret_cast<const __nv_bfloat16*>(residual);
  p.ldr = ldr;
  p.status = status;
  p.wait_flag = reinterpret_cast<const uint32_t*>(wait_flag);
  p.wait_target = reinterpret_cast<const uint32_t*>(wait_target);
  p.wait_world = wait_flag != nullptr ? wait_world : 0;
  p.wait_limit_ns = peer_wait_limit_ns();
  const long long tiles = (long long)p.tiles_m * p.tiles_n;
  if (tiles > 0x7fffffff) return -21;
  const int pairs = tiles < 74 ? (int)tiles : 74;          // 148 SMs
  if (act == 2) return launch_persist<2>(mx, mw, mx2, mw2, mo, p, pairs, stream);
  if (act == 1) return launch_persist<3>(mx, mw, mx2, mw2, mo, p, pairs, stream);
  if (act == 3) return launch_persist<4>(mx, mw, mx2, mw2, mo, p, pairs, stream);
  return residual != nullptr ? launch_persist<1>(mx, mw, mx2, mw2, mo, p, pairs, stream) : launch_persist<0>(mx, mw, mx2, mw2, mo, p, pairs, stream);
}
