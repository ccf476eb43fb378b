// Matrix product for a handful of tokens: out[t, f] = sum_k X[t, k] W[f, k] (+ sum_r X2[t, r] W2[f, r]) (+ residual),
// with the epilogues of gemm_tcgen05.cu (plain, residual, GELU, interleaved SwiGLU, xIELU), for M <= 32, and for narrow weights at
// token counts whose 32-token tiles (the grid's second dimension) still fit one wave.
//
// What bounds it: the weight is read once (2 F K bytes) and used M times, so this is a stream of HBM at 2 M FLOP per
// weight; and it runs in a chain of small launches, so the time from the predecessor's end to the last store counts as
// much as the bandwidth.  A 128-feature tensor-memory tile leaves most SMs without work at the layer sizes (F = 2048
// gives 16 tiles, 64 CTAs with a cluster split), and pays for tensor-map fetch, tensor-memory allocation, a cluster
// barrier pair and a staged TMA store in every launch.  Here a CTA owns 16 or 32 features, its warps split the
// reduction, weights go from global memory straight into the registers that warp-level tensor instructions read,
// and the warps' partial sums meet once in shared memory.
//
// Fragment layout: mma.m16n8k16 wants for lane (g = lane / 4, t = lane % 4) the reduction indices {2t, 2t+1, 2t+8, 2t+9} of
// rows g and g + 8.  The order of the reduction is free as long as both operands agree, so a lane reads 16 consecutive
// bytes (8 indices) of a row at 8 t and feeds two instructions with them: 64 contiguous bytes per row and step, no
// shared memory, no shuffles.
//
// Ticks of few rows (FUSE): a layer of a decode tick was ten launches, of which the RMSNorms with the gated rows' adapter inputs (2.5 us of a
// one-row layer's 43, 3.6 us each with six rows) and the adapter inputs of the output and down projections (1.2 and 2.1 us) do next to
// nothing.  Here the product does it itself: a CTA normalises the rows into shared memory while its first weights are on their way (a row is
// 4 KB, from L2), and the first CTAs of the grid form T = gate * x A^T, which the others wait for behind their main loop (bounded; a
// CTA only waits for ones with a lower index, which run before it) and only where a row is gated; without one the adapter's weights are not
// read at all.  Six launches a layer, in ticks of up to eight rows (few_fused_pays in tah_b200/ops/cuda.py: above that all CTAs' norms of all rows cost more
// than the launches).
#include <cuda.h>

#include "common.cuh"

namespace tahb {

struct FewParams {
  const __nv_bfloat16 *W, *X, *W2, *X2, *residual;
  __nv_bfloat16* out;
  int M, F, K, R;
  long long ldw, ldx, ldw2, ldx2, ldo, ldr;
  int act;               // 0 none, 1 GELU, 2 SwiGLU of interleaved rows, 3 xIELU
  int stacked;           // SwiGLU of a weight with all gate rows in front of the up rows: how many gate rows; 0: interleaved
  float act_up, act_low;
  int early;             // the weights are constants of the launch chain: read them ahead of the dependency wait
  // FUSE
  const __nv_bfloat16* norm_w;   // RMSNorm in front of the product, or null
  float eps;
  const __nv_bfloat16* A;        // adapter: T [M, R] = gate * x A^T is what X2 points at
  __nv_bfloat16* T;
  const int* gate;               // [M]
  int t_ctas;                    // CTAs that form T
  unsigned long long* sync;      // CTAs of T done and, in the high half, CTAs that look at it no more; zero between launches
  int* status;
};

__device__ __forceinline__ void mma_16816(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint4 ld_stream(const void* p) {
  uint4 v;
  asm volatile("ld.global.nc.L1::no_allocate.L2::256B.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}

__device__ __forceinline__ unsigned long long ld_acquire(const unsigned long long* p) {
  unsigned long long v;
  asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
// Every CTA of a launch with gated rows, those that form T included, leaves once, when it will not look at the counters again; the last one
// finds all of T counted and puts them back to zero.  So they are zero behind every launch, also one whose wait for T ran out (the
// CTAs of T then leave behind the others).  A CTA of T counts and leaves in one step: one word, T's CTAs in the low half.
__device__ __forceinline__ void few_leave(unsigned long long* sync, unsigned long long formed) {
  if (atomicAdd(sync, (1ull << 32) + formed) >> 32 == gridDim.x - 1) *sync = 0;
}
constexpr int FEW_ROWS_MOST = 96 * 1024;       // of shared memory for normalised rows: two CTAs per SM

// T[r] = gate[r] ? x[r] A^T : 0 for a decode tick of many rows, of which a few are gated.  What bounds it: latency; a row's product is R dot
// products of K, and as dot products of one row at a time (lora_a_rows_kernel in elementwise.cu) 14 gated rows of 256 read A 14 times: 3.5 to 6.6 us
// a launch, four launches a layer.  Here the gated rows are gathered, 16 at a time, into the token side of warp-level tensor
// instructions; 16 outputs per cluster of eight CTAs that split the reduction, so that a warp holds all it needs of A in registers, read
// ahead of the dependency wait; the partial sums meet in the first CTA's shared memory, in a fixed order.  256 rows, 192 outputs of 2048, us, rows
// of dot products / this: 1 gated row 4.1 / 2.9, 14 5.3 / 3.0; 64 outputs of 6144: 4.2 / 3.2, 5.1 / 3.3.  27 KB of shared memory and 256 threads
// fit an SM beside a CTA of the one-tile GEMM, so that the start-up stands under its tail.  Small adapters and ticks of up to 32 rows keep the dot products
// (lora_gated_pays in tah_b200/ops/cuda.py).
constexpr int LG_WARPS = 8, LG_CL = 8, LG_STEPS = 4, LG_NT = 2, LG_TOK = 8 * LG_NT, LG_PITCH = 17;
struct LoraGatedParams {
  const __nv_bfloat16 *x, *A;
  __nv_bfloat16* T;
  const int* gate;
  int M, K, R;
  long long ldx, ldt;
};
__global__ void __launch_bounds__(LG_WARPS * 32) lora_gated_kernel(const LoraGatedParams p) {
  __shared__ float red[LG_WARPS * LG_TOK * LG_PITCH];
  __shared__ float part[2][LG_CL][LG_TOK * 16];               // [buffer][CTA of the cluster], used in the first CTA
  __shared__ short rows[1024];
  __shared__ int counts[32];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const int rank = (int)cluster_ctarank(), f0 = (int)(blockIdx.x / LG_CL) * 16;
  const int steps = p.K >> 5, c0 = steps * rank / LG_CL, cn = steps * (rank + 1) / LG_CL - c0;
  const int s0 = c0 + cn * warp / LG_WARPS, s1 = c0 + cn * (warp + 1) / LG_WARPS;
  uint4 a[LG_STEPS][2];
#pragma unroll
  for (int i = 0; i < LG_STEPS; ++i)
#pragma unroll
    for (int h = 0; h < 2; ++h)
      a[i][h] = s0 + i < s1 ? ld_stream(p.A + (size_t)min(f0 + 8 * h + g, p.R - 1) * p.K + t * 8 + (s0 + i) * 32) : make_uint4(0u, 0u, 0u, 0u);
  cluster_sync_all();                                         // the first CTA's shared memory exists before anyone writes to it
  pdl_wait();
  // the gated rows, in order
  unsigned m[4];
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    const int r = (warp + c * LG_WARPS) * 32 + lane;
    m[c] = __ballot_sync(0xffffffffu, r < p.M && p.gate[r] != 0);
    if (lane == 0) counts[warp + c * LG_WARPS] = __popc(m[c]);
  }
  __syncthreads();
  const int n = __reduce_add_sync(0xffffffffu, counts[lane]);
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    const int chunk = warp + c * LG_WARPS, r = chunk * 32 + lane;
    const int before = __reduce_add_sync(0xffffffffu, lane < chunk ? counts[lane] : 0);
    if (m[c] >> lane & 1u) {
      rows[before + __popc(m[c] & ((1u << lane) - 1u))] = (short)r;
    } else if (r < p.M && r % LG_CL == rank && blockIdx.y == 0) {     // zeros for the others, rows dealt out to the CTAs of the cluster
      uint4* dst = reinterpret_cast<uint4*>(p.T + (size_t)r * p.ldt + f0);
      dst[0] = make_uint4(0u, 0u, 0u, 0u);
      if (f0 + 8 < p.R) dst[1] = make_uint4(0u, 0u, 0u, 0u);
    }
  }
  __syncthreads();
  const uint32_t part0 = dsmem_addr(smem_u32(&part[0][rank][0]), 0);
  const int stride = LG_TOK * gridDim.y;
  for (int base = LG_TOK * blockIdx.y, pass = 0; base < n; base += stride, ++pass) {
    float acc[LG_NT][4];
#pragma unroll
    for (int j = 0; j < LG_NT; ++j)
#pragma unroll
      for (int c = 0; c < 4; ++c) acc[j][c] = 0.f;
    uint4 x[LG_STEPS][LG_NT];
#pragma unroll
    for (int j = 0; j < LG_NT; ++j) {
      const __nv_bfloat16* src = p.x + (size_t)rows[min(base + 8 * j + g, n - 1)] * p.ldx + t * 8;
#pragma unroll
      for (int i = 0; i < LG_STEPS; ++i)
        x[i][j] = s0 + i < s1 ? *reinterpret_cast<const uint4*>(src + (s0 + i) * 32) : make_uint4(0u, 0u, 0u, 0u);
    }
#pragma unroll
    for (int i = 0; i < LG_STEPS; ++i)
#pragma unroll
      for (int j = 0; j < LG_NT; ++j) {
        mma_16816(acc[j], a[i][0].x, a[i][1].x, a[i][0].y, a[i][1].y, x[i][j].x, x[i][j].y);
        mma_16816(acc[j], a[i][0].z, a[i][1].z, a[i][0].w, a[i][1].w, x[i][j].z, x[i][j].w);
      }
    if (base + stride >= n) pdl_launch_dependents();
#pragma unroll
    for (int j = 0; j < LG_NT; ++j)
#pragma unroll
      for (int c = 0; c < 4; ++c) red[(warp * LG_TOK + 8 * j + 2 * t + (c & 1)) * LG_PITCH + g + 8 * (c >> 1)] = acc[j][c];
    __syncthreads();
    if (tid < LG_TOK * 16) {
      float v = 0.f;
#pragma unroll
      for (int k = 0; k < LG_WARPS; ++k) v += red[(k * LG_TOK + tid / 16) * LG_PITCH + tid % 16];
      st_dsmem_f32(part0 + ((pass & 1) * LG_CL * LG_TOK * 16 + tid) * 4, v);
    }
    cluster_sync_all();       // two buffers: a CTA writes the one of pass + 2 behind the barrier that follows the reading of this one
    if (rank == 0 && tid < LG_TOK * 16) {
      float v = 0.f;
#pragma unroll
      for (int k = 0; k < LG_CL; ++k) v += part[pass & 1][k][tid];
      const int tok = base + tid / 16, f = f0 + tid % 16;
      if (tok < n && f < p.R) p.T[(size_t)rows[tok] * p.ldt + f] = __float2bfloat16_rn(v);
    }
  }
}

template <int NT, int MT>
struct FewCfg {
  static constexpr int ST = 4 / MT;                        // steps of 32 reduction indices per buffer, two buffers: 64 registers
  static constexpr int PITCH = 16 * MT + 4;                // floats per token in the reduction area: no bank conflicts
  static constexpr int red_bytes(int warps) { return warps * 8 * NT * PITCH * 4; }
};

// FUSE: 1 with the adapter input of the gated rows, 2 with the RMSNorm in front as well
template <int NT, int MT, int NW, int FUSE>
__global__ void __launch_bounds__(NW * 32)
gemm_few_kernel(const FewParams p) {
  using C = FewCfg<NT, MT>;
  constexpr int ST = C::ST, FT = 16 * MT;
  extern __shared__ __align__(16) float red[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const bool forms_t = FUSE && (int)blockIdx.x < p.t_ctas;
  const int F = forms_t ? p.R : p.F;
  const int f0 = (FUSE && !forms_t ? (int)blockIdx.x - p.t_ctas : (int)blockIdx.x) * FT;
  const int tok0 = blockIdx.y * 8 * NT, M = min(p.M - tok0, 8 * NT);          // this CTA's tokens
  const int steps = p.K >> 5, s0 = steps * warp / NW, s1 = steps * (warp + 1) / NW;

  auto row_of = [&](int m, int h) {            // weight row of this lane's feature
    const int v = min(f0 + 16 * m + 8 * h + g, F - 1);
    return (size_t)(p.stacked && !forms_t ? (v >> 1) + (v & 1) * p.stacked : v);
  };
  const __nv_bfloat16* wr[MT][2];
#pragma unroll
  for (int m = 0; m < MT; ++m)
#pragma unroll
    for (int h = 0; h < 2; ++h) wr[m][h] = (forms_t ? p.A + row_of(m, h) * p.K : p.W + row_of(m, h) * p.ldw) + t * 8;

  uint4 w[2][ST][MT][2];
  auto fetch = [&](uint4 (&b)[ST][MT][2], int s) {
#pragma unroll
    for (int i = 0; i < ST; ++i)
#pragma unroll
      for (int m = 0; m < MT; ++m)
#pragma unroll
        for (int h = 0; h < 2; ++h)
          b[i][m][h] = s + i < s1 ? ld_stream(wr[m][h] + (size_t)(s + i) * 32) : make_uint4(0u, 0u, 0u, 0u);
  };
  bool gated = false;
  if constexpr (FUSE) {
    if (!forms_t) {
      fetch(w[0], s0);
      fetch(w[1], s0 + ST);
    }
    uint4* nw = reinterpret_cast<uint4*>(red);                     // [K / 8] norm weights, then the rows
    if constexpr (FUSE == 2)
      for (int i = threadIdx.x; i < p.K / 8; i += NW * 32) nw[i] = reinterpret_cast<const uint4*>(p.norm_w)[i];
    pdl_wait();
    gated = p.t_ctas > 0 && __any_sync(0xffffffffu, lane < M && p.gate[lane] != 0);
    if (forms_t) {
      if (!gated) return;                                          // nobody reads T
      fetch(w[0], s0);
      fetch(w[1], s0 + ST);
    }
    if constexpr (FUSE == 2) {
      __syncthreads();                                             // the norm weights
      const int nvec = p.K / 8, pitch = nvec + 4;                  // 64 bytes between rows: no bank conflicts between fragments
      for (int r = warp; r < M; r += NW) {
        const uint4* src = reinterpret_cast<const uint4*>(p.X + (size_t)r * p.ldx);
        uint4* dst = nw + nvec + r * pitch;
        float ss = 0.f;
        for (int i0 = lane; i0 < nvec; i0 += 256) {
          uint4 v[8];
#pragma unroll
          for (int u = 0; u < 8; ++u) v[u] = i0 + u * 32 < nvec ? src[i0 + u * 32] : make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
          for (int u = 0; u < 8; ++u) {
            if (i0 + u * 32 < nvec) dst[i0 + u * 32] = v[u];
            const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&v[u]);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              const float2 f = __bfloat1622float2(h[j]);
              ss += f.x * f.x + f.y * f.y;
            }
          }
        }
        const float rstd = rsqrtf(warp_sum(ss) / (float)p.K + p.eps);
#pragma unroll 4
        for (int i = lane; i < nvec; i += 32) {                    // what this lane wrote
          uint4 v = dst[i];
          const uint4 wv = nw[i];
          __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&v);
          const __nv_bfloat162* wh = reinterpret_cast<const __nv_bfloat162*>(&wv);
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const float2 f = __bfloat1622float2(h[j]), q = __bfloat1622float2(wh[j]);
            h[j] = __floats2bfloat162_rn(q.x * bf16_round(f.x * rstd), q.y * bf16_round(f.y * rstd));
          }
          dst[i] = v;
        }
      }
      __syncthreads();
    }
  } else {
    if (!p.early) pdl_wait();
    fetch(w[0], s0);
    fetch(w[1], s0 + ST);
    if (p.early) pdl_wait();
  }

  float acc[MT][NT][4];
#pragma unroll
  for (int m = 0; m < MT; ++m)
#pragma unroll
    for (int j = 0; j < NT; ++j)
#pragma unroll
      for (int c = 0; c < 4; ++c) acc[m][j][c] = 0.f;

  const __nv_bfloat16* xr[NT];
#pragma unroll
  for (int j = 0; j < NT; ++j) {
    const int r = min(8 * j + g, M - 1);
    if constexpr (FUSE == 2) xr[j] = reinterpret_cast<const __nv_bfloat16*>(red) + p.K + r * (p.K + 32) + t * 8;
    else xr[j] = p.X + (size_t)(tok0 + r) * p.ldx + t * 8;
  }

  auto multiply = [&](const uint4 (&b)[MT][2], const uint4 (&x)[NT]) {
#pragma unroll
    for (int j = 0; j < NT; ++j)
#pragma unroll
      for (int m = 0; m < MT; ++m) {
        mma_16816(acc[m][j], b[m][0].x, b[m][1].x, b[m][0].y, b[m][1].y, x[j].x, x[j].y);
        mma_16816(acc[m][j], b[m][0].z, b[m][1].z, b[m][0].w, b[m][1].w, x[j].z, x[j].w);
      }
  };
  auto consume = [&](uint4 (&b)[ST][MT][2], int s) {
    uint4 x[ST][NT];
#pragma unroll
    for (int i = 0; i < ST; ++i)
#pragma unroll
      for (int j = 0; j < NT; ++j)
        x[i][j] = s + i < s1 ? *reinterpret_cast<const uint4*>(xr[j] + (size_t)(s + i) * 32) : make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
    for (int i = 0; i < ST; ++i) multiply(b[i], x[i]);
  };
  for (int s = s0; s < s1; s += 2 * ST) {
    consume(w[0], s);
    if (s + 2 * ST < s1) fetch(w[0], s + 2 * ST);
    if (s + ST < s1) {
      consume(w[1], s + ST);
      if (s + 3 * ST < s1) fetch(w[1], s + 3 * ST);
    }
  }
  // the K-extension: R / 32 more steps, one warp each in turn
  int ext = p.R >> 5;
  if constexpr (FUSE) {
    if (forms_t || !gated) {
      ext = 0;
    } else {
      if (threadIdx.x == 0) {
        unsigned long long t0 = 0;
        for (uint32_t spins = 0; (int)(uint32_t)ld_acquire(p.sync) < p.t_ctas;) {
          if ((++spins & 0xff) == 0) {
            const unsigned long long now = globaltimer_ns();
            if (t0 == 0) t0 = now;
            else if (now - t0 > WAIT_TIMEOUT_NS) {
              atomicCAS(p.status, 0, STATUS_TIMEOUT_ACCUM);
              break;
            }
          }
        }
      }
      __syncthreads();
      if (threadIdx.x == 0) few_leave(p.sync, 0);
    }
  }
  for (int s = warp; s < ext; s += NW) {
    uint4 b[MT][2], x[NT];
#pragma unroll
    for (int m = 0; m < MT; ++m)
#pragma unroll
      for (int h = 0; h < 2; ++h)
        b[m][h] = ld_stream(p.W2 + row_of(m, h) * p.ldw2 + t * 8 + s * 32);
#pragma unroll
    for (int j = 0; j < NT; ++j)
      x[j] = __ldcg(reinterpret_cast<const uint4*>(p.X2 + (size_t)(tok0 + min(8 * j + g, M - 1)) * p.ldx2 + t * 8 + s * 32));
    multiply(b, x);
  }

  pdl_launch_dependents();

  if constexpr (FUSE == 2) __syncthreads();          // the sums take the place of the rows
  // the warps' sums meet: [warp][token][feature]
#pragma unroll
  for (int m = 0; m < MT; ++m)
#pragma unroll
    for (int j = 0; j < NT; ++j)
#pragma unroll
      for (int c = 0; c < 4; ++c)
        red[(warp * 8 * NT + 8 * j + 2 * t + (c & 1)) * C::PITCH + 16 * m + g + 8 * (c >> 1)] = acc[m][j][c];
  __syncthreads();
  auto total = [&](int tok, int f) {
    float v = 0.f;
#pragma unroll
    for (int k = 0; k < NW; ++k) v += red[(k * 8 * NT + tok) * C::PITCH + f];
    return v;
  };
  if constexpr (FUSE) {
    if (forms_t) {
      for (int o = threadIdx.x; o < M * FT; o += NW * 32) {
        const int tok = o / FT, f = f0 + o % FT;
        if (f < p.R) p.T[(size_t)tok * p.R + f] = __float2bfloat16_rn(p.gate[tok] != 0 ? total(tok, o % FT) : 0.f);
      }
      __threadfence();
      __syncthreads();
      if (threadIdx.x == 0) few_leave(p.sync, 1);
      return;
    }
  }
  if (p.act == 2) {
    for (int o = threadIdx.x; o < M * (FT / 2); o += NW * 32) {
      const int tok = o / (FT / 2), f = o % (FT / 2);
      if (f0 + 2 * f >= F) continue;
      const float gate = bf16_round(total(tok, 2 * f)), up = bf16_round(total(tok, 2 * f + 1));
      p.out[(size_t)(tok0 + tok) * p.ldo + f0 / 2 + f] = __float2bfloat16_rn(bf16_round(silu(gate)) * up);
    }
    return;
  }
  for (int o = threadIdx.x; o < M * FT; o += NW * 32) {
    const int tok = o / FT, f = f0 + o % FT;
    if (f >= F) continue;
    float v = total(tok, o % FT);
    if (p.residual != nullptr) v = bf16_round(v) + __bfloat162float(p.residual[(size_t)(tok0 + tok) * p.ldr + f]);
    if (p.act == 1) {
      const float z = bf16_round(v);
      v = 0.5f * z * (1.0f + erff(z * 0.70710678118654752f));
    } else if (p.act == 3) {
      const float z = bf16_round(v);
      v = fmaf(0.5f, z, z > 0.f ? p.act_up * z * z : p.act_low * (ex2_approx(z * 1.4426950408889634f) - 1.0f - z));
    }
    p.out[(size_t)(tok0 + tok) * p.ldo + f] = __float2bfloat16_rn(v);
  }
}

// norm weights and normalised rows
static int few_rows_bytes(int M, int K) { return K * 2 + M * (K * 2 + 64); }

template <int NT, int MT, int NW, int FUSE>
static int launch_few(FewParams& p, cudaStream_t stream) {
  int bytes = FewCfg<NT, MT>::red_bytes(NW);
  static_assert(FewCfg<NT, MT>::red_bytes(NW) <= 48 * 1024, "no opt-in for more shared memory");
  auto kern = gemm_few_kernel<NT, MT, NW, FUSE>;
  if constexpr (FUSE) {
    p.t_ctas = (p.R + 16 * MT - 1) / (16 * MT);
    if constexpr (FUSE == 2) {
      static bool configured = false;
      if (!configured) {
        if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, FEW_ROWS_MOST) != cudaSuccess) return -10;
        configured = true;
      }
      const int rows = few_rows_bytes(p.M, p.K);
      bytes = bytes > rows ? bytes : rows;
    }
  }
  return launch_chain(kern, dim3((FUSE ? p.t_ctas : 0) + (p.F + 16 * MT - 1) / (16 * MT), (p.M + 8 * NT - 1) / (8 * NT)), dim3(NW * 32), bytes, stream,
                      p) == cudaSuccess ? 0 : -12;
}

// The split by sizes, see tahb_gemm_few.
template <int FUSE>
static int dispatch_few(FewParams& p, cudaStream_t stream) {
  const int tiles = (p.F + 15) / 16, M = p.M, K = p.K;
#define TAHB_FEW(NT_)                                                                         \
  {                                                                                           \
    if (tiles >= 4 * 148) return launch_few<NT_, 2, 4, FUSE>(p, stream);                      \
    if (NT_ == 1 && K <= 2048) return launch_few<1, 2, 16, FUSE>(p, stream);                  \
    if (tiles <= 148 || K >= 4096) return launch_few<NT_, 1, 16, FUSE>(p, stream);            \
    return launch_few<NT_, 1, 8, FUSE>(p, stream);                                            \
  }
  if (M <= 8) TAHB_FEW(1)
  if (M <= 16) TAHB_FEW(2)
  if constexpr (FUSE == 2) return -22;
  else TAHB_FEW(4)
#undef TAHB_FEW
}

}  // namespace tahb

using namespace tahb;

// Same operands as tahb_gemm (act as its `dual`: 0 plain, 1 SwiGLU of stacked rows, 3 GELU, 4 interleaved SwiGLU; 5 xIELU with act_up /
// act_low); F counts weight rows.  K and R multiples of 32, W / X / W2 / X2 on 16-byte boundaries with row pitches that are
// multiples of 8 elements.
//
// The split, measured with weights out of HBM (us, M = 1 / 12 / 32; in brackets the tcgen05 form it takes the place of):
//   F x K          2048 x 2048          4096 x 2048          2048 x 6144           12288 x 2048 SwiGLU     151936 x 2048
//   1 tile, 16 w   2.8 / 3.2 / 4.1      5.6 / 6.2 / 8.2      5.9 / 6.4 / 8.6       16 / 18 / 24            144 / 167 / 230
//   1 tile, 8 w    3.4 / 3.5 / 4.8      4.4 / 4.7 / 6.2      8.8 / 9.3 / 13.9      12.5 / 13.4 / 18.0      92 / 124 / 174
//   2 tiles, 16 w  2.4 / 3.5 / 5.2      4.0 / 4.9 / 6.5      6.8 / 9.1 / 13.5      11.1 / 14.1 / 18.8      99 / 133 / 189
//   2 tiles, 4 w   6.9 / 7.9 / 9.8      7.6 / 8.9 / 12.0     19 / 22 / 27          9.7 / 11.4 / 13.1       90 / 98 / 131
//   (tcgen05)      13.1 / 13.3 / 9.4    13.7 / 13.8 / 9.9    33.5 / 33.5 / 19.7    14.2 / 14.2 / 15.0      120 / 122 / 125
// Tiles of 16 features: about 16 warps per SM keep enough bytes in flight, more only add partial sums.  With four times as many
// tiles as SMs, four warps a CTA and two tiles are the streaming form (activations read once per 32 features).  Up to 8 tokens a
// reduction of 2048 lies in the two register buffers of 16 warps x 2 tiles: every weight byte is requested before the first wait.
extern "C" int tahb_gemm_few(const void* W, const void* X, void* out, const void* residual, const void* W2, const void* X2, int M, int F,
                             int K, int R, long long ldw, long long ldx, long long ldo, long long ldr, long long ldw2, long long ldx2,
                             int act, float act_up, float act_low, int early, cudaStream_t stream) {
  if (M <= 0 || F <= 0) return 0;
  if (K <= 0 || K % 32 || R % 32 || ((act == 1 || act == 4) && (F % 2 || residual != nullptr))) return -20;
  auto odd = [](const void* p, long long ld) { return (reinterpret_cast<uintptr_t>(p) & 15) || (ld & 7); };
  if (odd(W, ldw) || odd(X, ldx) || (R > 0 && (odd(W2, ldw2) || odd(X2, ldx2)))) return -2;
  FewParams p;
  p.W = reinterpret_cast<const __nv_bfloat16*>(W);
  p.X = reinterpret_cast<const __nv_bfloat16*>(X);
  p.W2 = reinterpret_cast<const __nv_bfloat16*>(W2);
  p.X2 = reinterpret_cast<const __nv_bfloat16*>(X2);
  p.residual = reinterpret_cast<const __nv_bfloat16*>(residual);
  p.out = reinterpret_cast<__nv_bfloat16*>(out);
  p.M = M; p.F = F; p.K = K; p.R = R;
  p.ldw = ldw; p.ldx = ldx; p.ldw2 = ldw2; p.ldx2 = ldx2; p.ldo = ldo; p.ldr = ldr;
  p.act = act == 3 ? 1 : (act == 1 || act == 4) ? 2 : act == 5 ? 3 : 0;
  p.stacked = act == 1 ? F / 2 : 0;
  p.act_up = act_up; p.act_low = act_low;
  p.early = early;
  p.t_ctas = 0;
  return dispatch_few<0>(p, stream);
}

// The same for up to 32 tokens (16 with norm_w) with what stands around it in a decode tick: norm_w != null: X goes through RMSNorm (norm_w, eps) first;
// R > 0: out += T B^T with T = gate * x A^T (A [R, K], B [F, R], T [M, R], all contiguous; T is written where a row is gated).
// act as above.  sync: eight bytes, zero, on their own boundary, for this stream's launches alone.
extern "C" int tahb_gemm_few_fused(const void* W, const void* X, void* out, const void* residual, const void* norm_w, float eps, const void* A,
                                   const void* B, void* T, const int* gate, void* sync, int M, int F, int K, int R, long long ldw,
                                   long long ldx, long long ldo, long long ldr, int act, int* status, cudaStream_t stream) {
  if (M <= 0 || F <= 0) return 0;
  if (M > (norm_w != nullptr ? 16 : 32) || K <= 0 || K % 64 || R % 64 || ((act == 1 || act == 4) && (F % 2 || residual != nullptr))) return -20;
  if (act != 0 && act != 1 && act != 4) return -29;
  if (R > 0 && (A == nullptr || B == nullptr || T == nullptr || gate == nullptr || sync == nullptr)) return -27;
  if (norm_w != nullptr && few_rows_bytes(M, K) > FEW_ROWS_MOST) return -22;
  auto odd = [](const void* p, long long ld) { return (reinterpret_cast<uintptr_t>(p) & 15) || (ld & 7); };
  if (odd(W, ldw) || odd(X, ldx) || odd(norm_w, 0) || odd(A, 0) || odd(B, 0) || odd(T, 0) || (reinterpret_cast<uintptr_t>(sync) & 7)) return -2;
  FewParams p = {};
  p.W = reinterpret_cast<const __nv_bfloat16*>(W);
  p.X = reinterpret_cast<const __nv_bfloat16*>(X);
  p.W2 = reinterpret_cast<const __nv_bfloat16*>(B);
  p.X2 = reinterpret_cast<const __nv_bfloat16*>(T);
  p.residual = reinterpret_cast<const __nv_bfloat16*>(residual);
  p.out = reinterpret_cast<__nv_bfloat16*>(out);
  p.M = M; p.F = F; p.K = K; p.R = R;
  p.ldw = ldw; p.ldx = ldx; p.ldw2 = R; p.ldx2 = R; p.ldo = ldo; p.ldr = ldr;
  p.act = act ? 2 : 0;
  p.stacked = act == 1 ? F / 2 : 0;
  p.norm_w = reinterpret_cast<const __nv_bfloat16*>(norm_w);
  p.eps = eps;
  p.A = reinterpret_cast<const __nv_bfloat16*>(A);
  p.T = reinterpret_cast<__nv_bfloat16*>(T);
  p.gate = gate;
  p.sync = reinterpret_cast<unsigned long long*>(sync);
  p.status = status;
  return norm_w != nullptr ? dispatch_few<2>(p, stream) : dispatch_few<1>(p, stream);
}

// T [M, R] = gate[r] ? x[r] A^T : 0 (see lora_gated_kernel).  M <= 1024, K a multiple of 64 up to 8192, R of 8; everything on 16-byte boundaries;
// A is a constant of the launch chain.
extern "C" int tahb_lora_gated(const void* x, const void* A, void* T, const int* gate, int M, int K, int R, long long ldx, long long ldt,
                               cudaStream_t stream) {
  if (M <= 0 || R <= 0) return 0;
  if (M > 1024 || K <= 0 || K % 64 || K > 32 * LG_CL * LG_WARPS * LG_STEPS || R % 8 || gate == nullptr) return -20;
  auto odd = [](const void* p, long long ld) { return (reinterpret_cast<uintptr_t>(p) & 15) || (ld & 7); };
  if (odd(x, ldx) || odd(A, K) || odd(T, ldt)) return -2;
  LoraGatedParams p;
  p.x = reinterpret_cast<const __nv_bfloat16*>(x);
  p.A = reinterpret_cast<const __nv_bfloat16*>(A);
  p.T = reinterpret_cast<__nv_bfloat16*>(T);
  p.gate = gate;
  p.M = M; p.K = K; p.R = R;
  p.ldx = ldx; p.ldt = ldt;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((R + 15) / 16 * LG_CL, M <= 64 ? 1 : 2);       // gated rows come 16 at a time, rarely more than 32
  cfg.blockDim = dim3(LG_WARPS * 32);
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = LG_CL;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl_enabled() ? 2 : 1;
  return cudaLaunchKernelEx(&cfg, lora_gated_kernel, p) == cudaSuccess ? 0 : -12;
}
