// Backward kernels of the memory-bound training ops: RMSNorm and SwiGLU.  Each reads its inputs
// once and writes its outputs once (bf16 in / out, fp32 math).
#include "common.cuh"

namespace tahb {

// ---------------------------------------------------------------------------------------------
// RMSNorm backward.  y = w * (x * rstd),  rstd = rsqrt(mean(x^2) + eps).  With gn = gy * w:
//     gx = rstd * (gn - xn * mean(gn * xn)),   gw = sum_rows gy * xn,   xn = x * rstd.
// A CTA of 256 threads walks rows blockIdx, + gridDim, ...; thread t owns columns 8t..8t+7 (+ 2048 k), keeps its slice of gw in
// registers over those rows and adds it to the fp32 gw buffer once at the end.  Bound: HBM (2048 columns, 3072 rows: 38 MB, 6 us); a
// row is a chain of load, block reduction and store, so the next row is on its way while one is reduced, and two CTAs per SM share
// the rows evenly.  32 rows in turn per CTA without that: 39 us at 3072 rows (96 CTAs), now 12.3 us.
// FEW: 3 to 64 rows (of a second pass, say) go to one cluster of eight CTAs, whose sums meet in a fixed order through distributed shared
// memory: the gradients of a few rows repeat themselves bit by bit.  64 rows 8.4 us, with atomics 3.9, in two CTAs 19.
// ---------------------------------------------------------------------------------------------
constexpr int RMSB_GRID = 296, RMSB_FEW_ROWS = 64, RMSB_FEW_CTAS = 8;      // two additions to a zeroed sum have no order

template <int VPT, bool FEW>
__global__ void __launch_bounds__(256) rmsnorm_bwd_kernel(const __nv_bfloat16* __restrict__ x,
                                                          const __nv_bfloat16* __restrict__ w,
                                                          const __nv_bfloat16* __restrict__ gy,
                                                          __nv_bfloat16* __restrict__ gx, float* __restrict__ gw,
                                                          int M, int H, float eps) {
  __shared__ float red[2][8];
  const int nvec = H / 8;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  float wv[VPT][8], gwa[VPT][8];
#pragma unroll
  for (int i = 0; i < VPT; ++i) {
    const int idx = tid + i * 256;
#pragma unroll
    for (int j = 0; j < 8; ++j) { gwa[i][j] = 0.f; wv[i][j] = 0.f; }
    if (idx < nvec) {
      const uint4 u = *reinterpret_cast<const uint4*>(w + idx * 8);
      const __nv_bfloat162* h2 = reinterpret_cast<const __nv_bfloat162*>(&u);
#pragma unroll
      for (int j = 0; j < 4; ++j) { const float2 f = __bfloat1622float2(h2[j]); wv[i][2 * j] = f.x; wv[i][2 * j + 1] = f.y; }
    }
  }
  uint4 nx[VPT], ng[VPT];
  auto fetch = [&](int row) {
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      const int idx = tid + i * 256;
      if (idx < nvec) {
        nx[i] = *reinterpret_cast<const uint4*>(x + (size_t)row * H + idx * 8);
        ng[i] = *reinterpret_cast<const uint4*>(gy + (size_t)row * H + idx * 8);
      }
    }
  };
  if ((int)blockIdx.x < M) fetch(blockIdx.x);
  for (int row = blockIdx.x; row < M; row += gridDim.x) {
    const size_t off = (size_t)row * H;
    float xv[VPT][8], gv[VPT][8];
    float ss = 0.f, dot = 0.f;
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      const int idx = tid + i * 256;
      if (idx < nvec) {
        const uint4 ux = nx[i], ug = ng[i];
        const __nv_bfloat162* hx = reinterpret_cast<const __nv_bfloat162*>(&ux);
        const __nv_bfloat162* hg = reinterpret_cast<const __nv_bfloat162*>(&ug);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float2 fx = __bfloat1622float2(hx[j]), fg = __bfloat1622float2(hg[j]);
          xv[i][2 * j] = fx.x; xv[i][2 * j + 1] = fx.y;
          gv[i][2 * j] = fg.x; gv[i][2 * j + 1] = fg.y;
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          ss += xv[i][j] * xv[i][j];
          dot += gv[i][j] * wv[i][j] * xv[i][j];
        }
      }
    }
    if (row + (int)gridDim.x < M) fetch(row + gridDim.x);
    ss = warp_sum(ss);
    dot = warp_sum(dot);
    __syncthreads();
    if (lane == 0) { red[0][warp] = ss; red[1][warp] = dot; }
    __syncthreads();
    float tss = 0.f, tdot = 0.f;
#pragma unroll
    for (int k = 0; k < 8; ++k) { tss += red[0][k]; tdot += red[1][k]; }
    const float rstd = rsqrtf(tss / (float)H + eps);
    const float c = tdot * rstd * rstd / (float)H;          // mean(gn * xn) * rstd, applied to x
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      const int idx = tid + i * 256;
      if (idx < nvec) {
        uint4 o;
        __nv_bfloat162* o2 = reinterpret_cast<__nv_bfloat162*>(&o);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float a = rstd * (gv[i][2 * j] * wv[i][2 * j] - xv[i][2 * j] * c);
          const float b = rstd * (gv[i][2 * j + 1] * wv[i][2 * j + 1] - xv[i][2 * j + 1] * c);
          o2[j] = __floats2bfloat162_rn(a, b);
        }
        *reinterpret_cast<uint4*>(gx + off + idx * 8) = o;
#pragma unroll
        for (int j = 0; j < 8; ++j) gwa[i][j] += gv[i][j] * xv[i][j] * rstd;
      }
    }
  }
  if (gw != nullptr) {
    // a thread owns eight neighbouring columns: by way of shared memory a warp's additions fall into one 128-byte line instead of eight
    __shared__ float slice[256 * 8];
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      __syncthreads();
#pragma unroll
      for (int j = 0; j < 8; ++j) slice[tid * 8 + j] = gwa[i][j];
      if constexpr (FEW) {
        cluster_sync_all();
        const int c = blockIdx.x * 256 + tid;                 // CTA k of the cluster adds up columns 256 k ..
        float sum = 0.f;
#pragma unroll
        for (int k = 0; k < RMSB_FEW_CTAS; ++k) sum += ld_dsmem_f32(smem_u32(&slice[c]), k);
        if (i * 2048 + c < H) gw[i * 2048 + c] += sum;
        cluster_sync_all();                                   // the others have read this CTA's slice
      } else {
        __syncthreads();
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const int c = j * 256 + tid;
          if (i * 2048 + c < H) atomicAdd(gw + i * 2048 + c, slice[c]);
        }
      }
    }
  }
}

// ---------------------------------------------------------------------------------------------
// SwiGLU backward on a [M, 2I] gate|up tensor: out = silu(g) * u,
//     d_gate = gy * u * sig(g) * (1 + g * (1 - sig(g))),   d_up = gy * silu(g).
// ---------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(256) swiglu_bwd_kernel(const __nv_bfloat16* __restrict__ gu,
                                                         const __nv_bfloat16* __restrict__ gy,
                                                         __nv_bfloat16* __restrict__ dgu, long long M, int I) {
  const long long nvec = M * (I / 8);
  for (long long v = blockIdx.x * (long long)blockDim.x + threadIdx.x; v < nvec; v += (long long)gridDim.x * blockDim.x) {
    const long long r = v / (I / 8);
    const int c = (int)(v % (I / 8)) * 8;
    const uint4 ug = *reinterpret_cast<const uint4*>(gu + r * 2 * I + c);
    const uint4 uu = *reinterpret_cast<const uint4*>(gu + r * 2 * I + I + c);
    const uint4 uy = *reinterpret_cast<const uint4*>(gy + r * I + c);
    const __nv_bfloat162* hg = reinterpret_cast<const __nv_bfloat162*>(&ug);
    const __nv_bfloat162* hu = reinterpret_cast<const __nv_bfloat162*>(&uu);
    const __nv_bfloat162* hy = reinterpret_cast<const __nv_bfloat162*>(&uy);
    uint4 og, ou;
    __nv_bfloat162* o_g = reinterpret_cast<__nv_bfloat162*>(&og);
    __nv_bfloat162* o_u = reinterpret_cast<__nv_bfloat162*>(&ou);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 g = __bfloat1622float2(hg[j]), u = __bfloat1622float2(hu[j]), y = __bfloat1622float2(hy[j]);
      const float s0 = 1.0f / (1.0f + __expf(-g.x)), s1 = 1.0f / (1.0f + __expf(-g.y));
      o_g[j] = __floats2bfloat162_rn(y.x * u.x * s0 * (1.0f + g.x * (1.0f - s0)), y.y * u.y * s1 * (1.0f + g.y * (1.0f - s1)));
      o_u[j] = __floats2bfloat162_rn(y.x * g.x * s0, y.y * g.y * s1);
    }
    *reinterpret_cast<uint4*>(dgu + r * 2 * I + c) = og;
    *reinterpret_cast<uint4*>(dgu + r * 2 * I + I + c) = ou;
  }
}

// ---------------------------------------------------------------------------------------------
// Backward of the per-head QK RMSNorm + rotate-half RoPE (forward: qk_norm_rope_kv_kernel in
// elementwise.cu).  Lane l owns elements l*EPL..+EPL-1 of a head.
//   n = w * (x * rstd),  y = n * cos + rot(n) * sin      (q and k heads; v heads pass through)
//   gn = gy * cos +/- partner(gy) * sin ;  gx = rstd * (gn*w - xn * mean(gn*w*xn)) ;  gw += gn * xn
// The weight gradients are summed per CTA in shared memory and added to the fp32 buffers once.
// A CTA takes a token at a time (several CTAs up to 64 tokens), a warp four of its heads with all their loads in flight and the sines and
// cosines once for them (once per CTA, by way of shared memory, 38 us: a barrier per token).  Bound: HBM (3072 tokens of 16 + 16 heads: 75 MB, 11 us); a warp per
// head with one in flight and its own sincosf: 50 us, now 34.4 us.
// ---------------------------------------------------------------------------------------------
struct QkRopeBwdParams {
  const __nv_bfloat16* qkv;      // [M, (nq + 2 nkv) * HD] forward input
  const __nv_bfloat16* q_w;
  const __nv_bfloat16* k_w;
  const __nv_bfloat16* gq;       // [M, nq * HD]
  const __nv_bfloat16* gk;       // [M, nkv * HD]
  const __nv_bfloat16* gv;       // [M, nkv * HD]
  __nv_bfloat16* gqkv;           // [M, (nq + 2 nkv) * HD]
  float* gq_w;                   // [HD] fp32, added to
  float* gk_w;
  const int* pos;
  int M, nq, nkv;
  float eps, log2_theta;
};

constexpr int QKB_U = 4, QKB_WARPS = 8;
template <int HD, bool WIDE>
__global__ void __launch_bounds__(QKB_WARPS * 32) qk_norm_rope_bwd_kernel(const QkRopeBwdParams p) {
  constexpr int EPL = HD / 32;
  using Piece = QkvPiece<EPL, WIDE ? EPL * 2 : 2>;
  __shared__ float s_gw[2][HD];
  for (int i = threadIdx.x; i < 2 * HD; i += blockDim.x) (&s_gw[0][0])[i] = 0.f;
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int heads = p.nq + 2 * p.nkv, per = (heads + gridDim.y - 1) / gridDim.y, first = blockIdx.y * per, last = min(heads, first + per);
  const bool upper = lane >= 16;
  float gw_q[EPL], gw_k[EPL];
  float inv[EPL];
#pragma unroll
  for (int i = 0; i < EPL; ++i) inv[i] = exp2f(-(2.0f * (float)((lane & 15) * EPL + i) / (float)HD) * p.log2_theta);
  Piece wq, wk;
  wq.load(p.q_w + lane * EPL);
  wk.load(p.k_w + lane * EPL);
#pragma unroll
  for (int i = 0; i < EPL; ++i) gw_q[i] = gw_k[i] = 0.f;
  for (int t = blockIdx.x; t < p.M; t += gridDim.x) {
    float2 cs[EPL];
    const float posf = (float)p.pos[t];
    for (int h0 = first + warp; h0 < last; h0 += QKB_U * QKB_WARPS) {
      Piece xin[QKB_U], gin[QKB_U];
#pragma unroll
      for (int u = 0; u < QKB_U; ++u) {
        const int h = h0 + u * QKB_WARPS;
        if (h >= last) continue;
        if (h < p.nq + p.nkv) xin[u].load(p.qkv + ((size_t)t * heads + h) * HD + lane * EPL);
        gin[u].load((h < p.nq ? p.gq + ((size_t)t * p.nq + h) * HD
                              : h < p.nq + p.nkv ? p.gk + ((size_t)t * p.nkv + h - p.nq) * HD
                                                 : p.gv + ((size_t)t * p.nkv + h - p.nq - p.nkv) * HD) + lane * EPL);
      }
      if (h0 == first + warp) {                      // once per token, with the first loads on their way
#pragma unroll
        for (int i = 0; i < EPL; ++i) {
          const float ang = posf * inv[i];
          cs[i] = make_float2(bf16_round(cosf(ang)), bf16_round(sinf(ang)));
        }
      }
#pragma unroll
      for (int u = 0; u < QKB_U; ++u) {
        const int h = h0 + u * QKB_WARPS;
        if (h >= last) continue;
        Piece out = gin[u];
        if (h < p.nq + p.nkv) {
          const bool is_q = h < p.nq;
          float x[EPL], gn[EPL], wv[EPL], ss = 0.f;
#pragma unroll
          for (int i = 0; i < EPL; ++i) {
            x[i] = __bfloat162float(xin[u].v[i]);
            wv[i] = __bfloat162float(is_q ? wq.v[i] : wk.v[i]);
            ss += x[i] * x[i];
          }
          const float rstd = rsqrtf(warp_sum(ss) / (float)HD + p.eps);
          float dot = 0.f;
#pragma unroll
          for (int i = 0; i < EPL; ++i) {
            const float gy = __bfloat162float(gin[u].v[i]), part = __shfl_xor_sync(0xffffffffu, gy, 16);
            gn[i] = gy * cs[i].x + (upper ? -part : part) * cs[i].y;
            x[i] *= rstd;
            dot += gn[i] * wv[i] * x[i];
          }
          dot = warp_sum(dot) / (float)HD;
#pragma unroll
          for (int i = 0; i < EPL; ++i) {
            out.v[i] = __float2bfloat16_rn(rstd * (gn[i] * wv[i] - x[i] * dot));
            if (is_q) gw_q[i] += gn[i] * x[i];
            else gw_k[i] += gn[i] * x[i];
          }
        }
        out.store(p.gqkv + ((size_t)t * heads + h) * HD + lane * EPL);
      }
    }
  }
#pragma unroll
  for (int i = 0; i < EPL; ++i) {
    atomicAdd(&s_gw[0][lane * EPL + i], gw_q[i]);
    atomicAdd(&s_gw[1][lane * EPL + i], gw_k[i]);
  }
  __syncthreads();
  for (int i = threadIdx.x; i < HD; i += blockDim.x) {
    if (p.gq_w != nullptr) atomicAdd(p.gq_w + i, s_gw[0][i]);
    if (p.gk_w != nullptr) atomicAdd(p.gk_w + i, s_gw[1][i]);
  }
}

// d[row] = sum over hd of a[row][.] * b[row][.]: what the attention backward subtracts from every score gradient of a query head.  A lane
// takes 16 bytes of each, hd / 8 lanes share a row.  HBM bound; the sum replaces two fp32 copies, their product and its reduction.
__global__ void __launch_bounds__(256) rows_dot_kernel(const uint4* __restrict__ a, const uint4* __restrict__ b, float* __restrict__ d,
                                                       long long rows, int lanes) {
  const long long i = blockIdx.x * 256ll + threadIdx.x;
  const long long row = i / lanes;
  float s = 0.f;
  if (row < rows) {
    const uint4 u = a[i], v = b[i];
    const __nv_bfloat162 *x = reinterpret_cast<const __nv_bfloat162*>(&u), *y = reinterpret_cast<const __nv_bfloat162*>(&v);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 f = __bfloat1622float2(x[j]), g = __bfloat1622float2(y[j]);
      s += f.x * g.x + f.y * g.y;
    }
  }
  for (int o = lanes >> 1; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if (row < rows && i % lanes == 0) d[row] = s;
}

// Block-diagonal adapter factor of a fused projection, [F, n r]: rows begin[j] .. end[j] of columns j r .. (j + 1) r hold
// B_j [., r] * scale, everything else is zero.
struct BlockDiagParams {
  const __nv_bfloat16* b[4];
  int begin[4], end[4];
  int n, r, F;
  float scale;
  __nv_bfloat16* out;
};
__global__ void __launch_bounds__(256) block_diag_kernel(const BlockDiagParams p) {
  const int per = p.n * p.r / 8;                     // pieces of eight columns in a row
  const long long i = blockIdx.x * 256ll + threadIdx.x;
  if (i >= (long long)p.F * per) return;
  const int row = (int)(i / per), col = (int)(i % per) * 8, j = col / p.r;
  uint4 v = make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    if (k != j || k >= p.n || row < p.begin[k] || row >= p.end[k]) continue;
    v = *reinterpret_cast<const uint4*>(p.b[k] + (size_t)(row - p.begin[k]) * p.r + (col - k * p.r));
    __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&v);
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const float2 f = __bfloat1622float2(h[c]);
      h[c] = __floats2bfloat162_rn(f.x * p.scale, f.y * p.scale);
    }
  }
  *reinterpret_cast<uint4*>(p.out + (size_t)row * p.n * p.r + col) = v;
}

}  // namespace tahb

using namespace tahb;

// Backward of tahb_qk_norm_rope_kv for contiguous tensors.  gq_w / gk_w: fp32 [hd] the kernel adds into.
extern "C" int tahb_qk_norm_rope_bwd(const void* qkv, const void* q_w, const void* k_w, const void* gq, const void* gk,
                                     const void* gv, void* gqkv, float* gq_w, float* gk_w, const int* pos, int M,
                                     int nq, int nkv, int hd, float eps, float theta, cudaStream_t stream) {
  if (M <= 0) return 0;
  QkRopeBwdParams p;
  p.qkv = reinterpret_cast<const __nv_bfloat16*>(qkv);
  p.q_w = reinterpret_cast<const __nv_bfloat16*>(q_w);
  p.k_w = reinterpret_cast<const __nv_bfloat16*>(k_w);
  p.gq = reinterpret_cast<const __nv_bfloat16*>(gq);
  p.gk = reinterpret_cast<const __nv_bfloat16*>(gk);
  p.gv = reinterpret_cast<const __nv_bfloat16*>(gv);
  p.gqkv = reinterpret_cast<__nv_bfloat16*>(gqkv);
  p.gq_w = gq_w;
  p.gk_w = gk_w;
  p.pos = pos;
  p.M = M; p.nq = nq; p.nkv = nkv;
  p.eps = eps;
  p.log2_theta = log2f(theta);
  uintptr_t at = 0;
  for (const void* q : {qkv, q_w, k_w, gq, gk, gv, (const void*)gqkv}) at |= reinterpret_cast<uintptr_t>(q);
  const bool wide = at % (hd / 16) == 0;
  // two CTAs per SM, whose sums meet in the weight gradients' few lines
  const dim3 grid(M < 296 ? M : 296, qk_head_groups(M, nq + 2 * nkv, QKB_WARPS, 128));
#define TAHB_QKB(HD_)                                                                          \
  (wide ? (void)(qk_norm_rope_bwd_kernel<HD_, true><<<grid, QKB_WARPS * 32, 0, stream>>>(p)) \
        : (void)(qk_norm_rope_bwd_kernel<HD_, false><<<grid, QKB_WARPS * 32, 0, stream>>>(p)))
  if (hd == 128) TAHB_QKB(128);
  else if (hd == 64) TAHB_QKB(64);
  else return -2;
  return cudaGetLastError() == cudaSuccess ? 0 : -3;
}

// x, gy, gx: [M, H] bf16 contiguous; w [H] bf16; gw: fp32 [H] that the kernel ADDS into (or null).
extern "C" int tahb_rmsnorm_bwd(const void* x, const void* w, const void* gy, void* gx, float* gw, int M, int H,
                                float eps, cudaStream_t stream) {
  if (M <= 0) return 0;
  if (H % 8) return -1;
  const int nvec = H / 8;
  auto X = reinterpret_cast<const __nv_bfloat16*>(x);
  auto W = reinterpret_cast<const __nv_bfloat16*>(w);
  auto GY = reinterpret_cast<const __nv_bfloat16*>(gy);
  auto GX = reinterpret_cast<__nv_bfloat16*>(gx);
#define TAHB_RMSB(VPT_)                                                                                                   \
  {                                                                                                                       \
    if (M > RMSB_FEW_ROWS || M <= 2) {                                                                                              \
      rmsnorm_bwd_kernel<VPT_, false><<<M < RMSB_GRID ? M : RMSB_GRID, 256, 0, stream>>>(X, W, GY, GX, gw, M, H, eps);     \
    } else {                                                                                                              \
      cudaLaunchAttribute attr = {};                                                                                      \
      attr.id = cudaLaunchAttributeClusterDimension;                                                                      \
      attr.val.clusterDim.x = RMSB_FEW_CTAS;                                                                              \
      attr.val.clusterDim.y = attr.val.clusterDim.z = 1;                                                                  \
      cudaLaunchConfig_t cfg = {};                                                                                        \
      cfg.gridDim = dim3(RMSB_FEW_CTAS);                                                                                  \
      cfg.blockDim = dim3(256);                                                                                           \
      cfg.stream = stream;                                                                                                \
      cfg.attrs = &attr;                                                                                                  \
      cfg.numAttrs = 1;                                                                                                   \
      if (cudaLaunchKernelEx(&cfg, rmsnorm_bwd_kernel<VPT_, true>, X, W, GY, GX, gw, M, H, eps) != cudaSuccess) return -3; \
    }                                                                                                                     \
  }
  if (nvec <= 256) TAHB_RMSB(1)
  else if (nvec <= 512) TAHB_RMSB(2)
  else if (nvec <= 1024) TAHB_RMSB(4)
  else return -2;
#undef TAHB_RMSB
  return cudaGetLastError() == cudaSuccess ? 0 : -3;
}

// gu, dgu: [M, 2I] bf16 contiguous (gate | up); gy: [M, I].
extern "C" int tahb_swiglu_bwd(const void* gu, const void* gy, void* dgu, long long M, int I, cudaStream_t stream) {
  if (M <= 0) return 0;
  if (I % 8) return -1;
  const long long nvec = M * (I / 8);
  long long blocks = (nvec + 255) / 256;
  if (blocks > 148 * 16) blocks = 148 * 16;
  swiglu_bwd_kernel<<<(int)blocks, 256, 0, stream>>>(reinterpret_cast<const __nv_bfloat16*>(gu),
                                                     reinterpret_cast<const __nv_bfloat16*>(gy),
                                                     reinterpret_cast<__nv_bfloat16*>(dgu), M, I);
  return cudaGetLastError() == cudaSuccess ? 0 : -3;
}

// d [rows] fp32 = row sums of a * b, both [rows, hd] bf16 contiguous on 16-byte boundaries, hd 64 or 128.
extern "C" int tahb_rows_dot(const void* a, const void* b, float* d, long long rows, int hd, cudaStream_t stream) {
  if (rows <= 0) return 0;
  if (hd != 64 && hd != 128) return -1;
  const long long blocks = (rows * (hd / 8) + 255) / 256;
  rows_dot_kernel<<<(unsigned)blocks, 256, 0, stream>>>(reinterpret_cast<const uint4*>(a), reinterpret_cast<const uint4*>(b), d, rows, hd / 8);
  return cudaGetLastError() == cudaSuccess ? 0 : -3;
}

// out [F, n r] from n <= 4 factors (see BlockDiagParams); r a multiple of 8, pointers on 16-byte boundaries.
extern "C" int tahb_block_diag(void* const* b, const int* begin, const int* end, int n, int r, int F, float scale, void* out, cudaStream_t stream) {
  if (F <= 0) return 0;
  if (n < 1 || n > 4 || r <= 0 || r % 8) return -1;
  BlockDiagParams p = {};
  for (int j = 0; j < n; ++j) {
    p.b[j] = reinterpret_cast<const __nv_bfloat16*>(b[j]);
    p.begin[j] = begin[j];
    p.end[j] = end[j];
  }
  p.n = n; p.r = r; p.F = F;
  p.scale = scale;
  p.out = reinterpret_cast<__nv_bfloat16*>(out);
  const long long blocks = ((long long)F * (n * r / 8) + 255) / 256;
  block_diag_kernel<<<(unsigned)blocks, 256, 0, stream>>>(p);
  return cudaGetLastError() == cudaSuccess ? 0 : -3;
}
