// Paged-KV decode attention over all iteration caches of a row, and a plain varlen duo-causal
// attention used as the bring-up / reference path for packed prefill.
//
// Decode: one query token per row.  A row at iteration depth d attends every entry of its own
// sequence in caches 0..d (its own K/V was appended to cache d before this kernel runs), which
// is the duo-causal rule for the newest position.  The caches are paged; cache c of one layer is
//   [page][2 (K,V)][n_kv_heads][page_size][HD]  bf16
// with a page table pt[c][row][i] and a length len[c][row].
//
// Work split: an item is (KV head, row, split), one CTA; its pages go to its two to four warps in turn.  All G = nq / nkv query
// heads that share the KV head are handled together, so K / V are read once, straight from global memory into the registers that
// warp-level tensor instructions read (a page and a half of a warp's in flight; no shared memory ring):
//
//     scores [16 entries][8 columns] = K Q^T      a lane reads 16 consecutive bytes of a K row and of Q at the same dims: the order
//                                                 of a reduction is free as long as both operands agree (see gemm_few.cu)
//     O^T [16 dims][8 columns] += V^T P           a lane reads eight dims of four entries and pairs them
//
// Column = (part, head): P in fp32 is the sum of three bf16 parts, exactly, and the parts take columns that one or two heads leave
// empty, so nothing of a probability is lost.  Online softmax in base 2; the warps merge through shared memory; with n_split > 1
// partial (m, l, acc) go to a workspace and a second kernel merges.
//
// What bounds it: HBM, and for short rows the chain of dependent loads of an item (length, page number, page).  The kernel before had
// four copy-fed warps per item on fp32 multiply-adds, 190 instructions for four entries of a warp, and was bound by their issue:
// us, 16 heads on 8 KV heads, before and now: 1 row at 60 entries 4.6 and 3.5, 6 rows at 220 10.0 and 8.5, 20 rows at 1300 34.7 and 29.4,
// 256 rows at 80 31.9 and 25.6, at 600 116 and 109 (5.9 TB/s).
#include "common.cuh"
#include "tah_b200_noalloc.h"

namespace tahb {

constexpr int MAX_CACHES = 4;

struct DecodeAttnParams {
  const __nv_bfloat16* q;       // [rows, nq, HD]
  __nv_bfloat16* out;           // [rows, nq, HD]
  const __nv_bfloat16* cache[MAX_CACHES];
  const int* page_table[MAX_CACHES];
  const int* len[MAX_CACHES];
  const int* depth;             // [rows] (nullptr: every row sees n_caches caches)
  float* ws;                    // [rows, nq, n_split, HD + 2]  (n_split > 1)
  int n_caches, rows, nq, nkv, page_size, max_pages[MAX_CACHES], n_split;
  float scale_log2;             // softmax scale * log2(e)
};

constexpr int ATT_PAGE = 16;

// Warps of the decode kernel that fit an SM without spills.
constexpr int att_resident_warps(int hd, int G) { return 3 * G > 8 ? (hd == 64 ? 12 : 8) : hd == 64 ? 16 : 12; }

template <int HD, int G>
struct AttCfg {
  static constexpr int STEPS = HD / 32;             // 16-byte pieces of a K row per lane
  static constexpr int HALVES = HD / 64;
  static constexpr int COLS = 3 * G;                // (part, head): see decode_attn_kernel
  static constexpr int TILES = (COLS + 7) / 8;
  static constexpr int PITCH = HD + 4;              // floats per column in the merge area
  static constexpr int WARPS = att_resident_warps(HD, G);
};

// Maps the i-th visible page of a row (pages of cache 0 first, then cache 1, ...) to its cache and
// to the page index inside that cache.
__device__ __forceinline__ void locate_page(int i, const int* seg_pages, int& c, int& local) {
  c = 0;
  local = i;
#pragma unroll
  for (int cc = 0; cc < MAX_CACHES - 1; ++cc)
    if (c == cc && local >= seg_pages[cc]) { local -= seg_pages[cc]; c = cc + 1; }
}

// c += A B.  The tensor core truncates where it adds to its accumulator: a product of its own per step and a rounded addition
// keep the sums as close to the exact ones as fp32 multiply-adds are.
__device__ __forceinline__ void att_mma_add(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  float d0, d1, d2, d3;
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%10, %10, %10, %10};"
               : "=f"(d0), "=f"(d1), "=f"(d2), "=f"(d3)
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.f));
  c[0] += d0; c[1] += d1; c[2] += d2; c[3] += d3;
}
__device__ __forceinline__ uint4 att_ld(const __nv_bfloat16* p) {
  uint4 v;
  asm volatile("ld.global.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}
// 8x8 tile of 16-bit values: lane (g, t) gives row g, columns 2t and 2t + 1, and gets column g, rows 2t and 2t + 1
__device__ __forceinline__ uint32_t att_transpose(uint32_t v) {
  uint32_t r;
  asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(r) : "r"(v));
  return r;
}
// part 0, 1, 2 of x: x = part 0 + part 1 + part 2 exactly, eight bits each
__device__ __forceinline__ float bf16_part(float x, int part) {
  const float hi = bf16_round(x), r1 = x - hi, mid = bf16_round(r1);
  return part == 0 ? hi : part == 1 ? mid : part == 2 ? r1 - mid : 0.f;
}

template <int HD, int G, int NW>
__global__ void __launch_bounds__(NW * 32, AttCfg<HD, G>::WARPS / NW) decode_attn_kernel(const DecodeAttnParams p) {
  pdl_wait();
  using C = AttCfg<HD, G>;
  constexpr int S = C::STEPS, NH = C::HALVES, NT = C::TILES;
  static_assert(C::PITCH % 4 == 0, "a column's 16-byte pieces");
  __shared__ __align__(16) float part[NW][C::COLS][C::PITCH];      // written as float4
  __shared__ float part_ml[NW][G][2];
  const int kvh = blockIdx.x, row = blockIdx.y, split = blockIdx.z;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;

  int seg_len[MAX_CACHES], seg_pages[MAX_CACHES];
  int total_pages = 0;
  const int visible = p.depth ? min(p.depth[row] + 1, p.n_caches) : p.n_caches;
#pragma unroll
  for (int c = 0; c < MAX_CACHES; ++c) {
    seg_len[c] = (c < visible) ? p.len[c][row] : 0;
    seg_pages[c] = (seg_len[c] + ATT_PAGE - 1) / ATT_PAGE;
    total_pages += seg_pages[c];
  }
  const int ppc = (total_pages + p.n_split - 1) / p.n_split;
  const int pb = split * ppc;
  const int pe = min(total_pages, pb + ppc);
  const int n = pe - pb > warp ? (pe - pb - warp + NW - 1) / NW : 0;      // pages pb + warp, + NW, ... are this warp's

  // 32 of the warp's pages at a time, one per lane: K block of this head, entries that are visible in it
  const __nv_bfloat16* blk = nullptr;
  int entries = 0;
  auto look_up = [&](int i) {
    const int pg = pb + warp + NW * (i + lane);
    if (pg >= pe) return;
    int c, local;
    locate_page(pg, seg_pages, c, local);
    int len = seg_len[0];
#pragma unroll
    for (int cc = 1; cc < MAX_CACHES; ++cc) if (c == cc) len = seg_len[cc];
    const int page = p.page_table[c][(size_t)row * p.max_pages[c] + local];
    blk = p.cache[c] + ((size_t)page * 2 * p.nkv + kvh) * (ATT_PAGE * HD);
    entries = len - local * ATT_PAGE;
  };
  auto block_of = [&](int i) {
    return reinterpret_cast<const __nv_bfloat16*>(__shfl_sync(0xffffffffu, reinterpret_cast<unsigned long long>(blk), i & 31));
  };
  uint4 kx[S], ky[S], v[NH][4];
  auto load_k = [&](const __nv_bfloat16* b) {           // entries g and g + 8
#pragma unroll
    for (int s = 0; s < S; ++s) {
      kx[s] = att_ld(b + g * HD + s * 32 + t * 8);
      ky[s] = att_ld(b + (g + 8) * HD + s * 32 + t * 8);
    }
  };
  auto load_v = [&](const __nv_bfloat16* b) {           // entries 2t, 2t + 1, 2t + 8, 2t + 9
    b += (size_t)p.nkv * (ATT_PAGE * HD);
#pragma unroll
    for (int h = 0; h < NH; ++h)
#pragma unroll
      for (int e = 0; e < 4; ++e) v[h][e] = att_ld(b + (2 * t + (e & 1) + 8 * (e >> 1)) * HD + h * 64 + g * 8);
  };
  look_up(0);
  if (n > 0) {
    const __nv_bfloat16* b = block_of(0);
    load_k(b);
    load_v(b);
  }

  // column g of the score tile: head g % G
  uint4 q[S];
  const __nv_bfloat16* qs = p.q + ((size_t)row * p.nq + kvh * G + g % G) * HD + t * 8;
  if ((reinterpret_cast<uintptr_t>(p.q) & 15) == 0) {
#pragma unroll
    for (int s = 0; s < S; ++s) q[s] = *reinterpret_cast<const uint4*>(qs + s * 32);
  } else {
#pragma unroll
    for (int s = 0; s < S; ++s) {
      __nv_bfloat16* e = reinterpret_cast<__nv_bfloat16*>(&q[s]);
#pragma unroll
      for (int j = 0; j < 8; ++j) e[j] = qs[s * 32 + j];
    }
  }

  // this lane's columns 2t and 2t + 1: maximum, its entries' share of the weight, and O
  float m[2] = {-INFINITY, -INFINITY}, l[2] = {0.f, 0.f}, acc[NT][NH][4][4];
#pragma unroll
  for (int a = 0; a < NT * NH * 16; ++a) (&acc[0][0][0][0])[a] = 0.f;

  for (int i = 0; i < n; ++i) {
    float sc[4] = {0.f, 0.f, 0.f, 0.f};                 // entries g (0, 1) and g + 8 (2, 3), columns 2t and 2t + 1
#pragma unroll
    for (int s = 0; s < S; ++s) {
      att_mma_add(sc, kx[s].x, ky[s].x, kx[s].y, ky[s].y, q[s].x, q[s].y);
      att_mma_add(sc, kx[s].z, ky[s].z, kx[s].w, ky[s].w, q[s].z, q[s].w);
    }
    const int have = __shfl_sync(0xffffffffu, entries, i & 31);
    const bool more = i + 1 < n;
    if (more && ((i + 1) & 31) == 0) look_up(i + 1);
    const __nv_bfloat16* next = block_of(i + 1);
    if (more) load_k(next);
#pragma unroll
    for (int c = 0; c < 4; ++c) sc[c] = g + 8 * (c >> 1) < have ? sc[c] * p.scale_log2 : -INFINITY;
    const float mx[2] = {fmaxf(sc[0], sc[2]), fmaxf(sc[1], sc[3])};
    if (__any_sync(0xffffffffu, mx[0] > m[0] || mx[1] > m[1])) {
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        float top = fmaxf(m[c], mx[c]);
#pragma unroll
        for (int o = 4; o < 32; o <<= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, o));
        const float f = m[c] == -INFINITY ? 0.f : exp2f(m[c] - top);
        m[c] = top;
        l[c] *= f;
#pragma unroll
        for (int a = 0; a < NT * NH * 8; ++a) (&acc[0][0][0][0])[2 * a + c] *= f;
      }
    }
    float w[4];
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      w[c] = sc[c] == -INFINITY ? 0.f : exp2f(sc[c] - m[c & 1]);
      l[c & 1] += w[c];
    }
    uint32_t b[NT][2];
#pragma unroll
    for (int a = 0; a < NT; ++a)
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        const __nv_bfloat162 pair = __floats2bfloat162_rn(bf16_part(w[2 * r], (8 * a + 2 * t) / G), bf16_part(w[2 * r + 1], (8 * a + 2 * t + 1) / G));
        b[a][r] = att_transpose(*reinterpret_cast<const uint32_t*>(&pair));
      }
    if (have < ATT_PAGE) {                              // what lies behind the last entry may be NaN bits
#pragma unroll
      for (int h = 0; h < NH; ++h)
#pragma unroll
        for (int e = 0; e < 4; ++e)
          if (2 * t + (e & 1) + 8 * (e >> 1) >= have) v[h][e] = make_uint4(0u, 0u, 0u, 0u);
    }
#pragma unroll
    for (int h = 0; h < NH; ++h) {
      const uint32_t* e0 = reinterpret_cast<const uint32_t*>(&v[h][0]);
      const uint32_t* e1 = reinterpret_cast<const uint32_t*>(&v[h][1]);
      const uint32_t* e2 = reinterpret_cast<const uint32_t*>(&v[h][2]);
      const uint32_t* e3 = reinterpret_cast<const uint32_t*>(&v[h][3]);
#pragma unroll
      for (int d = 0; d < 4; ++d) {                     // rows g and g + 8 of the tile: dims 8 g + 2 d and 8 g + 2 d + 1
        const uint32_t a0 = __byte_perm(e0[d], e1[d], 0x5410), a1 = __byte_perm(e0[d], e1[d], 0x7632);
        const uint32_t a2 = __byte_perm(e2[d], e3[d], 0x5410), a3 = __byte_perm(e2[d], e3[d], 0x7632);
#pragma unroll
        for (int a = 0; a < NT; ++a) att_mma_add(acc[a][h][d], a0, a1, a2, a3, b[a][0], b[a][1]);
      }
    }
    if (more) load_v(next);
  }

  pdl_launch_dependents();
  // the warps meet in shared memory
#pragma unroll
  for (int c = 0; c < 2; ++c) {
#pragma unroll
    for (int o = 4; o < 32; o <<= 1) l[c] += __shfl_xor_sync(0xffffffffu, l[c], o);
    if (g == 0 && 2 * t + c < G) {
      part_ml[warp][2 * t + c][0] = m[c];
      part_ml[warp][2 * t + c][1] = l[c];
    }
#pragma unroll
    for (int a = 0; a < NT; ++a) {
      const int col = 8 * a + 2 * t + c;
      if (col >= C::COLS) continue;
#pragma unroll
      for (int h = 0; h < NH; ++h) {
        float4* dst = reinterpret_cast<float4*>(&part[warp][col][h * 64 + g * 8]);
        dst[0] = make_float4(acc[a][h][0][c], acc[a][h][0][2 + c], acc[a][h][1][c], acc[a][h][1][2 + c]);
        dst[1] = make_float4(acc[a][h][2][c], acc[a][h][2][2 + c], acc[a][h][3][c], acc[a][h][3][2 + c]);
      }
    }
  }
  __syncthreads();
  for (int idx = tid; idx < G * HD; idx += NW * 32) {
    const int hg = idx / HD, d = idx % HD;
    float mx = -INFINITY;
#pragma unroll
    for (int w = 0; w < NW; ++w) mx = fmaxf(mx, part_ml[w][hg][0]);
    float num = 0.f, den = 0.f;
#pragma unroll
    for (int w = 0; w < NW; ++w) {
      const float mw = part_ml[w][hg][0];
      const float f = (mw == -INFINITY) ? 0.f : exp2f(mw - mx);
      const float hi = part[w][hg][d], v = hi + (part[w][G + hg][d] + part[w][2 * G + hg][d]);
      num += f * (fabsf(v) < INFINITY ? v : hi);        // an infinite entry: its products with the parts of one weight may cancel
      den += f * part_ml[w][hg][1];
    }
    const int head = kvh * G + hg;
    if (p.n_split == 1) {
      p.out[((size_t)row * p.nq + head) * HD + d] = __float2bfloat16_rn(den > 0.f ? num / den : 0.f);
    } else {
      float* w = p.ws + (((size_t)row * p.nq + head) * p.n_split + split) * (HD + 2);
      w[d] = num;
      if (d == 0) { w[HD] = mx; w[HD + 1] = den; }
    }
  }
}

template <int HD>
__global__ void decode_attn_merge_kernel(const float* ws, __nv_bfloat16* out, int n_split) {
  pdl_launch_dependents();
  pdl_wait();
  const int rh = blockIdx.x;   // row * nq + head
  const float* w = ws + (size_t)rh * n_split * (HD + 2);
  for (int d = threadIdx.x; d < HD; d += blockDim.x) {
    float mx = -INFINITY;
    for (int s = 0; s < n_split; ++s) mx = fmaxf(mx, w[s * (HD + 2) + HD]);
    float num = 0.f, den = 0.f;
    for (int s = 0; s < n_split; ++s) {
      const float ms = w[s * (HD + 2) + HD];
      const float f = (ms == -INFINITY) ? 0.f : exp2f(ms - mx);
      num += f * w[s * (HD + 2) + d];
      den += f * w[s * (HD + 2) + HD + 1];
    }
    out[(size_t)rh * HD + d] = __float2bfloat16_rn(den > 0.f ? num / den : 0.f);
  }
}

// ---------------------------------------------------------------------------------------------
// Plain varlen duo-causal attention over packed tokens (CUDA cores, one warp per (token, head)).
// Query token i attends, in up to three segments s, KV rows  seg_base[s][i] + j  for
// j < seg_count[s][i]  of the packed K/V tensors k[s]/v[s]  ([n, nkv, HD]).  Callers derive
// (base, count) from the duo-causal rule: segment 0 = depth-0 K/V of the same sequence up to the
// query's position, segment 1 = deeper K/V of the same sequence up to the query's own entry.
// ---------------------------------------------------------------------------------------------
struct VarlenAttnParams {
  const __nv_bfloat16* q;
  __nv_bfloat16* out;
  const __nv_bfloat16* k[3];
  const __nv_bfloat16* v[3];
  const int* seg_base[3];
  const int* seg_count[3];
  int n_q, nq, nkv, n_seg;
  float scale_log2;
};

template <int HD>
__global__ void __launch_bounds__(128) varlen_attn_naive_kernel(const VarlenAttnParams p) {
  constexpr int EPL = HD / 32;
  const int wg = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (wg >= p.n_q * p.nq) return;
  const int t = wg / p.nq, h = wg % p.nq;
  const int kvh = h / (p.nq / p.nkv);
  float qv[EPL], acc[EPL];
#pragma unroll
  for (int i = 0; i < EPL; ++i) {
    qv[i] = __bfloat162float(p.q[((size_t)t * p.nq + h) * HD + lane * EPL + i]) * p.scale_log2;
    acc[i] = 0.f;
  }
  float m = -INFINITY, l = 0.f;
  for (int s = 0; s < p.n_seg; ++s) {
    const int base = p.seg_base[s][t], cnt = p.seg_count[s][t];
    for (int j = 0; j < cnt; ++j) {
      const size_t off = ((size_t)(base + j) * p.nkv + kvh) * HD + lane * EPL;
      float dot = 0.f;
#pragma unroll
      for (int i = 0; i < EPL; ++i) dot += qv[i] * __bfloat162float(p.k[s][off + i]);
      dot = warp_sum(dot);
      const float mx = fmaxf(m, dot);
      const float corr = (m == -INFINITY) ? 0.f : exp2f(m - mx);
      const float pw = exp2f(dot - mx);
      l = l * corr + pw;
#pragma unroll
      for (int i = 0; i < EPL; ++i) acc[i] = acc[i] * corr + pw * __bfloat162float(p.v[s][off + i]);
      m = mx;
    }
  }
#pragma unroll
  for (int i = 0; i < EPL; ++i)
    p.out[((size_t)t * p.nq + h) * HD + lane * EPL + i] = __float2bfloat16_rn(l > 0.f ? acc[i] / l : 0.f);
}

// Estimated cost of `items` (row, KV head) items of up to `pages` pages, every one cut into `split` parts of `warps` warps: microseconds when
// all are that long plus microseconds when their lengths are spread.  A CTA takes the start of an item (length, page number, page: dependent
// loads) and its warps' pages in turn, a page at its latency or, with enough warps on the chip, at its share of HBM; a split adds the merge
// kernel.  Equal items run in waves; uneven ones fill the SMs as they end, and behind them the longest one stands alone.  Fitted to 1 to 256
// rows of 60 to 2099 entries, equal and spread from a quarter to all of them, in all six geometries: the choice among 2 to 4 warps and 1 to 4
// parts is 0.9 % behind the best for each on average.
static double decode_estimate(int hd, int G, long long items, int pages, int split, int warps) {
  constexpr double START = 4.5, HBM_KB = 6500.0, MEAN = 0.5, ALONE = 0.65;
  const long long n = items * split, resident = 148ll * (att_resident_warps(hd, G) / warps);
  const int whole = (pages + split - 1) / split;
  const double steps = 0.5 * ((whole + warps - 1) / warps + (double)pages / split / warps);
  const double latency = hd == 128 ? (3 * G > 8 ? 1.7 : 2.1) : (3 * G > 8 ? 1.45 : 1.9), page = ATT_PAGE * hd * 4 / 1000.0 / HBM_KB;
  auto wave = [&](long long ctas) { return ctas > 0 ? START + steps * fmax(latency, ctas * warps * page) : 0.0; };
  const double equal = n / resident * wave(resident) + wave(n % resident), moved = n * warps * steps * MEAN * page, turns = (double)n / resident;
  const double spread = n <= resident ? START + fmax(steps * latency, moved)
                                      : fmax(turns * (START + MEAN * steps * latency), turns * START + moved) + ALONE * (START + steps * latency);
  return equal + spread + (split > 1 ? 2.0 * (6.2 + 0.0007 * n) : 0.0);
}

static int decode_warps(int hd, int G, long long items, int pages, int split) {
  int best = 4;
  for (int w = 3; w >= 2; --w)          // three of eight resident warps fit no more items than four: they are never taken there
    if (decode_estimate(hd, G, items, pages, split, w) < decode_estimate(hd, G, items, pages, split, best)) best = w;
  return best;
}

// Two to four warps per item, by the estimate: with four, 444 items of heads of 128 run at once, with three 592, with two 888.  Four / the
// number taken, us, 8 KV heads of two heads of 128: 64 rows at 60 entries 10.2 / 8.0 (three), at 300 23.4 / 17.5, at 1024 61.6 / 46.1 (spread
// from a quarter of that 41.8 / 39.5); 96 rows at 140 17.2 / 14.1 (two); 256 rows at 60 25.2 / 21.4 (two); 128 rows at 1024 96.6 / 87.7 (three;
// spread 63.4 / 69.1, the other way round).
template <int HD, int G>
static int launch_decode(const DecodeAttnParams& p, cudaStream_t stream) {
  const dim3 grid(p.nkv, p.rows, p.n_split);
  int pages = 0;
  for (int c = 0; c < p.n_caches; ++c) pages = p.max_pages[c] > pages ? p.max_pages[c] : pages;
  const int warps = decode_warps(HD, G, (long long)p.nkv * p.rows, pages, p.n_split);
  constexpr int THREE = AttCfg<HD, G>::WARPS == 8 ? 4 : 3;
  cudaError_t e = warps == 2   ? launch_chain(decode_attn_kernel<HD, G, 2>, grid, dim3(64), 0, stream, p)
                  : warps == 3 ? launch_chain(decode_attn_kernel<HD, G, THREE>, grid, dim3(32 * THREE), 0, stream, p)
                               : launch_chain(decode_attn_kernel<HD, G, 4>, grid, dim3(128), 0, stream, p);
  if (e == cudaSuccess && p.n_split > 1)
    e = launch_chain(decode_attn_merge_kernel<HD>, dim3(p.rows * p.nq), dim3(HD), 0, stream, p.ws, p.out, p.n_split);
  return e == cudaSuccess ? 0 : -3;
}

}  // namespace tahb

using namespace tahb;

// Workspace floats needed by tahb_decode_attn when n_split > 1.
extern "C" long long tahb_decode_attn_ws_floats(int rows, int nq, int hd, int n_split) {
  return n_split > 1 ? (long long)rows * nq * n_split * (hd + 2) : 0;
}

// The number of warps per item that a launch takes.
extern "C" int tahb_decode_attn_warps(int rows, int nq, int nkv, int hd, int pages, int n_split) {
  return decode_warps(hd, nq / nkv, (long long)rows * nkv, pages, n_split);
}

// How many parts (1 to 4) every (row, KV head) item is best cut into when rows hold up to `pages` pages; no launch, no GPU needed.
extern "C" int tahb_decode_attn_split(int rows, int nq, int nkv, int hd, int pages) {
  if (rows <= 0 || nkv <= 0 || nq < nkv) return 1;
  const int G = nq / nkv;
  const long long items = (long long)rows * nkv;
  auto cost = [&](int s) { return decode_estimate(hd, G, items, pages, s, decode_warps(hd, G, items, pages, s)); };
  int best = 1;
  for (int s = 2; s <= 4; ++s)
    if (cost(s) < cost(best)) best = s;
  return best;
}

extern "C" int tahb_decode_attn(const void* q, void* out, void* const* caches, const int* const* page_tables,
                                const int* const* lens, const int* max_pages, int n_caches, const int* depth,
                                int rows, int nq, int nkv, int hd, int page_size, float scale, int n_split,
                                float* ws, int* status, cudaStream_t stream) {
  if (rows <= 0) return 0;
  if (page_size != ATT_PAGE) return -5;
  if (n_caches < 1 || n_caches > MAX_CACHES) return -1;
  if (n_split < 1) n_split = 1;
  if (n_split > 1 && ws == nullptr) return -4;
  DecodeAttnParams p;
  p.q = reinterpret_cast<const __nv_bfloat16*>(q);
  p.out = reinterpret_cast<__nv_bfloat16*>(out);
  for (int c = 0; c < MAX_CACHES; ++c) {
    const int cc = c < n_caches ? c : 0;
    p.cache[c] = reinterpret_cast<const __nv_bfloat16*>(caches[cc]);
    p.page_table[c] = page_tables[cc];
    p.len[c] = lens[cc];
    p.max_pages[c] = max_pages[cc];
  }
  p.depth = depth;
  p.ws = ws;
  (void)status;                 // no wait in this kernel can run out
  p.n_caches = n_caches; p.rows = rows; p.nq = nq; p.nkv = nkv; p.page_size = page_size; p.n_split = n_split;
  p.scale_log2 = scale * 1.4426950408889634f;
  const int G = nq / nkv;
  if (nq % nkv) return -2;
#define TAHB_DEC(HD_, G_) if (hd == HD_ && G == G_) return launch_decode<HD_, G_>(p, stream);
  TAHB_DEC(128, 1) TAHB_DEC(128, 2) TAHB_DEC(128, 4)
  TAHB_DEC(64, 1) TAHB_DEC(64, 2) TAHB_DEC(64, 4)
#undef TAHB_DEC
  return -2;
}

// ---------------------------------------------------------------------------------------------
// Allocation-free variant (declared and documented in tah_b200_noalloc.h).
// ---------------------------------------------------------------------------------------------
constexpr long long NOALLOC_WS_FLOATS = 1ll << 20;     // 4 MiB of scratch per GPU
static __device__ __align__(256) float g_noalloc_ws[NOALLOC_WS_FLOATS];

extern "C" long long tahb_decode_attn_noalloc_capacity(void) { return NOALLOC_WS_FLOATS; }

// In host code `g_noalloc_ws` is only a handle for the symbol, not an address a kernel can use:
// the device address is looked up once per device and cached here.
static float* noalloc_ws_for_current_device(void) {
  constexpr int MAX_DEVICES = 64;
  static float* cached[MAX_DEVICES] = {nullptr};
  int dev = -1;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= MAX_DEVICES) return nullptr;
  if (cached[dev] == nullptr) {
    float* ptr = nullptr;
    if (cudaGetSymbolAddress(reinterpret_cast<void**>(&ptr), g_noalloc_ws) != cudaSuccess) return nullptr;
    cached[dev] = ptr;
  }
  return cached[dev];
}

extern "C" int tahb_decode_attn_noalloc(const void* q, void* out, void* const* caches,
                                        const int* const* page_tables, const int* const* lens,
                                        const int* max_pages, int n_caches, const int* depth, int rows, int nq,
                                        int nkv, int hd, int page_size, float scale, int n_split, int* status,
                                        cudaStream_t stream) {
  if (n_split < 1) n_split = 1;
  const long long need = tahb_decode_attn_ws_floats(rows, nq, hd, n_split);
  if (need > NOALLOC_WS_FLOATS) return -7;     // request exceeds the built-in scratch area
  float* ws = noalloc_ws_for_current_device();
  if (ws == nullptr) return -8;
  return tahb_decode_attn(q, out, caches, page_tables, lens, max_pages, n_caches, depth, rows, nq, nkv, hd,
                          page_size, scale, n_split, ws, status, stream);
}

extern "C" int tahb_varlen_attn_naive(const void* q, void* out, void* const* ks, void* const* vs,
                                      const int* const* bases, const int* const* counts, int n_seg, int n_q, int nq,
                                      int nkv, int hd, float scale, cudaStream_t stream) {
  if (n_q <= 0) return 0;
  if (n_seg < 1 || n_seg > 3) return -1;
  VarlenAttnParams p;
  p.q = reinterpret_cast<const __nv_bfloat16*>(q);
  p.out = reinterpret_cast<__nv_bfloat16*>(out);
  for (int s = 0; s < 3; ++s) {
    const int ss = s < n_seg ? s : 0;
    p.k[s] = reinterpret_cast<const __nv_bfloat16*>(ks[ss]);
    p.v[s] = reinterpret_cast<const __nv_bfloat16*>(vs[ss]);
    p.seg_base[s] = bases[ss];
    p.seg_count[s] = counts[ss];
  }
  p.n_q = n_q; p.nq = nq; p.nkv = nkv; p.n_seg = n_seg;
  p.scale_log2 = scale * 1.4426950408889634f;
  const long long warps = (long long)n_q * nq;
  const int blocks = (int)((warps + 3) / 4);
  if (hd == 128) varlen_attn_naive_kernel<128><<<blocks, 128, 0, stream>>>(p);
  else if (hd == 64) varlen_attn_naive_kernel<64><<<blocks, 128, 0, stream>>>(p);
  else return -2;
  return cudaGetLastError() == cudaSuccess ? 0 : -3;
}
