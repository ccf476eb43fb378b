// Shared device helpers for the sm_100a kernels: mbarrier, TMA, tcgen05/TMEM and cluster PTX
// wrappers, a bounded-wait policy, and small numeric utilities.
//
// Bounded waits: no wait in this library spins forever.  Every mbarrier wait polls with
// try_wait and gives up after WAIT_TIMEOUT_NS of wall time; the thread that gives up records a
// code in the kernel's status word (a device int the host passes in and reads back) and raises a
// CTA-wide abort flag that makes all later waits return at once, so the kernel runs to its end,
// releases its tensor memory and returns.  The output of such a launch is undefined; the host
// raises an error when it sees a non-zero status.
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <type_traits>

namespace tahb {

constexpr unsigned long long WAIT_TIMEOUT_NS = 2000000000ull;  // 2 s

enum Status : int {
  STATUS_OK = 0,
  STATUS_TIMEOUT_TMA_FULL = 1,
  STATUS_TIMEOUT_STAGE_EMPTY = 2,
  STATUS_TIMEOUT_ACCUM = 3,
  STATUS_TIMEOUT_PEER_FLAG = 4,
  STATUS_BAD_INDEX = 5,
};

// ---------------------------------------------------------------------------------------------
// Programmatic dependent launch.  The kernels of the per-layer decode chain are launched with the
// programmatic-stream-serialization attribute: a kernel tells the scheduler at its very start that
// its successor may be launched (pdl_launch_dependents), does the set-up that touches no global
// memory, and then waits until its predecessor has completed and flushed (pdl_wait) before its
// first global access.  Launch latency, CTA scheduling and set-up of kernel N+1 thus overlap the
// tail of kernel N.  Every such kernel executes pdl_wait on every path, so completion of a kernel
// implies completion of all kernels before it.  Both instructions are no-ops in a kernel launched
// without the attribute.
//
// Kernels of a few microseconds release their successor late, when their loads have arrived and only arithmetic
// and stores are left: released at its start, a chain of such kernels piles several waiting grids up on the SMs,
// and a tick of one row (336 launches) took 2.06 ms instead of 1.50 ms; 20 rows 3.51 and 3.04 ms.
// ---------------------------------------------------------------------------------------------
__device__ __forceinline__ void pdl_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// 1 unless the environment variable TAH_B200_PDL is "0" (defined in elementwise.cu)
int pdl_enabled();
// Limit of the waits on flags that another GPU advances, in nanoseconds (defined in elementwise.cu; default
// WAIT_TIMEOUT_NS, changed with tahb_set_peer_wait_limit_ns).  Kernels receive it as a launch parameter.
unsigned long long peer_wait_limit_ns();

// Launch `kern` with (or without) the programmatic-stream-serialization attribute.
template <typename... KArgs, typename... Args>
inline cudaError_t launch_chain(void (*kern)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream,
                                Args&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl_enabled() ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kern, static_cast<KArgs>(args)...);
}

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ unsigned long long globaltimer_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// One lane of a converged warp.  Loops that issue copies and tensor instructions belong to a lane elected so: behind a test of the lane's number the
// compiler wraps every such instruction in a loop over the active lanes (a tensor instruction 57 against about 15 cycles; attention with two
// heads per CTA over 8192 tokens: forward 339 / 289 us, dQ 577 / 398, dK / dV 848 / 768).
__device__ __forceinline__ bool elect_one() {
  uint32_t pred = 0;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "elect.sync _|p, 0xffffffff;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(pred));
  return pred != 0;
}

// ---------------------------------------------------------------------------------------------
// mbarrier
// ---------------------------------------------------------------------------------------------
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}
__device__ __forceinline__ void mbar_fence_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}

// Bounded wait.  `abort_flag` lives in shared memory; `status` in global memory.
__device__ __forceinline__ void mbar_wait(uint64_t* bar, uint32_t parity, volatile int* abort_flag, int* status,
                                          int code) {
  if (mbar_try_wait(bar, parity)) return;
  unsigned long long t0 = 0;
  uint32_t spins = 0;
  while (true) {
    if (*abort_flag) return;
    if (mbar_try_wait(bar, parity)) return;
    if ((++spins & 0x3ff) == 0) {
      unsigned long long now = globaltimer_ns();
      if (t0 == 0) t0 = now;
      else if (now - t0 > WAIT_TIMEOUT_NS) {
        *abort_flag = 1;
        atomicCAS(status, 0, code);
        return;
      }
    }
  }
}

// As mbar_wait, for the loops of a converged warp whose every step a wait stands in: nothing but the barrier is looked at while it answers at once.
// False, in all lanes alike, once this CTA has given up and the barrier is not there yet: the caller leaves its loop.
__device__ __forceinline__ bool mbar_wait_tight(uint64_t* bar, uint32_t parity, volatile int* abort_flag, int* status, int code) {
  if (__all_sync(0xffffffffu, mbar_try_wait(bar, parity))) return true;
  unsigned long long t0 = 0;
#pragma unroll 1
  for (uint32_t spins = 1;; ++spins) {
    if (__any_sync(0xffffffffu, *abort_flag != 0)) return false;
    if (__all_sync(0xffffffffu, mbar_try_wait(bar, parity))) return true;
    if ((spins & 0x3ff) == 0) {
      const unsigned long long now = globaltimer_ns();
      if (t0 == 0) t0 = now;
      else if (__any_sync(0xffffffffu, now - t0 > WAIT_TIMEOUT_NS)) {
        *abort_flag = 1;
        atomicCAS(status, 0, code);
        return false;
      }
    }
  }
}

// For copies and products that are on their way in a CTA that may have given up: they are waited for whatever the flag says (bounded).
__device__ __forceinline__ void mbar_drain(uint64_t* bar, uint32_t parity) {
  const unsigned long long t0 = globaltimer_ns();
  while (!mbar_try_wait(bar, parity) && globaltimer_ns() - t0 < WAIT_TIMEOUT_NS) {}
}

// Bounded wait of ONE thread until flag[q] has reached target[q] (wrap-around safe) for every q <
// world.  The flags are local device memory that peers advance over NVLink after they have stored
// rows into this GPU's memory; target[] is local state.  Returns false after a timeout (status set).
__device__ __forceinline__ bool wait_peer_rows(const uint32_t* flag, const uint32_t* target, int world, int* status,
                                               unsigned long long limit_ns = WAIT_TIMEOUT_NS) {
  if (limit_ns == 0) limit_ns = WAIT_TIMEOUT_NS;
  unsigned long long t0 = 0;
  uint32_t spins = 0;
  for (int q = 0; q < world; ++q) {
    const uint32_t want = target[q];
    while (true) {
      uint32_t v;
      asm volatile("ld.acquire.sys.global.u32 %0, [%1];" : "=r"(v) : "l"(flag + q) : "memory");
      if ((int32_t)(v - want) >= 0) break;
      if ((++spins & 0xff) == 0) {
        const unsigned long long now = globaltimer_ns();
        if (t0 == 0) t0 = now;
        else if (now - t0 > limit_ns) {
          atomicCAS(status, 0, STATUS_TIMEOUT_PEER_FLAG);
          return false;
        }
      }
    }
  }
  return true;
}

// ---------------------------------------------------------------------------------------------
// TMA (no multicast anywhere in this library)
// ---------------------------------------------------------------------------------------------
__device__ __forceinline__ void prefetch_tensormap(const void* tmap) {
  asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(tmap)) : "memory");
}
// 2D tiled load: coordinates (x = innermost element index, y = row).  x * elemsize must be a
// multiple of 16 bytes; callers only pass multiples of 64 bf16 elements.
__device__ __forceinline__ void tma_load_2d(void* smem_dst, const void* tmap, int x, int y, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
      ::"r"(smem_u32(smem_dst)), "l"(reinterpret_cast<uint64_t>(tmap)), "r"(smem_u32(bar)), "r"(x), "r"(y)
      : "memory");
}

__device__ __forceinline__ void tma_load_3d(void* smem_dst, const void* tmap, int x, int y, int z, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
      ::"r"(smem_u32(smem_dst)), "l"(reinterpret_cast<uint64_t>(tmap)), "r"(smem_u32(bar)), "r"(x), "r"(y), "r"(z)
      : "memory");
}

// Untiled bulk copy global -> shared (both addresses 16-byte aligned, size a multiple of 16).
__device__ __forceinline__ void bulk_load(void* smem_dst, const void* gsrc, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
               ::"r"(smem_u32(smem_dst)), "l"(reinterpret_cast<uint64_t>(gsrc)), "r"(bytes), "r"(smem_u32(bar))
               : "memory");
}

// 2D tiled store shared -> global (bulk async group); rows/columns outside the tensor are clipped.
__device__ __forceinline__ void tma_store_2d(const void* tmap, const void* smem_src, int x, int y) {
  asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%2, %3}], [%1];"
               ::"l"(reinterpret_cast<uint64_t>(tmap)), "r"(smem_u32(smem_src)), "r"(x), "r"(y)
               : "memory");
}
__device__ __forceinline__ void tma_store_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
// returns once the committed bulk stores have finished READING shared memory
__device__ __forceinline__ void tma_store_wait_read() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }
// orders this thread's generic-proxy shared-memory writes before later async-proxy (TMA) reads
__device__ __forceinline__ void fence_proxy_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void named_bar_sync(int id, int nthreads) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(nthreads) : "memory");
}

// ---------------------------------------------------------------------------------------------
// tcgen05 / tensor memory
// ---------------------------------------------------------------------------------------------
__device__ __forceinline__ void tmem_alloc(uint32_t* smem_result, uint32_t ncols) {  // whole warp
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(smem_result)),
               "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void tmem_relinquish() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {  // whole warp
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// Shared-memory matrix descriptor for a K-major bf16 tile stored as rows of 64 elements (128 B)
// with the 128-byte swizzle TMA applies: 8-row groups are 1024 B apart (SBO), the tile base is
// 1024-byte aligned, descriptor version 1 (Blackwell), layout type 2 = SWIZZLE_128B.
__device__ __forceinline__ uint64_t umma_desc_sw128(uint32_t smem_addr) {
  uint64_t d = 0;
  d |= static_cast<uint64_t>((smem_addr & 0x3FFFF) >> 4);
  d |= static_cast<uint64_t>(1) << 16;    // leading byte offset (unused for swizzled K-major)
  d |= static_cast<uint64_t>(64) << 32;   // stride byte offset 1024 >> 4
  d |= static_cast<uint64_t>(1) << 46;    // version
  d |= static_cast<uint64_t>(2) << 61;    // SWIZZLE_128B
  return d;
}

// Instruction descriptor: bf16 x bf16 -> fp32, both operands K-major, M x N tile.
__host__ __device__ constexpr uint32_t umma_idesc_bf16(int m, int n) {
  return (1u << 4) | (1u << 7) | (1u << 10) | (static_cast<uint32_t>(n >> 3) << 17) |
         (static_cast<uint32_t>(m >> 4) << 24);
}

// D[tmem] (+)= A[smem] * B[smem]^T ; issued by one thread.
__device__ __forceinline__ void umma_bf16(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc,
                                          uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(tmem_d), "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
      : "memory");
}
// mbarrier arrives when all tcgen05 ops issued so far by this thread have completed.
__device__ __forceinline__ void umma_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
               : "memory");
}

// 32 lanes x 32 columns of fp32: thread i of the warp gets row (lane base + i), columns c..c+31.
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, float* v) {
  uint32_t* r = reinterpret_cast<uint32_t*>(v);
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
        "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
        "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr));
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float* v) {
  uint32_t* r = reinterpret_cast<uint32_t*>(v);
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
}
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, float* v) {
  uint32_t* r = reinterpret_cast<uint32_t*>(v);
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr));
}
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// ---------------------------------------------------------------------------------------------
// thread-block cluster
// ---------------------------------------------------------------------------------------------
__device__ __forceinline__ uint32_t cluster_ctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ float ld_dsmem_f32(uint32_t local_smem_addr, uint32_t rank) {
  uint32_t raddr;
  float v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(raddr) : "r"(local_smem_addr), "r"(rank));
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(raddr) : "memory");
  return v;
}

__device__ __forceinline__ uint32_t dsmem_addr(uint32_t local_smem_addr, uint32_t rank) {
  uint32_t raddr;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(raddr) : "r"(local_smem_addr), "r"(rank));
  return raddr;
}
__device__ __forceinline__ void st_dsmem_v4(uint32_t cluster_addr, float4 v) {
  asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};"
               ::"r"(cluster_addr), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w)
               : "memory");
}
__device__ __forceinline__ void st_dsmem_u32(uint32_t cluster_addr, uint32_t v) {
  asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(cluster_addr), "r"(v) : "memory");
}
__device__ __forceinline__ void st_dsmem_f32(uint32_t cluster_addr, float v) {
  asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(cluster_addr), "f"(v) : "memory");
}
__device__ __forceinline__ float4 ld_dsmem_v4(uint32_t local_smem_addr, uint32_t rank) {
  uint32_t raddr;
  float4 v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(raddr) : "r"(local_smem_addr), "r"(rank));
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
               : "r"(raddr)
               : "memory");
  return v;
}

// ---------------------------------------------------------------------------------------------
// numerics
// ---------------------------------------------------------------------------------------------
__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
// 2^x on the special-function unit, no range fix-up (2^-inf = +0, denormal results flush to 0)
__device__ __forceinline__ float ex2_approx(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float bf16_round(float x) { return __bfloat162float(__float2bfloat16_rn(x)); }
// x * sigmoid(x) with the approximate exponential and the approximate division (a reciprocal and a multiply: the
// IEEE division is a dozen instructions, which made the SwiGLU epilogue of a 128 x 256 tile cost as much as its
// main loop).  Relative error ~2^-21, far below the bf16 rounding that follows every use.
__device__ __forceinline__ float silu(float x) { return __fdividef(x, 1.0f + __expf(-x)); }

// EPL consecutive bf16 of a lane, moved BYTES (a power of two from 2 on) at a time: everything they lie on has to start on such a boundary.
// 2 also takes words of 4 bytes, off their boundary shifted out of the words around the piece (loads) or with one element at each end (stores).
template <int EPL, int BYTES = EPL * 2>
struct alignas(EPL * 2) QkvPiece {
  static_assert(BYTES >= 2 && BYTES <= EPL * 2 && BYTES <= 16, "words of a piece");
  __nv_bfloat16 v[EPL];
  using Word = typename std::conditional<
      BYTES == 16, uint4, typename std::conditional<BYTES == 8, uint2, typename std::conditional<BYTES == 4, uint32_t, __nv_bfloat16>::type>::type>::type;
  __device__ __forceinline__ __nv_bfloat162& pair(int i) { return reinterpret_cast<__nv_bfloat162*>(v)[i]; }
  __device__ __forceinline__ void load(const __nv_bfloat16* src) {
    if constexpr (BYTES == 2) {
      uint32_t* o = reinterpret_cast<uint32_t*>(v);
      const uint32_t odd = (uint32_t)(reinterpret_cast<uintptr_t>(src) & 2) / 2;
      const uint32_t* w = reinterpret_cast<const uint32_t*>(src - odd);
      uint32_t a = w[0];
#pragma unroll
      for (int i = 0; i < EPL / 2; ++i) {
        const uint32_t b = i + 1 < EPL / 2 || odd ? w[i + 1] : 0u;      // the last word of an odd piece holds its last element
        o[i] = __funnelshift_r(a, b, odd * 16);
        a = b;
      }
    } else {
#pragma unroll
      for (int i = 0; i < EPL * 2 / BYTES; ++i) reinterpret_cast<Word*>(v)[i] = reinterpret_cast<const Word*>(src)[i];
    }
  }
  __device__ __forceinline__ void store(__nv_bfloat16* dst) const {
    if constexpr (BYTES == 2) {
      const uint32_t* o = reinterpret_cast<const uint32_t*>(v);
      if (reinterpret_cast<uintptr_t>(dst) & 2) {
        dst[0] = v[0];
#pragma unroll
        for (int i = 0; i + 1 < EPL / 2; ++i) reinterpret_cast<uint32_t*>(dst + 1)[i] = __funnelshift_r(o[i], o[i + 1], 16);
        dst[EPL - 1] = v[EPL - 1];
      } else {
#pragma unroll
        for (int i = 0; i < EPL / 2; ++i) reinterpret_cast<uint32_t*>(dst)[i] = o[i];
      }
    } else {
#pragma unroll
      for (int i = 0; i < EPL * 2 / BYTES; ++i) reinterpret_cast<Word*>(dst)[i] = reinterpret_cast<const Word*>(v)[i];
    }
  }
};

// How many CTAs the heads of a token are dealt out to: one head per warp while tokens x CTAs stay below `most`, else half as many, ...
inline int qk_head_groups(int tokens, int heads, int warps, int most) {
  int g = (heads + warps - 1) / warps;
  while (g > 1 && (long long)tokens * g > most) g = (g + 1) / 2;
  return g;
}

struct __align__(16) bf16x8 {
  __nv_bfloat162 v[4];
};

}  // namespace tahb
