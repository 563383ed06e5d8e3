// BF16 tensor-core kernels of the learned warm start (sm_100a): the network
// that predicts an initial flow field from the case parameters is trained
// and evaluated with these kernels only.
//
//   ffnn_gemm     C[M,N] = A[M,K] * B[N,K]^T (+ bias, SiLU), BF16 operands,
//                 FP32 accumulation in tensor memory (tcgen05.mma, one
//                 elected thread per CTA, operands staged in shared memory
//                 in the canonical K-major core-matrix layout, completion
//                 through an mbarrier, accumulator read back with
//                 tcgen05.ld): k_gemm_rows for many rows against one small
//                 matrix, else k_gemm_bf16 (with split-K and FP32 atomics
//                 where a caller asks for it; the network does not).
//   ffnn_wgrad    G[N,K] += X[R,N]^T Y[R,K], the weight gradients.
//   element-wise  SiLU backward and mean-squared-error gradient, each also
//                 with the bias gradient in the same pass (the network's
//                 form), column sums, transposes, casts, Adam.
//
// Every device wait is bounded: on time-out the kernel sets the error word,
// waits (bounded) for its own tensor-core work, frees its tensor memory and
// returns; the host reads the word with ffnn_error().
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/finflo_nn.h"

namespace {

constexpr int GM = 128;        // rows of a CTA tile (tcgen05 M)
constexpr int GKT = 64;        // K elements staged per iteration (4 MMAs of K = 16)
constexpr int GTHREADS = 128;  // 4 warps: one per 32 TMEM lanes
constexpr long kSpin = 1L << 26;

__device__ int g_err;          // first error of any kernel of this file

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}\n"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}

// Bounded wait for one phase of an mbarrier; false on time-out.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity) {
  for (long it = 0; it < kSpin; it++)
    if (mbar_try_wait(bar, parity)) return true;
  return false;
}

// Shared-memory matrix descriptor, K-major without swizzle: core matrices
// of 8 rows x 16 bytes; lbo = byte distance of the two core matrices along
// K that one MMA (K = 16) reads, sbo = byte distance of 8-row groups.
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
  uint64_t d = 0;
  d |= (uint64_t)((addr >> 4) & 0x3FFFu);
  d |= (uint64_t)((lbo >> 4) & 0x3FFFu) << 16;
  d |= (uint64_t)((sbo >> 4) & 0x3FFFu) << 32;
  d |= (uint64_t)1 << 46;   // descriptor version of sm_100
  return d;                 // base offset 0, legacy LBO mode, no swizzle
}

// Instruction descriptor of kind::f16: BF16 A and B (K-major), FP32 D.
__host__ __device__ constexpr uint32_t instr_desc(int m, int n) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}

__device__ __forceinline__ void mma_bf16(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                         uint32_t accumulate) {
  uint32_t z = 0;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %6, %7, %8}, p;\n\t}\n" ::"r"(tmem_d),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate), "r"(z), "r"(z), "r"(z), "r"(z)
      : "memory");
}

__device__ __forceinline__ void mma_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar)
               : "memory");
}

__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void proxy_fence() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

__device__ __forceinline__ void tmem_ld8(uint32_t taddr, float v[8]) {
  uint32_t r[8];
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 8; i++) v[i] = __uint_as_float(r[i]);
}

__device__ __forceinline__ float silu(float z) { return z / (1.f + __expf(-z)); }

}  // namespace

namespace {

struct GemmArgs {
  const __nv_bfloat16* A;   // [M, K] row-major (K contiguous), lda elements per row
  const __nv_bfloat16* B;   // [N, K] row-major, ldb
  int lda, ldb, M, N, K;
  int nt;                   // columns of a CTA tile: multiple of 16, <= 256
  int ksplit;               // K elements per split (a multiple of GKT)
  const float* bias;        // [N] or null
  int act;                  // 0: none, 1: SiLU on the bf16 output
  float* zf;                // FP32 output (pre-activation) or null
  int ldz;
  int atomic;               // 1: zf += (split-K partial sums)
  __nv_bfloat16* yb;        // BF16 output (after the activation) or null
  int ldy;
};

// Shared memory of one stage: A tile [128 x 64] then B tile [nt x 64], each in
// core-matrix order: element (r, k) at (r/8)*1024 + (k/8)*128 + (r%8)*16 + (k%8)*2.
constexpr uint32_t kLBO = 128, kSBO = (GKT / 8) * 128;

__device__ __forceinline__ uint32_t core_off(int r, int c8) { return (r >> 3) * kSBO + c8 * kLBO + (r & 7) * 16; }

__global__ void __launch_bounds__(GTHREADS) k_gemm_bf16(GemmArgs g) {
  extern __shared__ __align__(1024) unsigned char smem[];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int m0 = blockIdx.x * GM, n0 = blockIdx.y * g.nt;
  const int kb = blockIdx.z * g.ksplit, ke = min(g.K, kb + g.ksplit);
  const uint32_t abytes = GM * GKT * 2, bbytes = g.nt * GKT * 2, sbytes = abytes + bbytes;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + 2 * sbytes);
  uint32_t* tslot = reinterpret_cast<uint32_t*>(bars + 2);
  const uint32_t sbase = smem_u32(smem), bar0 = smem_u32(bars), bar1 = bar0 + 8;
  uint32_t ncol = 32;
  while ((int)ncol < g.nt) ncol <<= 1;
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tslot)), "r"(ncol)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (tid == 0) {
    mbar_init(bar0, 1);
    mbar_init(bar1, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tslot;
  const uint32_t idesc = instr_desc(GM, g.nt);
  const int nk = ke > kb ? (ke - kb + GKT - 1) / GKT : 0;
  bool ok = true;
  for (int it = 0; it < nk && ok; it++) {
    const int b = it & 1;
    if (it >= 2) {   // the MMAs that read this stage two iterations ago are done
      bool w = mbar_wait(b ? bar1 : bar0, ((it >> 1) - 1) & 1);
      if (__syncthreads_or(!w)) { ok = false; break; }
    }
    const int k0 = kb + it * GKT, klen = min(GKT, ke - k0);
    const int nc8 = klen >> 3;
    unsigned char* sa = smem + b * sbytes;
    unsigned char* sb = sa + abytes;
    // A tile: 128 rows x nc8 chunks of 8 elements (16 bytes), zero past M
    for (int q = tid; q < GM * nc8; q += GTHREADS) {
      const int r = q / nc8, c8 = q % nc8;
      uint4 v = make_uint4(0, 0, 0, 0);
      if (m0 + r < g.M) v = *reinterpret_cast<const uint4*>(g.A + (size_t)(m0 + r) * g.lda + k0 + c8 * 8);
      *reinterpret_cast<uint4*>(sa + core_off(r, c8)) = v;
    }
    for (int q = tid; q < g.nt * nc8; q += GTHREADS) {
      const int r = q / nc8, c8 = q % nc8;
      uint4 v = make_uint4(0, 0, 0, 0);
      if (n0 + r < g.N) v = *reinterpret_cast<const uint4*>(g.B + (size_t)(n0 + r) * g.ldb + k0 + c8 * 8);
      *reinterpret_cast<uint4*>(sb + core_off(r, c8)) = v;
    }
    proxy_fence();   // generic-proxy stores -> visible to the tensor core's reads
    __syncthreads();
    if (tid == 0) {
      tc_fence_after();
      const uint32_t a_addr = sbase + b * sbytes, b_addr = a_addr + abytes;
      for (int s = 0; s < (klen >> 4); s++) {
        const uint64_t ad = smem_desc(a_addr + s * 2 * kLBO, kLBO, kSBO);
        const uint64_t bd = smem_desc(b_addr + s * 2 * kLBO, kLBO, kSBO);
        mma_bf16(tmem, ad, bd, idesc, (it > 0 || s > 0) ? 1u : 0u);
      }
      mma_commit(b ? bar1 : bar0);
    }
  }
  // the last commit tracks every MMA issued before it
  bool done = nk == 0;
  if (nk > 0) {
    const int last = nk - 1;
    done = mbar_wait((last & 1) ? bar1 : bar0, (last >> 1) & 1);
  }
  if (__syncthreads_or(!done || !ok)) {
    if (tid == 0) atomicCAS(&g_err, 0, 1);
    ok = false;
  }
  tc_fence_after();
  if (ok && nk > 0) {
    const int row = m0 + warp * 32 + lane;
    for (int c = 0; c < g.nt / 8; c++) {
      float v[8];
      tmem_ld8(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)(c * 8), v);
      if (row >= g.M) continue;
#pragma unroll
      for (int j = 0; j < 8; j++) {
        const int col = n0 + c * 8 + j;
        if (col >= g.N) break;
        float z = v[j] + (g.bias ? g.bias[col] : 0.f);
        if (g.zf) {
          if (g.atomic) atomicAdd(g.zf + (size_t)row * g.ldz + col, z);
          else g.zf[(size_t)row * g.ldz + col] = z;
        }
        if (g.yb) g.yb[(size_t)row * g.ldy + col] = __float2bfloat16_rn(g.act == 1 ? silu(z) : z);
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(ncol) : "memory");
}


// ---- many rows against one small matrix --------------------------------------
// Z[M,N] = A[M,K] B[N,K]^T for the decoder's layers and their input gradients:
// M up to a million rows, N and K at most 256.  These are bound by memory (K =
// 32: 6 flop a byte), so what counts is that every byte moves once and in
// whole lines.  A CTA keeps B in shared memory and walks over its 128-row
// tiles; the accumulator goes from tensor memory through a per-warp
// transpose in shared memory to the outputs, 128 contiguous bytes a row
// (k_gemm_bf16 stores eight columns a lane, one row a lane, and sets up
// tensor memory and barriers for every tile).  1,048,576 x 32 x 32 with both
// outputs, B200: 459 -> 63 us.
// Four (N <= 64), three or two CTAs an SM overlap one another's loads, MMAs
// and stores.
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, float v[32]) {
  uint32_t r[32];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];\n"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
        "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
        "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 32; i++) v[i] = __uint_as_float(r[i]);
}

constexpr int TPAD = 36;   // floats a row of the per-warp transpose (32 + 4: 16-byte rows, few bank conflicts)

// Shared memory of k_gemm_rows: B in core-matrix order, one A tile, the four warps' transposes, barrier and TMEM slot.
inline size_t gemm_rows_smem(int n, int k) {
  const int nt = (n + 15) / 16 * 16;
  return (size_t)nt * k * 2 + (size_t)GM * k * 2 + 4 * 32 * TPAD * 4 + 64;
}

__global__ void __launch_bounds__(GTHREADS) k_gemm_rows(GemmArgs g) {
  extern __shared__ __align__(1024) unsigned char smem[];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t kb8 = g.K >> 3, sbo = kb8 * 128;   // 8-row groups lie K/8 core matrices apart
  unsigned char* sb = smem;
  unsigned char* sa = sb + (size_t)g.nt * g.K * 2;
  float* st = reinterpret_cast<float*>(sa + (size_t)GM * g.K * 2) + warp * 32 * TPAD;
  uint64_t* bar = reinterpret_cast<uint64_t*>(sa + (size_t)GM * g.K * 2 + 4 * 32 * TPAD * 4);
  uint32_t* tslot = reinterpret_cast<uint32_t*>(bar + 1);
  const uint32_t a_addr = smem_u32(sa), b_addr = smem_u32(sb), bar0 = smem_u32(bar);
  uint32_t ncol = 32;
  while ((int)ncol < g.nt) ncol <<= 1;
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tslot)), "r"(ncol)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (tid == 0) {
    mbar_init(bar0, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  for (int q = tid; q < g.nt * (int)kb8; q += GTHREADS) {
    const int r = q / kb8, c8 = q % kb8;
    uint4 v = make_uint4(0, 0, 0, 0);
    if (r < g.N) v = *reinterpret_cast<const uint4*>(g.B + (size_t)r * g.ldb + c8 * 8);
    *reinterpret_cast<uint4*>(sb + (r >> 3) * sbo + c8 * 128 + (r & 7) * 16) = v;
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tslot, idesc = instr_desc(GM, g.nt);
  const int tiles = (g.M + GM - 1) / GM;
  bool ok = true;
  uint32_t par = 0;
  for (int t = blockIdx.x; t < tiles; t += gridDim.x, par ^= 1) {
    const int m0 = t * GM;
    for (int q = tid; q < GM * (int)kb8; q += GTHREADS) {
      const int r = q / kb8, c8 = q % kb8;
      uint4 v = make_uint4(0, 0, 0, 0);
      if (m0 + r < g.M) v = __ldg(reinterpret_cast<const uint4*>(g.A + (size_t)(m0 + r) * g.lda + c8 * 8));
      *reinterpret_cast<uint4*>(sa + (r >> 3) * sbo + c8 * 128 + (r & 7) * 16) = v;
    }
    proxy_fence();   // generic-proxy stores -> visible to the tensor core's reads
    tc_fence_before();   // the previous tile's tensor-memory reads are done
    __syncthreads();
    if (tid == 0) {
      tc_fence_after();
      for (int s = 0; s < (g.K >> 4); s++)
        mma_bf16(tmem, smem_desc(a_addr + s * 256, 128, sbo), smem_desc(b_addr + s * 256, 128, sbo), idesc, s > 0 ? 1u : 0u);
      mma_commit(bar0);
    }
    const bool w = mbar_wait(bar0, par);
    if (__syncthreads_or(!w)) { ok = false; break; }
    tc_fence_after();
    const int r0 = m0 + warp * 32;
    for (int c0 = 0; c0 < g.nt; c0 += 32) {
      // 32 rows x 32 columns of this warp: row a lane -> transpose -> 8 lanes a row
      const int nc = min(32, g.nt - c0);
      float v[32];
      if (nc == 32) {
        tmem_ld32(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)c0, v);
      } else {
        for (int h = 0; h < 2; h++) tmem_ld8(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)(c0 + 8 * h), v + 8 * h);
      }
      __syncwarp();
#pragma unroll
      for (int q = 0; q < 8; q++)
        if (4 * q < nc)
          *reinterpret_cast<float4*>(st + lane * TPAD + 4 * q) = make_float4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
      __syncwarp();
      const int c = (lane & 7) * 4, col = c0 + c;
      if (c < nc && col < g.N) {
        float bs[4] = {0.f, 0.f, 0.f, 0.f};
        if (g.bias)
#pragma unroll
          for (int q = 0; q < 4; q++) bs[q] = __ldg(g.bias + col + q);
#pragma unroll
        for (int rr = 0; rr < 32; rr += 4) {
          const int r = rr + (lane >> 3), row = r0 + r;
          if (row >= g.M) continue;
          float4 z = *reinterpret_cast<const float4*>(st + r * TPAD + c);
          z.x += bs[0]; z.y += bs[1]; z.z += bs[2]; z.w += bs[3];
          if (g.zf) *reinterpret_cast<float4*>(g.zf + (size_t)row * g.ldz + col) = z;
          if (g.yb) {
            if (g.act == 1) { z.x = silu(z.x); z.y = silu(z.y); z.z = silu(z.z); z.w = silu(z.w); }
            __nv_bfloat162 y0 = __floats2bfloat162_rn(z.x, z.y), y1 = __floats2bfloat162_rn(z.z, z.w);
            uint2 y;
            y.x = *reinterpret_cast<uint32_t*>(&y0);
            y.y = *reinterpret_cast<uint32_t*>(&y1);
            *reinterpret_cast<uint2*>(g.yb + (size_t)row * g.ldy + col) = y;
          }
        }
      }
    }
  }
  if (!ok && tid == 0) atomicCAS(&g_err, 0, 1);
  tc_fence_before();
  __syncthreads();
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(ncol) : "memory");
}

// ---- weight gradients ----------------------------------------------------------
// G[N,K] += X[R,N]^T Y[R,K], the sum running over the R rows (all voxels of the
// batch): both operands are read once, row by row as they lie, and turned in
// registers, 8 rows x 8 columns a thread, into the K-major core matrices the
// tensor core reads -- no transposed copies (two launches and 4 bytes of
// traffic an element before the GEMM even began).  blockIdx.y takes 128 of the
// N columns; each CTA a share of the rows, added with FP32 atomics.
// 1,048,576 rows, N = K = 32: 375 us (two transposes, a split GEMM) -> 90 us.
struct WgradArgs {
  const __nv_bfloat16 *X, *Y;
  int ldx, ldy, rows, N, K, per, kst, nst;   // per: rows of a CTA, a multiple of kst; kst: rows of a stage; nst: stages
  float* G;
  int ldg;
};

// A stage of 64 rows, two of them; where its blocks would leave half of the
// threads idle, one of 128 rows (loads overlap the waits all the same, since
// a thread holds its next block in registers).
inline void wgrad_stage(WgradArgs& g) {
  const bool small = GKT / 8 * (min(g.N, GM) + g.K) / 8 <= GTHREADS / 2;
  g.kst = small ? 2 * GKT : GKT;
  g.nst = small ? 1 : 2;
}
// bytes between column groups of 8: 16 more than the core matrices take, so that the 16-byte stores of neighbouring
// lanes (one offset of their core matrices) fall on different banks; 64 more between the operands
__host__ __device__ __forceinline__ uint32_t wgrad_sbo(int kst) { return kst / 8 * kLBO + 16; }
__host__ __device__ __forceinline__ uint32_t wgrad_stage_bytes(int kst, int kt) {
  return (GM + kt) / 8 * wgrad_sbo(kst) + 64;
}

// 8 rows x 8 columns of a row-major operand in registers (rows past nrow zero) ...
struct Block8 {
  uint32_t w[8][4];
};
__device__ __forceinline__ void block_load(Block8& t, const __nv_bfloat16* src, size_t ld, int nrow) {
#pragma unroll
  for (int r = 0; r < 8; r++) {
    uint4 v = make_uint4(0, 0, 0, 0);
    if (r < nrow) v = __ldg(reinterpret_cast<const uint4*>(src + r * ld));
    t.w[r][0] = v.x; t.w[r][1] = v.y; t.w[r][2] = v.z; t.w[r][3] = v.w;
  }
}
// ... and transposed into the core matrix at dst, 16 bytes a column
__device__ __forceinline__ void block_store(const Block8& t, unsigned char* dst) {
#pragma unroll
  for (int c = 0; c < 8; c++) {
    const uint32_t sel = (c & 1) ? 0x7632u : 0x5410u;
    uint4 o;
    o.x = __byte_perm(t.w[0][c >> 1], t.w[1][c >> 1], sel);
    o.y = __byte_perm(t.w[2][c >> 1], t.w[3][c >> 1], sel);
    o.z = __byte_perm(t.w[4][c >> 1], t.w[5][c >> 1], sel);
    o.w = __byte_perm(t.w[6][c >> 1], t.w[7][c >> 1], sel);
    *reinterpret_cast<uint4*>(dst + c * 16) = o;
  }
}

__global__ void __launch_bounds__(GTHREADS) k_wgrad(WgradArgs g) {
  extern __shared__ __align__(1024) unsigned char smem[];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int n0 = blockIdx.y * GM, nn = min(GM, g.N - n0), kt = (g.K + 15) / 16 * 16;
  const uint32_t sbo = wgrad_sbo(g.kst), abytes = GM / 8 * sbo + 64, sbytes = wgrad_stage_bytes(g.kst, kt);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + g.nst * sbytes);
  uint32_t* tslot = reinterpret_cast<uint32_t*>(bars + 2);
  const uint32_t sbase = smem_u32(smem), bar0 = smem_u32(bars);
  uint32_t ncol = 32;
  while ((int)ncol < kt) ncol <<= 1;
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tslot)), "r"(ncol)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (tid == 0) {
    mbar_init(bar0, 1);
    mbar_init(bar0 + 8, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  for (uint32_t q = tid * 16; q < g.nst * sbytes; q += GTHREADS * 16)   // rows past N and K stay zero
    *reinterpret_cast<uint4*>(smem + q) = make_uint4(0, 0, 0, 0);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tslot, idesc = instr_desc(GM, kt);
  const int rb = blockIdx.x * g.per, re = min(g.rows, rb + g.per);
  const int nk = re > rb ? (re - rb + g.kst - 1) / g.kst : 0, na = nn >> 3, ncg = na + (g.K >> 3);
  // a stage is kst / 8 row groups x ncg column groups of 8 x 8 blocks, dealt out thread by thread; lanes run along
  // the columns, so a row is read in whole lines.  A thread loads its next block (of the next stage after its last
  // of this one) before it waits for anything.
  const int nblk = g.kst / 8 * ncg;
  Block8 cur, nxt;
  auto load = [&](Block8& t, int it, int q) {
    const int rg = q / ncg, cg = q - rg * ncg, r = rb + it * g.kst + rg * 8, nr = max(0, min(8, re - r));
    if (cg < na) block_load(t, g.X + (size_t)r * g.ldx + n0 + cg * 8, g.ldx, nr);
    else block_load(t, g.Y + (size_t)r * g.ldy + (cg - na) * 8, g.ldy, nr);
  };
  if (nk > 0 && tid < nblk) load(cur, 0, tid);
  bool ok = true;
  for (int it = 0; it < nk && ok; it++) {
    const int b = it % g.nst;
    if (it >= g.nst) {   // the MMAs that read this stage last are done
      const bool w = mbar_wait(bar0 + 8 * b, (it / g.nst - 1) & 1);
      if (__syncthreads_or(!w)) { ok = false; break; }
    }
    unsigned char *sa = smem + b * sbytes, *sb = sa + abytes;
    for (int q = tid; q < nblk; q += GTHREADS) {
      if (q + GTHREADS < nblk) load(nxt, it, q + GTHREADS);
      else if (it + 1 < nk) load(nxt, it + 1, tid);
      const int rg = q / ncg, cg = q - rg * ncg;
      block_store(cur, (cg < na ? sa + cg * sbo : sb + (cg - na) * sbo) + rg * kLBO);
      cur = nxt;
    }
    proxy_fence();
    __syncthreads();
    if (tid == 0) {
      tc_fence_after();
      const uint32_t aa = sbase + b * sbytes, ba = aa + abytes;
      for (int s = 0; s < g.kst / 16; s++)
        mma_bf16(tmem, smem_desc(aa + s * 2 * kLBO, kLBO, sbo), smem_desc(ba + s * 2 * kLBO, kLBO, sbo), idesc,
                 (it > 0 || s > 0) ? 1u : 0u);
      mma_commit(bar0 + 8 * b);
    }
  }
  bool done = true;   // the last commit tracks every MMA before it
  if (nk > 0) done = mbar_wait(bar0 + 8 * ((nk - 1) % g.nst), ((nk - 1) / g.nst) & 1);
  if (__syncthreads_or(!done || !ok)) {
    if (tid == 0) atomicCAS(&g_err, 0, 1);
    ok = false;
  }
  tc_fence_after();
  if (ok && nk > 0) {
    const int row = warp * 32 + lane;
    for (int c = 0; c < kt / 8; c++) {
      float v[8];
      tmem_ld8(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)(c * 8), v);
      if (row < nn)
#pragma unroll
        for (int j = 0; j < 8; j++)
          if (c * 8 + j < g.K) atomicAdd(g.G + (size_t)(n0 + row) * g.ldg + c * 8 + j, v[j]);
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(ncol) : "memory");
}

}  // namespace

namespace {

// dz = dy * silu'(z), written as BF16 (the next GEMM's operand) and FP32.
__global__ void k_silu_bwd(const float* __restrict__ dy, const float* __restrict__ z, long n, __nv_bfloat16* dzb,
                           float* dzf) {
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) {
    const float zi = z[i], s = 1.f / (1.f + __expf(-zi));
    const float d = dy[i] * s * (1.f + zi * (1.f - s));
    if (dzb) dzb[i] = __float2bfloat16_rn(d);
    if (dzf) dzf[i] = d;
  }
}

// Column sums of what a thread block has in registers: thread tid holds columns
// 4 (tid % c4) .. + 3 of every (blockDim / c4)-th row; one atomic a column.
__device__ __forceinline__ void add_columns(const float s[4], int c4, float* out) {
  __shared__ float red[256 * 4];
#pragma unroll
  for (int q = 0; q < 4; q++) red[threadIdx.x * 4 + q] = s[q];
  __syncthreads();
  for (int c = threadIdx.x; c < 4 * c4; c += blockDim.x) {
    float t = 0.f;
    for (int r = c >> 2; r < (int)blockDim.x; r += c4) t += red[r * 4 + (c & 3)];
    atomicAdd(out + c, t);
  }
}

__device__ __forceinline__ void put_bf16x4(__nv_bfloat16* p, const float d[4]) {
  __nv_bfloat162 a = __floats2bfloat162_rn(d[0], d[1]), b = __floats2bfloat162_rn(d[2], d[3]);
  uint2 y;
  y.x = *reinterpret_cast<uint32_t*>(&a);
  y.y = *reinterpret_cast<uint32_t*>(&b);
  *reinterpret_cast<uint2*>(p) = y;
}

// k_silu_bwd on [rows, cols] with the bias gradient in the same pass: out[c]
// += the column sums of dz (c4 = cols / 4, at most 64, a divisor of 256).
// The separate column-sum kernel re-read the 4 bytes an element that
// k_silu_bwd had just written for it, with 32 of its 128 threads at work
// where a layer has 32 columns (0.46 ms for 1,048,576 rows).
__global__ void __launch_bounds__(256) k_silu_bwd_bias(const float* __restrict__ dy, const float* __restrict__ z, int rows,
                                                       int c4, __nv_bfloat16* dzb, float* dzf, float* out) {
  const int c = threadIdx.x % c4, rstep = 256 / c4;
  float s[4] = {0.f, 0.f, 0.f, 0.f};
  for (long r = (long)blockIdx.x * rstep + threadIdx.x / c4; r < rows; r += (long)gridDim.x * rstep) {
    const size_t o = ((size_t)r * c4 + c) * 4;
    const float4 a = *reinterpret_cast<const float4*>(dy + o), b = *reinterpret_cast<const float4*>(z + o);
    const float dv[4] = {a.x, a.y, a.z, a.w}, zv[4] = {b.x, b.y, b.z, b.w};
    float d[4];
#pragma unroll
    for (int q = 0; q < 4; q++) {
      const float sg = 1.f / (1.f + __expf(-zv[q]));
      d[q] = dv[q] * sg * (1.f + zv[q] * (1.f - sg));
      s[q] += d[q];
    }
    put_bf16x4(dzb + o, d);
    if (dzf) *reinterpret_cast<float4*>(dzf + o) = make_float4(d[0], d[1], d[2], d[3]);
  }
  add_columns(s, c4, out);
}

// out[c] += sum over rows of x[r * ld + c] (bias gradients).
__global__ void k_colsum(const float* __restrict__ x, int rows, int cols, int ld, float* out) {
  const int c = blockIdx.y * blockDim.x + threadIdx.x;
  if (c >= cols) return;
  float s = 0.f;
  for (int r = blockIdx.x; r < rows; r += gridDim.x) s += x[(size_t)r * ld + c];
  atomicAdd(out + c, s);
}

// out[c * ldo + r] = in[r * ldi + c] for r < rows, c < cols; rows padded
// with zeros up to rows_pad (so that the transposed operand's K is a
// multiple of the GEMM's K step).
__global__ void k_transpose_bf16(const __nv_bfloat16* __restrict__ in, int rows, int cols, int ldi,
                                 __nv_bfloat16* out, int ldo, int rows_pad) {
  __shared__ __nv_bfloat16 t[32][33];
  const int r0 = blockIdx.x * 32, c0 = blockIdx.y * 32;
  for (int y = threadIdx.y; y < 32; y += blockDim.y) {
    const int r = r0 + y, c = c0 + threadIdx.x;
    t[y][threadIdx.x] = (r < rows && c < cols) ? in[(size_t)r * ldi + c] : __float2bfloat16_rn(0.f);
  }
  __syncthreads();
  for (int y = threadIdx.y; y < 32; y += blockDim.y) {
    const int c = c0 + y, r = r0 + threadIdx.x;
    if (c < cols && r < rows_pad) out[(size_t)c * ldo + r] = t[threadIdx.x][y];
  }
}

__global__ void k_f32_to_bf16(const float* __restrict__ in, long n, __nv_bfloat16* out) {
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x)
    out[i] = __float2bfloat16_rn(in[i]);
}

// Mean-squared error of pred [rows, ld] (first cols columns) against
// target [rows, cols]: loss += sum((p - t)^2) / count, grad = 2 (p - t) / count
// as BF16 [rows, ld] with zero padding columns (and as FP32 when gradf is set).
__global__ void k_mse(const float* __restrict__ pred, int ld, const float* __restrict__ tgt, int rows, int cols,
                      float inv_count, __nv_bfloat16* grad, float* gradf, float* loss) {
  float s = 0.f;
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < (long)rows * ld; i += (long)gridDim.x * blockDim.x) {
    const long r = i / ld;
    const int c = (int)(i % ld);
    float g = 0.f;
    if (c < cols) {
      const float d = pred[i] - tgt[r * cols + c];
      s += d * d;
      g = 2.f * d * inv_count;
    }
    grad[i] = __float2bfloat16_rn(g);
    if (gradf) gradf[i] = g;
  }
  for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0) atomicAdd(loss, s * inv_count);
}

// k_mse with the column sums of the gradient (the output layer's bias
// gradient) in the same pass; c4 = ld / 4 as in k_silu_bwd_bias.
__global__ void __launch_bounds__(256) k_mse_bias(const float* __restrict__ pred, int c4, const float* __restrict__ tgt,
                                                  int rows, int cols, float inv_count, __nv_bfloat16* grad, float* gradf,
                                                  float* loss, float* out) {
  const int c = threadIdx.x % c4, rstep = 256 / c4;
  float s[4] = {0.f, 0.f, 0.f, 0.f}, l = 0.f;
  for (long r = (long)blockIdx.x * rstep + threadIdx.x / c4; r < rows; r += (long)gridDim.x * rstep) {
    const size_t o = ((size_t)r * c4 + c) * 4;
    const float4 a = *reinterpret_cast<const float4*>(pred + o);
    const float pv[4] = {a.x, a.y, a.z, a.w};
    float g[4];
#pragma unroll
    for (int q = 0; q < 4; q++) {
      g[q] = 0.f;
      if (4 * c + q < cols) {
        const float d = pv[q] - __ldg(tgt + r * cols + 4 * c + q);
        l += d * d;
        g[q] = 2.f * d * inv_count;
        s[q] += g[q];
      }
    }
    put_bf16x4(grad + o, g);
    if (gradf) *reinterpret_cast<float4*>(gradf + o) = make_float4(g[0], g[1], g[2], g[3]);
  }
  add_columns(s, c4, out);
  for (int o = 16; o > 0; o >>= 1) l += __shfl_down_sync(0xffffffffu, l, o);
  if ((threadIdx.x & 31) == 0) atomicAdd(loss, l * inv_count);
}

// Adam on FP32 master weights w [n]; w16 gets the BF16 copy and, when
// rows > 0, w16t the BF16 transpose of w viewed as [rows, n / rows].
__global__ void k_adam(float* w, const float* __restrict__ g, float* m, float* v, long n, float lr, float b1,
                       float b2, float eps, float c1, float c2, float wd, __nv_bfloat16* w16, __nv_bfloat16* w16t,
                       int rows) {
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) {
    const float gi = g[i] + wd * w[i];
    const float mi = b1 * m[i] + (1.f - b1) * gi, vi = b2 * v[i] + (1.f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    const float wi = w[i] - lr * (mi * c1) / (sqrtf(vi * c2) + eps);
    w[i] = wi;
    if (w16) w16[i] = __float2bfloat16_rn(wi);
    if (w16t && rows > 0) {
      const long cols = n / rows, r = i / cols, c = i % cols;
      w16t[c * rows + r] = __float2bfloat16_rn(wi);
    }
  }
}

int g_smem_set[64], g_rows_set[64], g_wgrad_set[64];   // the kernels' shared memory is granted, per device

// What a GEMM kernel with tiles of nt columns is launched with: its
// tensor-memory columns, and its shared memory, at least `need` and so much
// that the CTAs resident on one SM never ask for more than its 512 columns.
struct GemmPlan {
  int nt, ncol;
  size_t smem;
};
GemmPlan gemm_plan(int nt, size_t need) {
  int ncol = 32;
  while (ncol < nt) ncol <<= 1;
  const size_t least = ncol >= 256 ? 80 * 1024 : (ncol >= 128 ? 48 * 1024 : (ncol >= 64 ? 28 * 1024 : 0));
  return {nt, ncol, need < least ? least : need};
}

inline int blocks_for(long n, int t) { return (int)min((n + t - 1) / t, (long)148 * 16); }

}  // namespace

extern "C" {

int ffnn_gemm(const void* A, int lda, const void* B, int ldb, int M, int N, int K, const float* bias, int act,
              float* zf, int ldz, int atomic, void* yb, int ldy, int ksplit, void* stream) {
  if (!A || !B || M < 1 || N < 1 || K < 16 || (K % 16) || (lda % 8) || (ldb % 8) || lda < K || ldb < K)
    return FFNN_ERR_ARG;
  if (((uintptr_t)A & 15) || ((uintptr_t)B & 15) || (!zf && !yb) || (atomic && !zf)) return FFNN_ERR_ARG;
  if (ksplit <= 0 || ksplit >= K) ksplit = K;
  else ksplit = (ksplit + GKT - 1) / GKT * GKT;
  if (ksplit < K && !atomic) return FFNN_ERR_ARG;   // partial sums need the atomic epilogue
  // many rows, a matrix that fits beside one A tile, whole 16-byte rows of the outputs: k_gemm_rows.  Below a
  // wave of tiles the per-tile kernel's extra CTAs count for more (measured equal at 4,096 rows).
  const bool rows_ok = M >= 4096 && N <= 256 && N % 4 == 0 && K <= 256 && !atomic && ksplit == K &&
                       (!zf || (ldz % 4 == 0 && ((uintptr_t)zf & 15) == 0)) &&
                       (!yb || (ldy % 4 == 0 && ((uintptr_t)yb & 7) == 0));
  GemmArgs g;
  g.A = (const __nv_bfloat16*)A; g.B = (const __nv_bfloat16*)B;
  g.lda = lda; g.ldb = ldb; g.M = M; g.N = N; g.K = K;
  g.ksplit = ksplit;
  g.bias = bias; g.act = act; g.zf = zf; g.ldz = ldz; g.atomic = atomic;
  g.yb = (__nv_bfloat16*)yb; g.ldy = ldy;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return FFNN_ERR_CUDA;
  const int wide = N <= 256 ? (N + 15) / 16 * 16 : 256;
  if (rows_ok) {
    const GemmPlan p = gemm_plan(wide, gemm_rows_smem(N, K));
    if (p.smem <= 200 * 1024) {   // 210 KB at N, K = 256: the kernel below
      if (!g_rows_set[dev]) {
        if (cudaFuncSetAttribute(k_gemm_rows, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024) != cudaSuccess)
          return FFNN_ERR_CUDA;
        g_rows_set[dev] = 1;
      }
      g.nt = p.nt;
      const int per_sm = min(p.ncol >= 256 ? 2 : (p.ncol >= 128 ? 4 : 8), max(1, (int)(220 * 1024 / p.smem)));
      k_gemm_rows<<<min((M + GM - 1) / GM, 148 * per_sm), GTHREADS, p.smem, (cudaStream_t)stream>>>(g);
      return cudaGetLastError() == cudaSuccess ? 0 : FFNN_ERR_CUDA;
    }
  }
  // columns of a CTA tile: as many as fit, but 32 where the tiles would leave SMs idle (a few rows: the K loop's
  // loads are the whole time, 16 x 256 x 512 took 106 us in one CTA)
  const bool few = (long)((M + GM - 1) / GM) * ((N + wide - 1) / wide) < 74;
  const int nt = few ? min(wide, 32) : wide;
  const GemmPlan p = gemm_plan(nt, 2 * (size_t)(GM + nt) * GKT * 2 + 64);
  if (!g_smem_set[dev]) {
    if (cudaFuncSetAttribute(k_gemm_bf16, cudaFuncAttributeMaxDynamicSharedMemorySize, 100 * 1024) != cudaSuccess)
      return FFNN_ERR_CUDA;
    g_smem_set[dev] = 1;
  }
  g.nt = p.nt;
  dim3 grid((M + GM - 1) / GM, (N + g.nt - 1) / g.nt, (K + ksplit - 1) / ksplit);
  k_gemm_bf16<<<grid, GTHREADS, p.smem, (cudaStream_t)stream>>>(g);
  return cudaGetLastError() == cudaSuccess ? 0 : FFNN_ERR_CUDA;
}

int ffnn_wgrad(const void* X, int ldx, const void* Y, int ldy, int rows, int N, int K, float* G, int ldg, void* stream) {
  if (!X || !Y || !G || rows < 1 || N < 8 || K < 8 || (N % 8) || (K % 8) || K > 256 || (ldx % 8) || (ldy % 8) || ldx < N ||
      ldy < K || ldg < K || ((uintptr_t)X & 15) || ((uintptr_t)Y & 15))
    return FFNN_ERR_ARG;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return FFNN_ERR_CUDA;
  const int kt = (K + 15) / 16 * 16, mt = (N + GM - 1) / GM;
  WgradArgs g;
  g.X = (const __nv_bfloat16*)X; g.Y = (const __nv_bfloat16*)Y;
  g.ldx = ldx; g.ldy = ldy; g.rows = rows; g.N = N; g.K = K; g.G = G; g.ldg = ldg;
  wgrad_stage(g);
  const size_t sm = gemm_plan(kt, g.nst * (size_t)wgrad_stage_bytes(g.kst, kt) + 64).smem;
  if (!g_wgrad_set[dev]) {
    if (cudaFuncSetAttribute(k_wgrad, cudaFuncAttributeMaxDynamicSharedMemorySize, 120 * 1024) != cudaSuccess)
      return FFNN_ERR_CUDA;
    g_wgrad_set[dev] = 1;
  }
  // five CTAs an SM, at least 4 x 64 rows each (their setup and atomics)
  const int share = (rows + 148 * 5 / mt - 1) / max(1, 148 * 5 / mt);
  g.per = max(4 * GKT, (share + g.kst - 1) / g.kst * g.kst);
  k_wgrad<<<dim3((rows + g.per - 1) / g.per, mt), GTHREADS, sm, (cudaStream_t)stream>>>(g);
  return cudaGetLastError() == cudaSuccess ? 0 : FFNN_ERR_CUDA;
}

static int c4_of(int cols) {   // the fused column sums' column groups, 0 where they don't fit
  const int c4 = cols / 4;
  return cols % 4 == 0 && c4 >= 1 && c4 <= 64 && 256 % c4 == 0 ? c4 : 0;
}

int ffnn_silu_bwd_bias(const float* dy, const float* z, int rows, int cols, void* dzb, float* dzf, float* gbias,
                       void* stream) {
  const int c4 = c4_of(cols);
  if (!dy || !z || !dzb || !gbias || rows < 1 || !c4 || ((uintptr_t)dy & 15) || ((uintptr_t)z & 15) || ((uintptr_t)dzb & 7) ||
      ((uintptr_t)dzf & 15))
    return FFNN_ERR_ARG;
  const long nb = ((long)rows * c4 + 255) / 256;
  k_silu_bwd_bias<<<(int)min(nb, 148L * 8), 256, 0, (cudaStream_t)stream>>>(dy, z, rows, c4, (__nv_bfloat16*)dzb, dzf, gbias);
  return cudaGetLastError() == cudaSuccess ? 0 : FFNN_ERR_CUDA;
}

int ffnn_mse_bias(const float* pred, int ld, const float* tgt, int rows, int cols, void* grad, float* gradf, float* loss,
                  float* gbias, void* stream) {
  const int c4 = c4_of(ld);
  if (!pred || !tgt || !grad || !loss || !gbias || rows < 1 || cols < 1 || ld < cols || !c4 || ((uintptr_t)pred & 15) ||
      ((uintptr_t)grad & 7) || ((uintptr_t)gradf & 15))
    return FFNN_ERR_ARG;
  const long nb = ((long)rows * c4 + 255) / 256;
  k_mse_bias<<<(int)min(nb, 148L * 8), 256, 0, (cudaStream_t)stream>>>(pred, c4, tgt, rows, cols, 1.f / ((float)rows * cols),
                                                                       (__nv_bfloat16*)grad, gradf, loss, gbias);
  return cudaGetLastError() == cudaSuccess ? 0 : FFNN_ERR_CUDA;
}

int ffnn_silu_bwd(const float* dy, const float* z, long n, void* dzb, float* dzf, void* stream) {
  if (n <= 0) return 0;
  k_silu_bwd<<<blocks_for(n, 256), 256, 0, (cudaStream_t)stream>>>(dy, z, n, (__nv_bfloat16*)dzb, dzf);
  return cudaGetLastError() == cudaSuccess ? 0 : FFNN_ERR_CUDA;
}

int ffnn_colsum(const float* x, int rows, int cols, int ld, float* out, void* stream) {
  if (rows <= 0 || cols <= 0) return 0;
  dim3 grid(min(rows, 1024), (cols + 127) / 128);
  k_colsum<<<grid, 128, 0, (cudaStream_t)stream>>>(x, rows, cols, ld, out);
  return cudaGetLastError() == cudaSuccess ? 0 : FFNN_ERR_CUDA;
}

int ffnn_transpose(const void* in, int rows, int cols, int ldi, void* out, int ldo, int rows_pad, void* stream) {
  if (rows_pad < rows || ldo < rows_pad) return FFNN_ERR_ARG;
  dim3 grid((rows_pad + 31) / 32, (cols + 31) / 32);
  k_transpose_bf16<<<grid, dim3(32, 8), 0, (cudaStream_t)stream>>>((const __nv_bfloat16*)in, rows, cols, ldi,
                                                                  (__nv_bfloat16*)out, ldo, rows_pad);
  return cudaGetLastError() == cudaSuccess ? 0 : FFNN_ERR_CUDA;
}

int ffnn_to_bf16(const float* in, long n, void* out, void* stream) {
  if (n <= 0) return 0;
  k_f32_to_bf16<<<blocks_for(n, 256), 256, 0, (cudaStream_t)stream>>>(in, n, (__nv_bfloat16*)out);
  return cudaGetLastError() == cudaSuccess ? 0 : FFNN_ERR_CUDA;
}

int ffnn_mse(const float* pred, int ld, const float* tgt, int rows, int cols, void* grad, float* gradf, float* loss,
             void* stream) {
  if (rows <= 0 || cols <= 0 || ld < cols) return FFNN_ERR_ARG;
  long n = (long)rows * ld;
  k_mse<<<blocks_for(n, 256), 256, 0, (cudaStream_t)stream>>>(pred, ld, tgt, rows, cols, 1.f / ((float)rows * cols),
                                                              (__nv_bfloat16*)grad, gradf, loss);
  return cudaGetLastError() == cudaSuccess ? 0 : FFNN_ERR_CUDA;
}

int ffnn_adam(float* w, const float* g, float* m, float* v, long n, float lr, float b1, float b2, float eps,
              int step, float wd, void* w16, void* w16t, int rows, void* stream) {
  if (n <= 0 || step < 1) return FFNN_ERR_ARG;
  const float c1 = 1.f / (1.f - powf(b1, (float)step)), c2 = 1.f / (1.f - powf(b2, (float)step));
  k_adam<<<blocks_for(n, 256), 256, 0, (cudaStream_t)stream>>>(w, g, m, v, n, lr, b1, b2, eps, c1, c2, wd,
                                                               (__nv_bfloat16*)w16, (__nv_bfloat16*)w16t, rows);
  return cudaGetLastError() == cudaSuccess ? 0 : FFNN_ERR_CUDA;
}

int ffnn_error(int reset) {
  int e = 0;
  if (cudaMemcpyFromSymbol(&e, g_err, sizeof(int)) != cudaSuccess) return FFNN_ERR_CUDA;
  if (reset) {
    int z = 0;
    if (cudaMemcpyToSymbol(g_err, &z, sizeof(int)) != cudaSuccess) return FFNN_ERR_CUDA;
  }
  return e ? FFNN_ERR_TIMEOUT : 0;
}

}  // extern "C"
