// BF16 tensor-core GEMM for the warm-start network, on the 5th-generation
// tensor cores (tcgen05): C[M x N] = alpha * A[M x K] B[K x N] with FP32
// accumulation in tensor memory, plus a fused epilogue (bias, ReLU, a 0/1
// mask from a BF16 array, FP32 and/or BF16 output).
//
// One CTA (128 threads) computes a 128 x BN tile, BN = 128 or 256 (the wide
// tile reads each A chunk once for twice the output and is chosen when the
// grid of wide tiles still fills every SM).  The K dimension runs in chunks
// of 64 through S shared-memory stages, refilled LAG chunks after the MMAs
// that read them were issued (BN = 128: S = 3, LAG = 1, two CTAs per SM;
// BN = 256: S = 4, LAG = 2, one CTA per SM, so that chunk c's MMAs are
// issued while chunk c - 1's still run): at chunk c the threads fetch chunk
// c + S - LAG into the stage chunk c - LAG used (16-byte cp.async copies from
// global memory when the operand is K-contiguous, element loads otherwise).
// Each stage holds A (128 x 64) and B (BN x 64) in the K-major, non-swizzled
// canonical layout of the UMMA
// descriptors -- core matrices of 8 rows x 16 bytes, the two 8-element K
// halves of a 16-wide slab LBO = 128 B apart, consecutive 8-row groups SBO =
// 256 B apart.  One elected thread issues four tcgen05.mma (K = 16 each) per
// chunk into the TMEM accumulator and commits them to the stage's mbarrier;
// a stage is refilled only after its mbarrier reports the MMAs that read it
// complete.  The epilogue reads the accumulator with tcgen05.ld (warp w owns
// TMEM lanes 32w..32w+31 = tile rows).  A and B are read through element
// strides, so either operand may be used transposed.  Waits are bounded: on
// a timeout the kernel records an error, frees its TMEM and returns.
//
// When each operand has a contiguous dimension and 16-byte aligned rows, the
// TMA form at the end of this file (k_gemm_group) replaces the threads' copies
// with tensor-map copies into 128-byte-swizzled stages and splits the CTA into
// producer and MMA warps; the form here runs what is left (other strides).
#pragma once

#include <cuda.h>  // CUtensorMap (the type only; maps are encoded through the runtime's driver entry point)
#include <cuda_bf16.h>

#include <cstdint>

namespace b2p {

constexpr int kGemmBM = 128;
constexpr int kGemmBK = 64;
constexpr int kGemmThreads = 128;
constexpr unsigned kMbarSpinLimit = 1u << 24;

// Tile shape: BN output columns (= TMEM columns), S stages of A 16 KB + B
// BN x 64 x 2 bytes.  BN = 128: three stages (96 KB), at most two CTAs per
// SM (2 x 128 TMEM columns <= 512).  BN = 256: four stages (192 KB), one CTA
// per SM.
template <int BN>
struct GemmTile {
  static constexpr int kStages = BN == 256 ? 4 : 3;
  static constexpr int kLag = BN == 256 ? 2 : 1;  // stage refill lag, in chunks
  static constexpr int kAhead = kStages - kLag;   // chunks in flight ahead of the MMAs
  static constexpr int kStageBytes = (kGemmBM + BN) * kGemmBK * 2;
  static constexpr int kSmemBytes = kStages * kStageBytes;
  static_assert(BN == 128 || BN == 256, "tile width");
  static_assert(kSmemBytes <= 200 * 1024, "stages exceed the shared-memory budget");
};

struct GemmArgs {
  int32_t M, N, K;
  const __nv_bfloat16* A;
  int64_t sam, sak;  // A(m, k) = A[m * sam + k * sak]
  const __nv_bfloat16* B;
  int64_t sbk, sbn;  // B(k, n) = B[k * sbk + n * sbn]
  float alpha;
  const float* bias;  // bias[n] added after alpha, or NULL
  int32_t relu;
  const __nv_bfloat16* mask;  // C(m, n) *= (mask[m * ldm + n] > 0), or NULL
  int64_t ldm;
  float* cf;  // FP32 output C[m * ldcf + n], or NULL
  int64_t ldcf;
  __nv_bfloat16* cb;  // BF16 output, or NULL
  int64_t ldcb;
  int32_t* error;  // set to 1 on an mbarrier timeout (page-locked host memory)
};

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// UMMA shared-memory descriptor, K-major, no swizzle.
__device__ __forceinline__ uint64_t umma_desc(uint32_t addr, uint32_t lbo_bytes, uint32_t sbo_bytes) {
  uint64_t d = 0;
  d |= static_cast<uint64_t>((addr >> 4) & 0x3FFF);
  d |= static_cast<uint64_t>((lbo_bytes >> 4) & 0x3FFF) << 16;
  d |= static_cast<uint64_t>((sbo_bytes >> 4) & 0x3FFF) << 32;
  d |= static_cast<uint64_t>(1) << 46;  // descriptor version (Blackwell)
  // base offset 0, legacy LBO mode, layout type 0 = SWIZZLE_NONE
  return d;
}

// Instruction descriptor: kind::f16, BF16 x BF16 -> F32, both K-major, M = 128,
// N = n (a multiple of 16 up to 256).
__host__ __device__ constexpr uint32_t umma_idesc_bf16(int n) {
  return (1u << 4)                                   // D format F32
         | (1u << 7)                                 // A format BF16
         | (1u << 10)                                // B format BF16
         | (static_cast<uint32_t>(n >> 3) << 17)     // N / 8
         | (static_cast<uint32_t>(kGemmBM >> 4) << 24);  // M / 16
}

// byte offset of element (r, k) of a row-major-in-K chunk of 64 columns
__device__ __forceinline__ uint32_t chunk_offset(int r, int k, int rows) {
  const int s = k >> 4, kk = k & 15;
  return static_cast<uint32_t>(s * (rows / 8) * 256 + (r >> 3) * 256 + (kk >> 3) * 128 + (r & 7) * 16 + (kk & 7) * 2);
}

// Copy the rows [r0, r0 + rows) x K columns [k0, k0 + 64) of an operand
// X(r, k) = X[r * sr + k * sk] into the canonical layout, zero-filling past
// R and K.  vec: sk == 1 and 16-byte aligned rows, so one thread moves one
// 8-element core-matrix row (16 bytes) per step as an asynchronous cp.async
// (source size 0 past the edge: the hardware writes zeros); the caller waits
// for them with cp.async.wait_group.  Otherwise single elements, stored
// directly, row index fastest when sr == 1 (a transposed operand) for
// coalescing.
__device__ __forceinline__ void stage_operand(unsigned char* dst, const __nv_bfloat16* X, int64_t sr, int64_t sk,
                                              int r0, int R, int k0, int K, int rows, bool vec, int tid) {
  if (vec) {
    for (int e = tid; e < rows * (kGemmBK / 8); e += kGemmThreads) {
      const int r = e / (kGemmBK / 8), k = (e % (kGemmBK / 8)) * 8;
      const int gr = r0 + r, gk = k0 + k;
      const bool in = gr < R && gk < K;
      const __nv_bfloat16* src = in ? X + gr * sr + gk : X;
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst + chunk_offset(r, k, rows))),
                   "l"(src), "r"(in ? 16 : 0)
                   : "memory");
    }
    return;
  }
  const bool row_fast = sr == 1;
  for (int e = tid; e < rows * kGemmBK; e += kGemmThreads) {
    const int r = row_fast ? e % rows : e / kGemmBK, k = row_fast ? e / rows : e % kGemmBK;
    const int gr = r0 + r, gk = k0 + k;
    __nv_bfloat16 v = __float2bfloat16(0.0f);
    if (gr < R && gk < K) v = X[gr * sr + gk * sk];
    *reinterpret_cast<__nv_bfloat16*>(dst + chunk_offset(r, k, rows)) = v;
  }
}

// vectorised staging applies: unit K stride, K and the row stride multiples
// of 8 elements, 16-byte aligned base
__host__ __device__ inline bool stage_vec_ok(const void* X, int64_t sr, int64_t sk, int K) {
  return sk == 1 && K % 8 == 0 && sr % 8 == 0 && (reinterpret_cast<uintptr_t>(X) & 15) == 0;
}

__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t phase) {
  for (unsigned spin = 0; spin < kMbarSpinLimit; ++spin) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(bar), "r"(phase)
        : "memory");
    if (done) return true;
  }
  return false;
}

// Epilogue of one 128 x BN tile, 32 columns at a time: tcgen05.ld gives a
// thread one tile row (TMEM lane), which goes through the warp's 4 KB of
// `stage` (16-byte chunks XOR-swizzled by row, conflict-free both ways) to
// come back as four columns of eight rows, so that the bias is loaded once,
// and mask and outputs move as whole row segments (128 bytes of FP32); alpha,
// bias, ReLU and the 0/1 mask are applied in FP32.  Written from the row
// layout with every option tested per column, this took 228 cycles a column:
// 14,600 of the 21,600 cycles of a 512 x 512 x 512 product in 128 x 64 tiles
// (2,070 here).
template <int BN>
__device__ __forceinline__ void gemm_epilogue(const GemmArgs& ga, uint32_t tmem, int m0, int n0, unsigned char* stage) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int M = ga.M, N = ga.N, relu = ga.relu;
  const float alpha = ga.alpha;
  const float* __restrict__ bias = ga.bias;
  const __nv_bfloat16* __restrict__ mask = ga.mask;
  float* __restrict__ cf = ga.cf;
  __nv_bfloat16* __restrict__ cb = ga.cb;
  const int64_t ldm = ga.ldm, ldcf = ga.ldcf, ldcb = ga.ldcb;
  const auto aligned = [](const void* p, int bytes, int64_t ld) {
    return ld % 4 == 0 && (reinterpret_cast<uintptr_t>(p) & (bytes - 1)) == 0;
  };
  const bool vec = (!cf || aligned(cf, 16, ldcf)) && (!cb || aligned(cb, 8, ldcb)) && (!mask || aligned(mask, 8, ldm));
  const bool rows_in = vec && m0 + kGemmBM <= M;
  float4* tile = reinterpret_cast<float4*>(stage) + warp * 256;  // 32 rows x 8 chunks of 4 columns
  const int quad = lane & 7, sub = lane >> 3;
  for (int c0 = 0; c0 < BN && n0 + c0 < N; c0 += 32) {
    uint32_t r[32];
    const uint32_t taddr = tmem + (static_cast<uint32_t>(warp * 32) << 16) + static_cast<uint32_t>(c0);
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
        "%15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
          "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
          "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int q = 0; q < 8; ++q)
      tile[lane * 8 + (q ^ (lane & 7))] =
          make_float4(__uint_as_float(r[4 * q]), __uint_as_float(r[4 * q + 1]), __uint_as_float(r[4 * q + 2]),
                      __uint_as_float(r[4 * q + 3]));
    __syncwarp();
    const int gn = n0 + c0 + 4 * quad, gm0 = m0 + warp * 32 + sub;
    if (rows_in && n0 + c0 + 32 <= N) {
      // straight-line: each option is one branch around 32 independent
      // operations (a warp per scheduler has only its own parallelism to
      // hide latencies with)
      float4 v[8];
#pragma unroll
      for (int it = 0; it < 8; ++it) {
        const int row = it * 4 + sub;
        v[it] = tile[row * 8 + (quad ^ (row & 7))];
      }
#pragma unroll
      for (int it = 0; it < 8; ++it)
        v[it] = make_float4(v[it].x * alpha, v[it].y * alpha, v[it].z * alpha, v[it].w * alpha);
      if (bias) {
        const float b0 = bias[gn], b1 = bias[gn + 1], b2 = bias[gn + 2], b3 = bias[gn + 3];
#pragma unroll
        for (int it = 0; it < 8; ++it)
          v[it] = make_float4(v[it].x + b0, v[it].y + b1, v[it].z + b2, v[it].w + b3);
      }
      if (relu) {
#pragma unroll
        for (int it = 0; it < 8; ++it)
          v[it] = make_float4(v[it].x > 0.0f ? v[it].x : 0.0f, v[it].y > 0.0f ? v[it].y : 0.0f,
                              v[it].z > 0.0f ? v[it].z : 0.0f, v[it].w > 0.0f ? v[it].w : 0.0f);
      }
      if (mask) {
        const __nv_bfloat16* src = mask + gm0 * ldm + gn;
        uint2 w[8];
#pragma unroll
        for (int it = 0; it < 8; ++it) w[it] = *reinterpret_cast<const uint2*>(src + it * 4 * ldm);
#pragma unroll
        for (int it = 0; it < 8; ++it) {
          const __nv_bfloat162 w0 = *reinterpret_cast<const __nv_bfloat162*>(&w[it].x);
          const __nv_bfloat162 w1 = *reinterpret_cast<const __nv_bfloat162*>(&w[it].y);
          v[it] = make_float4(__low2float(w0) > 0.0f ? v[it].x : 0.0f, __high2float(w0) > 0.0f ? v[it].y : 0.0f,
                              __low2float(w1) > 0.0f ? v[it].z : 0.0f, __high2float(w1) > 0.0f ? v[it].w : 0.0f);
        }
      }
      if (cf) {
        float* dst = cf + gm0 * ldcf + gn;
#pragma unroll
        for (int it = 0; it < 8; ++it) *reinterpret_cast<float4*>(dst + it * 4 * ldcf) = v[it];
      }
      if (cb) {
        __nv_bfloat16* dst = cb + gm0 * ldcb + gn;
#pragma unroll
        for (int it = 0; it < 8; ++it) {
          const __nv_bfloat162 h0 = __floats2bfloat162_rn(v[it].x, v[it].y), h1 = __floats2bfloat162_rn(v[it].z, v[it].w);
          uint2 h;
          h.x = *reinterpret_cast<const uint32_t*>(&h0);
          h.y = *reinterpret_cast<const uint32_t*>(&h1);
          *reinterpret_cast<uint2*>(dst + it * 4 * ldcb) = h;
        }
      }
    } else {
      for (int it = 0; it < 8; ++it) {
        const int row = it * 4 + sub, gm = gm0 + it * 4;
        const float4 t = tile[row * 8 + (quad ^ (row & 7))];
        const float v[4] = {t.x, t.y, t.z, t.w};
        if (gm >= M) break;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          if (gn + q >= N) break;
          float o = v[q] * alpha;
          if (bias) o += bias[gn + q];
          if (relu) o = o > 0.0f ? o : 0.0f;
          if (mask && !(__bfloat162float(mask[gm * ldm + gn + q]) > 0.0f)) o = 0.0f;
          if (cf) cf[gm * ldcf + gn + q] = o;
          if (cb) cb[gm * ldcb + gn + q] = __float2bfloat16(o);
        }
      }
    }
    __syncwarp();
  }
}

template <int BN>
__global__ void __launch_bounds__(kGemmThreads) k_gemm_bf16_tc(GemmArgs g) {
  constexpr int kGemmBN = BN;
  constexpr int kGemmStages = GemmTile<BN>::kStages;
  constexpr int kGemmStageBytes = GemmTile<BN>::kStageBytes;
  constexpr int kLag = GemmTile<BN>::kLag, kAhead = GemmTile<BN>::kAhead;
  extern __shared__ __align__(1024) unsigned char smem[];
  __shared__ __align__(8) uint64_t mbar[kGemmStages];
  __shared__ uint32_t tmem_base_sh;
  __shared__ int failed_sh;
  const int tid = threadIdx.x, warp = tid >> 5;
  const int m0 = blockIdx.x * kGemmBM, n0 = blockIdx.y * kGemmBN;

  if (tid == 0) {
#pragma unroll
    for (int st = 0; st < kGemmStages; ++st)
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&mbar[st])) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    failed_sh = 0;
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_sh)),
                 "r"(kGemmBN)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = tmem_base_sh;
  const uint32_t idesc = umma_idesc_bf16(kGemmBN);
  const int nchunks = (g.K + kGemmBK - 1) / kGemmBK;
  const bool vec_a = stage_vec_ok(g.A, g.sam, g.sak, g.K), vec_b = stage_vec_ok(g.B, g.sbn, g.sbk, g.K);
  uint32_t phase[kGemmStages] = {};  // parity of each stage's next completion
  auto stage_a = [&](int st) { return smem + st * kGemmStageBytes; };
  auto stage_b = [&](int st) { return smem + st * kGemmStageBytes + kGemmBM * kGemmBK * 2; };
  auto fetch = [&](int ch) {  // chunk ch into stage ch % kGemmStages, as one cp.async group
    const int st = ch % kGemmStages, k0 = ch * kGemmBK;
    stage_operand(stage_a(st), g.A, g.sam, g.sak, m0, g.M, k0, g.K, kGemmBM, vec_a, tid);
    stage_operand(stage_b(st), g.B, g.sbn, g.sbk, n0, g.N, k0, g.K, kGemmBN, vec_b, tid);
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  // prologue: the first kAhead chunks in flight
  for (int c = 0; c < kAhead; ++c)
    if (c < nchunks) fetch(c);
  for (int ch = 0; ch < nchunks; ++ch) {
    const int st = ch % kGemmStages;
    const int ahead = ch + kAhead;  // the chunk fetched in this step
    if (ahead < nchunks) {
      // its stage was last read by chunk ch - kLag's MMAs: refill it once
      // they are done (a stage not used yet needs no wait)
      const int nx = ahead % kGemmStages;
      if (ch >= kLag) {
        if (!mbar_wait(smem_u32(&mbar[nx]), phase[nx])) failed_sh = 1;
        phase[nx] ^= 1u;
      }
      __syncthreads();
      if (failed_sh) break;
      fetch(ahead);
      asm volatile("cp.async.wait_group %0;" ::"n"(kAhead) : "memory");  // chunk ch has landed
    } else {
      asm volatile("cp.async.wait_group 0;" ::: "memory");
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncthreads();
    if (tid == 0) {
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t a_base = smem_u32(stage_a(st)), b_base = smem_u32(stage_b(st));
#pragma unroll
      for (int s = 0; s < kGemmBK / 16; ++s) {
        const uint64_t da = umma_desc(a_base + s * (kGemmBM / 8) * 256, 128, 256);
        const uint64_t db = umma_desc(b_base + s * (kGemmBN / 8) * 256, 128, 256);
        const uint32_t acc = (ch > 0 || s > 0) ? 1u : 0u;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "setp.ne.b32 p, %4, 0;\n\t"
            "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %6, %7, %8}, p;\n\t}"
            :
            : "r"(tmem), "l"(da), "l"(db), "r"(idesc), "r"(acc), "r"(0u), "r"(0u), "r"(0u), "r"(0u)
            : "memory");
      }
      asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                       smem_u32(&mbar[st]))
                   : "memory");
    }
  }
  // the last commit tracks every MMA issued before it
  if (nchunks > 0 && !failed_sh) {
    const int st = (nchunks - 1) % kGemmStages;
    if (!mbar_wait(smem_u32(&mbar[st]), phase[st])) failed_sh = 1;
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  if (!failed_sh) {
    gemm_epilogue<kGemmBN>(g, tmem, m0, n0, smem);
  } else if (tid == 0) {
    *const_cast<volatile int32_t*>(g.error) = 1;
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kGemmBN) : "memory");
}


// ---------------------------------------------------------------------------
// TMA form, for operands with one contiguous dimension -- K (A row-major
// M x K, B stored N x K) or the other one (A stored K x M, B stored K x N) --
// and 16-byte aligned rows.  128 x BN tiles, brought in by the tensor memory
// accelerator (cp.async.bulk.tensor.2d, zero-filled past the edges) into
// 128-byte-swizzled stages, K-major (one 64 x rows box an operand and chunk)
// or MN-major (one box of 64 x 64 for every 64 rows of the tile).  The CTA's
// roles are split: warp 0 issues the copies, warp 1 the MMAs (one lane each,
// the other lanes following in step so that no lane spins beside them), and
// all four warps run the epilogue.  Each stage has a "full" mbarrier (the
// copies' bytes arrived) and an "empty" one (the MMAs that read it
// completed); the producer refills a stage once it is empty, so all stages
// are in flight while the tensor core works.  Every wait is bounded: on a
// timeout the kernel records an error, waits (bounded) for the copies it
// issued, frees its TMEM and returns.
//
// One launch runs a group of up to two independent products and the two
// small reductions that go with a layer's backward pass (the bias gradient's
// column sums, the loss), each on blocks of its own: a 512 x 512 x 512
// product alone is 32 tiles, a fifth of the SMs, and mostly launch and
// pipeline latency.  Launches overlap their set-up with the previous
// kernel's tail (programmatic dependent launch).
//
// Measured on the network's training step (batch 512, 512-wide layers; the
// backward products' operands are not K-contiguous): 765 us a step in
// element-copied stages with separate reductions, 61 us here.

// Most stages of a tile shape (the launch takes fewer where K is shorter, or
// where two CTAs are to share an SM).
template <int BN>
struct GemmTmaTile {
  static constexpr int kABytes = kGemmBM * kGemmBK * 2;  // 16 KB
  static constexpr int kBBytes = BN * kGemmBK * 2;
  static constexpr int kStageBytes = kABytes + kBBytes;
  static constexpr int kMaxStages = BN == 256 ? 4 : BN == 128 ? 6 : 8;
  static constexpr int kSharedStages = BN == 256 ? 4 : BN == 128 ? 3 : 4;  // two CTAs per SM up to BN = 128
  // + 1 KB so that the stages can start on a 1,024-byte boundary (the
  // period of the 128-byte swizzle)
  __host__ __device__ static constexpr int smem_bytes(int stages) { return stages * kStageBytes + 1024; }
};
constexpr int kGemmMaxStages = 8;

struct GemmProblem {
  alignas(64) CUtensorMap a;
  alignas(64) CUtensorMap b;
  GemmArgs g;
  int32_t first, blocks;  // its blocks of the grid
  int32_t tiles_m;
  int32_t a_mn, b_mn;  // the operand's contiguous dimension is M / N, not K
};

// out[c] = sum_r x[r * cols + c], rows in order.
struct GroupColsum {
  const float* x;
  float* out;
  int32_t rows, cols;
  int32_t first, blocks;
};

// *loss = 0.5 * sum(partial) * inv_rows (in order), *accum += that * weight.
struct GroupLoss {
  const double* partial;
  double* loss;
  double* accum;
  double inv_rows, weight;
  int32_t count;
  int32_t first, blocks;
};

struct GemmGroup {
  GemmProblem p[2];
  GroupColsum colsum;
  GroupLoss loss;
  int32_t problems;
  int32_t stages;
};

__device__ __forceinline__ void gemm_pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void gemm_pdl_launch() { asm volatile("griddepcontrol.launch_dependents;" :::); }

// UMMA shared-memory descriptor, 128-byte swizzle.  K-major: rows of 64 BF16
// (128 bytes) as the copies wrote them, 8-row groups SBO = 1,024 bytes apart,
// LBO unused (1); the address advances by 32 bytes per K = 16 step inside the
// 128-byte row.  MN-major: K rows of 64 M / N elements (128 bytes), groups of
// 8 K rows SBO = 1,024 bytes apart, blocks of 64 M / N elements LBO = 64 x 128
// bytes apart; the address advances by 16 rows per K = 16 step.  The swizzle
// is applied to the absolute address bits.
__device__ __forceinline__ uint64_t umma_desc_sw128(uint32_t addr, int mn) {
  uint64_t d = 0;
  d |= static_cast<uint64_t>((addr >> 4) & 0x3FFF);
  d |= static_cast<uint64_t>(mn ? (kGemmBK * 128) >> 4 : 1) << 16;  // LBO
  d |= static_cast<uint64_t>(1024 >> 4) << 32;                      // SBO
  d |= static_cast<uint64_t>(1) << 46;                              // descriptor version (Blackwell)
  d |= static_cast<uint64_t>(2) << 61;                              // layout type SWIZZLE_128B
  return d;
}

__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
          dst),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(bar)
      : "memory");
}

// One operand's rows [r0, r0 + rows) x K columns [k0, k0 + 64) of a chunk.
__device__ __forceinline__ void tma_load_operand(uint32_t dst, const CUtensorMap* map, int mn, int rows, int r0, int k0,
                                                 uint32_t bar) {
  if (!mn) {
    tma_load_2d(dst, map, k0, r0, bar);
  } else {
    for (int q = 0; q < rows; q += 64) tma_load_2d(dst + q * kGemmBK * 2, map, r0 + q, k0, bar);
  }
}

// Column sums of 32 columns (cols and c0 multiples of 4): the rows staged in
// shared memory, up to `room` at a time, a thread's sixteen 16-byte loads all
// in flight before the first is stored; one thread per column adds them in
// order.  (Stored as they arrive, the loads wait for one another: 19,100
// cycles for 512 rows against 2,850.)
__device__ __forceinline__ void group_colsum(const GroupColsum& j, float4* stage, int room) {
  constexpr int kLoads = 16, kRows = kGemmThreads / 8;  // rows a step of all threads covers
  const int c0 = (blockIdx.x - j.first) * 32, quad = threadIdx.x & 7, sub = threadIdx.x >> 3;
  const bool in = c0 + 4 * quad < j.cols;
  const float* src = j.x + c0 + 4 * quad;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  float s = 0.0f;
  for (int r0 = 0; r0 < j.rows; r0 += room) {
    const int cnt = j.rows - r0 < room ? j.rows - r0 : room;
    for (int r = sub; r < cnt; r += kLoads * kRows) {
      float4 v[kLoads];
#pragma unroll
      for (int q = 0; q < kLoads; ++q) {
        const int row = r + q * kRows;
        if (in && row < cnt)
          v[q] = __ldcg(reinterpret_cast<const float4*>(src + static_cast<int64_t>(r0 + row) * j.cols));
      }
#pragma unroll
      for (int q = 0; q < kLoads; ++q)
        if (r + q * kRows < cnt) stage[(r + q * kRows) * 8 + quad] = v[q];
    }
    __syncthreads();
    if (warp == 0) {
      const float* col = reinterpret_cast<const float*>(stage) + lane;
#pragma unroll 16
      for (int r = 0; r < cnt; ++r) s += col[r * 32];
    }
    __syncthreads();
  }
  if (warp == 0 && c0 + lane < j.cols) j.out[c0 + lane] = s;
}

__device__ __forceinline__ void group_loss(const GroupLoss& j, double* stage) {
  for (int i = threadIdx.x; i < j.count; i += kGemmThreads) stage[i] = __ldcg(j.partial + i);
  __syncthreads();
  if (threadIdx.x != 0) return;
  double s = 0.0;
#pragma unroll 8
  for (int i = 0; i < j.count; ++i) s += stage[i];
  const double l = 0.5 * s * j.inv_rows;
  if (j.loss) *j.loss = l;
  if (j.accum) *j.accum += l * j.weight;
}

template <int BN>
__global__ void __launch_bounds__(kGemmThreads) k_gemm_group(const __grid_constant__ GemmGroup G) {
  using Tile = GemmTmaTile<BN>;
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  __shared__ __align__(8) uint64_t full[kGemmMaxStages], empty[kGemmMaxStages], done;
  __shared__ uint32_t tmem_base_sh;
  __shared__ int failed_sh, issued_sh, consumed_sh;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int blk = blockIdx.x;
  if (blk >= G.loss.first && blk < G.loss.first + G.loss.blocks) {
    gemm_pdl_wait();
    gemm_pdl_launch();
    group_loss(G.loss, reinterpret_cast<double*>(smem_raw));
    return;
  }
  if (blk >= G.colsum.first && blk < G.colsum.first + G.colsum.blocks) {
    gemm_pdl_wait();
    gemm_pdl_launch();
    group_colsum(G.colsum, reinterpret_cast<float4*>(smem_raw), Tile::smem_bytes(G.stages) / 128);
    return;
  }
  const GemmProblem& P = G.p[G.problems > 1 && blk >= G.p[1].first ? 1 : 0];
  const GemmArgs& g = P.g;
  const int S = G.stages;
  const int tile = blk - P.first;
  const int m0 = tile % P.tiles_m * kGemmBM, n0 = tile / P.tiles_m * BN;
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;  // stage 0, 1,024-byte aligned
  const int nchunks = (g.K + kGemmBK - 1) / kGemmBK;

  if (tid == 0) {
    for (int st = 0; st < S; ++st) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&full[st])) : "memory");
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&empty[st])) : "memory");
    }
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&done)) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    failed_sh = 0;
    issued_sh = 0;
    consumed_sh = 0;
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&P.a)) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&P.b)) : "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_sh)),
                 "r"(BN)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = tmem_base_sh;
  // everything above is this CTA's own; the operands, and what the outputs
  // overwrite, belong to the kernels before
  gemm_pdl_wait();
  gemm_pdl_launch();

  if (warp == 0) {
    // producer warp (lane 0 issues): chunk ch into stage ch % S once the MMAs
    // of chunk ch - S are done
    int ch = 0, st = 0;
    uint32_t round = 0;
    for (; ch < nchunks; ++ch) {
      bool ok = true;
      if (round > 0) ok = mbar_wait(smem_u32(&empty[st]), (round - 1) & 1);
      if (!__all_sync(0xffffffffu, ok) || *reinterpret_cast<volatile int*>(&failed_sh)) {
        if (lane == 0) failed_sh = 1;
        break;
      }
      if (lane == 0) {
        const uint32_t sa = base + st * Tile::kStageBytes, sb = sa + Tile::kABytes;
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(&full[st])),
                     "r"(Tile::kStageBytes)
                     : "memory");
        tma_load_operand(sa, &P.a, P.a_mn, kGemmBM, m0, ch * kGemmBK, smem_u32(&full[st]));
        tma_load_operand(sb, &P.b, P.b_mn, BN, n0, ch * kGemmBK, smem_u32(&full[st]));
      }
      __syncwarp();
      if (++st == S) st = 0, ++round;
    }
    if (lane == 0) issued_sh = ch;
  } else if (warp == 1) {
    // MMA warp (lane 0 issues): four K = 16 steps per chunk, then commit the
    // stage back
    const uint32_t idesc = umma_idesc_bf16(BN) | (P.a_mn ? 1u << 15 : 0u) | (P.b_mn ? 1u << 16 : 0u);
    const uint32_t step_a = P.a_mn ? 16 * 128 : 32, step_b = P.b_mn ? 16 * 128 : 32;
    int ch = 0, st = 0;
    uint32_t round = 0;
    for (; ch < nchunks; ++ch) {
      const bool ok = mbar_wait(smem_u32(&full[st]), round & 1);
      if (!__all_sync(0xffffffffu, ok)) {
        if (lane == 0) failed_sh = 1;
        break;
      }
      if (lane == 0) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t sa = base + st * Tile::kStageBytes, sb = sa + Tile::kABytes;
#pragma unroll
        for (int s = 0; s < kGemmBK / 16; ++s) {
          const uint64_t da = umma_desc_sw128(sa + s * step_a, P.a_mn), db = umma_desc_sw128(sb + s * step_b, P.b_mn);
          const uint32_t acc = (ch > 0 || s > 0) ? 1u : 0u;
          asm volatile(
              "{\n\t.reg .pred p;\n\t"
              "setp.ne.b32 p, %4, 0;\n\t"
              "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %6, %7, %8}, p;\n\t}"
              :
              : "r"(tmem), "l"(da), "l"(db), "r"(idesc), "r"(acc), "r"(0u), "r"(0u), "r"(0u), "r"(0u)
              : "memory");
        }
        asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                         smem_u32(&empty[st]))
                     : "memory");
      }
      __syncwarp();
      if (++st == S) st = 0, ++round;
    }
    if (lane == 0) {
      consumed_sh = ch;
      // tracks every MMA issued before it
      asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                       smem_u32(&done))
                   : "memory");
    }
    __syncwarp();
  }
  if (!mbar_wait(smem_u32(&done), 0u)) failed_sh = 1;
  __syncthreads();
  __syncwarp();  // the producer and MMA lanes rejoin their warps before tcgen05.ld
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  if (!failed_sh) {
    gemm_epilogue<BN>(g, tmem, m0, n0, smem_raw + (base - raw));
  } else if (tid == 0) {
    *const_cast<volatile int32_t*>(g.error) = 1;
    // copies issued but not consumed still write into shared memory: wait for them
    for (int ch = consumed_sh; ch < issued_sh; ++ch)
      mbar_wait(smem_u32(&full[ch % S]), static_cast<uint32_t>((ch / S) & 1));
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(BN) : "memory");
}

}  // namespace b2p
