// The learned warm-start network: forward, loss, backward and Adam kernels
// around the tcgen05 BF16 GEMM (mlp_gemm.cuh), and the C ABI of
// include/b2p_mlp.h.  Every reduction runs in a fixed order, so training is
// deterministic for a given seed.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <cudaTypedefs.h>  // PFN_cuTensorMapEncodeTiled

#include <algorithm>
#include <cmath>
#include <cstring>
#include <mutex>
#include <numeric>
#include <optional>
#include <random>
#include <vector>

#include "../../include/b2p_mlp.h"
#include "mlp_gemm.cuh"
#include "pdhg_host_common.h"

namespace b2p {
namespace {

constexpr int kEw = 256;  // threads of the elementwise kernels
constexpr int kLossBlocks = 148;

inline int ew_blocks(int64_t n) { return static_cast<int>(std::max<int64_t>(1, std::min<int64_t>((n + kEw - 1) / kEw, 148 * 16))); }

// minibatch rows r <- samples perm[offset + r]: FP32 inputs to BF16, targets copied
__global__ void k_gather(int32_t rows, int32_t din, int32_t dout, const float* __restrict__ x,
                         const float* __restrict__ y, const int32_t* __restrict__ perm, int64_t offset,
                         __nv_bfloat16* __restrict__ xb, float* __restrict__ yt) {
  gemm_pdl_wait();
  gemm_pdl_launch();
  const int64_t nin = static_cast<int64_t>(rows) * din, nout = static_cast<int64_t>(rows) * dout;
  for (int64_t e = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; e < nin + nout;
       e += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    if (e < nin) {
      const int64_t r = e / din, c = e % din;
      const int64_t s = perm ? perm[offset + r] : offset + r;
      xb[e] = __float2bfloat16(x[s * din + c]);
    } else if (yt) {
      const int64_t f = e - nin, r = f / dout, c = f % dout;
      const int64_t s = perm ? perm[offset + r] : offset + r;
      yt[f] = y[s * dout + c];
    }
  }
}

// d = out - target; G = d / rows (FP32 and BF16); per-block sums of d^2
__global__ void __launch_bounds__(kEw) k_mse_grad(int64_t count, float inv_rows, const float* __restrict__ out,
                                                  const float* __restrict__ target, float* __restrict__ gf,
                                                  __nv_bfloat16* __restrict__ gb, double* __restrict__ partial) {
  gemm_pdl_wait();
  gemm_pdl_launch();
  double s = 0.0;
  for (int64_t e = blockIdx.x * static_cast<int64_t>(kEw) + threadIdx.x; e < count;
       e += static_cast<int64_t>(gridDim.x) * kEw) {
    const float d = out[e] - target[e];
    const float gv = d * inv_rows;
    gf[e] = gv;
    gb[e] = __float2bfloat16(gv);
    s += static_cast<double>(d) * static_cast<double>(d);
  }
  __shared__ double red[kEw];
  red[threadIdx.x] = s;
  __syncthreads();
  for (int w = kEw / 2; w > 0; w >>= 1) {
    if (static_cast<int>(threadIdx.x) < w) red[threadIdx.x] += red[threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x == 0) partial[blockIdx.x] = red[0];
}

// Adam (decoupled weight decay on the entries flagged in `decay`), then the
// BF16 copy of the parameters.  Four parameters a thread (every width is a
// multiple of 8, so n is of 4): 540,000 parameters in one wave of 16-byte
// accesses instead of two of 4-byte ones, 10.3 -> 7.5 us.
__global__ void __launch_bounds__(kEw) k_adam(int64_t n4, float4* __restrict__ p, const float4* __restrict__ g,
                                              float4* __restrict__ m, float4* __restrict__ v,
                                              const uchar4* __restrict__ decay, float lr, float b1, float b2, float c1,
                                              float c2, float eps, float wd, uint2* __restrict__ pb) {
  gemm_pdl_wait();
  gemm_pdl_launch();
  const auto one = [&](float gi, float& mo, float& vo, float& po, bool dec) {
    const float mi = b1 * mo + (1.0f - b1) * gi;
    const float vi = b2 * vo + (1.0f - b2) * gi * gi;
    mo = mi;
    vo = vi;
    const float mh = mi * c1, vh = vi * c2;
    float pi = po - lr * (mh / (sqrtf(vh) + eps));
    if (wd > 0.0f && dec) pi -= lr * wd * po;
    po = pi;
  };
  for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < n4;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const float4 gi = g[i];
    float4 mi = m[i], vi = v[i], pi = p[i];
    const uchar4 d = decay[i];
    one(gi.x, mi.x, vi.x, pi.x, d.x);
    one(gi.y, mi.y, vi.y, pi.y, d.y);
    one(gi.z, mi.z, vi.z, pi.z, d.z);
    one(gi.w, mi.w, vi.w, pi.w, d.w);
    m[i] = mi;
    v[i] = vi;
    p[i] = pi;
    const __nv_bfloat162 h0 = __floats2bfloat162_rn(pi.x, pi.y), h1 = __floats2bfloat162_rn(pi.z, pi.w);
    pb[i] = make_uint2(*reinterpret_cast<const uint32_t*>(&h0), *reinterpret_cast<const uint32_t*>(&h1));
  }
}

__global__ void k_to_bf16(int64_t n, const float* __restrict__ src, __nv_bfloat16* __restrict__ dst) {
  for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < n;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x)
    dst[i] = __float2bfloat16(src[i]);
}

int gemm_sms[64] = {};  // SM count per device, set with the attributes

// cuTensorMapEncodeTiled through the runtime's driver entry point (no link
// against the driver library); NULL if the driver does not offer it.
PFN_cuTensorMapEncodeTiled_v12000 tensor_map_encoder() {
  static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q = cudaDriverEntryPointSymbolNotFound;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
  });
  return fn;
}

// How the TMA form reads an operand X(r, k) = X[r * sr + k * sk], r < R,
// k < K: 0 = K-major, 1 = MN-major, -1 = not at all (a tensor map wants one
// contiguous dimension and rows of a multiple of 16 bytes on a 16-byte
// aligned base).
int operand_major(const void* X, int64_t sr, int64_t sk, int R, int K) {
  const auto rows_ok = [&](int64_t stride, int64_t inner) {
    return stride >= inner && stride % 8 == 0 && stride < (int64_t{1} << 38);
  };
  if (K <= 0 || (reinterpret_cast<uintptr_t>(X) & 15) != 0) return -1;
  if (sk == 1 && rows_ok(sr, K)) return 0;
  if (sr == 1 && rows_ok(sk, R)) return 1;
  return -1;
}

// Tensor map of such an operand, zeros past the edges, 128-byte swizzle:
// boxes of 64 K columns x box_rows rows (K-major) or 64 rows x 64 K columns
// (MN-major).
bool encode_operand(CUtensorMap* map, const __nv_bfloat16* X, int64_t sr, int64_t sk, int R, int K, int mn,
                    int box_rows) {
  const auto fn = tensor_map_encoder();
  if (!fn) return false;
  const cuuint64_t dims[2] = {static_cast<cuuint64_t>(mn ? R : K), static_cast<cuuint64_t>(mn ? K : R)};
  const cuuint64_t strides[1] = {static_cast<cuuint64_t>(mn ? sk : sr) * 2};
  const cuuint32_t box[2] = {64, static_cast<cuuint32_t>(mn ? kGemmBK : box_rows)};
  const cuuint32_t elem[2] = {1, 1};
  return fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<__nv_bfloat16*>(X), dims, strides, box, elem,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

void set_gemm_attributes() {
  static std::once_flag once[64];
  int dev = 0;
  B2P_CUDA(cudaGetDevice(&dev));
  cudaError_t err = cudaSuccess;
  std::call_once(once[dev & 63], [&] {
    err = cudaFuncSetAttribute(k_gemm_bf16_tc<128>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               GemmTile<128>::kSmemBytes);
    if (err == cudaSuccess)
      err = cudaFuncSetAttribute(k_gemm_bf16_tc<256>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 GemmTile<256>::kSmemBytes);
    const auto group = [&](auto* fn, int bytes) {
      if (err == cudaSuccess) err = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    };
    group(k_gemm_group<64>, GemmTmaTile<64>::smem_bytes(GemmTmaTile<64>::kMaxStages));
    group(k_gemm_group<128>, GemmTmaTile<128>::smem_bytes(GemmTmaTile<128>::kMaxStages));
    group(k_gemm_group<256>, GemmTmaTile<256>::smem_bytes(GemmTmaTile<256>::kMaxStages));
    if (err == cudaSuccess) err = cudaDeviceGetAttribute(&gemm_sms[dev & 63], cudaDevAttrMultiProcessorCount, dev);
  });
  B2P_CUDA(err);
}

// Launch with programmatic dependent launch (the kernel waits for the one
// before it itself).
template <typename... KArgs, typename... Args>
void launch_pdl(void (*kern)(KArgs...), unsigned grid, unsigned block, size_t smem, cudaStream_t stream,
                const Args&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  B2P_CUDA(cudaLaunchKernelEx(&cfg, kern, static_cast<KArgs>(args)...));
}

template <int BN>
void launch_group_bn(GemmGroup& gr, cudaStream_t stream, int sms) {
  using Tile = GemmTmaTile<BN>;
  int next = 0, chunks = 2;
  for (int i = 0; i < gr.problems; ++i) {
    GemmProblem& p = gr.p[i];
    p.tiles_m = (p.g.M + kGemmBM - 1) / kGemmBM;
    p.first = next;
    p.blocks = p.tiles_m * ((p.g.N + BN - 1) / BN);
    next += p.blocks;
    chunks = std::max(chunks, (p.g.K + kGemmBK - 1) / kGemmBK);
  }
  gr.colsum.first = next;
  next += gr.colsum.blocks;
  gr.loss.first = next;
  next += gr.loss.blocks;
  // one CTA per SM has the whole shared memory for its stages
  gr.stages = std::min(chunks, next <= sms ? Tile::kMaxStages : Tile::kSharedStages);
  if (next > 0)
    launch_pdl(k_gemm_group<BN>, static_cast<unsigned>(next), kGemmThreads, Tile::smem_bytes(gr.stages), stream, gr);
}

void launch_gemm_strided(const GemmArgs& g, cudaStream_t stream, int sms) {
  const int64_t mt = (g.M + kGemmBM - 1) / kGemmBM;
  if (mt * ((g.N + 255) / 256) >= sms) {
    const dim3 grid(static_cast<unsigned>(mt), (g.N + 255) / 256);
    k_gemm_bf16_tc<256><<<grid, kGemmThreads, GemmTile<256>::kSmemBytes, stream>>>(g);
  } else {
    const dim3 grid(static_cast<unsigned>(mt), (g.N + 127) / 128);
    k_gemm_bf16_tc<128><<<grid, kGemmThreads, GemmTile<128>::kSmemBytes, stream>>>(g);
  }
  B2P_CUDA(cudaGetLastError());
}

// Up to two independent products and the reductions of `jobs` (its colsum and
// loss; blocks 0 = none) in one launch.  The widest tiles that still give
// every SM a CTA, else the narrowest (128 x 64: a product too small to fill
// the GPU is bound by its pipeline's latency, which more and shorter tiles
// share out: 512 x 512 x 512 takes 6.4 us
// in 32 tiles).  A product whose strides a tensor map cannot describe
// runs the cp.async form by itself.
void launch_group(const GemmArgs* g, int count, GemmGroup jobs, cudaStream_t stream) {
  int dev = 0;
  B2P_CUDA(cudaGetDevice(&dev));
  const int sms = gemm_sms[dev & 63];
  GemmGroup& gr = jobs;
  gr.problems = 0;
  int64_t tiles256 = 0, tiles128 = 0;
  for (int i = 0; i < count; ++i) {
    if (g[i].M <= 0 || g[i].N <= 0) continue;
    const int64_t mt = (g[i].M + kGemmBM - 1) / kGemmBM;
    tiles256 += mt * ((g[i].N + 255) / 256);
    tiles128 += mt * ((g[i].N + 127) / 128);
  }
  const int bn = tiles256 >= sms ? 256 : tiles128 >= sms ? 128 : 64;
  for (int i = 0; i < count; ++i) {
    const GemmArgs& a = g[i];
    if (a.M <= 0 || a.N <= 0) continue;
    GemmProblem& p = gr.p[gr.problems];
    const int ma = operand_major(a.A, a.sam, a.sak, a.M, a.K), mb = operand_major(a.B, a.sbn, a.sbk, a.N, a.K);
    if (ma >= 0 && mb >= 0 && encode_operand(&p.a, a.A, a.sam, a.sak, a.M, a.K, ma, kGemmBM) &&
        encode_operand(&p.b, a.B, a.sbn, a.sbk, a.N, a.K, mb, bn)) {
      p.g = a;
      p.a_mn = ma;
      p.b_mn = mb;
      ++gr.problems;
    } else {
      launch_gemm_strided(a, stream, sms);
    }
  }
  if (bn == 256) launch_group_bn<256>(gr, stream, sms);
  else if (bn == 128) launch_group_bn<128>(gr, stream, sms);
  else launch_group_bn<64>(gr, stream, sms);
}

void launch_gemm(const GemmArgs& g, cudaStream_t stream) { launch_group(&g, 1, GemmGroup{}, stream); }

// A page-locked word that a GEMM's timeout sets and the host reads once the
// stream is synchronised: no memset before the call, no copy after it.
class ErrorWord {
 public:
  ErrorWord() : word_(static_cast<volatile int32_t*>(PinnedCache::get(sizeof(int32_t)))) { *word_ = 0; }
  ~ErrorWord() { PinnedCache::put(const_cast<int32_t*>(word_), sizeof(int32_t)); }
  ErrorWord(const ErrorWord&) = delete;
  ErrorWord& operator=(const ErrorWord&) = delete;
  int32_t* device() const { return const_cast<int32_t*>(word_); }
  // Waits for the stream; throws if a wait of its kernels timed out.
  void check(cudaStream_t stream) {
    B2P_CUDA(cudaStreamSynchronize(stream));
    if (!*word_) return;
    *word_ = 0;
    throw Error(B2P_ERR_CUDA, "tensor-core GEMM: mbarrier wait timed out");
  }

 private:
  volatile int32_t* word_;
};

// Buffers of one call on a stream, from the device's stream-ordered pool: a
// cudaMalloc / cudaFree pair costs 30 us to milliseconds a call and waits for
// the whole device.  The pool keeps what it gets back, so large buffers
// (training sets, long predictions), whose copies over the bus take far longer
// than the pair, are allocated and go back to the device with the call.
class CallBuffers {
 public:
  static constexpr size_t kPooledMost = size_t(64) << 20;
  CallBuffers(int dev, cudaStream_t stream) : dev_(dev), stream_(stream) {}
  ~CallBuffers() {
    for (void* p : pooled_) cudaFreeAsync(p, stream_);
    for (void* p : allocated_) cudaFree(p);
  }
  CallBuffers(const CallBuffers&) = delete;
  CallBuffers& operator=(const CallBuffers&) = delete;
  template <class T>
  T* get(size_t count) {
    if (!count) return nullptr;
    void* p = nullptr;
    const size_t bytes = count * sizeof(T);
    if (bytes <= kPooledMost) {
      B2P_CUDA(cudaMallocFromPoolAsync(&p, bytes, device_pool(dev_), stream_));
      pooled_.push_back(p);
    } else {
      B2P_CUDA(cudaMalloc(&p, bytes));
      allocated_.push_back(p);
    }
    return static_cast<T*>(p);
  }

 private:
  int dev_;
  cudaStream_t stream_;
  std::vector<void*> pooled_, allocated_;
};

template <class T>
T* dalloc(size_t count) {
  void* p = nullptr;
  if (count) B2P_CUDA(cudaMalloc(&p, count * sizeof(T)));
  return static_cast<T*>(p);
}

struct Mlp {
  int device = 0;
  cudaStream_t stream = nullptr;
  std::vector<int32_t> w;  // widths, L + 1 entries
  int L = 0;
  int32_t max_batch = 0;
  int64_t nparams = 0;
  std::vector<int64_t> woff, boff;
  int64_t step = 0;
  float *params = nullptr, *grads = nullptr, *adam_m = nullptr, *adam_v = nullptr;
  uint8_t* decay = nullptr;
  __nv_bfloat16* pbf = nullptr;               // BF16 copy of params
  std::vector<__nv_bfloat16*> act;            // act[l]: max_batch x w[l], l = 0 .. L-1
  float* out = nullptr;                       // max_batch x w[L]
  float* target = nullptr;                    // max_batch x w[L]
  float *gf[2] = {nullptr, nullptr};          // gradient ping-pong, max_batch x max width
  __nv_bfloat16* gb[2] = {nullptr, nullptr};
  double* partial = nullptr;                  // kLossBlocks
  double* d_loss = nullptr;                   // [0] last loss, [1..] epoch sums
  std::optional<ErrorWord> error;             // once there is a device
  std::vector<void*> owned;

  ~Mlp() {
    if (device >= 0) cudaSetDevice(device);
    for (void* p : owned) cudaFree(p);
    if (stream) cudaStreamDestroy(stream);
  }

  template <class T>
  T* alloc(size_t count) {
    T* p = dalloc<T>(count);
    if (p) owned.push_back(p);
    return p;
  }

  void create(const int32_t* widths, int32_t layers, int32_t mb, int32_t dev) {
    if (!widths || layers < 1) throw Error(B2P_ERR_INVALID, "network needs at least one layer");
    if (mb < 1) throw Error(B2P_ERR_INVALID, "max_batch must be positive");
    device = pick_device(dev);
    B2P_CUDA(cudaSetDevice(device));
    B2P_CUDA(cudaStreamCreateWithFlags(&stream, cudaStreamNonBlocking));
    L = layers;
    max_batch = mb;
    w.assign(widths, widths + layers + 1);
    int32_t wmax = 0;
    for (int32_t x : w) {
      if (x < 8 || x % 8 != 0 || x > 65536) throw Error(B2P_ERR_INVALID, "every width must be a multiple of 8");
      wmax = std::max(wmax, x);
    }
    woff.resize(L);
    boff.resize(L);
    for (int l = 0; l < L; ++l) {
      woff[l] = nparams;
      nparams += static_cast<int64_t>(w[l + 1]) * w[l];
      boff[l] = nparams;
      nparams += w[l + 1];
    }
    params = alloc<float>(nparams);
    grads = alloc<float>(nparams);
    adam_m = alloc<float>(nparams);
    adam_v = alloc<float>(nparams);
    pbf = alloc<__nv_bfloat16>(nparams);
    decay = alloc<uint8_t>(nparams);
    B2P_CUDA(cudaMemsetAsync(params, 0, sizeof(float) * nparams, stream));
    B2P_CUDA(cudaMemsetAsync(pbf, 0, sizeof(__nv_bfloat16) * nparams, stream));
    std::vector<uint8_t> hd(nparams, 0);
    for (int l = 0; l < L; ++l) std::fill(hd.begin() + woff[l], hd.begin() + boff[l], uint8_t(1));
    B2P_CUDA(cudaMemcpyAsync(decay, hd.data(), nparams, cudaMemcpyHostToDevice, stream));
    act.resize(L);
    for (int l = 0; l < L; ++l) act[l] = alloc<__nv_bfloat16>(static_cast<size_t>(mb) * w[l]);
    out = alloc<float>(static_cast<size_t>(mb) * w[L]);
    target = alloc<float>(static_cast<size_t>(mb) * w[L]);
    for (int i = 0; i < 2; ++i) {
      gf[i] = alloc<float>(static_cast<size_t>(mb) * wmax);
      gb[i] = alloc<__nv_bfloat16>(static_cast<size_t>(mb) * wmax);
    }
    partial = alloc<double>(kLossBlocks);
    error.emplace();
    set_gemm_attributes();
    reset_moments();
    B2P_CUDA(cudaStreamSynchronize(stream));
  }

  void reset_moments() {
    B2P_CUDA(cudaMemsetAsync(adam_m, 0, sizeof(float) * nparams, stream));
    B2P_CUDA(cudaMemsetAsync(adam_v, 0, sizeof(float) * nparams, stream));
    step = 0;
  }

  GemmArgs gemm_base() const {
    GemmArgs g{};
    g.alpha = 1.0f;
    g.error = error->device();
    return g;
  }

  // forward on rows of act[0]; result in `y` (FP32, rows x w[L])
  void forward(int32_t rows, float* y, cudaStream_t s) {
    for (int l = 0; l < L; ++l) {
      GemmArgs g = gemm_base();
      g.M = rows;
      g.N = w[l + 1];
      g.K = w[l];
      g.A = act[l];
      g.sam = w[l];
      g.sak = 1;
      g.B = pbf + woff[l];
      g.sbk = 1;
      g.sbn = w[l];
      g.bias = params + boff[l];
      if (l + 1 < L) {
        g.relu = 1;
        g.cb = act[l + 1];
        g.ldcb = w[l + 1];
      } else {
        g.cf = y;
        g.ldcf = w[L];
      }
      launch_gemm(g, s);
    }
  }

  // loss of the forward output `out` against `target`, then all gradients
  void loss_backward(int32_t rows, double* accum, double weight) {
    const int64_t cnt = static_cast<int64_t>(rows) * w[L];
    const int nb = static_cast<int>(std::min<int64_t>(kLossBlocks, (cnt + kEw - 1) / kEw));
    launch_pdl(k_mse_grad, nb, kEw, 0, stream, cnt, 1.0f / static_cast<float>(rows), out, target, gf[0], gb[0], partial);
    int cur = 0;
    for (int l = L - 1; l >= 0; --l) {
      const int32_t wo = w[l + 1], wi = w[l];
      GemmArgs g[2];
      int count = 0;
      if (l > 0) {
        // G_{l-1} = (G W_l) masked by relu'(h_l)  (rows x wi, K = wo)
        GemmArgs& h = g[count++] = gemm_base();
        h.M = rows;
        h.N = wi;
        h.K = wo;
        h.A = gb[cur];
        h.sam = wo;
        h.sak = 1;
        h.B = pbf + woff[l];
        h.sbk = wi;
        h.sbn = 1;
        h.mask = act[l];
        h.ldm = wi;
        h.cf = gf[cur ^ 1];
        h.ldcf = wi;
        h.cb = gb[cur ^ 1];
        h.ldcb = wi;
      }
      // dW_l = G^T h_l  (wo x wi, K = rows)
      GemmArgs& d = g[count++] = gemm_base();
      d.M = wo;
      d.N = wi;
      d.K = rows;
      d.A = gb[cur];
      d.sam = 1;
      d.sak = wo;
      d.B = act[l];
      d.sbk = wi;
      d.sbn = 1;
      d.cf = grads + woff[l];
      d.ldcf = wi;
      // the bias gradient, and, beside the last layer, the loss
      GemmGroup jobs{};
      jobs.colsum = GroupColsum{gf[cur], grads + boff[l], rows, wo, 0, (wo + 31) / 32};
      if (l == L - 1) jobs.loss = GroupLoss{partial, d_loss, accum, 1.0 / rows, weight, nb, 0, 1};
      launch_group(g, count, jobs, stream);
      cur ^= 1;
    }
  }

  void check_error() { error->check(stream); }

  void set_params(const float* hp) {
    B2P_CUDA(cudaSetDevice(device));
    B2P_CUDA(cudaMemcpyAsync(params, hp, sizeof(float) * nparams, cudaMemcpyHostToDevice, stream));
    k_to_bf16<<<ew_blocks(nparams), kEw, 0, stream>>>(nparams, params, pbf);
    B2P_CUDA(cudaGetLastError());
    reset_moments();
    B2P_CUDA(cudaStreamSynchronize(stream));
  }

  void get_params(float* hp) {
    B2P_CUDA(cudaSetDevice(device));
    B2P_CUDA(cudaMemcpyAsync(hp, params, sizeof(float) * nparams, cudaMemcpyDeviceToHost, stream));
    B2P_CUDA(cudaStreamSynchronize(stream));
  }

  void forward_host(const float* x, int64_t batch, float* y) {
    B2P_CUDA(cudaSetDevice(device));
    if (batch < 0) throw Error(B2P_ERR_INVALID, "negative batch");
    CallBuffers buf(device, stream);
    float* dx = buf.get<float>(static_cast<size_t>(batch) * w[0]);
    float* dy = buf.get<float>(static_cast<size_t>(batch) * w[L]);
    if (batch) {
      B2P_CUDA(cudaMemcpyAsync(dx, x, sizeof(float) * batch * w[0], cudaMemcpyHostToDevice, stream));
      forward_dev(dx, batch, dy, stream);
      B2P_CUDA(cudaMemcpyAsync(y, dy, sizeof(float) * batch * w[L], cudaMemcpyDeviceToHost, stream));
    }
    check_error();
  }

  // chunks of max_batch rows through the activation buffers
  void forward_dev(const float* dx, int64_t batch, float* dy, cudaStream_t s) {
    for (int64_t r0 = 0; r0 < batch; r0 += max_batch) {
      const int32_t rows = static_cast<int32_t>(std::min<int64_t>(max_batch, batch - r0));
      launch_pdl(k_gather, ew_blocks(static_cast<int64_t>(rows) * w[0]), kEw, 0, s, rows, w[0], w[L], dx, nullptr,
                 nullptr, r0, act[0], nullptr);
      forward(rows, dy + r0 * w[L], s);
    }
  }

  void loss_grad(const float* x, const float* y, int32_t batch, double* loss, float* grad) {
    B2P_CUDA(cudaSetDevice(device));
    if (batch < 1 || batch > max_batch) throw Error(B2P_ERR_INVALID, "batch must be in [1, max_batch]");
    CallBuffers buf(device, stream);
    float* dx = buf.get<float>(static_cast<size_t>(batch) * w[0]);
    float* dy = buf.get<float>(static_cast<size_t>(batch) * w[L]);
    LossGuard guard{*this, buf.get<double>(1)};
    B2P_CUDA(cudaMemcpyAsync(dx, x, sizeof(float) * batch * w[0], cudaMemcpyHostToDevice, stream));
    B2P_CUDA(cudaMemcpyAsync(dy, y, sizeof(float) * batch * w[L], cudaMemcpyHostToDevice, stream));
    launch_pdl(k_gather, ew_blocks(static_cast<int64_t>(batch) * (w[0] + w[L])), kEw, 0, stream, batch, w[0], w[L], dx,
               dy, nullptr, 0, act[0], target);
    forward(batch, out, stream);
    loss_backward(batch, nullptr, 0.0);
    double hl = 0;
    B2P_CUDA(cudaMemcpyAsync(&hl, d_loss, sizeof(double), cudaMemcpyDeviceToHost, stream));
    if (grad) B2P_CUDA(cudaMemcpyAsync(grad, grads, sizeof(float) * nparams, cudaMemcpyDeviceToHost, stream));
    check_error();
    if (loss) *loss = hl;
  }

  // d_loss for the time of one call
  struct LossGuard {
    Mlp& net;
    LossGuard(Mlp& n, double* p) : net(n) { net.d_loss = p; }
    ~LossGuard() { net.d_loss = nullptr; }
  };

  void train(const float* x, const float* y, int64_t count, const b2p_mlp_train_options& o, float* epoch_loss) {
    B2P_CUDA(cudaSetDevice(device));
    if (count < 1) throw Error(B2P_ERR_INVALID, "no training samples");
    if (o.epochs < 0 || o.batch < 1 || o.batch > max_batch) throw Error(B2P_ERR_INVALID, "bad epochs / batch");
    if (count > INT32_MAX) throw Error(B2P_ERR_TOO_LARGE, "too many samples");
    const int32_t bs = static_cast<int32_t>(std::min<int64_t>(o.batch, count));
    const int64_t steps_per_epoch = count / bs;
    const int64_t total = steps_per_epoch * o.epochs;
    CallBuffers buf(device, stream);
    float* dx = buf.get<float>(static_cast<size_t>(count) * w[0]);
    float* dy = buf.get<float>(static_cast<size_t>(count) * w[L]);
    int32_t* dperm = buf.get<int32_t>(static_cast<size_t>(count));
    double* dl = buf.get<double>(1 + std::max(o.epochs, 1));
    LossGuard guard{*this, dl};
    B2P_CUDA(cudaMemcpyAsync(dx, x, sizeof(float) * count * w[0], cudaMemcpyHostToDevice, stream));
    B2P_CUDA(cudaMemcpyAsync(dy, y, sizeof(float) * count * w[L], cudaMemcpyHostToDevice, stream));
    B2P_CUDA(cudaMemsetAsync(dl, 0, sizeof(double) * (1 + std::max(o.epochs, 1)), stream));
    std::mt19937_64 rng(o.seed);
    std::vector<int32_t> perm(count);
    int64_t t = 0;
    for (int ep = 0; ep < o.epochs; ++ep) {
      std::iota(perm.begin(), perm.end(), 0);
      std::shuffle(perm.begin(), perm.end(), rng);
      B2P_CUDA(cudaMemcpyAsync(dperm, perm.data(), sizeof(int32_t) * count, cudaMemcpyHostToDevice, stream));
      for (int64_t sidx = 0; sidx < steps_per_epoch; ++sidx, ++t) {
        launch_pdl(k_gather, ew_blocks(static_cast<int64_t>(bs) * (w[0] + w[L])), kEw, 0, stream, bs, w[0], w[L], dx,
                   dy, dperm, sidx * bs, act[0], target);
        forward(bs, out, stream);
        loss_backward(bs, dl + 1 + ep, 1.0 / static_cast<double>(steps_per_epoch));
        ++step;
        const double frac = total > 1 ? static_cast<double>(t) / static_cast<double>(total - 1) : 1.0;
        const double lr = o.lr_final + 0.5 * (o.lr - o.lr_final) * (1.0 + std::cos(M_PI * frac));
        const double c1 = 1.0 / (1.0 - std::pow(static_cast<double>(o.beta1), static_cast<double>(step)));
        const double c2 = 1.0 / (1.0 - std::pow(static_cast<double>(o.beta2), static_cast<double>(step)));
        launch_pdl(k_adam, ew_blocks(nparams / 4), kEw, 0, stream, nparams / 4, reinterpret_cast<float4*>(params),
                   reinterpret_cast<const float4*>(grads), reinterpret_cast<float4*>(adam_m),
                   reinterpret_cast<float4*>(adam_v), reinterpret_cast<const uchar4*>(decay),
                   static_cast<float>(lr), o.beta1, o.beta2, static_cast<float>(c1), static_cast<float>(c2), o.eps,
                   o.weight_decay, reinterpret_cast<uint2*>(pbf));
      }
    }
    std::vector<double> hl(1 + std::max(o.epochs, 1));
    B2P_CUDA(cudaMemcpyAsync(hl.data(), dl, sizeof(double) * hl.size(), cudaMemcpyDeviceToHost, stream));
    check_error();
    if (epoch_loss)
      for (int ep = 0; ep < o.epochs; ++ep) epoch_loss[ep] = static_cast<float>(hl[1 + ep]);
  }
};

Mlp* as_mlp(b2p_mlp* h) {
  if (!h) throw Error(B2P_ERR_INVALID, "network is NULL");
  return reinterpret_cast<Mlp*>(h);
}

}  // namespace
}  // namespace b2p

using namespace b2p;

extern "C" {

b2p_mlp_train_options b2p_mlp_default_train_options(void) {
  b2p_mlp_train_options o{};
  o.epochs = 200;
  o.batch = 512;
  o.lr = 1e-3f;
  o.lr_final = 1e-5f;
  o.beta1 = 0.9f;
  o.beta2 = 0.999f;
  o.eps = 1e-8f;
  o.weight_decay = 0.0f;
  o.seed = 0;
  return o;
}

int b2p_mlp_create(const int32_t* widths, int32_t num_layers, int32_t max_batch, int32_t device, b2p_mlp** out) {
  return guarded([&] {
    if (!out) throw Error(B2P_ERR_INVALID, "out is NULL");
    *out = nullptr;
    Mlp* m = new Mlp();
    try {
      m->create(widths, num_layers, max_batch, device);
    } catch (...) {
      delete m;
      throw;
    }
    *out = reinterpret_cast<b2p_mlp*>(m);
  });
}

int b2p_mlp_destroy(b2p_mlp* net) {
  return guarded([&] { delete reinterpret_cast<Mlp*>(net); });
}

int b2p_mlp_num_params(const b2p_mlp* net, int64_t* count) {
  return guarded([&] {
    if (!net || !count) throw Error(B2P_ERR_INVALID, "NULL argument");
    *count = reinterpret_cast<const Mlp*>(net)->nparams;
  });
}

int b2p_mlp_set_params(b2p_mlp* net, const float* params) {
  return guarded([&] {
    if (!params) throw Error(B2P_ERR_INVALID, "params is NULL");
    as_mlp(net)->set_params(params);
  });
}

int b2p_mlp_get_params(b2p_mlp* net, float* params) {
  return guarded([&] {
    if (!params) throw Error(B2P_ERR_INVALID, "params is NULL");
    as_mlp(net)->get_params(params);
  });
}

int b2p_mlp_forward(b2p_mlp* net, const float* x, int64_t batch, float* y) {
  return guarded([&] {
    if ((!x || !y) && batch > 0) throw Error(B2P_ERR_INVALID, "NULL buffer");
    as_mlp(net)->forward_host(x, batch, y);
  });
}

int b2p_mlp_forward_device(b2p_mlp* net, const float* x, int64_t batch, float* y, void* stream) {
  return guarded([&] {
    Mlp* m = as_mlp(net);
    if ((!x || !y) && batch > 0) throw Error(B2P_ERR_INVALID, "NULL buffer");
    if (batch < 0) throw Error(B2P_ERR_INVALID, "negative batch");
    B2P_CUDA(cudaSetDevice(m->device));
    cudaStream_t s = stream ? static_cast<cudaStream_t>(stream) : m->stream;
    // the activation buffers belong to the network's stream: order the caller's stream after it
    if (s != m->stream) {
      cudaEvent_t ev;
      B2P_CUDA(cudaEventCreateWithFlags(&ev, cudaEventDisableTiming));
      B2P_CUDA(cudaEventRecord(ev, m->stream));
      B2P_CUDA(cudaStreamWaitEvent(s, ev, 0));
      B2P_CUDA(cudaEventDestroy(ev));
    }
    m->forward_dev(x, batch, y, s);
    if (s != m->stream) {
      cudaEvent_t ev;
      B2P_CUDA(cudaEventCreateWithFlags(&ev, cudaEventDisableTiming));
      B2P_CUDA(cudaEventRecord(ev, s));
      B2P_CUDA(cudaStreamWaitEvent(m->stream, ev, 0));
      B2P_CUDA(cudaEventDestroy(ev));
    }
  });
}

int b2p_mlp_loss_grad(b2p_mlp* net, const float* x, const float* target, int32_t batch, double* loss, float* grad) {
  return guarded([&] {
    if (!x || !target) throw Error(B2P_ERR_INVALID, "NULL buffer");
    as_mlp(net)->loss_grad(x, target, batch, loss, grad);
  });
}

int b2p_mlp_train(b2p_mlp* net, const float* x, const float* target, int64_t count,
                  const b2p_mlp_train_options* opts, float* epoch_loss) {
  return guarded([&] {
    if (!x || !target) throw Error(B2P_ERR_INVALID, "NULL buffer");
    const b2p_mlp_train_options o = opts ? *opts : b2p_mlp_default_train_options();
    as_mlp(net)->train(x, target, count, o, epoch_loss);
  });
}

int b2p_mlp_gemm_bf16(int32_t M, int32_t N, int32_t K, const uint16_t* A, int64_t sam, int64_t sak,
                      const uint16_t* B, int64_t sbk, int64_t sbn, float alpha, const float* bias, int32_t relu,
                      const uint16_t* mask, int64_t ldm, float* cf, int64_t ldcf, uint16_t* cb, int64_t ldcb,
                      void* stream) {
  return guarded([&] {
    if (M < 0 || N < 0 || K < 0) throw Error(B2P_ERR_INVALID, "negative size");
    if ((!A || !B) && K > 0) throw Error(B2P_ERR_INVALID, "NULL operand");
    if (!cf && !cb) throw Error(B2P_ERR_INVALID, "no output");
    int dev = 0;
    B2P_CUDA(cudaGetDevice(&dev));
    int major = 0;
    B2P_CUDA(cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, dev));
    if (major != 10) throw Error(B2P_ERR_NO_DEVICE, "tcgen05 GEMM needs an sm_100 device");
    set_gemm_attributes();
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    ErrorWord error;
    GemmArgs g{};
    g.M = M;
    g.N = N;
    g.K = K;
    g.A = reinterpret_cast<const __nv_bfloat16*>(A);
    g.sam = sam;
    g.sak = sak;
    g.B = reinterpret_cast<const __nv_bfloat16*>(B);
    g.sbk = sbk;
    g.sbn = sbn;
    g.alpha = alpha;
    g.bias = bias;
    g.relu = relu;
    g.mask = reinterpret_cast<const __nv_bfloat16*>(mask);
    g.ldm = ldm;
    g.cf = cf;
    g.ldcf = ldcf;
    g.cb = reinterpret_cast<__nv_bfloat16*>(cb);
    g.ldcb = ldcb;
    g.error = error.device();
    try {
      launch_gemm(g, s);
      error.check(s);
    } catch (...) {
      cudaStreamSynchronize(s);  // nothing still writes the word when it goes back
      throw;
    }
  });
}

int b2p_mlp_gemm_bf16_time(int32_t M, int32_t N, int32_t K, const uint16_t* A, int64_t sam, int64_t sak,
                           const uint16_t* B, int64_t sbk, int64_t sbn, float* cf, int64_t ldcf, int32_t reps,
                           double* ms_per_launch) {
  return guarded([&] {
    if (M <= 0 || N <= 0 || K <= 0 || reps <= 0) throw Error(B2P_ERR_INVALID, "sizes and reps must be positive");
    if (!A || !B || !cf || !ms_per_launch) throw Error(B2P_ERR_INVALID, "NULL argument");
    int dev = 0, major = 0;
    B2P_CUDA(cudaGetDevice(&dev));
    B2P_CUDA(cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, dev));
    if (major != 10) throw Error(B2P_ERR_NO_DEVICE, "tcgen05 GEMM needs an sm_100 device");
    set_gemm_attributes();
    cudaStream_t s = nullptr;
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    ErrorWord error;
    struct Cleanup {
      cudaStream_t& s;
      cudaEvent_t &e0, &e1;
      ~Cleanup() {
        if (s) cudaStreamSynchronize(s);
        if (e0) cudaEventDestroy(e0);
        if (e1) cudaEventDestroy(e1);
        if (s) cudaStreamDestroy(s);
      }
    } cleanup{s, e0, e1};
    B2P_CUDA(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking));
    B2P_CUDA(cudaEventCreate(&e0));
    B2P_CUDA(cudaEventCreate(&e1));
    GemmArgs g{};
    g.M = M;
    g.N = N;
    g.K = K;
    g.A = reinterpret_cast<const __nv_bfloat16*>(A);
    g.sam = sam;
    g.sak = sak;
    g.B = reinterpret_cast<const __nv_bfloat16*>(B);
    g.sbk = sbk;
    g.sbn = sbn;
    g.alpha = 1.0f;
    g.cf = cf;
    g.ldcf = ldcf;
    g.error = error.device();
    launch_gemm(g, s);  // warm-up (module load, attributes)
    B2P_CUDA(cudaEventRecord(e0, s));
    for (int r = 0; r < reps; ++r) launch_gemm(g, s);
    B2P_CUDA(cudaEventRecord(e1, s));
    B2P_CUDA(cudaEventSynchronize(e1));
    float ms = 0;
    B2P_CUDA(cudaEventElapsedTime(&ms, e0, e1));
    error.check(s);
    *ms_per_launch = static_cast<double>(ms) / reps;
  });
}

}  // extern "C"
