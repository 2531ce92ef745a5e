// Kernels of the learned join-order prior (join_prior.h): one forward (and
// back to every layer's deltas) of all layers, and one weight gradient + Adam
// update.  The MLP is tiny (41,473 fp32 parameters) and stays in fp32, so it
// runs on CUDA cores, bound by latency: what matters is how many SMs and
// warps share a batch and how many dependent steps each takes.
#include "join_prior.h"

#include <algorithm>
#include <cmath>
#include <cstring>

#include "capi_internal.h"

namespace kdb {
namespace {

constexpr int kIn = JoinPrior::kIn;
constexpr int kHid = JoinPrior::kHid;
constexpr int kPassThreads = 512;  // forward / deltas
constexpr int kShares = 8;         // parts of a layer's inputs; two warps share one, half of the rows each
static_assert(kPassThreads / 32 == 2 * kShares, "two warps per share");
constexpr int kPitch = kHid + 4;   // floats per weight row in shared memory: rows four banks apart
constexpr int kMaxTileRows = 8;
constexpr int kGradThreads = 512;
constexpr int kGradWarps = kGradThreads / 32;
constexpr int64_t kParams = JoinPrior::kParams;

// Shared memory of a forward / deltas CTA working on R rows at a time.
template <int R>
struct PassSmem {
  float w[(kIn + 2 * kHid) * kPitch];  // W1, W2, W3
  float b[3 * kHid];
  float w4[kHid];
  float x[R * kIn];
  float h[3][R * kHid];
  float d[2][R * kHid];
  float part[kShares * R * kHid];
  float t[R];
  float dy[R];
};
static_assert(sizeof(PassSmem<kMaxTileRows>) <= 227 * 1024, "fits an SM");

__device__ __forceinline__ float WarpSum(float s) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  return s;
}

__device__ __forceinline__ void CopyAsync16(float* dst, const float* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
                   static_cast<uint32_t>(__cvta_generic_to_shared(dst))),
               "l"(src)
               : "memory");
}
// ROWS weight rows of kHid floats into rows of kPitch floats, as one group
template <int ROWS>
__device__ __forceinline__ void CopyRowsAsync(float* dst, const float* src) {
  for (int i = threadIdx.x; i < ROWS * (kHid / 4); i += kPassThreads)
    CopyAsync16(dst + (i / (kHid / 4)) * kPitch + 4 * (i % (kHid / 4)), src + 4 * i);
  asm volatile("cp.async.commit_group;" ::: "memory");
}
template <int LEFT>
__device__ __forceinline__ void WaitCopies() {
  asm volatile("cp.async.wait_group %0;" ::"n"(LEFT) : "memory");
  __syncthreads();
}

// Sums the shares of R x kHid outputs in their order from `first` on,
// and hands each to done(row, column, sum); ends with a barrier.
template <int R, typename FIRST, typename DONE>
__device__ __forceinline__ void SumShares(const float* part, FIRST first, DONE done) {
  __syncthreads();
  for (int o = threadIdx.x; o < R * kHid; o += kPassThreads) {
    const int r = o / kHid, j = o % kHid;
    float s = first(j);
#pragma unroll
    for (int w = 0; w < kShares; w++) s += part[w * R * kHid + o];
    done(r, j, s);
  }
  __syncthreads();
}

// A warp's share of in (R x K) times W (K x kHid): one eighth of the inputs,
// half of the rows.  A lane owns 4 neighbouring outputs: a weight row is one
// 16-byte load per lane, an input is the same word for the whole warp.
template <int R, int K>
__device__ __forceinline__ void DenseShare(const float* W, const float* in, float* part) {
  constexpr int kShare = K / kShares, H = R / 2;
  const int lane = threadIdx.x & 31, share = (threadIdx.x >> 5) % kShares, r0 = (threadIdx.x >> 5) / kShares * H;
  const int k0 = share * kShare;
  float acc[H][4];
#pragma unroll
  for (int r = 0; r < H; r++) acc[r][0] = acc[r][1] = acc[r][2] = acc[r][3] = 0.f;
#pragma unroll
  for (int k = 0; k < kShare; k += 4) {
    float4 v[H];
#pragma unroll
    for (int r = 0; r < H; r++) v[r] = *reinterpret_cast<const float4*>(in + (r0 + r) * K + k0 + k);
#pragma unroll
    for (int i = 0; i < 4; i++) {
      const float4 w = *reinterpret_cast<const float4*>(W + (k0 + k + i) * kPitch + 4 * lane);
#pragma unroll
      for (int r = 0; r < H; r++) {
        const float s = i == 0 ? v[r].x : i == 1 ? v[r].y : i == 2 ? v[r].z : v[r].w;
        acc[r][0] = fmaf(s, w.x, acc[r][0]);
        acc[r][1] = fmaf(s, w.y, acc[r][1]);
        acc[r][2] = fmaf(s, w.z, acc[r][2]);
        acc[r][3] = fmaf(s, w.w, acc[r][3]);
      }
    }
  }
#pragma unroll
  for (int r = 0; r < H; r++)
    *reinterpret_cast<float4*>(part + (share * R + r0 + r) * kHid + 4 * lane) =
        make_float4(acc[r][0], acc[r][1], acc[r][2], acc[r][3]);
}

// A warp's share of dz (R x kHid) times W transposed: one eighth of the
// columns, half of the rows.  A lane owns outputs lane + 32 i, whose weight
// rows lie four banks apart.
template <int R>
__device__ __forceinline__ void DeltaShare(const float* W, const float* dz, float* part) {
  constexpr int kShare = kHid / kShares, H = R / 2;
  const int lane = threadIdx.x & 31, share = (threadIdx.x >> 5) % kShares, r0 = (threadIdx.x >> 5) / kShares * H;
  const int j0 = share * kShare;
  float acc[H][4];
#pragma unroll
  for (int r = 0; r < H; r++) acc[r][0] = acc[r][1] = acc[r][2] = acc[r][3] = 0.f;
#pragma unroll
  for (int j = 0; j < kShare; j += 4) {
    float4 v[H];
#pragma unroll
    for (int r = 0; r < H; r++) v[r] = *reinterpret_cast<const float4*>(dz + (r0 + r) * kHid + j0 + j);
#pragma unroll
    for (int i = 0; i < 4; i++) {
      const float4 w = *reinterpret_cast<const float4*>(W + (lane + 32 * i) * kPitch + j0 + j);
#pragma unroll
      for (int r = 0; r < H; r++)
        acc[r][i] = fmaf(v[r].w, w.w, fmaf(v[r].z, w.z, fmaf(v[r].y, w.y, fmaf(v[r].x, w.x, acc[r][i]))));
    }
  }
#pragma unroll
  for (int r = 0; r < H; r++)
#pragma unroll
    for (int i = 0; i < 4; i++) part[(share * R + r0 + r) * kHid + lane + 32 * i] = acc[r][i];
}

// Forward of every layer for tiles of R rows and, with targets, back to
// every layer's pre-activation deltas.  Each CTA brings all weights into its
// shared memory once (in the order the layers need them) and walks its
// tiles; the 16 warps split each layer's inputs and rows.  X, T and Y are host memory
// mapped into the device (a batch is read and its outputs written once, over
// the link, without separate copies).  For the weight gradients the inputs,
// the activations and the deltas go to `keep`.
template <int R>
__global__ void __launch_bounds__(kPassThreads, 1)
    PriorPass(const float* __restrict__ P, const float* __restrict__ X, const float* __restrict__ T, int64_t n,
              float* __restrict__ Y, const PriorKeep keep) {
  extern __shared__ __align__(16) unsigned char prior_smem[];
  PassSmem<R>& s = *reinterpret_cast<PassSmem<R>*>(prior_smem);
  float* const W1 = s.w;
  float* const W2 = s.w + kIn * kPitch;
  float* const W3 = W2 + kHid * kPitch;
  CopyRowsAsync<kIn>(W1, P + JoinPrior::kOffW1);
  CopyRowsAsync<kHid>(W2, P + JoinPrior::kOffW2);
  CopyRowsAsync<kHid>(W3, P + JoinPrior::kOffW3);
  for (int j = threadIdx.x; j < kHid; j += kPassThreads) {
    s.b[j] = P[JoinPrior::kOffB1 + j];
    s.b[kHid + j] = P[JoinPrior::kOffB2 + j];
    s.b[2 * kHid + j] = P[JoinPrior::kOffB3 + j];
    s.w4[j] = P[JoinPrior::kOffW4 + j];
  }
  const float b4 = P[JoinPrior::kOffB4];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t tiles = (n + R - 1) / R;
  for (int64_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
    const int64_t row0 = tile * R;
    for (int i = threadIdx.x; i < R * (kIn / 4); i += kPassThreads) {
      const int64_t row = row0 + i / (kIn / 4);
      float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
      if (row < n) {
        v = reinterpret_cast<const float4*>(X)[row0 * (kIn / 4) + i];
        if (T) reinterpret_cast<float4*>(keep.x)[row0 * (kIn / 4) + i] = v;
      }
      reinterpret_cast<float4*>(s.x)[i] = v;
    }
    // (with the inputs: a read over the link takes about 2 us)
    if (T && threadIdx.x >= kPassThreads - R) {
      const int r = threadIdx.x - (kPassThreads - R);
      s.t[r] = row0 + r < n ? T[row0 + r] : 0.f;
    }
    // layer l's activations: to shared memory, and kept when training
    auto relu = [&](int l) {
      return [&, l](int r, int j, float v) {
        v = fmaxf(v, 0.f);
        s.h[l][r * kHid + j] = v;
        if (T && row0 + r < n) keep.h[l][(row0 + r) * kHid + j] = v;
      };
    };
    WaitCopies<2>();
    DenseShare<R, kIn>(W1, s.x, s.part);
    SumShares<R>(s.part, [&](int j) { return s.b[j]; }, relu(0));
    WaitCopies<1>();
    DenseShare<R, kHid>(W2, s.h[0], s.part);
    SumShares<R>(s.part, [&](int j) { return s.b[kHid + j]; }, relu(1));
    WaitCopies<0>();
    DenseShare<R, kHid>(W3, s.h[1], s.part);
    SumShares<R>(s.part, [&](int j) { return s.b[2 * kHid + j]; }, relu(2));
    // head: one warp per row
    for (int r = warp; r < R; r += kPassThreads / 32) {
      const float4 h = *reinterpret_cast<const float4*>(s.h[2] + r * kHid + 4 * lane);
      const float4 w = *reinterpret_cast<const float4*>(s.w4 + 4 * lane);
      const float y = WarpSum((h.x * w.x + h.y * w.y) + (h.z * w.z + h.w * w.w)) + b4;
      if (lane == 0) {
        float dy = 0.f;
        if (row0 + r < n) {
          Y[row0 + r] = y;
          if (T) {
            dy = 2.f * (y - s.t[r]) / static_cast<float>(n);
            keep.dy[row0 + r] = dy;
          }
        }
        s.dy[r] = dy;
      }
    }
    if (!T) {
      __syncthreads();  // the next tile overwrites x
      continue;
    }
    __syncthreads();
    auto delta = [&](int l, float* to) {
      return [&, l, to](int r, int j, float v) {
        v = s.h[l][r * kHid + j] > 0.f ? v : 0.f;
        to[r * kHid + j] = v;
        if (row0 + r < n) keep.d[l][(row0 + r) * kHid + j] = v;
      };
    };
    for (int o = threadIdx.x; o < R * kHid; o += kPassThreads)
      delta(2, s.d[0])(o / kHid, o % kHid, s.dy[o / kHid] * s.w4[o % kHid]);
    __syncthreads();
    auto zero = [](int) { return 0.f; };
    DeltaShare<R>(W3, s.d[0], s.part);
    SumShares<R>(s.part, zero, delta(1, s.d[1]));
    DeltaShare<R>(W2, s.d[1], s.part);
    SumShares<R>(s.part, zero, delta(0, s.d[0]));
  }
}

// Gradient of mean((y - t)^2) over the batch and, with lr > 0, the Adam step
// (Kingma & Ba, beta1 0.9, beta2 0.999, eps 1e-8).  A CTA owns 16 x 32 weights
// of one layer over all rows: its 16 warps take every 16th row, eight rows'
// loads in flight, and their sums meet in shared memory in warp order, so the
// result is the same on every run and no per-CTA partials are written.
// Four more CTAs own the biases and the head.
constexpr int kGradK = 16, kGradJ = 32, kGradAhead = 8;
constexpr int kGradTiles1 = (kIn / kGradK) * (kHid / kGradJ);
constexpr int kGradTiles = (kHid / kGradK) * (kHid / kGradJ);
constexpr int kGradBlocks = kGradTiles1 + 2 * kGradTiles + 4;
static_assert(kGradK * kGradJ == kGradThreads, "one weight per thread");

__global__ void __launch_bounds__(kGradThreads)
    PriorGrad(float* __restrict__ P, const PriorKeep keep, int64_t n, float* __restrict__ m, float* __restrict__ v,
              float* __restrict__ grad, float lr, float c1, float c2) {
  __shared__ float part[kGradWarps * kGradThreads];
  __shared__ float head[kGradWarps];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  auto update = [&](int64_t p, float g) {
    if (grad) grad[p] = g;
    if (lr > 0.f) {
      const float mp = 0.9f * m[p] + 0.1f * g;
      const float vp = 0.999f * v[p] + 0.001f * g * g;
      m[p] = mp;
      v[p] = vp;
      P[p] -= lr * (mp / c1) / (sqrtf(vp / c2) + 1e-8f);
    }
  };
  int b = blockIdx.x;
  if (b < kGradTiles1 + 2 * kGradTiles) {
    int l = 0;
    if (b >= kGradTiles1) {
      b -= kGradTiles1;
      l = 1 + b / kGradTiles;
      b %= kGradTiles;
    }
    const int k0 = b / (kHid / kGradJ) * kGradK, j0 = b % (kHid / kGradJ) * kGradJ;
    const int width = l == 0 ? kIn : kHid;
    const float* in = (l == 0 ? keep.x : keep.h[l - 1]) + k0 + 4 * (lane >> 3);
    const float* dz = keep.d[l] + j0 + 4 * (lane & 7);
    float acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; i++) acc[i][0] = acc[i][1] = acc[i][2] = acc[i][3] = 0.f;
    auto add = [&](const float4& a, const float4& d) {
      const float x[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
      for (int i = 0; i < 4; i++) {
        acc[i][0] = fmaf(x[i], d.x, acc[i][0]);
        acc[i][1] = fmaf(x[i], d.y, acc[i][1]);
        acc[i][2] = fmaf(x[i], d.z, acc[i][2]);
        acc[i][3] = fmaf(x[i], d.w, acc[i][3]);
      }
    };
    int64_t r = warp;
    // (whole batches without a test per row: with one the compiler takes
    // the rows' loads one after the other, 125 us for 4096 rows)
    for (; r + (kGradAhead - 1) * kGradWarps < n; r += kGradAhead * kGradWarps) {
      float4 a[kGradAhead], d[kGradAhead];
#pragma unroll
      for (int u = 0; u < kGradAhead; u++) {
        a[u] = __ldcg(reinterpret_cast<const float4*>(in + (r + u * kGradWarps) * width));
        d[u] = __ldcg(reinterpret_cast<const float4*>(dz + (r + u * kGradWarps) * kHid));
      }
#pragma unroll
      for (int u = 0; u < kGradAhead; u++) add(a[u], d[u]);
    }
    for (; r < n; r += kGradWarps)
      add(*reinterpret_cast<const float4*>(in + r * width), *reinterpret_cast<const float4*>(dz + r * kHid));
#pragma unroll
    for (int i = 0; i < 4; i++)
      *reinterpret_cast<float4*>(part + warp * kGradThreads + (4 * (lane >> 3) + i) * kGradJ + 4 * (lane & 7)) =
          make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
    __syncthreads();
    float g = 0.f;
#pragma unroll
    for (int w = 0; w < kGradWarps; w++) g += part[w * kGradThreads + threadIdx.x];
    const int64_t off = l == 0 ? JoinPrior::kOffW1 : l == 1 ? JoinPrior::kOffW2 : JoinPrior::kOffW3;
    update(off + (k0 + threadIdx.x / kGradJ) * kHid + j0 + threadIdx.x % kGradJ, g);
    return;
  }
  // a layer's bias (the column sums of its deltas), or the head (the third
  // layer's activations weighted by dy, and dy's own sum)
  const int l = b - (kGradTiles1 + 2 * kGradTiles);
  const bool is_head = l == 3;
  const float* rows = (is_head ? keep.h[2] : keep.d[l]) + 4 * lane;
  float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
  float sum = 0.f;
  auto add = [&](const float4& x, float f) {
    acc.x = fmaf(f, x.x, acc.x);
    acc.y = fmaf(f, x.y, acc.y);
    acc.z = fmaf(f, x.z, acc.z);
    acc.w = fmaf(f, x.w, acc.w);
    sum += f;
  };
  int64_t r = warp;
  for (; r + (kGradAhead - 1) * kGradWarps < n; r += kGradAhead * kGradWarps) {
    float4 x[kGradAhead];
    float f[kGradAhead];
#pragma unroll
    for (int u = 0; u < kGradAhead; u++) {
      x[u] = __ldcg(reinterpret_cast<const float4*>(rows + (r + u * kGradWarps) * kHid));
      f[u] = is_head ? __ldcg(keep.dy + r + u * kGradWarps) : 1.f;
    }
#pragma unroll
    for (int u = 0; u < kGradAhead; u++) add(x[u], f[u]);
  }
  for (; r < n; r += kGradWarps)
    add(*reinterpret_cast<const float4*>(rows + r * kHid), is_head ? keep.dy[r] : 1.f);
  *reinterpret_cast<float4*>(part + warp * kHid + 4 * lane) = acc;
  if (lane == 0) head[warp] = sum;
  __syncthreads();
  if (threadIdx.x < kHid) {
    float g = 0.f;
    for (int w = 0; w < kGradWarps; w++) g += part[w * kHid + threadIdx.x];
    const int64_t off = l == 0   ? JoinPrior::kOffB1
                        : l == 1 ? JoinPrior::kOffB2
                        : l == 2 ? JoinPrior::kOffB3
                                 : JoinPrior::kOffW4;
    update(off + threadIdx.x, g);
  } else if (is_head && threadIdx.x == kHid) {
    float g = 0.f;
    for (int w = 0; w < kGradWarps; w++) g += head[w];
    update(JoinPrior::kOffB4, g);
  }
}

template <int R>
void LaunchPass(const float* p, const float* x, const float* t, int64_t n, float* y, const PriorKeep& keep, int sms,
                cudaStream_t s) {
  constexpr int kSmem = static_cast<int>(sizeof(PassSmem<R>));
  KDB_CUDA(cudaFuncSetAttribute(PriorPass<R>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem));
  const int grid = static_cast<int>(std::min<int64_t>((n + R - 1) / R, sms));
  PriorPass<R><<<grid, kPassThreads, kSmem, s>>>(p, x, t, n, y, keep);
  KDB_CUDA(cudaGetLastError());
}

uint64_t SplitMix(uint64_t& s) {
  uint64_t z = (s += 0x9E3779B97F4A7C15ULL);
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ULL;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBULL;
  return z ^ (z >> 31);
}

}  // namespace

JoinPrior::JoinPrior(int device, uint32_t seed) : device_(device) {
  KDB_CUDA(cudaSetDevice(device));
  KDB_CUDA(cudaStreamCreateWithFlags(&stream_, cudaStreamNonBlocking));
  KDB_CUDA(cudaDeviceGetAttribute(&sms_, cudaDevAttrMultiProcessorCount, device));
  KDB_CUDA(cudaMalloc(&p_, sizeof(float) * kParams));
  KDB_CUDA(cudaMalloc(&m_, sizeof(float) * kParams));
  KDB_CUDA(cudaMalloc(&v_, sizeof(float) * kParams));
  // inputs, three activations, three deltas and dy of a batch
  KDB_CUDA(cudaMalloc(&batch_, sizeof(float) * kMaxRows * (kIn + 6 * kHid + 1)));
  keep_.x = batch_;
  for (int l = 0; l < 3; l++) {
    keep_.h[l] = batch_ + kMaxRows * (kIn + l * kHid);
    keep_.d[l] = batch_ + kMaxRows * (kIn + (3 + l) * kHid);
  }
  keep_.dy = batch_ + kMaxRows * (kIn + 6 * kHid);
  // a batch's inputs, targets and outputs, and the gradient: read and
  // written by the kernels directly
  KDB_CUDA(cudaHostAlloc(&pinned_, sizeof(float) * (kMaxRows * (kIn + 2) + kParams), cudaHostAllocMapped));
  void* mapped = nullptr;
  KDB_CUDA(cudaHostGetDevicePointer(&mapped, pinned_, 0));
  mapped_ = static_cast<float*>(mapped);
  // He-uniform initialisation (bound sqrt(6 / fan_in)), zero biases
  std::vector<float> init(kParams, 0.f);
  uint64_t s = 0x6A09E667F3BCC909ULL ^ seed;
  auto fill = [&](int64_t off, int64_t count, int fan_in) {
    const double a = std::sqrt(6.0 / fan_in);
    for (int64_t i = 0; i < count; i++)
      init[off + i] = static_cast<float>((static_cast<double>(SplitMix(s) >> 11) * 0x1.0p-53 * 2.0 - 1.0) * a);
  };
  fill(kOffW1, kIn * kHid, kIn);
  fill(kOffW2, kHid * kHid, kHid);
  fill(kOffW3, kHid * kHid, kHid);
  fill(kOffW4, kHid, kHid);
  SetParams(init.data());
}

JoinPrior::~JoinPrior() {
  cudaSetDevice(device_);
  cudaStreamSynchronize(stream_);
  for (float* p : {p_, m_, v_, batch_}) cudaFree(p);
  cudaFreeHost(pinned_);
  cudaStreamDestroy(stream_);
}

void JoinPrior::SetParams(const float* p) {
  std::lock_guard<std::mutex> lock(mu_);
  KDB_CUDA(cudaSetDevice(device_));
  std::memcpy(pinned_, p, sizeof(float) * kParams);
  KDB_CUDA(cudaMemcpyAsync(p_, pinned_, sizeof(float) * kParams, cudaMemcpyHostToDevice, stream_));
  KDB_CUDA(cudaMemsetAsync(m_, 0, sizeof(float) * kParams, stream_));
  KDB_CUDA(cudaMemsetAsync(v_, 0, sizeof(float) * kParams, stream_));
  KDB_CUDA(cudaStreamSynchronize(stream_));
  step_ = 0;
}

void JoinPrior::GetParams(float* p) {
  std::lock_guard<std::mutex> lock(mu_);
  KDB_CUDA(cudaSetDevice(device_));
  KDB_CUDA(cudaMemcpyAsync(pinned_, p_, sizeof(float) * kParams, cudaMemcpyDeviceToHost, stream_));
  KDB_CUDA(cudaStreamSynchronize(stream_));
  std::memcpy(p, pinned_, sizeof(float) * kParams);
}

double JoinPrior::Run(const float* x, const float* t, int64_t n, float* grad, float lr, float* y) {
  if (n <= 0 || n > kMaxRows) throw Error(KDB_ERR_INVALID, "join prior batch must hold 1.." +
                                                              std::to_string(kMaxRows) + " rows");
  std::lock_guard<std::mutex> lock(mu_);
  KDB_CUDA(cudaSetDevice(device_));
  constexpr int64_t kOffT = kMaxRows * kIn, kOffY = kOffT + kMaxRows, kOffG = kOffY + kMaxRows;
  const float* py = pinned_ + kOffY;
  std::memcpy(pinned_, x, sizeof(float) * n * kIn);
  if (t) std::memcpy(pinned_ + kOffT, t, sizeof(float) * n);
  // Rows per tile: the fewest that let every tile have its own SM (a tile is
  // a chain of layers, so a batch is done soonest spread wide), else 8, the
  // CTAs walking their tiles with the weights in place.
  const float* mt = t ? mapped_ + kOffT : nullptr;
  if (n <= 2 * sms_) LaunchPass<2>(p_, mapped_, mt, n, mapped_ + kOffY, keep_, sms_, stream_);
  else if (n <= 4 * sms_) LaunchPass<4>(p_, mapped_, mt, n, mapped_ + kOffY, keep_, sms_, stream_);
  else LaunchPass<kMaxTileRows>(p_, mapped_, mt, n, mapped_ + kOffY, keep_, sms_, stream_);
  if (t) {
    float c1 = 1.f, c2 = 1.f;
    if (lr > 0.f) {
      step_++;
      c1 = static_cast<float>(1.0 - std::pow(0.9, static_cast<double>(step_)));
      c2 = static_cast<float>(1.0 - std::pow(0.999, static_cast<double>(step_)));
    }
    PriorGrad<<<kGradBlocks, kGradThreads, 0, stream_>>>(p_, keep_, n, m_, v_, grad ? mapped_ + kOffG : nullptr, lr, c1,
                                                         c2);
    KDB_CUDA(cudaGetLastError());
  }
  KDB_CUDA(cudaStreamSynchronize(stream_));
  if (grad) std::memcpy(grad, pinned_ + kOffG, sizeof(float) * kParams);
  double loss = 0;
  if (t)
    for (int64_t i = 0; i < n; i++) {
      const double d = static_cast<double>(py[i]) - t[i];
      loss += d * d;
    }
  if (y) std::memcpy(y, py, sizeof(float) * n);
  return t ? loss / static_cast<double>(n) : 0.0;
}

void JoinPrior::Forward(const float* x, int64_t n, float* y) {
  Run(x, nullptr, n, nullptr, 0.f, y);
}

double JoinPrior::Gradient(const float* x, const float* t, int64_t n, float* grad) {
  return Run(x, t, n, grad, 0.f, nullptr);
}

double JoinPrior::TrainStep(const float* x, const float* t, int64_t n, float lr) {
  if (!(lr > 0.f)) throw Error(KDB_ERR_INVALID, "learning rate must be positive");
  return Run(x, t, n, nullptr, lr, nullptr);
}

}  // namespace kdb

struct kdb_mlp {
  std::unique_ptr<kdb::JoinPrior> p;
  std::string err;
};

namespace {

template <typename F>
int MGuard(kdb_mlp* m, F&& f) {
  if (!m) return KDB_ERR_INVALID;
  try {
    f();
    return KDB_OK;
  } catch (const kdb::Error& e) {
    m->err = e.what();
    return e.code;
  } catch (const std::exception& e) {
    m->err = e.what();
    return KDB_ERR_CUDA;
  }
}

}  // namespace

extern "C" {

int32_t kdb_mlp_num_features(void) { return kdb::JoinPrior::kIn; }
int64_t kdb_mlp_num_params(void) { return kdb::JoinPrior::kParams; }

int kdb_mlp_create(kdb_ctx* ctx, uint32_t seed, kdb_mlp** out) {
  if (!ctx || !out) return KDB_ERR_INVALID;
  *out = nullptr;
  try {
    kdb::Context& c = *kdb_ctx_context(ctx);
    if (c.dry) throw kdb::Error(KDB_ERR_UNSUPPORTED, "the join prior needs a GPU context");
    auto m = std::make_unique<kdb_mlp>();
    m->p = std::make_unique<kdb::JoinPrior>(c.device, seed);
    *out = m.release();
    return KDB_OK;
  } catch (const kdb::Error& e) {
    kdb_ctx_set_error(ctx, e.what());
    return e.code;
  } catch (const std::exception& e) {
    kdb_ctx_set_error(ctx, e.what());
    return KDB_ERR_CUDA;
  }
}

const char* kdb_mlp_last_error(kdb_mlp* m) { return m ? m->err.c_str() : "null model"; }

int kdb_mlp_set_params(kdb_mlp* m, const float* params, int64_t n) {
  return MGuard(m, [&] {
    if (!params || n != kdb::JoinPrior::kParams) throw kdb::Error(KDB_ERR_INVALID, "wrong parameter count");
    m->p->SetParams(params);
  });
}

int kdb_mlp_get_params(kdb_mlp* m, float* params, int64_t n) {
  return MGuard(m, [&] {
    if (!params || n != kdb::JoinPrior::kParams) throw kdb::Error(KDB_ERR_INVALID, "wrong parameter count");
    m->p->GetParams(params);
  });
}

int kdb_mlp_forward(kdb_mlp* m, const float* x, int64_t n, float* y) {
  return MGuard(m, [&] {
    if (!x || !y) throw kdb::Error(KDB_ERR_INVALID, "null buffer");
    m->p->Forward(x, n, y);
  });
}

int kdb_mlp_gradient(kdb_mlp* m, const float* x, const float* t, int64_t n, float* grad, double* loss) {
  return MGuard(m, [&] {
    if (!x || !t || !grad) throw kdb::Error(KDB_ERR_INVALID, "null buffer");
    double l = m->p->Gradient(x, t, n, grad);
    if (loss) *loss = l;
  });
}

int kdb_mlp_train_step(kdb_mlp* m, const float* x, const float* t, int64_t n, float lr, double* loss) {
  return MGuard(m, [&] {
    if (!x || !t) throw kdb::Error(KDB_ERR_INVALID, "null buffer");
    double l = m->p->TrainStep(x, t, n, lr);
    if (loss) *loss = l;
  });
}

void kdb_mlp_free(kdb_mlp* m) { delete m; }

int kdb_ctx_set_skinner_policy(kdb_ctx* ctx, int32_t policy, kdb_mlp* prior, int32_t log_samples) {
  if (!ctx || policy < 0 || policy > 2) return KDB_ERR_INVALID;
  kdb::Context& c = *kdb_ctx_context(ctx);
  if (policy == 1 && !prior) {
    kdb_ctx_set_error(ctx, "the prior policy needs a model");
    return KDB_ERR_INVALID;
  }
  if (prior && prior->p->device() != c.device) {
    kdb_ctx_set_error(ctx, "the model lives on another device");
    return KDB_ERR_INVALID;
  }
  c.skinner_policy = policy;
  c.join_prior = prior ? prior->p.get() : nullptr;
  c.skinner_log = log_samples != 0;
  return KDB_OK;
}

}  // extern "C"
