// Batch normalisation of a row-major matrix in training, with the activation that follows it.
//
// Bound: HBM or, for the matrices of most layers (15 - 60 MB), L2.  Two passes over x forward (statistics; normalise,
// activate, store), two over x and the incoming gradient backward (column sums; input gradient), each pass one 16-byte
// vector of channels a thread with four rows in flight, backward two of x and two of the gradient; after the first pass of
// each direction a kernel of eight channels a CTA finishes the chunks' partial results.  Nothing is kept between the passes
// but the statistics: the normalised rows that the activation saw are made again from x.
//
// torch runs the two modules as three kernels forward and three backward.  The thirteen pairs of a UNet training step (two indoor
// scans of 120 000 voxels, fp16, SiLU): forward 1.68 -> 0.47 ms, backward 1.59 -> 0.73 ms.
//
// Statistics: a thread takes four rows at a time to their mean and squared deviations and merges these into its running
// pair, threads of a chunk are merged the same way (Chan, Golub, LeVeque: "Updating formulae and a pairwise algorithm for
// computing sample variances").  Of the chunks' pairs the mean of the means is taken in fp64, then the squared deviations
// within the chunks and of their means from it: no difference of large sums anywhere.
#include <algorithm>

#include "common.cuh"

namespace spc {
namespace {

constexpr int kThreads = 256;
constexpr int kAhead = 4;        // rows of a thread in flight
constexpr int kCtas = 4;         // CTAs a multiprocessor, all of them at once: a chunk each, few enough to merge in one launch
constexpr int kMostChunks = kCtas * 148;

template <typename T> struct Vec {
  static constexpr int N = 16 / sizeof(T);
  alignas(16) T v[N];
};

// 1 / (1 + exp(-z)).  For 16-bit features the reciprocal unit (1 ulp, as documented) on a quarter of the denominator, whose
// reciprocal is never below the normal numbers: 0.5 ulp more than the IEEE division at a quarter of its instructions.  The
// exponential is the accurate one: __expf's relative error grows with |z|, and with __fdividef bf16 results below z = -87.3
// came out as 0.  UNet training step 6.28 - 6.35 ms, with the IEEE division 6.60.
// Error against fp64 (2-norms; fp16 and bf16, 4 099 to 240 000 rows, 32 to 256 channels, gains of 1 and 4), this / with the IEEE
// division / of the two modules: results and input gradients the same to all digits, 2.07e-4 / 2.07e-4 / 2.7 - 3.2e-4 in fp16 and
// 1.66e-3 / 1.66e-3 / 2.1 - 2.7e-3 in bf16; the fp32 gradients of weight and bias 1.0 - 3.3e-7 / 0.9 - 3.2e-7 / 1.8 - 2.6e-4 in fp16
// and 1.3 - 2.2e-3 in bf16 for the modules, whose sums see rounded values.
template <typename T>
__device__ __forceinline__ float sigmoid(float z) {
  const float e = expf(-z);
  if (sizeof(T) != 2) return 1.f / (1.f + e);
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(fmaf(e, 0.25f, 0.25f)));
  return 0.25f * r;
}
template <typename T, int ACT>
__device__ __forceinline__ float activate(float z) {
  if (ACT == SPC_NORM_RELU) return z < 0.f ? 0.f : z;  // (NaN stays)
  if (ACT == SPC_NORM_SILU) return sizeof(T) == 2 ? z * sigmoid<T>(z) : z / (1.f + expf(-z));
  return z;
}
template <typename T, int ACT>
__device__ __forceinline__ float gradient(float z, float dy) {
  if (ACT == SPC_NORM_RELU) return z <= 0.f ? 0.f : dy;
  if (ACT == SPC_NORM_SILU) {
    const float s = sigmoid<T>(z);
    return dy * (s * (1.f + z * (1.f - s)));
  }
  return dy;
}

// Columns of a CTA: grid.y times `width` vectors; rows of a chunk are dealt to `lanes` threads a column vector.
struct Place {
  int width, lanes, cv, rl, col;
  long long lo, n;
};
template <int N>
__device__ __forceinline__ Place place(long long rows, int cols, long long chunk) {
  Place p;
  const int vecs = cols / N;
  p.width = min(vecs, kThreads);
  p.lanes = kThreads / p.width;
  p.cv = threadIdx.x % p.width;
  p.rl = threadIdx.x / p.width;
  p.col = (blockIdx.y * p.width + p.cv) * N;
  p.lo = blockIdx.x * chunk;
  p.n = min(rows - p.lo, chunk);
  if (p.rl >= p.lanes || p.col >= cols) p.n = 0;
  return p;
}

struct Moments {
  float n, mean, m2;
};
__device__ __forceinline__ void merge(Moments& a, float n, float mean, float m2) {
  if (n == 0.f) return;
  const float all = a.n + n, d = mean - a.mean, share = n / all;
  a.mean += d * share;
  a.m2 += m2 + d * d * a.n * share;
  a.n = all;
}

template <typename T>
__global__ void __launch_bounds__(kThreads, kCtas)
moments_kernel(const T* __restrict__ x, long long rows, int cols, long long chunk, float2* __restrict__ partial) {
  constexpr int N = Vec<T>::N;
  extern __shared__ float2 shared2[];  // [lanes][width * N]
  const Place p = place<N>(rows, cols, chunk);
  float n = 0.f, mean[N], m2[N];
#pragma unroll
  for (int v = 0; v < N; ++v) mean[v] = m2[v] = 0.f;
  const T* const at = x + p.lo * cols + p.col;
  long long r = p.rl;
  for (; r + (kAhead - 1) * p.lanes < p.n; r += kAhead * p.lanes) {
    Vec<T> q[kAhead];
#pragma unroll
    for (int u = 0; u < kAhead; ++u) q[u] = *reinterpret_cast<const Vec<T>*>(at + (r + u * p.lanes) * cols);
    const float share = kAhead / (n + kAhead), both = n * share;
    n += kAhead;
#pragma unroll
    for (int v = 0; v < N; ++v) {
      float f[kAhead];
#pragma unroll
      for (int u = 0; u < kAhead; ++u) f[u] = to_float(q[u].v[v]);
      const float g = 0.25f * ((f[0] + f[1]) + (f[2] + f[3]));
      float s = 0.f;
#pragma unroll
      for (int u = 0; u < kAhead; ++u) s = fmaf(f[u] - g, f[u] - g, s);
      const float d = g - mean[v];
      mean[v] = fmaf(d, share, mean[v]);
      m2[v] += fmaf(d * d, both, s);
    }
  }
  for (; r < p.n; r += p.lanes) {
    const Vec<T> q = *reinterpret_cast<const Vec<T>*>(at + r * cols);
    n += 1.f;
    const float share = 1.f / n;
#pragma unroll
    for (int v = 0; v < N; ++v) {
      const float f = to_float(q.v[v]), d = f - mean[v];
      mean[v] = fmaf(d, share, mean[v]);
      m2[v] = fmaf(d, f - mean[v], m2[v]);
    }
  }
  float* const counts = reinterpret_cast<float*>(shared2 + p.lanes * p.width * N);  // [lanes]
  if (p.rl < p.lanes) {
#pragma unroll
    for (int v = 0; v < N; ++v) shared2[(p.rl * p.width + p.cv) * N + v] = make_float2(mean[v], m2[v]);
    if (p.cv == 0) counts[p.rl] = n;
  }
  __syncthreads();
  for (int i = threadIdx.x; i < p.width * N; i += kThreads) {
    if (blockIdx.y * p.width * N + i >= cols) break;
    Moments a{0.f, 0.f, 0.f};
    for (int l = 0; l < p.lanes; ++l) {
      const float2 b = shared2[l * p.width * N + i];
      merge(a, counts[l], b.x, b.y);
    }
    partial[blockIdx.x * static_cast<long long>(cols) + blockIdx.y * p.width * N + i] = make_float2(a.mean, a.m2);
  }
}

// The finishing kernels: eight channels a CTA (64 bytes of a chunk's results), 32 threads a channel that hold the results of
// all their chunks at once, so that each kernel waits for memory once (a warp a channel, four loads ahead: 8 and 5 us).
constexpr int kFinishChannels = 8, kFinishLanes = kThreads / kFinishChannels;
constexpr int kHeld = (kMostChunks + kFinishLanes - 1) / kFinishLanes;
struct Held {
  float2 v[kHeld];
};
__device__ __forceinline__ Held held_chunks(const float2* partial, int chunks, int cols, int c, int first) {
  Held h;
#pragma unroll
  for (int i = 0; i < kHeld; ++i) {
    const int at = first + i * kFinishLanes;
    h.v[i] = at < chunks && c < cols ? __ldg(&partial[static_cast<long long>(at) * cols + c]) : make_float2(0.f, 0.f);
  }
  return h;
}
// Sum over the threads of a channel, for each of them.
__device__ __forceinline__ double channel_sum(double v) {
  __shared__ double sums[kThreads / 32][kFinishChannels];
  v += __shfl_xor_sync(0xffffffffu, v, 8);
  v += __shfl_xor_sync(0xffffffffu, v, 16);
  const int channel = threadIdx.x % kFinishChannels;
  __syncthreads();
  if ((threadIdx.x & 31) < kFinishChannels) sums[threadIdx.x >> 5][channel] = v;
  __syncthreads();
  double all = 0.;
#pragma unroll
  for (int w = 0; w < kThreads / 32; ++w) all += sums[w][channel];
  return all;
}

// The mean of the chunks' means, then their squared deviations and those of their means from it, in fp64; kept in fp32 as
// the user's running ones are.
__global__ void __launch_bounds__(kThreads)
finish_moments_kernel(const float2* __restrict__ partial, int chunks, long long chunk, long long rows, int cols, float eps, float momentum,
                      float* __restrict__ save_mean, float* __restrict__ save_invstd, float* __restrict__ running_mean,
                      float* __restrict__ running_var, long long* __restrict__ batches) {
  const int c = blockIdx.x * kFinishChannels + threadIdx.x % kFinishChannels, lane = threadIdx.x / kFinishChannels;
  if (blockIdx.x == 0 && threadIdx.x == 0 && batches != nullptr) *batches += 1;
  const Held h = held_chunks(partial, chunks, cols, c, lane);
  const double n = static_cast<double>(rows);
  const auto size = [&](int i) {
    const int at = lane + i * kFinishLanes;
    return at < chunks ? static_cast<double>(min(chunk, rows - at * chunk)) : 0.;
  };
  double sum = 0.;
#pragma unroll
  for (int i = 0; i < kHeld; ++i) sum += size(i) * h.v[i].x;
  const double mean = channel_sum(sum) / n;
  double m2 = 0.;
#pragma unroll
  for (int i = 0; i < kHeld; ++i) {
    const double d = h.v[i].x - mean;
    m2 += h.v[i].y + size(i) * d * d;
  }
  m2 = channel_sum(m2);
  if (lane != 0 || c >= cols) return;
  const double var = m2 / n;
  save_mean[c] = static_cast<float>(mean);
  save_invstd[c] = static_cast<float>(1. / sqrt(var + static_cast<double>(eps)));
  if (running_mean != nullptr) {
    running_mean[c] = (1.f - momentum) * running_mean[c] + momentum * static_cast<float>(mean);
    running_var[c] = (1.f - momentum) * running_var[c] + momentum * static_cast<float>(m2 / (n - 1.));
  }
}

template <int N>
struct Channel {
  float mean[N], gain[N], shift[N];
};
template <int N>
__device__ __forceinline__ Channel<N> channel(const float* mean, const float* invstd, const float* weight, const float* bias, int col) {
  Channel<N> c;
#pragma unroll
  for (int v = 0; v < N; ++v) {
    c.mean[v] = __ldg(mean + col + v);
    c.gain[v] = __ldg(invstd + col + v) * (weight != nullptr ? __ldg(weight + col + v) : 1.f);
    c.shift[v] = bias != nullptr ? __ldg(bias + col + v) : 0.f;
  }
  return c;
}

template <typename T, int ACT>
__global__ void __launch_bounds__(kThreads, kCtas)
normalize_kernel(const T* __restrict__ x, const float* __restrict__ mean, const float* __restrict__ invstd, const float* __restrict__ weight,
                 const float* __restrict__ bias, long long rows, int cols, long long chunk, T* __restrict__ y) {
  constexpr int N = Vec<T>::N;
  const Place p = place<N>(rows, cols, chunk);
  if (p.n <= p.rl) return;
  const Channel<N> c = channel<N>(mean, invstd, weight, bias, p.col);
  const T* const from = x + p.lo * cols + p.col;
  T* const to = y + p.lo * cols + p.col;
  const auto one = [&](const Vec<T>& q, long long r) {
    Vec<T> o;
#pragma unroll
    for (int v = 0; v < N; ++v) o.v[v] = from_float<T>(activate<T, ACT>(fmaf(to_float(q.v[v]) - c.mean[v], c.gain[v], c.shift[v])));
    *reinterpret_cast<Vec<T>*>(to + r * cols) = o;
  };
  long long r = p.rl;
  for (; r + (kAhead - 1) * p.lanes < p.n; r += kAhead * p.lanes) {
    Vec<T> q[kAhead];
#pragma unroll
    for (int u = 0; u < kAhead; ++u) q[u] = *reinterpret_cast<const Vec<T>*>(from + (r + u * p.lanes) * cols);
#pragma unroll
    for (int u = 0; u < kAhead; ++u) one(q[u], r + u * p.lanes);
  }
  for (; r < p.n; r += p.lanes) one(*reinterpret_cast<const Vec<T>*>(from + r * cols), r);
}

// Per chunk and channel: sum of dz and of dz (x - mean), dz the gradient at the normalisation's output.
template <typename T, int ACT>
__global__ void __launch_bounds__(kThreads, kCtas)
gradient_sums_kernel(const T* __restrict__ x, const T* __restrict__ dy, const float* __restrict__ mean, const float* __restrict__ invstd,
                     const float* __restrict__ weight, const float* __restrict__ bias, long long rows, int cols, long long chunk,
                     float2* __restrict__ partial) {
  constexpr int N = Vec<T>::N, AHEAD = 2;
  extern __shared__ float2 shared2[];
  const Place p = place<N>(rows, cols, chunk);
  float s0[N], s1[N];
#pragma unroll
  for (int v = 0; v < N; ++v) s0[v] = s1[v] = 0.f;
  if (p.n > p.rl) {
    const Channel<N> c = channel<N>(mean, invstd, weight, bias, p.col);
    const T* const from = x + p.lo * cols + p.col;
    const T* const grad = dy + p.lo * cols + p.col;
    const auto one = [&](const Vec<T>& q, const Vec<T>& g) {
#pragma unroll
      for (int v = 0; v < N; ++v) {
        const float d = to_float(q.v[v]) - c.mean[v];
        const float dz = gradient<T, ACT>(fmaf(d, c.gain[v], c.shift[v]), to_float(g.v[v]));
        s0[v] += dz;
        s1[v] = fmaf(dz, d, s1[v]);
      }
    };
    long long r = p.rl;
    for (; r + (AHEAD - 1) * p.lanes < p.n; r += AHEAD * p.lanes) {
      Vec<T> q[AHEAD], g[AHEAD];
#pragma unroll
      for (int u = 0; u < AHEAD; ++u) {
        q[u] = *reinterpret_cast<const Vec<T>*>(from + (r + u * p.lanes) * cols);
        g[u] = *reinterpret_cast<const Vec<T>*>(grad + (r + u * p.lanes) * cols);
      }
#pragma unroll
      for (int u = 0; u < AHEAD; ++u) one(q[u], g[u]);
    }
    for (; r < p.n; r += p.lanes) one(*reinterpret_cast<const Vec<T>*>(from + r * cols), *reinterpret_cast<const Vec<T>*>(grad + r * cols));
  }
  if (p.rl < p.lanes)
#pragma unroll
    for (int v = 0; v < N; ++v) shared2[(p.rl * p.width + p.cv) * N + v] = make_float2(s0[v], s1[v]);
  __syncthreads();
  for (int i = threadIdx.x; i < p.width * N; i += kThreads) {
    if (blockIdx.y * p.width * N + i >= cols) break;
    float a = 0.f, b = 0.f;
    for (int l = 0; l < p.lanes; ++l) {
      const float2 q = shared2[l * p.width * N + i];
      a += q.x;
      b += q.y;
    }
    partial[blockIdx.x * static_cast<long long>(cols) + blockIdx.y * p.width * N + i] = make_float2(a, b);
  }
}

__global__ void __launch_bounds__(kThreads)
finish_sums_kernel(const float2* __restrict__ partial, int chunks, long long rows, int cols, const float* __restrict__ invstd,
                   float* __restrict__ dweight, float* __restrict__ dbias, float2* __restrict__ means) {
  const int c = blockIdx.x * kFinishChannels + threadIdx.x % kFinishChannels, lane = threadIdx.x / kFinishChannels;
  const Held h = held_chunks(partial, chunks, cols, c, lane);
  double a = 0., b = 0.;
#pragma unroll
  for (int i = 0; i < kHeld; ++i) {
    a += h.v[i].x;
    b += h.v[i].y;
  }
  a = channel_sum(a);
  b = channel_sum(b);
  if (lane != 0 || c >= cols) return;
  const double inv = invstd[c];
  if (dweight != nullptr) dweight[c] = static_cast<float>(b * inv);
  if (dbias != nullptr) dbias[c] = static_cast<float>(a);
  means[c] = make_float2(static_cast<float>(a / rows), static_cast<float>(b * inv * inv / rows));
}

template <typename T, int ACT>
__global__ void __launch_bounds__(kThreads, kCtas)
input_gradient_kernel(const T* __restrict__ x, const T* __restrict__ dy, const float* __restrict__ mean, const float* __restrict__ invstd,
                      const float* __restrict__ weight, const float* __restrict__ bias, const float2* __restrict__ means, long long rows,
                      int cols, long long chunk, T* __restrict__ dx) {
  constexpr int N = Vec<T>::N, AHEAD = 2;
  const Place p = place<N>(rows, cols, chunk);
  if (p.n <= p.rl) return;
  const Channel<N> c = channel<N>(mean, invstd, weight, bias, p.col);
  float m0[N], m1[N];
#pragma unroll
  for (int v = 0; v < N; ++v) {
    const float2 m = __ldg(means + p.col + v);
    m0[v] = m.x;
    m1[v] = m.y;
  }
  const T* const from = x + p.lo * cols + p.col;
  const T* const grad = dy + p.lo * cols + p.col;
  T* const to = dx + p.lo * cols + p.col;
  const auto one = [&](const Vec<T>& q, const Vec<T>& g, long long r) {
    Vec<T> o;
#pragma unroll
    for (int v = 0; v < N; ++v) {
      const float d = to_float(q.v[v]) - c.mean[v];
      const float dz = gradient<T, ACT>(fmaf(d, c.gain[v], c.shift[v]), to_float(g.v[v]));
      o.v[v] = from_float<T>((dz - m0[v] - d * m1[v]) * c.gain[v]);
    }
    *reinterpret_cast<Vec<T>*>(to + r * cols) = o;
  };
  long long r = p.rl;
  for (; r + (AHEAD - 1) * p.lanes < p.n; r += AHEAD * p.lanes) {
    Vec<T> q[AHEAD], g[AHEAD];
#pragma unroll
    for (int u = 0; u < AHEAD; ++u) {
      q[u] = *reinterpret_cast<const Vec<T>*>(from + (r + u * p.lanes) * cols);
      g[u] = *reinterpret_cast<const Vec<T>*>(grad + (r + u * p.lanes) * cols);
    }
#pragma unroll
    for (int u = 0; u < AHEAD; ++u) one(q[u], g[u], r + u * p.lanes);
  }
  for (; r < p.n; r += p.lanes)
    one(*reinterpret_cast<const Vec<T>*>(from + r * cols), *reinterpret_cast<const Vec<T>*>(grad + r * cols), r);
}

// Evaluation mode: scale and shift for the store of the GEMM before the normalisation.  Latency of one launch (2 us), a CTA a
// normalisation; made for each pass, so that nobody has to notice when the statistics change.
constexpr int kMostFolds = 48;  // a launch's parameters are at most 4 KB
struct Folds {
  spc_norm_fold of[kMostFolds];
};
__device__ __forceinline__ float value_at(const void* p, int type, int c) {
  if (type == SPC_F16) return to_float(static_cast<const __half*>(p)[c]);
  if (type == SPC_BF16) return to_float(static_cast<const __nv_bfloat16*>(p)[c]);
  return static_cast<const float*>(p)[c];
}
__global__ void __launch_bounds__(kThreads)
fold_norms_kernel(const __grid_constant__ Folds folds) {
  const spc_norm_fold& f = folds.of[blockIdx.x];
  for (int c = threadIdx.x; c < f.channels; c += kThreads) {
    float scale = rsqrtf(value_at(f.var, f.types[1], c) + f.eps);
    if (f.weight != nullptr) scale *= value_at(f.weight, f.types[2], c);
    // (rounded after each step, as torch's functions of these tensors round)
    float shift = __fmul_rn(-value_at(f.mean, f.types[0], c), scale);
    if (f.bias != nullptr) shift = __fadd_rn(shift, value_at(f.bias, f.types[3], c));
    f.scale[c] = scale;
    f.shift[c] = shift;
  }
}

struct Plan {
  int chunks, across, lanes;  // chunks of rows, CTAs across the columns, threads a column vector
  long long chunk;
  size_t shared;
};
Plan plan(long long rows, int cols, int dtype) {
  Plan p;
  const int n = static_cast<int>(16 / dtype_size(dtype)), vecs = cols / n, width = std::min(vecs, kThreads);
  p.lanes = kThreads / width;
  p.across = (vecs + width - 1) / width;
  // a chunk gives each thread four rows at least; no more chunks than the chip holds CTAs
  const long long most = std::max(1, kMostChunks / p.across);
  p.chunk = std::max<long long>(static_cast<long long>(p.lanes) * kAhead, ceil_div(rows, most));
  p.chunks = static_cast<int>(ceil_div(rows, p.chunk));
  p.shared = static_cast<size_t>(p.lanes) * width * n * sizeof(float2) + p.lanes * sizeof(float);
  return p;
}

bool takes(int64_t rows, int cols, int dtype) {
  if (rows < 2 || cols <= 0 || (dtype != SPC_F16 && dtype != SPC_BF16 && dtype != SPC_F32)) return false;
  return cols % static_cast<int>(16 / dtype_size(dtype)) == 0 && cols <= 4096;
}
bool aligned(const void* a, const void* b, const void* c) {
  return ((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(b) | reinterpret_cast<uintptr_t>(c)) & 15u) == 0;
}

template <typename T, int ACT>
int forward(const void* x, const float* weight, const float* bias, float* running_mean, float* running_var, long long* batches, float momentum,
            float eps, void* y, float* save_mean, float* save_invstd, void* workspace, long long rows, int cols, int dtype, cudaStream_t st) {
  const Plan p = plan(rows, cols, dtype);
  float2* const partial = static_cast<float2*>(workspace);
  const dim3 grid(p.chunks, p.across);
  moments_kernel<T><<<grid, kThreads, p.shared, st>>>(static_cast<const T*>(x), rows, cols, p.chunk, partial);
  SPC_LAUNCH_OK();
  finish_moments_kernel<<<static_cast<unsigned>(ceil_div(cols, kFinishChannels)), kThreads, 0, st>>>(
      partial, p.chunks, p.chunk, rows, cols, eps, momentum, save_mean, save_invstd, running_mean, running_var, batches);
  SPC_LAUNCH_OK();
  normalize_kernel<T, ACT><<<grid, kThreads, 0, st>>>(static_cast<const T*>(x), save_mean, save_invstd, weight, bias, rows, cols, p.chunk,
                                                      static_cast<T*>(y));
  SPC_LAUNCH_OK();
  return SPC_OK;
}

template <typename T, int ACT>
int backward(const void* x, const void* dy, const float* weight, const float* bias, const float* save_mean, const float* save_invstd, void* dx,
             float* dweight, float* dbias, void* workspace, long long rows, int cols, int dtype, cudaStream_t st) {
  const Plan p = plan(rows, cols, dtype);
  float2* const partial = static_cast<float2*>(workspace);
  float2* const means = partial + static_cast<size_t>(p.chunks) * cols;
  const dim3 grid(p.chunks, p.across);
  gradient_sums_kernel<T, ACT><<<grid, kThreads, p.shared, st>>>(static_cast<const T*>(x), static_cast<const T*>(dy), save_mean, save_invstd,
                                                                 weight, bias, rows, cols, p.chunk, partial);
  SPC_LAUNCH_OK();
  finish_sums_kernel<<<static_cast<unsigned>(ceil_div(cols, kFinishChannels)), kThreads, 0, st>>>(partial, p.chunks, rows, cols, save_invstd,
                                                                                               dweight, dbias, means);
  SPC_LAUNCH_OK();
  if (dx == nullptr) return SPC_OK;
  input_gradient_kernel<T, ACT><<<grid, kThreads, 0, st>>>(static_cast<const T*>(x), static_cast<const T*>(dy), save_mean, save_invstd, weight,
                                                           bias, means, rows, cols, p.chunk, static_cast<T*>(dx));
  SPC_LAUNCH_OK();
  return SPC_OK;
}

}  // namespace
}  // namespace spc

using namespace spc;

extern "C" size_t spc_norm_act_workspace_bytes(int64_t rows, int cols, int dtype) {
  if (!takes(rows, cols, dtype)) return 0;
  return (static_cast<size_t>(plan(rows, cols, dtype).chunks) + 1) * cols * sizeof(float2);
}

extern "C" int spc_fold_norms(const spc_norm_fold* norms, int n, void* stream) {
  if (norms == nullptr || n < 0) return fail(SPC_ERR_INVALID_ARGUMENT, "fold_norms: bad arguments");
  for (int i = 0; i < n; ++i) {
    const spc_norm_fold& f = norms[i];
    if (!f.mean || !f.var || !f.scale || !f.shift || f.channels <= 0) return fail(SPC_ERR_INVALID_ARGUMENT, "fold_norms: bad arguments");
    for (int t : f.types)
      if (t != SPC_F16 && t != SPC_BF16 && t != SPC_F32) return fail(SPC_ERR_UNSUPPORTED, "fold_norms: unsupported dtype");
  }
  for (int first = 0; first < n; first += kMostFolds) {
    Folds folds{};
    const int count = std::min(n - first, kMostFolds);
    std::copy(norms + first, norms + first + count, folds.of);
    fold_norms_kernel<<<count, kThreads, 0, static_cast<cudaStream_t>(stream)>>>(folds);
    SPC_LAUNCH_OK();
  }
  return SPC_OK;
}

#define SPC_NORM_TYPES(CALL)                                                      \
  switch (dtype) {                                                                \
    case SPC_F16: SPC_NORM_ACTS(CALL, __half);                                    \
    case SPC_BF16: SPC_NORM_ACTS(CALL, __nv_bfloat16);                            \
    default: SPC_NORM_ACTS(CALL, float);                                          \
  }
#define SPC_NORM_ACTS(CALL, T)                                                    \
  return act == SPC_NORM_SILU ? CALL(T, SPC_NORM_SILU) : act == SPC_NORM_RELU ? CALL(T, SPC_NORM_RELU) : CALL(T, SPC_NORM_NONE)

extern "C" int spc_norm_act_forward(const void* x, const float* weight, const float* bias, float* running_mean, float* running_var,
                                    int64_t* batches, float momentum, float eps, int act, void* y, float* save_mean, float* save_invstd,
                                    void* workspace, size_t workspace_bytes, int64_t rows, int cols, int dtype, void* stream) {
  if (!x || !y || !save_mean || !save_invstd || !workspace || (running_mean == nullptr) != (running_var == nullptr) || act < SPC_NORM_NONE ||
      act > SPC_NORM_SILU)
    return fail(SPC_ERR_INVALID_ARGUMENT, "norm_act_forward: bad arguments");
  if (!takes(rows, cols, dtype) || !aligned(x, y, workspace)) return fail(SPC_ERR_UNSUPPORTED, "norm_act_forward: unsupported shape, dtype or alignment");
  if (workspace_bytes < spc_norm_act_workspace_bytes(rows, cols, dtype)) return fail(SPC_ERR_WORKSPACE_TOO_SMALL, "norm_act_forward: workspace");
#define SPC_CALL(T, A)                                                                                                                   \
  (forward<T, A>(x, weight, bias, running_mean, running_var, reinterpret_cast<long long*>(batches), momentum, eps, y, save_mean, save_invstd, \
                 workspace, rows, cols, dtype, static_cast<cudaStream_t>(stream)))
  SPC_NORM_TYPES(SPC_CALL)
#undef SPC_CALL
}

extern "C" int spc_norm_act_backward(const void* x, const void* dy, const float* weight, const float* bias, const float* save_mean,
                                     const float* save_invstd, int act, void* dx, float* dweight, float* dbias, void* workspace,
                                     size_t workspace_bytes, int64_t rows, int cols, int dtype, void* stream) {
  if (!x || !dy || !save_mean || !save_invstd || !workspace || act < SPC_NORM_NONE || act > SPC_NORM_SILU)
    return fail(SPC_ERR_INVALID_ARGUMENT, "norm_act_backward: bad arguments");
  if (!takes(rows, cols, dtype) || !aligned(x, dy, workspace) || !aligned(dx, nullptr, nullptr))
    return fail(SPC_ERR_UNSUPPORTED, "norm_act_backward: unsupported shape, dtype or alignment");
  if (workspace_bytes < spc_norm_act_workspace_bytes(rows, cols, dtype)) return fail(SPC_ERR_WORKSPACE_TOO_SMALL, "norm_act_backward: workspace");
#define SPC_CALL(T, A)                                                                                                                       \
  (backward<T, A>(x, dy, weight, bias, save_mean, save_invstd, dx, dweight, dbias, workspace, rows, cols, dtype, static_cast<cudaStream_t>(stream)))
  SPC_NORM_TYPES(SPC_CALL)
#undef SPC_CALL
}
