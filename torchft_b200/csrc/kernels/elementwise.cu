// Bandwidth-bound training kernels: SwiGLU, fused softmax cross-entropy (loss and
// gradient in one kernel), embedding gather / scatter-add, fused AdamW, and the DiLoCo
// outer step (pseudo-gradient, Nesterov update).  One pass over memory each, 16-byte
// vector accesses, fp32 math.
#include "common.cuh"

#include <cfloat>

namespace tft {

__device__ __forceinline__ void ew_unpack8(const uint4& u, float (&f)[8]) {
  const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&u);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    float2 t = __bfloat1622float2(h[i]);
    f[2 * i] = t.x;
    f[2 * i + 1] = t.y;
  }
}
__device__ __forceinline__ uint4 ew_pack8(const float (&f)[8]) {
  uint4 u;
  u.x = pack_bf16(f[0], f[1]);
  u.y = pack_bf16(f[2], f[3]);
  u.z = pack_bf16(f[4], f[5]);
  u.w = pack_bf16(f[6], f[7]);
  return u;
}

// ------------------------------------------------------------------ SwiGLU
// gu: [rows, 2*F] with the gate in columns [0,F) and the up projection in [F,2F).
__global__ void swiglu_fwd_kernel(const __nv_bfloat16* __restrict__ gu, __nv_bfloat16* __restrict__ out,
                                  long long rows, int F) {
  const int vec_per_row = F / 8;
  const long long total = rows * vec_per_row;
  for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < total;
       i += static_cast<long long>(gridDim.x) * blockDim.x) {
    const long long r = i / vec_per_row;
    const int c = static_cast<int>(i % vec_per_row) * 8;
    float g[8], u[8], o[8];
    ew_unpack8(*reinterpret_cast<const uint4*>(gu + r * 2 * F + c), g);
    ew_unpack8(*reinterpret_cast<const uint4*>(gu + r * 2 * F + F + c), u);
#pragma unroll
    for (int j = 0; j < 8; ++j) o[j] = g[j] / (1.f + __expf(-g[j])) * u[j];
    *reinterpret_cast<uint4*>(out + r * F + c) = ew_pack8(o);
  }
}

// dgu[:, :F] = dout * u * d silu(g);  dgu[:, F:] = dout * silu(g)
__global__ void swiglu_bwd_kernel(const __nv_bfloat16* __restrict__ gu, const __nv_bfloat16* __restrict__ dout,
                                  __nv_bfloat16* __restrict__ dgu, long long rows, int F) {
  const int vec_per_row = F / 8;
  const long long total = rows * vec_per_row;
  for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < total;
       i += static_cast<long long>(gridDim.x) * blockDim.x) {
    const long long r = i / vec_per_row;
    const int c = static_cast<int>(i % vec_per_row) * 8;
    float g[8], u[8], d[8], dg[8], du[8];
    ew_unpack8(*reinterpret_cast<const uint4*>(gu + r * 2 * F + c), g);
    ew_unpack8(*reinterpret_cast<const uint4*>(gu + r * 2 * F + F + c), u);
    ew_unpack8(*reinterpret_cast<const uint4*>(dout + r * F + c), d);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float s = 1.f / (1.f + __expf(-g[j]));
      const float silu = g[j] * s;
      du[j] = d[j] * silu;
      dg[j] = d[j] * u[j] * (s + silu * (1.f - s));
    }
    *reinterpret_cast<uint4*>(dgu + r * 2 * F + c) = ew_pack8(dg);
    *reinterpret_cast<uint4*>(dgu + r * 2 * F + F + c) = ew_pack8(du);
  }
}

// ------------------------------------------------------------------ cross entropy
// logits <- (softmax - onehot) * grad_scale, loss[row] = lse - z_target.  Rows whose target is ignore_index produce
// zero loss and zero gradient.
//
// Two kernels.  Rows of up to 32768 columns stay in the registers of one block between the two passes, eight 16-byte
// vectors a thread (xent_row_kernel).  Longer rows are read twice, the second time partly from L2 (xent_kernel): holding
// them in the registers of a cluster of CTAs reads memory once but costs a cluster barrier a row, and took 311 to 430 us
// where the two passes took 205 (2048 x 128256).
constexpr int XENT_VECS = 8;
constexpr int XENT_THREADS = 512;
constexpr int XENT_ROOM = XENT_THREADS * XENT_VECS;  // vectors of a row that one block takes

// Maximum and sum of exp(x - m) of a part of a row.  The maximum starts at the lowest finite number, so that differences from it
// are never those of two infinities: a part that is empty or all -inf has the sum 0.  The maximum passes over NaN and the sum
// does not, so NaN makes the row's loss and gradient NaN; +inf does too, and a row of nothing but -inf.
struct MaxSum {
  float m, s;
};
__device__ __forceinline__ MaxSum empty_part() { return {-FLT_MAX, 0.f}; }
__device__ __forceinline__ MaxSum combine(const MaxSum& a, const MaxSum& b) {
  MaxSum r;
  r.m = fmaxf(a.m, b.m);
  r.s = a.s * __expf(a.m - r.m) + b.s * __expf(b.m - r.m);
  return r;
}
__device__ __forceinline__ MaxSum warp_combine(MaxSum v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    MaxSum w;
    w.m = __shfl_xor_sync(0xffffffffu, v.m, o);
    w.s = __shfl_xor_sync(0xffffffffu, v.s, o);
    v = combine(v, w);
  }
  return v;
}

// Eight softmax values times the gradient's scale: exp(f - m) * unit with the row's maximum m and unit = scale / s.  Differences
// from the maximum are exact where they count, whatever the size of the logits.  From the log-sum-exp, which is rounded to the
// size of the maximum, exp(f - lse) is off by up to 3 % at logits of 1e6, and lse * log2(e) overflows in rows of the type's
// lowest value.  Two values at a time but for the exponential: both kernels are close to their issue rate here.
constexpr float kLog2e = 1.4426950408889634f;
__device__ __forceinline__ uint4 xent_grad(const uint4& u, float m, float unit) {
  float f[8];
  ew_unpack8(u, f);
  const float2 less_m = make_float2(-m, -m), log2e = make_float2(kLog2e, kLog2e), units = make_float2(unit, unit);
#pragma unroll
  for (int j = 0; j < 8; j += 2) {
    const float2 t = __fmul2_rn(__fadd2_rn(make_float2(f[j], f[j + 1]), less_m), log2e);
    const float2 g = __fmul2_rn(make_float2(exp2f(t.x), exp2f(t.y)), units);
    f[j] = g.x;
    f[j + 1] = g.y;
  }
  return ew_pack8(f);
}

// The target's part, left to the thread that writes the target's vector: it reads the logit before the gradient goes over it
// and takes 1 from the softmax there afterwards.  The vectors are stored as another type than the one element, so both
// accesses are fenced off from them for the compiler.
__device__ __forceinline__ float xent_target_logit(const __nv_bfloat16* at) {
  const float hot = __bfloat162float(*at);
  asm volatile("" ::: "memory");
  return hot;
}
__device__ __forceinline__ void xent_target(__nv_bfloat16* at, float hot, const MaxSum& r, float unit, float* loss) {
  asm volatile("" ::: "memory");
  *loss = (r.m - hot) + __logf(r.s);
  *at = __float2bfloat16((__expf(hot - r.m) - r.s) * unit);
}

// One block per row, as few threads as hold it: short rows then share an SM with more of their kind.  Bound by the launch
// below a few thousand rows; 10.5 us for 26 with two passes at 2048 x 4096, 25.7 for 63.8 at 4096 x 8192, 5.8 for 12.6 at
// 1024 x 1000, 213 for 282 at 8192 x 32000 (logits left in L2 by the call before where they fit).
__global__ void __launch_bounds__(XENT_THREADS, 2)
xent_row_kernel(__nv_bfloat16* __restrict__ logits, const long long* __restrict__ targets, float* __restrict__ loss, int V,
                int ld, float grad_scale, long long ignore_index) {
  __shared__ MaxSum part[32];  // one per warp
  const size_t row = blockIdx.x;
  const int n = V / 8, step = blockDim.x;
  uint4* z = reinterpret_cast<uint4*>(logits + row * ld) + threadIdx.x;
  const long long tgt = targets[row];
  const bool ignored = tgt == ignore_index || tgt < 0 || tgt >= V;
  const bool mine = !ignored && static_cast<int>(tgt) / 8 % step == static_cast<int>(threadIdx.x);
  const float hot = mine ? xent_target_logit(logits + row * ld + tgt) : 0.f;
  uint4 v[XENT_VECS];
#pragma unroll
  for (int k = 0; k < XENT_VECS; ++k)
    v[k] = static_cast<int>(threadIdx.x) + k * step < n ? z[k * step] : make_uint4(0xFF80FF80u, 0xFF80FF80u, 0xFF80FF80u, 0xFF80FF80u);  // -inf
  MaxSum r = empty_part();
#pragma unroll
  for (int k = 0; k < XENT_VECS; ++k) {
    float f[8];
    ew_unpack8(v[k], f);
#pragma unroll
    for (int j = 0; j < 8; ++j) r.m = fmaxf(r.m, f[j]);
  }
#pragma unroll
  for (int k = 0; k < XENT_VECS; ++k) {
    float f[8];
    ew_unpack8(v[k], f);
#pragma unroll
    for (int j = 0; j < 8; ++j) r.s += __expf(f[j] - r.m);
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
  r = warp_combine(r);
  if (warps > 1) {
    if (lane == 0) part[warp] = r;
    __syncthreads();
    r = warp_combine(lane < warps ? part[lane] : empty_part());
  }
  const float unit = (ignored ? 0.f : grad_scale) / r.s;
#pragma unroll
  for (int k = 0; k < XENT_VECS; ++k, z += step) {
    if (static_cast<int>(threadIdx.x) + k * step >= n) break;
    *z = xent_grad(v[k], r.m, unit);
  }
  if (mine) xent_target(logits + row * ld + tgt, hot, r, unit, loss + row);
  if (ignored && threadIdx.x == 0) loss[row] = 0.f;
}

// Pass 1: online maximum and sum of exponentials.  Pass 2 (in place): the gradient.  Two vectors a thread and round in flight,
// two blocks of 1024 per SM: 200 us at 2048 x 128256 (158 for one read and one write at the copy bandwidth), 241 with one.
// Four vectors and half the threads, or one block per SM, cost 5 % more.  With the target's element picked out inside the
// second loop the kernel spills at its 32 registers: 213.
constexpr int XENT_LONG_THREADS = 1024;
constexpr int XENT_LONG_VECS = 2;
__global__ void __launch_bounds__(XENT_LONG_THREADS, 2)
xent_kernel(__nv_bfloat16* __restrict__ logits, const long long* __restrict__ targets, float* __restrict__ loss, int V, int ld,
            float grad_scale, long long ignore_index) {
  __shared__ MaxSum part[32];
  constexpr int U = XENT_LONG_VECS, STEP = XENT_LONG_THREADS;
  const size_t row = blockIdx.x;
  const int n = V / 8;
  uint4* z = reinterpret_cast<uint4*>(logits + row * ld);
  const long long tgt = targets[row];
  const bool ignored = tgt == ignore_index || tgt < 0 || tgt >= V;
  const bool mine = !ignored && static_cast<int>(tgt) / 8 % STEP == static_cast<int>(threadIdx.x);
  const float hot = mine ? xent_target_logit(logits + row * ld + tgt) : 0.f;
  MaxSum r = empty_part();
  for (int i0 = threadIdx.x; i0 < n; i0 += U * STEP) {
    uint4 v[U];
#pragma unroll
    for (int u = 0; u < U; ++u)
      v[u] = i0 + u * STEP < n ? z[i0 + u * STEP] : make_uint4(0xFF80FF80u, 0xFF80FF80u, 0xFF80FF80u, 0xFF80FF80u);  // -inf
    float m = r.m;
#pragma unroll
    for (int u = 0; u < U; ++u) {
      float f[8];
      ew_unpack8(v[u], f);
#pragma unroll
      for (int j = 0; j < 8; ++j) m = fmaxf(m, f[j]);
    }
    float s = 0.f;
#pragma unroll
    for (int u = 0; u < U; ++u) {
      float f[8];
      ew_unpack8(v[u], f);
#pragma unroll
      for (int j = 0; j < 8; ++j) s += __expf(f[j] - m);
    }
    r.s = r.s * __expf(r.m - m) + s;
    r.m = m;
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  r = warp_combine(r);
  if (lane == 0) part[warp] = r;
  __syncthreads();
  r = warp_combine(part[lane]);
  const float unit = (ignored ? 0.f : grad_scale) / r.s;
  for (int i0 = threadIdx.x; i0 < n; i0 += U * STEP) {
    uint4 v[U];
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (i0 + u * STEP < n) v[u] = z[i0 + u * STEP];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int i = i0 + u * STEP;
      if (i < n) z[i] = xent_grad(v[u], r.m, unit);
    }
  }
  if (mine) xent_target(logits + row * ld + tgt, hot, r, unit, loss + row);
  if (ignored && threadIdx.x == 0) loss[row] = 0.f;
}

// ------------------------------------------------------------------ embedding
__global__ void embedding_fwd_kernel(const long long* __restrict__ tokens, const __nv_bfloat16* __restrict__ table,
                                     __nv_bfloat16* __restrict__ out, long long n_tokens, int dim) {
  const int vec = dim / 8;
  const long long total = n_tokens * vec;
  for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < total;
       i += static_cast<long long>(gridDim.x) * blockDim.x) {
    const long long t = i / vec;
    const int c = static_cast<int>(i % vec);
    reinterpret_cast<uint4*>(out + t * dim)[c] = reinterpret_cast<const uint4*>(table + tokens[t] * dim)[c];
  }
}

// dtable[tokens[t], :] += dout[t, :]   (bf16x2 atomics; dtable must be zeroed or hold earlier grads)
__global__ void embedding_bwd_kernel(const long long* __restrict__ tokens, const __nv_bfloat16* __restrict__ dout,
                                     __nv_bfloat16* __restrict__ dtable, long long n_tokens, int dim) {
  const int pairs = dim / 2;
  const long long total = n_tokens * pairs;
  for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < total;
       i += static_cast<long long>(gridDim.x) * blockDim.x) {
    const long long t = i / pairs;
    const int c = static_cast<int>(i % pairs);
    const __nv_bfloat162 v = reinterpret_cast<const __nv_bfloat162*>(dout + t * dim)[c];
    atomicAdd(reinterpret_cast<__nv_bfloat162*>(dtable + tokens[t] * dim) + c, v);
  }
}

// ------------------------------------------------------------------ tables of tensors
// Index of the tensor that chunk `c` belongs to: first[t] <= c < first[t + 1].
__device__ __forceinline__ int table_find(const int* first, int count, int c) {
  int lo = 0, hi = count - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (first[mid] <= c) lo = mid; else hi = mid - 1;
  }
  return lo;
}

// ------------------------------------------------------------------ AdamW
// p (bf16) updated in place from g (bf16) with fp32 moments; decoupled weight decay.
// bc1 = 1 - beta1^t, bc2 = 1 - beta2^t.  grad_scale multiplies g first (1/accumulation steps).
// One launch for up to kAdamMax tensors without memory in common, whose addresses travel as an argument; a block handles one
// chunk of one tensor.
// Bound by HBM: 22 bytes a parameter.  The launch for every tensor that this replaces cost a model of small tensors more
// than the update (see tft_adamw_multi).
constexpr int kAdamMax = 80;
constexpr int kAdamThreads = 256;
constexpr long long kAdamSmall = 1 << 23;  // elements of a lone tensor up to which <1, 1> is used

// A table of up to MAX tensors; a block takes VECS vectors of 8 elements per thread.  Two instances: <kAdamMax, 2>, and <1, 1>
// for a lone tensor of few elements, where one trip to memory behind another and the long argument are most of the time:
// 2.0 us for 2.9 at 4096 elements, 2.3 for 3.1 at 100 000, 8.9 for 9.8 at 3 million, 21.1 for 22.2 at 8.  From 16 on both move 6.3
// TB/s and more.
template <int MAX, int VECS>
struct AdamTable {
  static constexpr int kMax = MAX, kVecs = VECS, kChunk = kAdamThreads * 8 * VECS;  // elements per block
  __nv_bfloat16* p[MAX];
  const __nv_bfloat16* g[MAX];
  float* m[MAX];
  float* v[MAX];
  long long n[MAX];
  int first[MAX + 1];  // first chunk of every tensor; first[count] chunks in all
  int count;
};
struct AdamArgs {
  float lr, b1, b2, eps, wd, inv_bc1, inv_sqrt_bc2, grad_scale;
};
__device__ __forceinline__ void adamw_one(const AdamArgs& a, float& p, float g, float& m, float& v) {
  const float gr = g * a.grad_scale;
  m = a.b1 * m + (1.f - a.b1) * gr;
  v = a.b2 * v + (1.f - a.b2) * gr * gr;
  const float denom = sqrtf(v) * a.inv_sqrt_bc2 + a.eps;
  p = p * (1.f - a.lr * a.wd) - a.lr * (m * a.inv_bc1) / denom;
}

template <typename Table>
__global__ void __launch_bounds__(kAdamThreads)
adamw_kernel(const __grid_constant__ Table tab, const AdamArgs a) {
  const int t = Table::kMax == 1 ? 0 : table_find(tab.first, tab.count, blockIdx.x);
  __nv_bfloat16* p = tab.p[t];
  const __nv_bfloat16* g = tab.g[t];
  float *m = tab.m[t], *v = tab.v[t];
  const long long n = tab.n[t], e0 = static_cast<long long>(blockIdx.x - tab.first[t]) * Table::kChunk;
  const long long nvec = n / 8;
#pragma unroll
  for (int k = 0; k < Table::kVecs; ++k) {
    const long long i = e0 / 8 + k * kAdamThreads + threadIdx.x;
    if (i < nvec) {
      float pf[8], gf[8];
      ew_unpack8(reinterpret_cast<const uint4*>(p)[i], pf);
      ew_unpack8(reinterpret_cast<const uint4*>(g)[i], gf);
      const float4 m0 = reinterpret_cast<float4*>(m)[2 * i], m1 = reinterpret_cast<float4*>(m)[2 * i + 1];
      const float4 v0 = reinterpret_cast<float4*>(v)[2 * i], v1 = reinterpret_cast<float4*>(v)[2 * i + 1];
      float mf[8] = {m0.x, m0.y, m0.z, m0.w, m1.x, m1.y, m1.z, m1.w};
      float vf[8] = {v0.x, v0.y, v0.z, v0.w, v1.x, v1.y, v1.z, v1.w};
#pragma unroll
      for (int j = 0; j < 8; ++j) adamw_one(a, pf[j], gf[j], mf[j], vf[j]);
      reinterpret_cast<uint4*>(p)[i] = ew_pack8(pf);
      reinterpret_cast<float4*>(m)[2 * i] = make_float4(mf[0], mf[1], mf[2], mf[3]);
      reinterpret_cast<float4*>(m)[2 * i + 1] = make_float4(mf[4], mf[5], mf[6], mf[7]);
      reinterpret_cast<float4*>(v)[2 * i] = make_float4(vf[0], vf[1], vf[2], vf[3]);
      reinterpret_cast<float4*>(v)[2 * i + 1] = make_float4(vf[4], vf[5], vf[6], vf[7]);
    }
  }
  // tail (n not a multiple of 8), by the block that has the end of the tensor
  const long long tail = nvec * 8 + threadIdx.x;
  if (tail < n && e0 + Table::kChunk >= n) {
    float pf = __bfloat162float(p[tail]);
    adamw_one(a, pf, __bfloat162float(g[tail]), m[tail], v[tail]);
    p[tail] = __float2bfloat16(pf);
  }
}

// ------------------------------------------------------------------ DiLoCo outer step
// Both kernels read or write the live parameters where they are and the flat buckets (communication buffer, global
// weights, momentum) at the parameter's offset, so no pack or unpack copy runs around them.  A table of up to
// kOuterMax tensors travels as a kernel argument; a block handles one chunk of one tensor.
// Bound by HBM: 6 bytes a bf16 weight for the pseudo-gradient, 16 for the update (two bytes each of gradient, global
// weight and parameter, fp32 momentum in and out).  Every thread has four (update: two) 16-byte vectors of each
// stream in flight.  0.31 G bf16 weights in 21 tensors, whole synchronisation of one replica: 1.01 ms (22 bytes a
// weight, the copy bandwidth); one element per thread and round between pack and unpack copies took 2.57 ms.
constexpr int kOuterMax = 128;
constexpr int kOuterThreads = 256;

struct OuterTable {
  void* p[kOuterMax];         // live parameter (or its packed copy inside the communication bucket)
  long long off[kOuterMax];   // its first element inside the flat buckets
  long long n[kOuterMax];
  int first[kOuterMax + 1];   // first chunk of every tensor; first[count] chunks in all
  int count;
};

template <typename T>
struct Outer {
  static constexpr int VEC = 16 / sizeof(T);
  static constexpr int CHUNK = kOuterThreads * VEC * 4;  // elements per block
};
__device__ __forceinline__ void vec_unpack(const uint4& u, float (&f)[8]) { ew_unpack8(u, f); }
__device__ __forceinline__ void vec_unpack(const uint4& u, float (&f)[4]) {
  f[0] = __uint_as_float(u.x); f[1] = __uint_as_float(u.y); f[2] = __uint_as_float(u.z); f[3] = __uint_as_float(u.w);
}
__device__ __forceinline__ uint4 vec_pack(const float (&f)[8]) { return ew_pack8(f); }
__device__ __forceinline__ uint4 vec_pack(const float (&f)[4]) {
  return make_uint4(__float_as_uint(f[0]), __float_as_uint(f[1]), __float_as_uint(f[2]), __float_as_uint(f[3]));
}
template <typename T>
__device__ __forceinline__ float ld1(const T* p, long long i);
template <>
__device__ __forceinline__ float ld1<float>(const float* p, long long i) { return p[i]; }
template <>
__device__ __forceinline__ float ld1<__nv_bfloat16>(const __nv_bfloat16* p, long long i) { return __bfloat162float(p[i]); }
template <typename T>
__device__ __forceinline__ void st1(T* p, long long i, float v);
template <>
__device__ __forceinline__ void st1<float>(float* p, long long i, float v) { p[i] = v; }
template <>
__device__ __forceinline__ void st1<__nv_bfloat16>(__nv_bfloat16* p, long long i, float v) { p[i] = __float2bfloat16(v); }

// comm[off + i] = p[i] - global[off + i].  p may be comm + off itself.
template <typename T>
__global__ void __launch_bounds__(kOuterThreads)
pseudograd_kernel(const __grid_constant__ OuterTable tab, T* comm, const T* global_w) {
  constexpr int VEC = Outer<T>::VEC, CHUNK = Outer<T>::CHUNK;
  const int t = table_find(tab.first, tab.count, blockIdx.x);
  const T* p = static_cast<const T*>(tab.p[t]);
  const T* w = global_w + tab.off[t];
  T* out = comm + tab.off[t];
  const long long e0 = static_cast<long long>(blockIdx.x - tab.first[t]) * CHUNK, n = tab.n[t];
  const bool aligned = ((reinterpret_cast<uintptr_t>(p) | reinterpret_cast<uintptr_t>(w) | reinterpret_cast<uintptr_t>(out)) & 15) == 0;
  if (aligned && e0 + CHUNK <= n) {
    uint4 a[4], b[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const long long v = e0 / VEC + k * kOuterThreads + threadIdx.x;
      a[k] = reinterpret_cast<const uint4*>(p)[v];
      b[k] = reinterpret_cast<const uint4*>(w)[v];
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const long long v = e0 / VEC + k * kOuterThreads + threadIdx.x;
      float x[VEC], y[VEC];
      vec_unpack(a[k], x);
      vec_unpack(b[k], y);
#pragma unroll
      for (int j = 0; j < VEC; ++j) x[j] -= y[j];
      reinterpret_cast<uint4*>(out)[v] = vec_pack(x);
    }
    return;
  }
  // last chunk of a tensor, or a parameter that is a view at an odd address
  const long long e1 = n < e0 + CHUNK ? n : e0 + CHUNK;
  for (long long i = e0 + threadIdx.x; i < e1; i += kOuterThreads) st1<T>(out, i, ld1<T>(p, i) - ld1<T>(w, i));
}

struct OuterUpdate {
  float lr, mu;
  int nesterov, first;
};
__device__ __forceinline__ float outer_update(const OuterUpdate& u, float grad, float w, float& b) {
  float step = grad;
  if (u.mu != 0.f) {
    b = u.first ? grad : u.mu * b + grad;
    step = u.nesterov ? grad + u.mu * b : b;
  }
  return w - u.lr * step;
}

// g: averaged pseudo-gradient (flat).  global_w: old -> new global weights; buf: fp32 momentum; p: new parameters.
// p may be g + off itself.
template <typename T>
__global__ void __launch_bounds__(kOuterThreads)
nesterov_outer_kernel(const __grid_constant__ OuterTable tab, const T* g_flat, T* global_w, float* buf_flat,
                      const OuterUpdate u) {
  constexpr int VEC = Outer<T>::VEC, CHUNK = Outer<T>::CHUNK;
  const int t = table_find(tab.first, tab.count, blockIdx.x);
  T* p = static_cast<T*>(tab.p[t]);
  const T* g = g_flat + tab.off[t];
  T* w = global_w + tab.off[t];
  float* buf = buf_flat + tab.off[t];
  const long long e0 = static_cast<long long>(blockIdx.x - tab.first[t]) * CHUNK, n = tab.n[t];
  const bool load_buf = u.mu != 0.f && !u.first, store_buf = u.mu != 0.f;
  const bool aligned = ((reinterpret_cast<uintptr_t>(p) | reinterpret_cast<uintptr_t>(g) | reinterpret_cast<uintptr_t>(w) |
                         reinterpret_cast<uintptr_t>(buf)) & 15) == 0;
  if (aligned && e0 + CHUNK <= n) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      uint4 gv[2], wv[2];
      float4 bv[2][VEC / 4];
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        const long long v = e0 / VEC + (2 * h + k) * kOuterThreads + threadIdx.x;
        gv[k] = reinterpret_cast<const uint4*>(g)[v];
        wv[k] = reinterpret_cast<const uint4*>(w)[v];
#pragma unroll
        for (int q = 0; q < VEC / 4; ++q)
          bv[k][q] = load_buf ? reinterpret_cast<const float4*>(buf)[v * (VEC / 4) + q] : make_float4(0.f, 0.f, 0.f, 0.f);
      }
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        const long long v = e0 / VEC + (2 * h + k) * kOuterThreads + threadIdx.x;
        float x[VEC], y[VEC], b[VEC];
        vec_unpack(gv[k], x);
        vec_unpack(wv[k], y);
#pragma unroll
        for (int q = 0; q < VEC / 4; ++q) {
          b[4 * q] = bv[k][q].x; b[4 * q + 1] = bv[k][q].y; b[4 * q + 2] = bv[k][q].z; b[4 * q + 3] = bv[k][q].w;
        }
#pragma unroll
        for (int j = 0; j < VEC; ++j) y[j] = outer_update(u, x[j], y[j], b[j]);
        const uint4 packed = vec_pack(y);
        reinterpret_cast<uint4*>(w)[v] = packed;
        reinterpret_cast<uint4*>(p)[v] = packed;
        if (store_buf) {
#pragma unroll
          for (int q = 0; q < VEC / 4; ++q)
            reinterpret_cast<float4*>(buf)[v * (VEC / 4) + q] = make_float4(b[4 * q], b[4 * q + 1], b[4 * q + 2], b[4 * q + 3]);
        }
      }
    }
    return;
  }
  const long long e1 = n < e0 + CHUNK ? n : e0 + CHUNK;
  for (long long i = e0 + threadIdx.x; i < e1; i += kOuterThreads) {
    float b = load_buf ? buf[i] : 0.f;
    const float nw = outer_update(u, ld1<T>(g, i), ld1<T>(w, i), b);
    if (store_buf) buf[i] = b;
    st1<T>(w, i, nw);
    st1<T>(p, i, nw);
  }
}

// Calls launch(table, chunks) for runs of at most kOuterMax tensors.
template <typename T, typename Launch>
static int outer_launches(void* const* p, const long long* off, const long long* n, int count, Launch launch) {
  int launches = 0;
  for (int i = 0; i < count;) {
    OuterTable tab;
    tab.count = 0;
    tab.first[0] = 0;
    for (; i < count && tab.count < kOuterMax; ++i) {
      if (n[i] <= 0) continue;
      const int k = tab.count++;
      tab.p[k] = p[i];
      tab.off[k] = off[i];
      tab.n[k] = n[i];
      tab.first[k + 1] = tab.first[k] + static_cast<int>((n[i] + Outer<T>::CHUNK - 1) / Outer<T>::CHUNK);
    }
    if (tab.count == 0) break;
    launch(tab, tab.first[tab.count]);
    ++launches;
  }
  const cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? launches : -static_cast<int>(e);
}

// Launches for all of the tensors, in tables of one kind; returns how many.
template <typename Table>
static int adamw_launches(void* const* p, const void* const* g, float* const* m, float* const* v, const long long* n, int count,
                          const AdamArgs& args, cudaStream_t stream) {
  int launches = 0;
  for (int i = 0; i < count;) {
    Table tab;
    tab.count = 0;
    tab.first[0] = 0;
    uintptr_t low = UINTPTR_MAX, high = 0;  // all parameters of the table lie between
    for (; i < count && tab.count < Table::kMax; ++i) {
      if (n[i] <= 0) continue;
      // Parameters that share memory (tied weights, one listed twice) take their updates one after the other: the next launch
      const uintptr_t begin = reinterpret_cast<uintptr_t>(p[i]), end = begin + static_cast<uintptr_t>(n[i]) * sizeof(__nv_bfloat16);
      bool shared = false;
      if (begin < high && low < end)
        for (int k = 0; k < tab.count && !shared; ++k)
          shared = begin < reinterpret_cast<uintptr_t>(tab.p[k] + tab.n[k]) && reinterpret_cast<uintptr_t>(tab.p[k]) < end;
      if (shared) break;
      low = begin < low ? begin : low;
      high = end > high ? end : high;
      const int k = tab.count++;
      tab.p[k] = static_cast<__nv_bfloat16*>(p[i]);
      tab.g[k] = static_cast<const __nv_bfloat16*>(g[i]);
      tab.m[k] = m[i];
      tab.v[k] = v[i];
      tab.n[k] = n[i];
      tab.first[k + 1] = tab.first[k] + static_cast<int>((n[i] + Table::kChunk - 1) / Table::kChunk);
    }
    if (tab.count == 0) break;
    adamw_kernel<Table><<<tab.first[tab.count], kAdamThreads, 0, stream>>>(tab, args);
    ++launches;
  }
  return launches;
}

static inline int ew_grid(long long work_items, int threads) {
  long long b = (work_items + threads - 1) / threads;
  const long long cap = 148LL * 16;
  if (b > cap) b = cap;
  if (b < 1) b = 1;
  return static_cast<int>(b);
}

}  // namespace tft

using namespace tft;

TFT_API int tft_swiglu_fwd(const void* gu, void* out, long long rows, int F, cudaStream_t stream) {
  if (F % 8) return static_cast<int>(cudaErrorInvalidValue);
  swiglu_fwd_kernel<<<ew_grid(rows * (F / 8), 256), 256, 0, stream>>>(
      static_cast<const __nv_bfloat16*>(gu), static_cast<__nv_bfloat16*>(out), rows, F);
  return static_cast<int>(cudaGetLastError());
}

TFT_API int tft_swiglu_bwd(const void* gu, const void* dout, void* dgu, long long rows, int F,
                           cudaStream_t stream) {
  if (F % 8) return static_cast<int>(cudaErrorInvalidValue);
  swiglu_bwd_kernel<<<ew_grid(rows * (F / 8), 256), 256, 0, stream>>>(
      static_cast<const __nv_bfloat16*>(gu), static_cast<const __nv_bfloat16*>(dout),
      static_cast<__nv_bfloat16*>(dgu), rows, F);
  return static_cast<int>(cudaGetLastError());
}

// logits [rows, V] bf16 (row stride ld) become the gradient; loss[rows] fp32.
TFT_API int tft_xent(void* logits, const long long* targets, float* loss, int rows, int V, int ld,
                     float grad_scale, long long ignore_index, cudaStream_t stream) {
  if (V % 8 || ld % 8) return static_cast<int>(cudaErrorInvalidValue);
  auto* z = static_cast<__nv_bfloat16*>(logits);
  const int vecs = V / 8;
  if (vecs <= XENT_ROOM)
    xent_row_kernel<<<rows, (vecs + 32 * XENT_VECS - 1) / (32 * XENT_VECS) * 32, 0, stream>>>(z, targets, loss, V, ld, grad_scale,
                                                                                             ignore_index);
  else
    xent_kernel<<<rows, XENT_LONG_THREADS, 0, stream>>>(z, targets, loss, V, ld, grad_scale, ignore_index);
  return static_cast<int>(cudaGetLastError());
}

TFT_API int tft_embedding_fwd(const long long* tokens, const void* table, void* out, long long n_tokens, int dim,
                              cudaStream_t stream) {
  if (dim % 8) return static_cast<int>(cudaErrorInvalidValue);
  embedding_fwd_kernel<<<ew_grid(n_tokens * (dim / 8), 256), 256, 0, stream>>>(
      tokens, static_cast<const __nv_bfloat16*>(table), static_cast<__nv_bfloat16*>(out), n_tokens, dim);
  return static_cast<int>(cudaGetLastError());
}

TFT_API int tft_embedding_bwd(const long long* tokens, const void* dout, void* dtable, long long n_tokens, int dim,
                              cudaStream_t stream) {
  if (dim % 2) return static_cast<int>(cudaErrorInvalidValue);
  embedding_bwd_kernel<<<ew_grid(n_tokens * (dim / 2), 256), 256, 0, stream>>>(
      tokens, static_cast<const __nv_bfloat16*>(dout), static_cast<__nv_bfloat16*>(dtable), n_tokens, dim);
  return static_cast<int>(cudaGetLastError());
}

// One AdamW update of `count` tensors: n[i] elements at p[i], g[i], m[i], v[i], each at a 16-byte boundary.  Host arrays,
// read before the call returns.  Returns the number of launches, or -(CUDA error).  0.31 G parameters in 21 tensors: one
// launch of 1012 us for 21 of 1118 in all (22 bytes a parameter: 6.8 TB/s); four tensors of 0.65 G: 2112 us for 2322.
TFT_API int tft_adamw_multi(void* const* p, const void* const* g, float* const* m, float* const* v, const long long* n,
                            int count, float lr, float b1, float b2, float eps, float wd, int step, float grad_scale,
                            cudaStream_t stream) {
  for (int i = 0; i < count; ++i)
    if (n[i] > 0 && ((reinterpret_cast<uintptr_t>(p[i]) | reinterpret_cast<uintptr_t>(g[i]) | reinterpret_cast<uintptr_t>(m[i]) |
                      reinterpret_cast<uintptr_t>(v[i])) & 15))
      return -static_cast<int>(cudaErrorInvalidValue);
  const float bc1 = 1.f - powf(b1, static_cast<float>(step));
  const float bc2 = 1.f - powf(b2, static_cast<float>(step));
  const AdamArgs args = {lr, b1, b2, eps, wd, 1.f / bc1, 1.f / sqrtf(bc2), grad_scale};
  const bool small = count == 1 && n[0] <= kAdamSmall;
  const int launches = small ? adamw_launches<AdamTable<1, 1>>(p, g, m, v, n, count, args, stream)
                             : adamw_launches<AdamTable<kAdamMax, 2>>(p, g, m, v, n, count, args, stream);
  const cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? launches : -static_cast<int>(e);
}

TFT_API int tft_adamw(void* p, const void* g, float* m, float* v, long long n, float lr, float b1, float b2,
                      float eps, float wd, int step, float grad_scale, cudaStream_t stream) {
  const int r = tft_adamw_multi(&p, &g, &m, &v, &n, 1, lr, b1, b2, eps, wd, step, grad_scale, stream);
  return r < 0 ? -r : 0;
}

// The outer step over `count` tensors of one dtype: tensor i has n[i] elements at p[i] and, inside the flat buckets, at
// element off[i].  Host arrays, read before the call returns.  Returns the number of launches, or -(CUDA error).
TFT_API int tft_pseudograd(void* const* p, const long long* off, const long long* n, int count, void* comm,
                           const void* global_w, int is_bf16, cudaStream_t stream) {
  if (is_bf16)
    return outer_launches<__nv_bfloat16>(p, off, n, count, [&](const OuterTable& tab, int chunks) {
      pseudograd_kernel<__nv_bfloat16><<<chunks, kOuterThreads, 0, stream>>>(
          tab, static_cast<__nv_bfloat16*>(comm), static_cast<const __nv_bfloat16*>(global_w));
    });
  return outer_launches<float>(p, off, n, count, [&](const OuterTable& tab, int chunks) {
    pseudograd_kernel<float><<<chunks, kOuterThreads, 0, stream>>>(tab, static_cast<float*>(comm),
                                                                   static_cast<const float*>(global_w));
  });
}

TFT_API int tft_nesterov_outer(void* const* p, const long long* off, const long long* n, int count, const void* g,
                               void* global_w, float* buf, float lr, float mu, int nesterov, int first, int is_bf16,
                               cudaStream_t stream) {
  const OuterUpdate u = {lr, mu, nesterov, first};
  if (is_bf16)
    return outer_launches<__nv_bfloat16>(p, off, n, count, [&](const OuterTable& tab, int chunks) {
      nesterov_outer_kernel<__nv_bfloat16><<<chunks, kOuterThreads, 0, stream>>>(
          tab, static_cast<const __nv_bfloat16*>(g), static_cast<__nv_bfloat16*>(global_w), buf, u);
    });
  return outer_launches<float>(p, off, n, count, [&](const OuterTable& tab, int chunks) {
    nesterov_outer_kernel<float><<<chunks, kOuterThreads, 0, stream>>>(tab, static_cast<const float*>(g),
                                                                       static_cast<float*>(global_w), buf, u);
  });
}
