// Embedding, norms, rotation + cache write, gated activation, logit cap, row gather.
// One row (token) per block unless said otherwise; float32 arithmetic throughout.
#include "common.cuh"

#include <type_traits>

// ---------------------------------------------------------------------------------
// Embedding lookup with an optional weightless RMS norm: x[t] = rms0(table[ids[t]]).
// The residual stream x is float32 in both precisions.
template <typename T>
__global__ void embed_rmsnorm_kernel(const int* __restrict__ ids, const T* __restrict__ table,
                                     float* __restrict__ x, int hidden, int vocab, float eps,
                                     int normed, int* err) {
  pdl_wait();
  pdl_launch_dependents();
  __shared__ float scratch[33];
  const int t = blockIdx.x;
  int id = ids[t];
  if (id < 0 || id >= vocab) {
    if (threadIdx.x == 0) atomicOr(err, OMNIA_ERR_TOKEN_ID);
    id = 0;
  }
  const T* row = table + (size_t)id * hidden;
  float* out = x + (size_t)t * hidden;
  float ss = 0.f;
  for (int i = threadIdx.x; i < hidden; i += blockDim.x) {
    const float v = to_f32(row[i]);
    ss += v * v;
  }
  float scale = 1.f;
  if (normed) scale = rsqrtf(block_sum(ss, scratch) / (float)hidden + eps);
  for (int i = threadIdx.x; i < hidden; i += blockDim.x) out[i] = to_f32(row[i]) * scale;
}

extern "C" int omnia_embed_rmsnorm(const int* ids, const void* table, float* x, int tokens,
                                   int hidden, int vocab, float eps, int normed, int dtype,
                                   int* err, cudaStream_t stream) {
  if (tokens == 0) return 0;
  OMNIA_DISPATCH_DTYPE(dtype, (launch_pdl(embed_rmsnorm_kernel<T>, tokens, 256, 0, stream, 
                                  ids, (const T*)table, x, hidden, vocab, eps, normed, err)));
  return OMNIA_LAUNCH_RESULT();
}

// ---------------------------------------------------------------------------------
// Embedding with a hashed table of token pairs: x[t] = table[ids[t]] * scale + pairs[row], row =
// (before * mul_prev + ids[t] * mul_cur) mod buckets, `before` being the token ahead of t in its
// request, and row = buckets (the table's extra last row) at position 0. The token ahead of a
// portion's first token is read from `prev` [slots] (by the request's state slot); the block of that
// first token, having read it, leaves the portion's last token there. Rows of padding (position
// < 0) are zero. One block per token.
template <typename T>
__global__ void embed_pair_kernel(const int* __restrict__ ids, const int* __restrict__ positions,
                                  const int* __restrict__ cu_seqlens, const int* __restrict__ state_slots,
                                  int num_seqs, const T* __restrict__ table, const T* __restrict__ pairs,
                                  int* __restrict__ prev, float* __restrict__ x, int hidden, int vocab,
                                  long long buckets, long long mul_prev, long long mul_cur, float scale, int* err) {
  pdl_wait();
  pdl_launch_dependents();
  const int t = blockIdx.x;
  float* out = x + (size_t)t * hidden;
  const int pos = positions[t];
  if (pos < 0) {
    for (int i = threadIdx.x; i < hidden; i += blockDim.x) out[i] = 0.f;
    return;
  }
  int lo = 0, hi = num_seqs - 1;  // the request of this token: the last s with cu_seqlens[s] <= t
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (cu_seqlens[mid] <= t) lo = mid; else hi = mid - 1;
  }
  const int begin = cu_seqlens[lo], end = cu_seqlens[lo + 1];
  int id = ids[t];
  if (id < 0 || id >= vocab) {
    if (threadIdx.x == 0) atomicOr(err, OMNIA_ERR_TOKEN_ID);
    id = 0;
  }
  int before = 0;
  if (t > begin) {
    before = ids[t - 1];
  } else {
    const int slot = state_slots[lo];
    before = prev[slot];
    __syncthreads();  // every thread has read the slot before one of them writes it
    if (threadIdx.x == 0) prev[slot] = ids[end - 1];
  }
  if (before < 0 || before >= vocab) before = 0;
  const long long row = pos == 0 ? buckets : ((long long)before * mul_prev + (long long)id * mul_cur) % buckets;
  const T* a = table + (size_t)id * hidden;
  const T* b = pairs + (size_t)row * hidden;
  for (int i = threadIdx.x; i < hidden; i += blockDim.x) out[i] = to_f32(a[i]) * scale + to_f32(b[i]);
}

extern "C" int omnia_embed_pair(const int* ids, const int* positions, const int* cu_seqlens, const int* state_slots,
                                int num_seqs, const void* table, const void* pairs, int* prev, float* x, int tokens,
                                int hidden, int vocab, long long buckets, long long mul_prev, long long mul_cur,
                                float scale, int dtype, int* err, cudaStream_t stream) {
  if (tokens == 0) return 0;
  if (buckets < 1 || mul_prev < 0 || mul_cur < 0) return (int)cudaErrorInvalidValue;
  OMNIA_DISPATCH_DTYPE(dtype, (launch_pdl(embed_pair_kernel<T>, tokens, 256, 0, stream, ids, positions, cu_seqlens,
                                          state_slots, num_seqs, (const T*)table, (const T*)pairs, prev, x, hidden,
                                          vocab, buckets, mul_prev, mul_cur, scale, err)));
  return OMNIA_LAUNCH_RESULT();
}

// ---------------------------------------------------------------------------------
// h = x * rsqrt(mean(x^2) + eps) * w   (w may be null: weightless). x is float32.
template <typename T>
__global__ void rmsnorm_kernel(const float* __restrict__ x, const float* __restrict__ w,
                               T* __restrict__ h, int hidden, float eps) {
  pdl_wait();
  pdl_launch_dependents();
  __shared__ float scratch[33];
  const float* row = x + (size_t)blockIdx.x * hidden;
  T* out = h + (size_t)blockIdx.x * hidden;
  float ss = 0.f;
  for (int i = threadIdx.x; i < hidden; i += blockDim.x) ss += row[i] * row[i];
  const float scale = rsqrtf(block_sum(ss, scratch) / (float)hidden + eps);
  for (int i = threadIdx.x; i < hidden; i += blockDim.x) {
    float v = row[i] * scale;
    if (w) v *= w[i];
    out[i] = from_f32<T>(v);
  }
}

extern "C" int omnia_rmsnorm(const float* x, const float* w, void* h, int rows, int hidden,
                             float eps, int dtype, cudaStream_t stream) {
  if (rows == 0) return 0;
  OMNIA_DISPATCH_DTYPE(dtype,
                       (launch_pdl(rmsnorm_kernel<T>, rows, 256, 0, stream, x, w, (T*)h, hidden, eps)));
  return OMNIA_LAUNCH_RESULT();
}

// ---------------------------------------------------------------------------------
// The residual step of a block, in one pass over the row:
//   a  = branch                      (optionally normed: a * rsqrt(mean a^2 + eps_b) * wb)
//   x += a                           (float32, in place)
//   h  = x * rsqrt(mean x^2 + eps_o) * wo   (optional; wo may be null; norm_out == 2: h = x, only rounded
//        to the element type, for whoever reads the residual itself)
// The row is staged in shared memory as float32, so the branch is read once and x is
// read and written once.
template <typename T>
__global__ void add_rmsnorm_kernel(float* __restrict__ x, const T* __restrict__ branch,
                                   const float* __restrict__ wb, float eps_b, int norm_branch,
                                   const float* __restrict__ wo, float eps_o, int norm_out,
                                   T* __restrict__ h, int hidden) {
  pdl_wait();
  pdl_launch_dependents();
  extern __shared__ float row[];
  __shared__ float scratch[33];
  float* xr = x + (size_t)blockIdx.x * hidden;
  const T* br = branch + (size_t)blockIdx.x * hidden;
  float ss = 0.f;
  for (int i = threadIdx.x; i < hidden; i += blockDim.x) {
    const float a = to_f32(br[i]);
    row[i] = a;
    ss += a * a;
  }
  float scale_b = 1.f;
  if (norm_branch) scale_b = rsqrtf(block_sum(ss, scratch) / (float)hidden + eps_b);
  ss = 0.f;
  for (int i = threadIdx.x; i < hidden; i += blockDim.x) {
    float a = row[i];
    if (norm_branch) {
      a *= scale_b;
      if (wb) a *= wb[i];
    }
    const float v = xr[i] + a;
    xr[i] = v;
    row[i] = v;
    ss += v * v;
  }
  if (!norm_out) return;
  const float scale_o = norm_out == 2 ? 1.f : rsqrtf(block_sum(ss, scratch) / (float)hidden + eps_o);
  T* out = h + (size_t)blockIdx.x * hidden;
  for (int i = threadIdx.x; i < hidden; i += blockDim.x) {
    float v = row[i] * scale_o;
    if (wo && norm_out == 1) v *= wo[i];
    out[i] = from_f32<T>(v);
  }
}

// The same residual step with the whole row in registers: every load of the row (branch, x
// and both weights) is issued before the first reduction, so a row costs one memory round
// trip instead of three. hidden % 4 == 0 and hidden <= 4 * ITERS * blockDim.
template <typename T>
struct Vec4;
template <>
struct Vec4<float> {
  typedef float4 Packed;
  static __device__ __forceinline__ void unpack(const float4& t, float* v) { v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w; }
  static __device__ __forceinline__ void load(const float* p, float* v) {
    const float4 t = *reinterpret_cast<const float4*>(p);
    v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w;
  }
  static __device__ __forceinline__ void store(float* p, const float* v) {
    *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
  }
};
template <>
struct Vec4<__nv_bfloat16> {
  typedef uint2 Packed;
  static __device__ __forceinline__ void load(const __nv_bfloat16* p, float* v) { unpack(*reinterpret_cast<const uint2*>(p), v); }
  static __device__ __forceinline__ void unpack(const uint2& t, float* v) {
    const __nv_bfloat162 a = *reinterpret_cast<const __nv_bfloat162*>(&t.x);
    const __nv_bfloat162 b = *reinterpret_cast<const __nv_bfloat162*>(&t.y);
    v[0] = __low2float(a); v[1] = __high2float(a); v[2] = __low2float(b); v[3] = __high2float(b);
  }
  static __device__ __forceinline__ void store(__nv_bfloat16* p, const float* v) {
    __nv_bfloat162 a = __floats2bfloat162_rn(v[0], v[1]), b = __floats2bfloat162_rn(v[2], v[3]);
    uint2 t;
    t.x = *reinterpret_cast<unsigned*>(&a);
    t.y = *reinterpret_cast<unsigned*>(&b);
    *reinterpret_cast<uint2*>(p) = t;
  }
};

// LATE: the norms' weights are read where they are needed instead of up front. With many rows they come from L1,
// where the rows before left them, and what counts is how many rows an SM has in flight: 32 registers a thread instead
// of 48, and eight values a thread at every width (sixteen took 84). 2,048 rows of 4,096: 30.4 -> 17.3 us (100 MB: 15.4 at
// the copy rate), 600 rows of 4,096: 10.5 -> 7.1. With few rows a row is one chain of trips to memory, and the weights come
// up front: up to two rows an SM, and up to twelve where 256 threads or fewer make a row, since an SM holds a good part of
// those at once either way. Launch after launch (x and branch in L2), 600 / 1,200 / 2,048 rows of 2,048: late 4.5 / 5.9 /
// 7.8 us, up front 3.8 / 5.8 / 8.4; of 1,024: 3.1 / 4.5 / 4.8 and 2.7 / 3.7 / 5.3; 260 / 300 rows of 4,096 late 3.6 / 4.5 and
// up front 3.5 / 4.9. Few wide rows of float32 take sixteen values a thread (8 rows of 5,120: 3.2 us, 3.4 with eight).
template <typename T, int ITERS, bool LATE>
__global__ void __launch_bounds__(ITERS > 2 ? 512 : 1024, LATE ? 2 : 1) add_rmsnorm_reg_kernel(float* __restrict__ x, const T* __restrict__ branch,
                                       const float* __restrict__ wb, float eps_b, int norm_branch,
                                       const float* __restrict__ wo, float eps_o, int norm_out,
                                       T* __restrict__ h, int hidden) {
  pdl_wait();
  pdl_launch_dependents();
  __shared__ float scratch[33];
  float* xr = x + (size_t)blockIdx.x * hidden;
  const T* br = branch + (size_t)blockIdx.x * hidden;
  const bool weigh_b = norm_branch && wb, weigh_o = norm_out == 1 && wo;
  typename Vec4<T>::Packed a[ITERS];
  float xv[ITERS][4], gb[ITERS][4], go[ITERS][4];
#pragma unroll
  for (int it = 0; it < ITERS; ++it) {
    const int i = (it * blockDim.x + threadIdx.x) * 4;
    const bool live = i < hidden;
    a[it] = typename Vec4<T>::Packed{};
#pragma unroll
    for (int k = 0; k < 4; ++k) xv[it][k] = 0.f, gb[it][k] = go[it][k] = 1.f;
    if (live) {
      a[it] = *reinterpret_cast<const typename Vec4<T>::Packed*>(br + i);
      Vec4<float>::load(xr + i, xv[it]);
      if (!LATE && weigh_b) Vec4<float>::load(wb + i, gb[it]);
      if (!LATE && weigh_o) Vec4<float>::load(wo + i, go[it]);
    }
  }
  float ss = 0.f;
#pragma unroll
  for (int it = 0; it < ITERS; ++it) {
    float v[4];
    Vec4<T>::unpack(a[it], v);
#pragma unroll
    for (int k = 0; k < 4; ++k) ss += v[k] * v[k];
  }
  float scale_b = 1.f;
  if (norm_branch) scale_b = rsqrtf(block_sum(ss, scratch) / (float)hidden + eps_b);
  ss = 0.f;
#pragma unroll
  for (int it = 0; it < ITERS; ++it) {
    const int i = (it * blockDim.x + threadIdx.x) * 4;
    float v[4];
    Vec4<T>::unpack(a[it], v);
    if (LATE && weigh_b && i < hidden) Vec4<float>::load(wb + i, gb[it]);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      if (norm_branch) v[k] = v[k] * scale_b * gb[it][k];
      xv[it][k] += v[k];
      ss += xv[it][k] * xv[it][k];
    }
    if (i < hidden) Vec4<float>::store(xr + i, xv[it]);
  }
  if (!norm_out) return;
  const float scale_o = norm_out == 2 ? 1.f : rsqrtf(block_sum(ss, scratch) / (float)hidden + eps_o);
  T* out = h + (size_t)blockIdx.x * hidden;
#pragma unroll
  for (int it = 0; it < ITERS; ++it) {
    const int i = (it * blockDim.x + threadIdx.x) * 4;
    if (i >= hidden) continue;
    if (LATE && weigh_o) Vec4<float>::load(wo + i, go[it]);
    float v[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) v[k] = xv[it][k] * scale_o * go[it][k];
    Vec4<T>::store(out + i, v);
  }
}

extern "C" int omnia_add_rmsnorm(float* x, const void* branch, const float* wb, float eps_b,
                                 int norm_branch, const float* wo, float eps_o, int norm_out,
                                 void* h, int rows, int hidden, int dtype, cudaStream_t stream) {
  if (rows == 0) return 0;
  if (hidden % 4 == 0 && hidden <= 8192) {
    const bool wide = hidden > 2048, late = rows > (wide ? 2 : 12) * omnia_sm_count();
    const int threads = hidden <= 1024 ? 128 : hidden <= 2048 ? 256 : hidden <= 4096 ? 512 : 1024;  // eight values each
    OMNIA_DISPATCH_DTYPE(dtype, {
      auto launch = [&](auto* kernel, int threads) {
        launch_pdl(kernel, rows, threads, 0, stream, x, (const T*)branch, wb, eps_b, norm_branch, wo, eps_o, norm_out, (T*)h, hidden);
      };
      constexpr int FEW = sizeof(T) == 4 ? 4 : 2;
      if (late) launch(add_rmsnorm_reg_kernel<T, 2, true>, threads);
      else if (wide) launch(add_rmsnorm_reg_kernel<T, FEW, false>, threads * 2 / FEW);
      else launch(add_rmsnorm_reg_kernel<T, 2, false>, threads);
    });
    return OMNIA_LAUNCH_RESULT();
  }
  const size_t smem = (size_t)hidden * sizeof(float);
  if (smem > 200 * 1024) return (int)cudaErrorInvalidValue;
  OMNIA_DISPATCH_DTYPE(dtype, {
    if (smem > 48 * 1024)
      cudaFuncSetAttribute(add_rmsnorm_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)smem);
    launch_pdl(add_rmsnorm_kernel<T>, rows, 256, smem, stream, x, (const T*)branch, wb, eps_b,
                                                       norm_branch, wo, eps_o, norm_out, (T*)h,
                                                       hidden);
  });
  return OMNIA_LAUNCH_RESULT();
}

// ---------------------------------------------------------------------------------
// Per head of a projected row [.. q heads .. | .. k heads .. | .. v heads ..] (each
// group at its own column of `proj`): weightless RMS over the head (q and k; eps < 0
// skips it), half-split rotation of the first `rot` dims by angle pos * inv_freq[i]
// (inv_freq null: no rotation), then q goes to q_out and k, v go into cache pages
// [page][k|v][kv_head][offset][d] at slot_mapping[t] (slot < 0: nothing is stored).
// One warp per head, four heads per block; head_dim <= 256 and even.
template <typename T>
__global__ void qk_norm_rope_store_kernel(const T* __restrict__ proj, int row_stride, int q_col,
                                          int k_col, int v_col, int nq, int nkv, int d,
                                          float eps, const float* __restrict__ inv_freq, int rot,
                                          const int* __restrict__ positions,
                                          const long long* __restrict__ slot_mapping,
                                          T* __restrict__ q_out, T* __restrict__ pages,
                                          int page_size, long long num_slots, int* err) {
  pdl_wait();
  pdl_launch_dependents();
  const int t = blockIdx.x;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int hs = blockIdx.y * (blockDim.x >> 5) + warp;
  if (hs >= nq + 2 * nkv) return;
  const int kind = hs < nq ? 0 : (hs < nq + nkv ? 1 : 2);
  const int head = kind == 0 ? hs : (kind == 1 ? hs - nq : hs - nq - nkv);
  const T* src = proj + (size_t)t * row_stride + (kind == 0 ? q_col : kind == 1 ? k_col : v_col) +
                 (size_t)head * d;
  T* dst;
  if (kind == 0) {
    dst = q_out + ((size_t)t * nq + head) * d;
  } else {
    const long long slot = slot_mapping[t];
    if (slot < 0) return;
    if (slot >= num_slots) {
      if (lane == 0) atomicOr(err, OMNIA_ERR_SLOT);
      return;
    }
    const long long page = slot / page_size, off = slot % page_size;
    dst = pages + (((page * 2 + (kind == 2)) * nkv + head) * page_size + off) * d;
  }
  if (kind == 2) {
    for (int i = lane; i < d; i += 32) dst[i] = src[i];
    return;
  }
  // The head is staged in shared memory as float32: norm, then rotation, then one rounding.
  __shared__ float staged[4][256];
  float* v = staged[warp];
  float ss = 0.f;
  for (int i = lane; i < d; i += 32) {
    const float a = to_f32(src[i]);
    v[i] = a;
    ss += a * a;
  }
  float scale = 1.f;
  if (eps >= 0.f) scale = rsqrtf(warp_sum(ss) / (float)d + eps);
  __syncwarp();
  const int rhalf = inv_freq != nullptr ? rot / 2 : 0;
  const float pos = (float)positions[t];
  for (int i = lane; i < rhalf; i += 32) {
    float s, c;
    sincosf(pos * inv_freq[i], &s, &c);
    const float a = v[i] * scale, b = v[i + rhalf] * scale;
    dst[i] = from_f32<T>(a * c - b * s);
    dst[i + rhalf] = from_f32<T>(a * s + b * c);
  }
  for (int i = 2 * rhalf + lane; i < d; i += 32) dst[i] = from_f32<T>(v[i] * scale);
}

// The same step for head sizes that are multiples of 32 with full (or no) rotation: lane l owns
// VW = d / 32 contiguous dims, read and written as one vector; the rotation partner of a dim in
// the first half lives 16 lanes away.
template <typename T, int VW>
struct alignas(sizeof(T) * VW) HeadPack {
  T v[VW];
};

template <typename T, int VW>
__global__ void __launch_bounds__(256)
qk_norm_rope_store_vec_kernel(const T* __restrict__ proj, int row_stride, int q_col, int k_col, int v_col, int nq,
                              int nkv, float eps, const float* __restrict__ inv_freq,
                              const int* __restrict__ positions, const long long* __restrict__ slot_mapping,
                              T* __restrict__ q_out, T* __restrict__ pages, int page_size, long long num_slots,
                              int* err) {
  pdl_wait();
  pdl_launch_dependents();
  constexpr int d = 32 * VW;
  __shared__ float cos_s[d / 2], sin_s[d / 2];
  const int t = blockIdx.x;  // one block per token: the token's angles are computed once for all heads
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (inv_freq != nullptr) {
    const float pos = (float)positions[t];
    for (int i = threadIdx.x; i < d / 2; i += blockDim.x) sincosf(pos * inv_freq[i], &sin_s[i], &cos_s[i]);
  }
  __syncthreads();
  const long long slot = slot_mapping != nullptr ? slot_mapping[t] : -1;
  if (nkv > 0 && slot >= num_slots && threadIdx.x == 0) atomicOr(err, OMNIA_ERR_SLOT);
  for (int hs = warp; hs < nq + 2 * nkv; hs += blockDim.x >> 5) {
    const int kind = hs < nq ? 0 : (hs < nq + nkv ? 1 : 2);
    const int head = kind == 0 ? hs : (kind == 1 ? hs - nq : hs - nq - nkv);
    const T* src = proj + (size_t)t * row_stride + (kind == 0 ? q_col : kind == 1 ? k_col : v_col) + (size_t)head * d;
    T* dst;
    if (kind == 0) {
      dst = q_out + ((size_t)t * nq + head) * d;
    } else {
      if (slot < 0 || slot >= num_slots) continue;
      const long long page = slot / page_size, off = slot % page_size;
      dst = pages + (((page * 2 + (kind == 2)) * nkv + head) * page_size + off) * d;
    }
    HeadPack<T, VW> pack = *reinterpret_cast<const HeadPack<T, VW>*>(src + lane * VW);
    if (kind != 2) {
      float v[VW], ss = 0.f;
#pragma unroll
      for (int i = 0; i < VW; ++i) {
        v[i] = to_f32(pack.v[i]);
        ss += v[i] * v[i];
      }
      const float scale = eps >= 0.f ? rsqrtf(warp_sum(ss) / (float)d + eps) : 1.f;
#pragma unroll
      for (int i = 0; i < VW; ++i) {
        float mine = v[i] * scale;
        if (inv_freq != nullptr) {
          const float other = __shfl_xor_sync(0xffffffffu, mine, 16);
          const float c = cos_s[(lane & 15) * VW + i], sn = sin_s[(lane & 15) * VW + i];
          mine = lane < 16 ? mine * c - other * sn : other * sn + mine * c;
        }
        pack.v[i] = from_f32<T>(mine);
      }
    }
    *reinterpret_cast<HeadPack<T, VW>*>(dst + lane * VW) = pack;
  }
}

extern "C" int omnia_qk_norm_rope_store(const void* proj, int row_stride, int q_col, int k_col,
                                        int v_col, int nq, int nkv, int d, float eps,
                                        const float* inv_freq, int rot, const int* positions,
                                        const long long* slot_mapping, void* q_out, void* pages,
                                        int page_size, long long num_slots, int tokens, int dtype,
                                        int* err, cudaStream_t stream) {
  if (tokens == 0) return 0;
  if (d > 256 || (d & 1) || rot > d || (rot & 1)) return (int)cudaErrorInvalidValue;
  const int heads = nq + 2 * nkv;
  dim3 grid(tokens, (heads + 3) / 4);
  // Head sizes 64, 128, 256 with full or no rotation, and operands aligned for vector access.
  const bool vector_ok = (rot == d || inv_freq == nullptr) && (d == 64 || d == 128 || d == 256) &&
                         row_stride % 8 == 0 && q_col % 8 == 0 && k_col % 8 == 0 && v_col % 8 == 0 &&
                         ((uintptr_t)proj & 15) == 0 && ((uintptr_t)q_out & 15) == 0 && ((uintptr_t)pages & 15) == 0;
  if (vector_ok) {
    OMNIA_DISPATCH_DTYPE(dtype, {
      if (d == 64)
        launch_pdl(qk_norm_rope_store_vec_kernel<T, 2>, tokens, 256, 0, stream, (const T*)proj, row_stride, q_col, k_col,
                   v_col, nq, nkv, eps, inv_freq, positions, slot_mapping, (T*)q_out, (T*)pages, page_size, num_slots, err);
      else if (d == 128)
        launch_pdl(qk_norm_rope_store_vec_kernel<T, 4>, tokens, 256, 0, stream, (const T*)proj, row_stride, q_col, k_col,
                   v_col, nq, nkv, eps, inv_freq, positions, slot_mapping, (T*)q_out, (T*)pages, page_size, num_slots, err);
      else
        launch_pdl(qk_norm_rope_store_vec_kernel<T, 8>, tokens, 256, 0, stream, (const T*)proj, row_stride, q_col, k_col,
                   v_col, nq, nkv, eps, inv_freq, positions, slot_mapping, (T*)q_out, (T*)pages, page_size, num_slots, err);
    });
    return OMNIA_LAUNCH_RESULT();
  }
  OMNIA_DISPATCH_DTYPE(dtype, (launch_pdl(qk_norm_rope_store_kernel<T>, grid, 128, 0, stream, 
                                  (const T*)proj, row_stride, q_col, k_col, v_col, nq, nkv, d, eps,
                                  inv_freq, rot, positions, slot_mapping, (T*)q_out, (T*)pages,
                                  page_size, num_slots, err)));
  return OMNIA_LAUNCH_RESULT();
}

// ---------------------------------------------------------------------------------
// The general form of the step above, for a mixer whose projections have biases, whose head norms
// have a weight (one vector of the head's size, shared by the heads), whose values are of another
// width than its keys, and whose rotation may cover only the first `rot` dims of a head:
// per head of a projected row, bias added, RMS norm with weight (q and k; eps < 0: none), rotation
// of dims (i, i + rot / 2) by position * inv_freq[i]; q goes to q_out [tokens, nq, dk], k and v to
// the token's slot of the cache: key row (head h) at k_pages + page * page_stride + (h * page_size
// + offset) * dk, value row at v_pages + page * page_stride + (h * page_size + offset) * dv.
// One block per token, its warps taking the heads in turn.
// `whole`: the norm is one root mean square over all heads of q (and one over all heads of k) with
// weights of the whole projection's size; `interleaved`: the rotation pairs dims (2i, 2i + 1).
#define QKV_PREPARE_MAX_NORMED 512
template <typename T>
__global__ void __launch_bounds__(256)
qkv_prepare_kernel(const T* __restrict__ proj, int row_stride, int q_col, int k_col, int v_col,
                   int nq, int nkv, int dk, int dv, const T* __restrict__ bias,
                   const float* __restrict__ q_weight, const float* __restrict__ k_weight, float eps,
                   const float* __restrict__ inv_freq, int rot, const int* __restrict__ positions,
                   const long long* __restrict__ slot_mapping, T* __restrict__ q_out,
                   T* __restrict__ k_pages, T* __restrict__ v_pages, long long page_stride,
                   int page_size, long long num_slots, int whole, int interleaved, const T* __restrict__ other,
                   int other_stride, float lam, int* err) {
  pdl_wait();
  pdl_launch_dependents();
  // One block per token: the token's angles are worked out once for all its heads.
  __shared__ float cos_s[128], sin_s[128];
  __shared__ float staged[8][256];
  __shared__ float head_ss[QKV_PREPARE_MAX_NORMED];  // `whole`: every normed head's sum of squares
  const int t = blockIdx.x;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
  const int rhalf = inv_freq != nullptr ? rot / 2 : 0;
  {
    const float pos = (float)positions[t];
    for (int i = threadIdx.x; i < rhalf; i += blockDim.x) sincosf(pos * inv_freq[i], &sin_s[i], &cos_s[i]);
  }
  __syncthreads();
  const long long slot = slot_mapping != nullptr ? slot_mapping[t] : -1;
  if (nkv > 0 && slot >= num_slots && threadIdx.x == 0) atomicOr(err, OMNIA_ERR_SLOT);
  float* v = staged[warp];
  float whole_scale[2] = {1.f, 1.f};
  if (whole && eps >= 0.f) {
    // One root mean square over all heads of q, one over all heads of k: the heads' sums of squares
    // first, then every thread adds them in the heads' order.
    for (int hs = warp; hs < nq + nkv; hs += warps) {
      const int col = hs < nq ? q_col + hs * dk : k_col + (hs - nq) * dk;
      const T* src = proj + (size_t)t * row_stride + col;
      float ss = 0.f;
      for (int i = lane; i < dk; i += 32) {
        const float a = to_f32(src[i]) + (bias ? to_f32(bias[col + i]) : 0.f);
        ss += a * a;
      }
      ss = warp_sum(ss);
      if (lane == 0) head_ss[hs] = ss;
    }
    __syncthreads();
    float sq = 0.f, sk = 0.f;
    for (int h = 0; h < nq; ++h) sq += head_ss[h];
    for (int h = 0; h < nkv; ++h) sk += head_ss[nq + h];
    whole_scale[0] = rsqrtf(sq / (float)(nq * dk) + eps);
    if (nkv > 0) whole_scale[1] = rsqrtf(sk / (float)(nkv * dk) + eps);
  }
  for (int hs = warp; hs < nq + 2 * nkv; hs += warps) {
    const int kind = hs < nq ? 0 : (hs < nq + nkv ? 1 : 2);
    const int head = kind == 0 ? hs : (kind == 1 ? hs - nq : hs - nq - nkv);
    const int d = kind == 2 ? dv : dk;
    const int col = (kind == 0 ? q_col : kind == 1 ? k_col : v_col) + head * d;
    const T* src = proj + (size_t)t * row_stride + col;
    const T* b = bias ? bias + col : nullptr;
    T* dst;
    if (kind == 0) {
      dst = q_out + ((size_t)t * nq + head) * dk;
    } else {
      if (slot < 0 || slot >= num_slots) continue;
      const long long page = slot / page_size, off = slot % page_size;
      dst = (kind == 1 ? k_pages : v_pages) + page * page_stride + ((long long)head * page_size + off) * d;
    }
    if (kind == 2) {
      if (other != nullptr) {  // the token's values of another layer mixed in
        const T* o = other + (size_t)t * other_stride + head * d;
        for (int i = lane; i < d; i += 32) dst[i] = from_f32<T>((1.f - lam) * to_f32(src[i]) + lam * to_f32(o[i]));
        continue;
      }
      for (int i = lane; i < d; i += 32) dst[i] = from_f32<T>(to_f32(src[i]) + (b ? to_f32(b[i]) : 0.f));
      continue;
    }
    const float* w = kind == 0 ? q_weight : k_weight;
    if (w != nullptr && whole) w += head * d;  // a weight of the projection's size, not of the head's
    float ss = 0.f;
    for (int i = lane; i < d; i += 32) {
      const float a = to_f32(src[i]) + (b ? to_f32(b[i]) : 0.f);
      v[i] = a;
      ss += a * a;
    }
    const float scale = eps < 0.f ? 1.f : whole ? whole_scale[kind] : rsqrtf(warp_sum(ss) / (float)d + eps);
    __syncwarp();
    if (eps >= 0.f)
      for (int i = lane; i < d; i += 32) v[i] = v[i] * scale * (w ? w[i] : 1.f);
    __syncwarp();
    for (int i = lane; i < rhalf; i += 32) {
      const float c = cos_s[i], sn = sin_s[i];
      // Which two dims turn together: (i, i + rot / 2), or neighbours (2i, 2i + 1).
      const int i0 = interleaved ? 2 * i : i, i1 = interleaved ? 2 * i + 1 : i + rhalf;
      const float a0 = v[i0], a1 = v[i1];
      dst[i0] = from_f32<T>(a0 * c - a1 * sn);
      dst[i1] = from_f32<T>(a1 * c + a0 * sn);
    }
    for (int i = 2 * rhalf + lane; i < d; i += 32) dst[i] = from_f32<T>(v[i]);
    __syncwarp();  // the staging row is read before the warp's next head overwrites it
  }
}

// N consecutive elements as float32, by the widest loads there are for their bytes; and back, rounded once.
template <int BYTES>
using piece_t = std::conditional_t<BYTES == 4, unsigned, std::conditional_t<BYTES == 8, uint2, uint4>>;
template <typename T, int N>
__device__ __forceinline__ void load_row_piece(const T* src, float (&dst)[N]) {
  using V = piece_t<N * (int)sizeof(T)>;
  constexpr int EACH = (int)(sizeof(V) / sizeof(T));
#pragma unroll
  for (int at = 0; at < N; at += EACH) {
    const V v = *reinterpret_cast<const V*>(src + at);
    const T* e = reinterpret_cast<const T*>(&v);
#pragma unroll
    for (int i = 0; i < EACH; ++i) dst[at + i] = to_f32(e[i]);
  }
}
template <typename T, int N>
__device__ __forceinline__ void store_row_piece(T* dst, const float (&src)[N]) {
  using V = piece_t<N * (int)sizeof(T)>;
  constexpr int EACH = (int)(sizeof(V) / sizeof(T));
#pragma unroll
  for (int at = 0; at < N; at += EACH) {
    V v;
    T* e = reinterpret_cast<T*>(&v);
#pragma unroll
    for (int i = 0; i < EACH; ++i) e[i] = from_f32<T>(src[at + i]);
    *reinterpret_cast<V*>(dst + at) = v;
  }
}

// The same step for keys and values of one width, 32 * PL dims, and at most 8 * HPW heads (32): a warp has up to HPW heads, a
// lane PL neighbouring dims of each. Blocks stay and take every gridDim.x-th token: the norms' weights are read once, ahead of
// the wait for the kernel before, and a token's rows, position and slot are asked for while the token before it is worked
// on. The kernel above walks a warp's heads one after another, twice where the norm is over all of them, each a trip to L2
// by 2-byte loads: that, not its bytes, is what it takes its time for.
// A rotation's pairs are a lane's own (interleaved), or its and those of the lane rot / 2 dims further, which have to be a
// power of two of lanes.
template <typename T, int PL, int HPW>
__global__ void __launch_bounds__(256, PL == 8 ? 2 : 3)
qkv_prepare_vec_kernel(const T* __restrict__ proj, int row_stride, int q_col, int k_col, int v_col, int tokens, int nq, int nkv,
                       const T* __restrict__ bias, const float* __restrict__ q_weight, const float* __restrict__ k_weight,
                       float eps, const float* __restrict__ inv_freq, int rot, const int* __restrict__ positions,
                       const long long* __restrict__ slot_mapping, T* __restrict__ q_out, T* __restrict__ k_pages,
                       T* __restrict__ v_pages, long long page_stride, int page_size, long long num_slots, int whole,
                       int interleaved, const T* __restrict__ other, int other_stride, float lam, int* err) {
  constexpr int d = 32 * PL;
  using V = piece_t<PL * (int)sizeof(T)>;
  constexpr int PARTS = PL * (int)sizeof(T) / (int)sizeof(V);
  __shared__ float cos_s[2][d / 2], sin_s[2][d / 2], head_ss[2][32];  // two tokens' in turn: one barrier a token
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rhalf = inv_freq != nullptr ? rot / 2 : 0, normed = nq + nkv, heads = normed + nkv;
  auto column = [&](int hs) { return (hs < nq ? q_col + hs * d : hs < normed ? k_col + (hs - nq) * d : v_col + (hs - normed) * d) + lane * PL; };
  float w[HPW][PL];
#pragma unroll
  for (int j = 0; j < HPW; ++j) {
    const int hs = warp + 8 * j;
    const float* weight = hs < nq ? q_weight : k_weight;
#pragma unroll
    for (int e = 0; e < PL; ++e) w[j][e] = 1.f;
    if (hs < normed && eps >= 0.f && weight != nullptr)
      load_row_piece<float, PL>(weight + (whole ? (hs < nq ? hs : hs - nq) * d : 0) + lane * PL, w[j]);
  }
  const float freq = (int)threadIdx.x < rhalf ? inv_freq[threadIdx.x] : 0.f;
  pdl_wait();
  pdl_launch_dependents();
  V next[HPW][PARTS];
  int next_pos = 0;
  long long next_slot = -1;
  auto ask = [&](int t) {
    if (t >= tokens) return;
#pragma unroll
    for (int j = 0; j < HPW; ++j)
      if (warp + 8 * j < heads) {
        const V* src = reinterpret_cast<const V*>(proj + (size_t)t * row_stride + column(warp + 8 * j));
#pragma unroll
        for (int part = 0; part < PARTS; ++part) next[j][part] = src[part];
      }
    if ((int)threadIdx.x < rhalf) next_pos = positions[t];
    if (slot_mapping != nullptr) next_slot = slot_mapping[t];
  };
  ask(blockIdx.x);
  int turn = 0;
  for (int t = blockIdx.x; t < tokens; t += gridDim.x, turn ^= 1) {
    float a[HPW][PL];
#pragma unroll
    for (int j = 0; j < HPW; ++j)
#pragma unroll
      for (int e = 0; e < PL; ++e)
        a[j][e] = warp + 8 * j < heads ? to_f32(reinterpret_cast<const T*>(&next[j][e * sizeof(T) / sizeof(V)])[e % (sizeof(V) / sizeof(T))]) : 0.f;
    const int pos = next_pos;
    const long long slot = next_slot;
    ask(t + gridDim.x);
    if ((int)threadIdx.x < rhalf) sincosf((float)pos * freq, &sin_s[turn][threadIdx.x], &cos_s[turn][threadIdx.x]);
    if (nkv > 0 && slot >= num_slots && threadIdx.x == 0) atomicOr(err, OMNIA_ERR_SLOT);
    float scale[HPW];
#pragma unroll
    for (int j = 0; j < HPW; ++j) {
      const int hs = warp + 8 * j;
      if (bias != nullptr && hs < heads) {
        float b[PL];
        load_row_piece<T, PL>(bias + column(hs), b);
#pragma unroll
        for (int e = 0; e < PL; ++e) a[j][e] += b[e];
      }
      float ss = 0.f;
#pragma unroll
      for (int e = 0; e < PL; ++e) ss += a[j][e] * a[j][e];
      ss = warp_sum(ss);
      scale[j] = eps < 0.f ? 1.f : rsqrtf(ss / (float)d + eps);
      if (whole && lane == 0 && hs < normed) head_ss[turn][hs] = ss;
    }
    __syncthreads();
    if (whole && eps >= 0.f) {  // one root mean square over all heads of q, one over all heads of k
      const float ss = lane < normed ? head_ss[turn][lane] : 0.f;
      const float sq = warp_sum(lane < nq ? ss : 0.f), sk = warp_sum(lane < nq ? 0.f : ss);
      const float scale_q = rsqrtf(sq / (float)(nq * d) + eps), scale_k = nkv > 0 ? rsqrtf(sk / (float)(nkv * d) + eps) : 1.f;
#pragma unroll
      for (int j = 0; j < HPW; ++j) scale[j] = warp + 8 * j < nq ? scale_q : scale_k;
    }
    const bool stored = slot >= 0 && slot < num_slots;
    // (A 64-bit division is a hundred instructions a warp, and these set this kernel's pace: there are 24 heads of them.)
    const long long page = !stored ? 0 : slot <= 0xffffffffLL ? (unsigned)slot / (unsigned)page_size : slot / page_size;
    const long long off = stored ? slot - page * page_size : 0;
    const int apart = rhalf / PL;  // lanes to a rotation's other half
#pragma unroll
    for (int j = 0; j < HPW; ++j) {
      const int hs = warp + 8 * j;
      if (hs >= heads || (hs >= nq && !stored)) break;
      T* dst = hs < nq ? q_out + ((size_t)t * nq + hs) * d
                       : (hs < normed ? k_pages : v_pages) + page * page_stride + ((long long)(hs < normed ? hs - nq : hs - normed) * page_size + off) * d;
      if (hs >= normed) {
        if (other != nullptr) {  // the token's values of another layer mixed in
          float o[PL];
          load_row_piece<T, PL>(other + (size_t)t * other_stride + (hs - normed) * d + lane * PL, o);
#pragma unroll
          for (int e = 0; e < PL; ++e) a[j][e] = (1.f - lam) * a[j][e] + lam * o[e];
        }
        store_row_piece<T, PL>(dst + lane * PL, a[j]);
        continue;
      }
      if (eps >= 0.f) {
#pragma unroll
        for (int e = 0; e < PL; ++e) a[j][e] = a[j][e] * scale[j] * w[j][e];
      }
      if (rhalf > 0) {
        if (interleaved) {
#pragma unroll
          for (int e = 0; e < PL; e += 2) {
            const int i = (lane * PL + e) / 2;
            if (i >= rhalf) break;
            const float c = cos_s[turn][i], sn = sin_s[turn][i], a0 = a[j][e], a1 = a[j][e + 1];
            a[j][e] = a0 * c - a1 * sn;
            a[j][e + 1] = a1 * c + a0 * sn;
          }
        } else {
          const bool lower = lane < apart, turns = lane < 2 * apart;
#pragma unroll
          for (int e = 0; e < PL; ++e) {
            const float partner = __shfl_xor_sync(0xffffffffu, a[j][e], apart);
            if (!turns) continue;
            const int i = (lower ? lane : lane - apart) * PL + e;
            const float c = cos_s[turn][i], sn = sin_s[turn][i];
            a[j][e] = lower ? a[j][e] * c - partner * sn : a[j][e] * c + partner * sn;
          }
        }
      }
      store_row_piece<T, PL>(dst + lane * PL, a[j]);
    }
  }
}

template <typename T, int PL>
void launch_qkv_prepare_vec(int heads, int tokens, cudaStream_t stream, const T* proj, int row_stride, int q_col, int k_col,
                            int v_col, int nq, int nkv, const T* bias, const float* q_weight, const float* k_weight, float eps,
                            const float* inv_freq, int rot, const int* positions, const long long* slot_mapping, T* q_out,
                            T* k_pages, T* v_pages, long long page_stride, int page_size, long long num_slots, int whole,
                            int interleaved, const T* other, int other_stride, float lam, int* err) {
  const auto kernel = heads <= 8 ? qkv_prepare_vec_kernel<T, PL, 1> : heads <= 16 ? qkv_prepare_vec_kernel<T, PL, 2>
                    : heads <= 24 ? qkv_prepare_vec_kernel<T, PL, 3> : qkv_prepare_vec_kernel<T, PL, 4>;
  const int places = (PL == 8 ? 2 : 3) * omnia_sm_count();  // as many blocks an SM as the kernel's registers are bounded for
  launch_pdl(kernel, tokens < places ? tokens : places, 256, 0, stream, proj, row_stride, q_col, k_col, v_col, tokens, nq, nkv, bias, q_weight,
             k_weight, eps, inv_freq, rot, positions, slot_mapping, q_out, k_pages, v_pages, page_stride, page_size, num_slots, whole,
             interleaved, other, other_stride, lam, err);
}

extern "C" int omnia_qkv_prepare(const void* proj, int row_stride, int q_col, int k_col, int v_col, int nq, int nkv,
                                 int dk, int dv, const void* bias, const float* q_weight, const float* k_weight,
                                 float eps, const float* inv_freq, int rot, const int* positions,
                                 const long long* slot_mapping, void* q_out, void* k_pages, void* v_pages,
                                 long long page_stride, int page_size, long long num_slots, int tokens, int whole,
                                 int interleaved, const void* other, int other_stride, float lam, int dtype, int* err,
                                 cudaStream_t stream) {
  if (tokens == 0) return 0;
  if (dk > 256 || dv > 256 || rot > dk || (rot & 1) || (whole && nq + nkv > QKV_PREPARE_MAX_NORMED))
    return (int)cudaErrorInvalidValue;
  const int heads = nq + 2 * nkv;
  // Keys and values of 64, 128 or 256 dims, at most 32 heads, everything on 16 bytes, and a half-split rotation whose halves
  // are a power of two of a lane's dims: a lane's piece of a head then is one load, and its partner one exchange away.
  const int piece = dk / 32, apart = rot / 2 / (piece > 0 ? piece : 1);
  const uintptr_t starts = (uintptr_t)proj | (uintptr_t)bias | (uintptr_t)q_weight | (uintptr_t)k_weight | (uintptr_t)q_out |
                           (uintptr_t)k_pages | (uintptr_t)v_pages | (uintptr_t)other;
  const bool turns = inv_freq == nullptr || rot == 0 || interleaved || (piece > 0 && rot / 2 % piece == 0 && (apart & (apart - 1)) == 0);
  if (dk == dv && (dk == 64 || dk == 128 || dk == 256) && heads <= 32 && turns && (starts & 15) == 0 &&
      ((row_stride | q_col | k_col | v_col | other_stride) & 7) == 0 && (page_stride & 7) == 0) {
    OMNIA_DISPATCH_DTYPE(dtype, {
      const auto launch = dk == 64 ? launch_qkv_prepare_vec<T, 2> : dk == 128 ? launch_qkv_prepare_vec<T, 4> : launch_qkv_prepare_vec<T, 8>;
      launch(heads, tokens, stream, (const T*)proj, row_stride, q_col, k_col, v_col, nq, nkv, (const T*)bias, q_weight, k_weight, eps,
             inv_freq, rot, positions, slot_mapping, (T*)q_out, (T*)k_pages, (T*)v_pages, page_stride, page_size, num_slots, whole,
             interleaved, (const T*)other, other_stride, lam, err);
    });
    return OMNIA_LAUNCH_RESULT();
  }
  const int threads = heads >= 8 ? 256 : heads >= 4 ? 128 : 64;
  OMNIA_DISPATCH_DTYPE(dtype, (launch_pdl(qkv_prepare_kernel<T>, tokens, threads, 0, stream, (const T*)proj, row_stride, q_col,
                                          k_col, v_col, nq, nkv, dk, dv, (const T*)bias, q_weight, k_weight, eps,
                                          inv_freq, rot, positions, slot_mapping, (T*)q_out, (T*)k_pages, (T*)v_pages,
                                          page_stride, page_size, num_slots, whole, interleaved, (const T*)other, other_stride, lam, err)));
  return OMNIA_LAUNCH_RESULT();
}

// ---------------------------------------------------------------------------------
// angles[i][t] = (cos, sin)(positions[t] * inv_freq[i]): what a product's epilogue that rotates its
// own rows reads. It has a thread per row, so the tokens run along the table's rows: a warp's 32
// threads then read 32 neighbours. The same expression as in the kernel above, so a row rotates
// alike wherever it is rotated.
__global__ void rope_angles_kernel(const int* __restrict__ positions, const float* __restrict__ inv_freq, int half,
                                   int tokens, float2* __restrict__ out) {
  pdl_wait();
  pdl_launch_dependents();
  const long long index = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (index >= (long long)tokens * half) return;
  const int t = (int)(index / half), i = (int)(index % half);
  float sn, cs;
  sincosf((float)positions[t] * inv_freq[i], &sn, &cs);
  out[(size_t)i * tokens + t] = make_float2(cs, sn);
}

extern "C" int omnia_rope_angles(const int* positions, const float* inv_freq, int half, int tokens, void* out,
                                 cudaStream_t stream) {
  const long long total = (long long)tokens * half;
  if (total == 0) return 0;
  launch_pdl(rope_angles_kernel, (int)((total + 255) / 256), 256, 0, stream, positions, inv_freq, half, tokens,
             (float2*)out);
  return OMNIA_LAUNCH_RESULT();
}

// ---------------------------------------------------------------------------------
// act[t, i] = unit(gu[t, i], gu[t, inner + i]) in float32, rounded once, `limit` naming the unit (gated_unit in
// common.cuh; 0: silu(gate) * up). Sixteen bytes a thread (`wide`) where rows and halves start on sixteen: an element a thread
// with a 64-bit division for its row took 8.3 us for 264 rows of 6,144 bfloat16 (9.7 MB, from L2) and 15.2 for 300 of 12,288; so 4.0 and 6.0.
// Where an element a thread gives an SM no more than three blocks, the launch is the latency of one thread, and eight
// elements are one exponential after another: a row of 2,048 2.0 us by sixteen bytes, 1.6 so, 17 rows 2.0 and 1.65.
template <typename T>
__global__ void __launch_bounds__(256)
gated_rows_kernel(const T* __restrict__ gu, T* __restrict__ act, int inner, float alpha, float limit, int wide) {
  pdl_wait();
  pdl_launch_dependents();
  const T* gate = gu + (size_t)blockIdx.x * 2 * inner;
  const T* up = gate + inner;
  T* out = act + (size_t)blockIdx.x * inner;
  constexpr int VEC = 16 / (int)sizeof(T);
  const int first = blockIdx.y * blockDim.x + threadIdx.x, step = gridDim.y * blockDim.x;
  if (wide && inner % VEC == 0 && (((uintptr_t)gu | (uintptr_t)act) & 15) == 0) {
    for (int c = first * VEC; c < inner; c += step * VEC) {
      const uint4 pg = *reinterpret_cast<const uint4*>(gate + c), pu = *reinterpret_cast<const uint4*>(up + c);
      const T *g = reinterpret_cast<const T*>(&pg), *u = reinterpret_cast<const T*>(&pu);
      uint4 po;
      T* o = reinterpret_cast<T*>(&po);
#pragma unroll
      for (int e = 0; e < VEC; ++e) o[e] = from_f32<T>(gated_unit(to_f32(g[e]), to_f32(u[e]), alpha, limit));
      *reinterpret_cast<uint4*>(out + c) = po;
    }
    return;
  }
  for (int c = first; c < inner; c += step) out[c] = from_f32<T>(gated_unit(to_f32(gate[c]), to_f32(up[c]), alpha, limit));
}

// Up to this many elements a pass over them takes one a thread: three blocks an SM.
long long small_elements() { return 3LL * 256 * omnia_sm_count(); }

template <typename T>
void launch_gated_rows(const T* gu, T* act, int rows, int inner, float alpha, float limit, cudaStream_t stream) {
  const bool wide = (long long)rows * inner > small_elements();
  const int vec = wide && inner % (16 / (int)sizeof(T)) == 0 ? 16 / (int)sizeof(T) : 1, pieces = (inner / vec + 255) / 256;
  launch_pdl(gated_rows_kernel<T>, dim3(rows, pieces < 64 ? pieces : 64), 256, 0, stream, gu, act, inner, alpha, limit, (int)wide);
}

extern "C" int omnia_swiglu(const void* gu, void* act, int rows, int inner, int dtype,
                            cudaStream_t stream) {
  if (rows == 0 || inner == 0) return 0;
  OMNIA_DISPATCH_DTYPE(dtype, (launch_gated_rows<T>((const T*)gu, (T*)act, rows, inner, 1.f, 0.f, stream)));
  return OMNIA_LAUNCH_RESULT();
}

// ---------------------------------------------------------------------------------
// h = x rounded to the element type, for a part that reads the float32 residual itself.
template <typename T>
__global__ void round_rows_kernel(const float* __restrict__ x, T* __restrict__ h, long long total) {
  pdl_wait();
  pdl_launch_dependents();
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += stride) h[i] = from_f32<T>(x[i]);
}

extern "C" int omnia_round_rows(const float* x, void* h, long long total, int dtype, cudaStream_t stream) {
  if (total == 0) return 0;
  const long long most = 16LL * omnia_sm_count();
  const int blocks = (int)((total + 255) / 256 < most ? (total + 255) / 256 : most);
  OMNIA_DISPATCH_DTYPE(dtype, (launch_pdl(round_rows_kernel<T>, blocks, 256, 0, stream, x, (T*)h, total)));
  return OMNIA_LAUNCH_RESULT();
}

// ---------------------------------------------------------------------------------
// The clamped gated unit: g = min(gu[t, i], limit), u = clamp(gu[t, inner + i], -limit, limit);
// act[t, i] = g * sigmoid(alpha * g) * (u + 1), in float32, rounded once. limit < 0 selects a unit that clamps
// nothing (see gated_unit in common.cuh): -1 relu(gate) * up, -2 the tanh form of GELU, gelu(gate) * up.
extern "C" int omnia_clamped_glu(const void* gu, void* act, int rows, int inner, float alpha, float limit, int dtype,
                                 cudaStream_t stream) {
  if (rows == 0 || inner == 0) return 0;
  OMNIA_DISPATCH_DTYPE(dtype, (launch_gated_rows<T>((const T*)gu, (T*)act, rows, inner, alpha, limit, stream)));
  return OMNIA_LAUNCH_RESULT();
}

// ---------------------------------------------------------------------------------
// act = f(z) element by element, in float32, rounded once. kind 0: relu(z)^2; 1: the tanh form of
// GELU, 0.5 z (1 + tanh(sqrt(2/pi) (z + 0.044715 z^3))); 2: SiLU.
template <typename T>
__global__ void activation_kernel(const T* __restrict__ z, T* __restrict__ act, long long total, int kind, float first,
                                  float second) {
  pdl_wait();
  pdl_launch_dependents();
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x; idx < total; idx += stride) {
    const float v = to_f32(z[idx]);
    float y;
    if (kind == 0) {
      const float r = fmaxf(v, 0.f);
      y = r * r;
    } else if (kind == 1) {
      y = 0.5f * v * (1.f + tanhf(0.7978845608028654f * (v + 0.044715f * v * v * v)));
    } else if (kind == 2) {
      y = v / (1.f + expf(-v));
    } else if (kind == 3) {
      y = xielu(v, first, second);
    } else {
      y = gelu_erf(v);
    }
    act[idx] = from_f32<T>(y);
  }
}

// kind: 0 relu^2, 1 tanh-GELU, 2 SiLU, 3 xIELU with the constants `first` (above zero) and `second` (below), 4 exact GELU.
extern "C" int omnia_activation(const void* z, void* act, long long total, int kind, float first, float second, int dtype,
                                cudaStream_t stream) {
  if (total == 0) return 0;
  if (kind < 0 || kind > 4) return (int)cudaErrorInvalidValue;
  const long long most = 16LL * omnia_sm_count();
  const int blocks = (int)((total + 255) / 256 < most ? (total + 255) / 256 : most);
  OMNIA_DISPATCH_DTYPE(dtype, (launch_pdl(activation_kernel<T>, blocks, 256, 0, stream, (const T*)z, (T*)act,
                                          total, kind, first, second)));
  return OMNIA_LAUNCH_RESULT();
}

// ---------------------------------------------------------------------------------
// In place: out[t, c] *= sigmoid(gate[t, c]), the gate's rows `gate_stride` apart; float32, rounded once. A block
// per token; sixteen bytes a thread where both rows start on sixteen.
template <typename T>
__global__ void __launch_bounds__(256)
gate_rows_kernel(T* __restrict__ out, const T* __restrict__ gate, int gate_stride, int width) {
  pdl_wait();
  pdl_launch_dependents();
  T* o = out + (size_t)blockIdx.x * width;
  const T* g = gate + (size_t)blockIdx.x * gate_stride;
  constexpr int VEC = 16 / (int)sizeof(T);
  if (width % VEC == 0 && gate_stride % VEC == 0 && (((uintptr_t)out | (uintptr_t)gate) & 15) == 0) {
    for (int c = threadIdx.x * VEC; c < width; c += blockDim.x * VEC) {
      uint4 po = *reinterpret_cast<const uint4*>(o + c);
      const uint4 pg = *reinterpret_cast<const uint4*>(g + c);
      T* vo = reinterpret_cast<T*>(&po);
      const T* vg = reinterpret_cast<const T*>(&pg);
#pragma unroll
      for (int e = 0; e < VEC; ++e) vo[e] = from_f32<T>(to_f32(vo[e]) / (1.f + expf(-to_f32(vg[e]))));
      *reinterpret_cast<uint4*>(o + c) = po;
    }
    return;
  }
  for (int c = threadIdx.x; c < width; c += blockDim.x) o[c] = from_f32<T>(to_f32(o[c]) / (1.f + expf(-to_f32(g[c]))));
}

extern "C" int omnia_gate_rows(void* out, const void* gate, int gate_stride, int tokens, int width, int dtype,
                               cudaStream_t stream) {
  if (tokens == 0 || width == 0) return 0;
  OMNIA_DISPATCH_DTYPE(dtype, (launch_pdl(gate_rows_kernel<T>, tokens, 256, 0, stream, (T*)out, (const T*)gate, gate_stride,
                                          width)));
  return OMNIA_LAUNCH_RESULT();
}

// ---------------------------------------------------------------------------------
// out = sa * a + sb * b, the sum taken in float32 and rounded once: two branches that read the same
// input meet with a constant each.
template <typename T>
__global__ void scaled_sum_kernel(const T* __restrict__ a, float sa, const T* __restrict__ b, float sb, T* __restrict__ out,
                                  long long total) {
  pdl_wait();
  pdl_launch_dependents();
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x; idx < total; idx += stride)
    out[idx] = from_f32<T>(fmaf(sa, to_f32(a[idx]), sb * to_f32(b[idx])));
}

extern "C" int omnia_scaled_sum(const void* a, float sa, const void* b, float sb, void* out, long long total, int dtype,
                                cudaStream_t stream) {
  if (total == 0) return 0;
  const long long most = 16LL * omnia_sm_count();
  const int blocks = (int)((total + 255) / 256 < most ? (total + 255) / 256 : most);
  OMNIA_DISPATCH_DTYPE(dtype, (launch_pdl(scaled_sum_kernel<T>, blocks, 256, 0, stream, (const T*)a, sa, (const T*)b, sb,
                                          (T*)out, total)));
  return OMNIA_LAUNCH_RESULT();
}

// ---------------------------------------------------------------------------------
// logits = cap * tanh(z * multiplier / cap)  (cap <= 0: logits = z * multiplier), float32 out.
// Sixteen bytes of z a thread (`wide`) where both start on sixteen (64 rows of 151,936: 21 us an element a thread, 15 so);
// an element a thread where there are few, as for the gated units (4 rows of 512: 2.0 and 1.6 us, a row of 32,000 2.05 and 1.65).
template <typename T>
__global__ void __launch_bounds__(256)
softcap_kernel(const T* __restrict__ z, float* __restrict__ out, long long total, float multiplier, float cap, int wide) {
  pdl_wait();
  pdl_launch_dependents();
  constexpr int VEC = 16 / (int)sizeof(T);
  const long long at = (long long)blockIdx.x * blockDim.x + threadIdx.x, stride = (long long)gridDim.x * blockDim.x;
  auto capped = [&](T a) {
    const float v = to_f32(a) * multiplier;
    return cap > 0.f ? cap * tanhf(v / cap) : v;
  };
  const long long whole = wide && (((uintptr_t)z | (uintptr_t)out) & 15) == 0 ? total / VEC : 0;
  for (long long i = at; i < whole; i += stride) {
    const uint4 piece = reinterpret_cast<const uint4*>(z)[i];
    const T* a = reinterpret_cast<const T*>(&piece);
    float v[VEC];
#pragma unroll
    for (int e = 0; e < VEC; ++e) v[e] = capped(a[e]);
#pragma unroll
    for (int e = 0; e < VEC; e += 4)
      reinterpret_cast<float4*>(out + i * VEC)[e / 4] = make_float4(v[e], v[e + 1], v[e + 2], v[e + 3]);
  }
  for (long long i = whole * VEC + at; i < total; i += stride) out[i] = capped(z[i]);
}

extern "C" int omnia_softcap(const void* z, float* out, long long total, float multiplier,
                             float cap, int dtype, cudaStream_t stream) {
  if (total == 0) return 0;
  const long long pieces = (total + 255) / 256, most = 16LL * omnia_sm_count();
  OMNIA_DISPATCH_DTYPE(dtype, (launch_pdl(softcap_kernel<T>, (int)(pieces < most ? pieces : most), 256, 0, stream, (const T*)z, out,
                                          total, multiplier, cap, total > small_elements())));
  return OMNIA_LAUNCH_RESULT();
}

// ---------------------------------------------------------------------------------
// out[r] = src[rows[r]]  (rows of `width` elements)
template <typename T>
__global__ void gather_rows_kernel(const T* __restrict__ src, const int* __restrict__ rows,
                                   T* __restrict__ out, int width) {
  pdl_wait();
  pdl_launch_dependents();
  const T* s = src + (size_t)rows[blockIdx.x] * width;
  T* o = out + (size_t)blockIdx.x * width;
  for (int i = threadIdx.x; i < width; i += blockDim.x) o[i] = s[i];
}

extern "C" int omnia_gather_rows(const void* src, const int* rows, void* out, int count, int width,
                                 int dtype, cudaStream_t stream) {
  if (count == 0) return 0;
  OMNIA_DISPATCH_DTYPE(dtype, (launch_pdl(gather_rows_kernel<T>, count, 256, 0, stream, 
                                  (const T*)src, rows, (T*)out, width)));
  return OMNIA_LAUNCH_RESULT();
}

// ---------------------------------------------------------------------------------
// The state of requests about to run their first step: slot slots[s] of every tensor i (slots of bytes[i]) becomes
// from[i] (one slot's worth), or zeros. The slots' numbers travel in the launch itself: indices copied from pageable
// memory made the host wait for all earlier steps, and a fill for each tensor cost a launch each (a prompt of 2,048
// tokens through eight layers, two of them with state: the GPU stood idle for 0.4 ms between two such steps).
#define OMNIA_FILL_TENSORS 32
#define OMNIA_FILL_SLOTS 128
struct SlotFill {
  unsigned char* to[OMNIA_FILL_TENSORS];
  const unsigned char* from[OMNIA_FILL_TENSORS];
  long long bytes[OMNIA_FILL_TENSORS];
  int slots[OMNIA_FILL_SLOTS];
};
__global__ void fill_slots_kernel(const __grid_constant__ SlotFill fill) {
  pdl_wait();
  pdl_launch_dependents();
  const int i = blockIdx.y;
  const long long bytes = fill.bytes[i];
  unsigned char* to = fill.to[i] + fill.slots[blockIdx.z] * bytes;
  const unsigned char* from = fill.from[i];
  const long long at = blockIdx.x * (long long)blockDim.x + threadIdx.x, step = gridDim.x * (long long)blockDim.x;
  if (((bytes | reinterpret_cast<uintptr_t>(fill.to[i]) | reinterpret_cast<uintptr_t>(from)) & 15) == 0) {
    const uint4 zero = make_uint4(0, 0, 0, 0);
    for (long long c = at; c < bytes / 16; c += step)
      reinterpret_cast<uint4*>(to)[c] = from ? reinterpret_cast<const uint4*>(from)[c] : zero;
  } else {
    for (long long c = at; c < bytes; c += step) to[c] = from ? from[c] : 0;
  }
}

extern "C" int omnia_fill_slots(const void* const* to, const void* const* from, const long long* bytes, int tensors,
                                const int* slots, int count, cudaStream_t stream) {
  if (tensors == 0 || count == 0) return 0;
  if (tensors < 0 || tensors > OMNIA_FILL_TENSORS || count < 0 || count > OMNIA_FILL_SLOTS) return (int)cudaErrorInvalidValue;
  SlotFill fill = {};
  long long most = 0;
  for (int i = 0; i < tensors; ++i) {
    fill.to[i] = (unsigned char*)const_cast<void*>(to[i]), fill.from[i] = (const unsigned char*)from[i], fill.bytes[i] = bytes[i];
    most = bytes[i] > most ? bytes[i] : most;
  }
  for (int s = 0; s < count; ++s) fill.slots[s] = slots[s];
  const long long pieces = (most / 16 + 255) / 256;
  launch_pdl(fill_slots_kernel, dim3((unsigned)(pieces < 1 ? 1 : pieces > 64 ? 64 : pieces), tensors, count), 256, 0, stream, fill);
  return OMNIA_LAUNCH_RESULT();
}

// ---------------------------------------------------------------------------------
// A decode step's requests cut into pieces for the decode attention kernel, a block a piece and key/value head. Chunks at
// fixed positions give a short request's only chunk as much of the GPU as a long one's, and the last blocks run alone. Here a
// request is cut into equal parts of at most `size` tiles of 32 keys, `size` the least with which the parts of all
// requests fit into one or two times `places` (the blocks a head that the GPU holds at a time), and the parts are
// listed largest first: SMs are given blocks in turn, so each gets its share of every size. Which of the two is estimated:
// blocks an SM times their mean size, but no less than `chain` times the largest (a block's tiles come one after another, and an
// SM with fewer blocks than `chain` waits for memory most of the time), and PIECE_WAVE tiles of an SM's time for a
// second round of blocks (their starts). Without `chain`, 64 requests of 1,000 positions were 64 pieces: steps of eight
// layers with heads of 64 took 755 us, with it 648 (by chunks 652); heads of 128: 918, 867 (884).
// PIECE_WAVE from 0 to 52 and PIECE_LEAST from 1 to 8 made no difference beyond 1 % (16 to 100 requests of unequal lengths,
// two models), PIECE_LEAST 16 cost 6 to 12 %.
// (Positions kept in sight below a window are not counted: a request's first piece has their few tiles on top of its own.)
// Lengths are on the device alone in a replayed step, hence a kernel, once for all layers that see as far: one block, a warp
// for each of the two to find its size, a thread for each request to list its parts.
constexpr int PIECE_LEAST = 4, PIECE_ROUNDS = 2, PIECE_WAVE = 13, PIECE_THREADS = 256;
__global__ void __launch_bounds__(PIECE_THREADS)
decode_pieces_kernel(const int* __restrict__ seq_lens, int requests, int window, int run, int nkv, int places, int rounds, int chain, int sms,
                     DecodePiece* __restrict__ list) {
  __shared__ int tiles[PIECE_THREADS], parts[PIECE_THREADS], sizes[PIECE_THREADS];
  __shared__ int found[PIECE_ROUNDS], cost[PIECE_ROUNDS];
  pdl_wait();
  pdl_launch_dependents();
  const int r = threadIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int pos = r < requests ? seq_lens[r] - 1 : -1;
  int first = window > 0 ? max(0, pos - window + 1) : 0;
  if (run > 0 && pos >= 0) first = max(first, pos - pos % run);
  const int mine = pos < 0 ? 0 : pos / 32 - first / 32 + 1;
  tiles[r] = mine;
  __syncthreads();
  if (warp < rounds) {
    const int room = places * (warp + 1);
    int total = 0, most = 0, live = 0;
    for (int i = lane; i < PIECE_THREADS; i += 32) total += tiles[i], most = max(most, tiles[i]), live += tiles[i] > 0;
    total = __reduce_add_sync(0xffffffffu, total), most = __reduce_max_sync(0xffffffffu, most), live = __reduce_add_sync(0xffffffffu, live);
    auto needed = [&](int size) {
      int need = 0;
      for (int i = lane; i < PIECE_THREADS; i += 32) need += (tiles[i] + size - 1) / size;
      return (int)__reduce_add_sync(0xffffffffu, need);
    };
    int lo = max(PIECE_LEAST, (total + room - 1) / room), hi = max(lo, most);  // the least size that fits lies within
    while (lo < hi) {
      const int mid = (lo + hi) / 2;
      if (needed(mid) <= room) hi = mid; else lo = mid + 1;
    }
    const int count = needed(lo);
    if (lane == 0) {
      found[warp] = lo;
      const int blocks = count * nkv;
      cost[warp] = live > room || count == 0 ? 0x7fffffff
                                             : max((int)((long long)((blocks + sms - 1) / sms) * total / count), chain * lo) + PIECE_WAVE * warp;
    }
  }
  __syncthreads();
  int round = 0;
  for (int i = 1; i < rounds; ++i)
    if (cost[i] < cost[round]) round = i;
  const int size = found[round], count = (mine + size - 1) / size, part = count > 0 ? (mine + count - 1) / count : 0;
  parts[r] = count, sizes[r] = part;
  __syncthreads();
  int before = 0, all = 0;
  for (int i = 0; i < requests; ++i) {
    const int n = parts[i], s = sizes[i];
    all += n;
    if (s > part || (s == part && i < r)) before += n;
  }
  const int base = count > 0 ? mine / count : 0, longer = count > 0 ? mine - base * count : 0;  // the first `longer` parts have a tile more
  for (int i = 0; i < count; ++i) {
    const int tile = first / 32 + i * base + min(i, longer), next = tile + base + (i < longer);
    list[before + i] = DecodePiece{r, pos, max(first, tile * 32), min(pos, next * 32 - 1), i, count, before, 0};
  }
  for (int i = all + r; i < places * rounds; i += PIECE_THREADS) list[i].request = -1;
}

// list: room for rounds * places pieces of eight ints, on 16 bytes. At most 256 requests, no more than that room, and 2 rounds.
extern "C" int omnia_decode_pieces(const int* seq_lens, int requests, int window, int run, int nkv, int places, int rounds, int chain, int sms,
                                   void* list, cudaStream_t stream) {
  if (requests < 1 || requests > PIECE_THREADS || places < 1 || rounds < 1 || rounds > PIECE_ROUNDS || requests > rounds * places || chain < 0 || sms < 1 ||
      nkv < 1 || ((uintptr_t)list & 15))
    return (int)cudaErrorInvalidValue;
  launch_pdl(decode_pieces_kernel, 1, PIECE_THREADS, 0, stream, seq_lens, requests, window, run, nkv, places, rounds, chain, sms, (DecodePiece*)list);
  return OMNIA_LAUNCH_RESULT();
}
