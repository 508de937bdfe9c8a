// The recurrence of lightning.cu over a portion's tokens, a chunk of L tokens at a time on the tensor cores. With S the
// state ahead of a chunk and d the head's decay, token i of a chunk (from 0) of n:
//
//   o_i = d^(i+1) S^T q_i + sum_(j <= i) d^(i-j) (q_i . k_j) v_j
//   S  <- d^n S + sum_j d^(n-1-j) k_j v_j^T
//
// Token by token the chain of multiply-adds is as long as the portion; a chunk is four products, q k^T, its weighted
// lower triangle times v, q S, and k^T times the weighted v, some 6 us, and what bounds it is those products on a
// block's eight warps (a head's columns are the only other thing to share out). 16 heads of 128: 2,048 tokens 421 us
// -> 97, 600 + 300 + 5 tokens 165 -> 44, 32 tokens 13.2 -> 8.8, 16 tokens 9.4 -> 9.1. The activated q, k and v are
// bfloat16 as lightning.cu rounds them, so they are exact operands; everything else that enters a product (the weighted
// triangle, the weighted v, the state) is float32 and goes in as the sum of three bfloat16 numbers, 24 bits of mantissa
// for numbers from 2^-109 up. Sums and the carried state are float32, sixteen products at a time from zero and
// then added on the ordinary cores: the tensor cores' own running sum cuts off what does not fit instead of rounding
// it. From the result in 64 bits, after 2,048 tokens: outputs 1.1e-7 and state 1.4e-7 (token by token 1.2e-7 and
// 5.8e-7; with running sums 2e-6 both), after 128: 7.6e-8 and 6.5e-8 (6.0e-8 and 1.8e-7). The powers of the decay are
// made in float64 and rounded once.
//
// That holds for finite numbers of ordinary size. Where something is infinite or NaN (or overflows on its way through a
// product, or as a bfloat16), a chunk's products would carry it to tokens that come before it, since a weight of zero
// times it is NaN, and would make NaN of an infinity taken apart. Whatever went in, an output or the last state that is
// not finite comes of it; the block then walks its tokens once more, one by one as lightning.cu does, from the state in
// memory, which it writes only at its end.
//
// A block owns LIGHTNING_COLS value columns of one head of one request and walks its chunks in order; a column of S
// needs no other column. Warp w has 16 of the chunk's tokens for the first three products (the tokens dealt so that the
// two warps of a scheduler have equal shares of the triangle) and 16 of the state's rows for the last, whose float32
// values never leave its registers; the other warps read them as triples from shared memory. The next chunk's q, k
// and v come in by asynchronous copies meanwhile, activated and laid side by side by a kernel of their own (every
// block of a head would otherwise activate the same q and k again).
//
// Compiled per key width and columns: -DLIGHTNING_DK=<DK> (a multiple of 16), -DLIGHTNING_COLS=<16 or 32>.
#include "common.cuh"

#ifndef LIGHTNING_DK
#define LIGHTNING_DK 128
#endif
#ifndef LIGHTNING_COLS
#define LIGHTNING_COLS 32
#endif

namespace {

typedef __nv_bfloat16 bf16;

constexpr int N = LIGHTNING_DK, COLS = LIGHTNING_COLS;
static_assert(N % 16 == 0 && (COLS == 16 || COLS == 32), "sizes the tensor cores' tiles fit");
constexpr int NROW = N + 8, XROW = COLS + 8;  // rows of shared memory in elements: an odd number of 16-byte pieces

constexpr size_t smem_bytes(int L) {
  return sizeof(bf16) * (2 * (size_t)L * (2 * NROW + XROW) + 3 * N * XROW + 3 * L * XROW) + sizeof(float) * (L + 1);
}
constexpr int L = N <= 128 && smem_bytes(128) <= 227 * 1024 ? 128 : 64;
static_assert(smem_bytes(L) <= 227 * 1024, "a chunk fits shared memory");
constexpr int WARPS = L / 16, THREADS = 32 * WARPS;
// The state's tiles of 16 rows x 8 columns: MPW row tiles a warp, or several warps to a row tile.
constexpr int MT = N / 16, MPW = (MT + WARPS - 1) / WARPS;
constexpr int share(int warps_a_tile) {
  return warps_a_tile >= 4 && COLS >= 32 ? 4 : warps_a_tile >= 2 ? 2 : 1;
}
constexpr int CW = share(WARPS / MT);  // warps that share a row tile's columns
constexpr int NT = COLS / 8, NTW = NT / CW;

__device__ __forceinline__ uint32_t shared_address(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void copy16(const void* smem, const void* gmem, bool valid) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(shared_address(smem)), "l"(gmem), "r"(valid ? 16 : 0)
               : "memory");
}
__device__ __forceinline__ void ldmatrix(uint32_t* r, const bf16* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(shared_address(p)));
}
__device__ __forceinline__ void ldmatrix_t(uint32_t* r, const bf16* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(shared_address(p)));
}
// c = a b + c, c a sum of products of its own (`first`: from zero).
__device__ __forceinline__ void mma(float* c, const uint32_t* a, uint32_t b0, uint32_t b1, bool first) {
  if (first) c[0] = c[1] = c[2] = c[3] = 0.f;
  asm(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void add(float* sum, const float* c) {
#pragma unroll
  for (int e = 0; e < 4; ++e) sum[e] += c[e];
}
// (u, v) as three pairs of bfloat16 whose sum has 24 bits of mantissa.
__device__ __forceinline__ void split(float u, float v, uint32_t* part) {
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(u, v);
    part[i] = *reinterpret_cast<const uint32_t*>(&h);
    u -= __low2float(h), v -= __high2float(h);
  }
}

// q | k | v of the listed requests' projected rows, silu in float32, rounded to bfloat16 as lightning.cu does: rows [tokens,
// 2 heads DK + heads dv].
__global__ void lightning_act_kernel(const bf16* __restrict__ proj, int stride, int q_col, int k_col, int v_col, int qk, int width,
                                     const int* __restrict__ cu_seqlens, const int* __restrict__ entries, bf16* __restrict__ rows) {
  pdl_wait();
  pdl_launch_dependents();
  const int across = width / 8, seq = entries ? entries[blockIdx.y] : blockIdx.y;
  const long long last = (long long)cu_seqlens[seq + 1] * across;
  for (long long i = (long long)cu_seqlens[seq] * across + blockIdx.x * (long long)blockDim.x + threadIdx.x; i < last;
       i += gridDim.x * (long long)blockDim.x) {
    const int c = (int)(i % across) * 8;
    const bf16* src = proj + (i / across) * stride + (c < qk ? q_col + c : c < 2 * qk ? k_col + c - qk : v_col + c - 2 * qk);
    uint4 piece;
    bf16* e = reinterpret_cast<bf16*>(&piece);
    if ((reinterpret_cast<uintptr_t>(src) & 15) == 0) {
      piece = *reinterpret_cast<const uint4*>(src);
    } else {
#pragma unroll
      for (int k = 0; k < 8; ++k) e[k] = src[k];
    }
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const float x = __bfloat162float(e[k]);
      e[k] = __float2bfloat16_rn(__fdividef(x, 1.f + __expf(-x)));
    }
    reinterpret_cast<uint4*>(rows)[i] = piece;
  }
}

__global__ void __launch_bounds__(THREADS, 1)
lightning_chunk_kernel(const bf16* __restrict__ rows, int H, int dv, const float* __restrict__ decay, float* __restrict__ S_state,
                       const int* __restrict__ cu_seqlens, const int* __restrict__ state_slots, const int* __restrict__ entries,
                       float* __restrict__ o_raw) {
  extern __shared__ __align__(16) unsigned char chunk_smem[];
  bf16* stage0 = reinterpret_cast<bf16*>(chunk_smem);  // two stages of [L][NROW] k, [L][NROW] q, [L][XROW] v
  constexpr int STAGE = L * (2 * NROW + XROW);
  bf16* Ss = stage0 + 2 * STAGE;  // [3][N][XROW] the state in three parts
  bf16* Ws = Ss + 3 * N * XROW;   // [3][L][XROW] the weighted v in three parts
  float* power = reinterpret_cast<float*>(Ws + 3 * L * XROW);  // [L + 1] the decay's powers

  const int parts = dv / COLS, head = blockIdx.x / parts, col0 = (blockIdx.x % parts) * COLS;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int g = lane >> 2, t4 = lane & 3, mat = lane >> 3, r8 = lane & 7;
  for (int i = tid; i <= L; i += THREADS) {
    // By squaring, in float64.
    double p = 1.0, s = decay[head];
    for (int e = i; e; e >>= 1, s *= s)
      if (e & 1) p *= s;
    power[i] = (float)p;
  }
  pdl_wait();
  pdl_launch_dependents();
  const int seq = entries ? entries[blockIdx.y] : blockIdx.y;
  const int begin = cu_seqlens[seq], end = cu_seqlens[seq + 1];
  if (end <= begin) return;
  const int row_stride = 2 * H * N + H * dv;
  const bf16* q_rows = rows + head * N;
  const bf16* k_rows = rows + (H + head) * N;
  const bf16* v_rows = rows + 2 * H * N + head * dv + col0;

  auto fetch = [&](int t0, int n, int b) {
    bf16* Kd = stage0 + b * STAGE;
    bf16* Qd = Kd + L * NROW;
    bf16* Vd = Qd + L * NROW;
    const int fill = min(L, (n + 31) & ~31);  // rows past the portion's end are zeros, up to a whole block of keys
    for (int i = tid; i < fill * (N / 8); i += THREADS) {
      const int r = i / (N / 8), c = (i % (N / 8)) * 8;
      const size_t from = (size_t)(t0 + (r < n ? r : 0)) * row_stride + c;
      copy16(Kd + r * NROW + c, k_rows + from, r < n);
      copy16(Qd + r * NROW + c, q_rows + from, r < n);
    }
    for (int i = tid; i < fill * (COLS / 8); i += THREADS) {
      const int r = i / (COLS / 8), c = (i % (COLS / 8)) * 8;
      copy16(Vd + r * XROW + c, v_rows + (size_t)(t0 + (r < n ? r : 0)) * row_stride + c, r < n);
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  };

  // This warp's part of the state: row tiles m0, m0 + 1, ..., columns from c0.
  const int m0 = (warp / CW) * MPW, c0 = (warp % CW) * NTW * 8;
  float S[MPW][NTW][4];
  float* mine = S_state + ((size_t)state_slots[seq] * H + head) * N * dv + col0 + c0 + 2 * t4;
  auto read_state = [&]() {
#pragma unroll
    for (int m = 0; m < MPW; ++m)
#pragma unroll
      for (int nt = 0; nt < NTW; ++nt)
#pragma unroll
        for (int side = 0; side < 2; ++side) {
          float2 v = make_float2(0.f, 0.f);
          if (m0 + m < MT) v = *reinterpret_cast<const float2*>(mine + (size_t)((m0 + m) * 16 + g + 8 * side) * dv + nt * 8);
          S[m][nt][2 * side] = v.x, S[m][nt][2 * side + 1] = v.y;
        }
  };
  read_state();

  const int tile = WARPS == 8 && warp >= 4 ? 11 - warp : warp, row0 = tile * 16;
  const int chunks = (end - begin + L - 1) / L;
  fetch(begin, min(L, end - begin), 0);
  float probe = 0.f;  // NaN once something this thread made was not finite
  for (int c = 0; c < chunks; ++c) {
    const int t0 = begin + c * L, n = min(L, end - t0), b = c & 1;
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    __syncthreads();  // the chunk has arrived, and everybody is done with the last one
    if (c + 1 < chunks) fetch(t0 + L, min(L, end - t0 - L), b ^ 1);
    const bf16 *Kc = stage0 + b * STAGE, *Qc = Kc + L * NROW, *Vc = Qc + L * NROW;
#pragma unroll
    for (int m = 0; m < MPW; ++m)
      if (m0 + m < MT)
#pragma unroll
        for (int nt = 0; nt < NTW; ++nt)
#pragma unroll
          for (int side = 0; side < 2; ++side) {
            uint32_t part[3];
            split(S[m][nt][2 * side], S[m][nt][2 * side + 1], part);
#pragma unroll
            for (int p = 0; p < 3; ++p)
              *reinterpret_cast<uint32_t*>(Ss + (p * N + (m0 + m) * 16 + g + 8 * side) * XROW + c0 + nt * 8 + 2 * t4) = part[p];
          }
    const int key_rows = (n + 15) & ~15;
#pragma unroll 4
    for (int i = tid; i < key_rows * (COLS / 2); i += THREADS) {
      const int r = i / (COLS / 2), place = r * XROW + (i % (COLS / 2)) * 2;
      const float w = r < n ? power[n - 1 - r] : 0.f;
      const float2 v = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(Vc + place));
      uint32_t part[3];
      split(w * v.x, w * v.y, part);
#pragma unroll
      for (int p = 0; p < 3; ++p) *reinterpret_cast<uint32_t*>(Ws + p * L * XROW + place) = part[p];
    }
    __syncthreads();  // the state and the weighted v are complete as operands
    if (row0 < n) {
      uint32_t cf[N / 16][4];
#pragma unroll
      for (int ks = 0; ks < N / 16; ++ks) ldmatrix(cf[ks], Qc + (row0 + (mat & 1) * 8 + r8) * NROW + ks * 16 + (mat >> 1) * 8);
      float acc[NT][4];
#pragma unroll
      for (int nt = 0; nt < NT; ++nt) acc[nt][0] = acc[nt][1] = acc[nt][2] = acc[nt][3] = 0.f;
#pragma unroll
      for (int ks = 0; ks < N / 16; ++ks)
#pragma unroll
        for (int pair = 0; pair < NT / 2; ++pair) {
          const int place = (ks * 16 + (mat & 1) * 8 + r8) * XROW + pair * 16 + (mat >> 1) * 8;
          float sum[2][4];
#pragma unroll
          for (int p = 2; p >= 0; --p) {
            uint32_t s[4];
            ldmatrix_t(s, Ss + p * N * XROW + place);
            mma(sum[0], cf[ks], s[0], s[1], p == 2);
            mma(sum[1], cf[ks], s[2], s[3], p == 2);
          }
          add(acc[2 * pair], sum[0]);
          add(acc[2 * pair + 1], sum[1]);
        }
      const float ea = power[min(row0 + g + 1, L)], eb = power[min(row0 + g + 9, L)];
#pragma unroll
      for (int nt = 0; nt < NT; ++nt) acc[nt][0] *= ea, acc[nt][1] *= ea, acc[nt][2] *= eb, acc[nt][3] *= eb;
      // The keys in blocks of 32, up to this warp's last token.
      const int blocks = (min(row0 + 16, n) + 31) / 32;
#pragma unroll 1
      for (int kb = 0; kb < blocks; ++kb) {
        float p[4][4];
#pragma unroll
        for (int j = 0; j < 4; ++j) p[j][0] = p[j][1] = p[j][2] = p[j][3] = 0.f;
#pragma unroll
        for (int ks = 0; ks < N / 16; ++ks)
#pragma unroll
          for (int j2 = 0; j2 < 2; ++j2) {
            uint32_t bm[4];
            ldmatrix(bm, Kc + (kb * 32 + j2 * 16 + (mat >> 1) * 8 + r8) * NROW + ks * 16 + (mat & 1) * 8);
            float sum[2][4];
            mma(sum[0], cf[ks], bm[0], bm[1], true);
            mma(sum[1], cf[ks], bm[2], bm[3], true);
            add(p[2 * j2], sum[0]);
            add(p[2 * j2 + 1], sum[1]);
          }
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const int key = kb * 32 + j * 8 + 2 * t4 + e;
            p[j][e] = key <= row0 + g ? p[j][e] * power[row0 + g - key] : 0.f;
            p[j][2 + e] = key <= row0 + g + 8 ? p[j][2 + e] * power[row0 + g + 8 - key] : 0.f;
          }
#pragma unroll
        for (int kk = 0; kk < 2; ++kk) {
          uint32_t part[4][3];
          split(p[2 * kk][0], p[2 * kk][1], part[0]);
          split(p[2 * kk][2], p[2 * kk][3], part[1]);
          split(p[2 * kk + 1][0], p[2 * kk + 1][1], part[2]);
          split(p[2 * kk + 1][2], p[2 * kk + 1][3], part[3]);
#pragma unroll
          for (int pair = 0; pair < NT / 2; ++pair) {
            uint32_t xv[4];
            ldmatrix_t(xv, Vc + (kb * 32 + kk * 16 + (mat & 1) * 8 + r8) * XROW + pair * 16 + (mat >> 1) * 8);
            float sum[2][4];
#pragma unroll
            for (int s = 2; s >= 0; --s) {
              const uint32_t a[4] = {part[0][s], part[1][s], part[2][s], part[3][s]};
              mma(sum[0], a, xv[0], xv[1], s == 2);
              mma(sum[1], a, xv[2], xv[3], s == 2);
            }
            add(acc[2 * pair], sum[0]);
            add(acc[2 * pair + 1], sum[1]);
          }
        }
      }
#pragma unroll
      for (int side = 0; side < 2; ++side) {
        const int r = row0 + g + 8 * side;
        if (r >= n) continue;
        float* out = o_raw + (size_t)(t0 + r) * H * dv + head * dv + col0 + 2 * t4;
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) {
          *reinterpret_cast<float2*>(out + nt * 8) = make_float2(acc[nt][2 * side], acc[nt][2 * side + 1]);
          probe = fmaf(acc[nt][2 * side + 1], 0.f, fmaf(acc[nt][2 * side], 0.f, probe));
        }
      }
    }
    const float kept = power[n];
#pragma unroll
    for (int m = 0; m < MPW; ++m) {
      if (m0 + m >= MT) continue;
#pragma unroll
      for (int nt = 0; nt < NTW; ++nt)
#pragma unroll
        for (int e = 0; e < 4; ++e) S[m][nt][e] *= kept;
#pragma unroll 2
      for (int ks = 0; ks < key_rows / 16; ++ks) {
        uint32_t bt[4];
        ldmatrix_t(bt, Kc + (ks * 16 + (mat >> 1) * 8 + r8) * NROW + (m0 + m) * 16 + (mat & 1) * 8);
        if constexpr (NTW == 1) {
          // One tile of eight columns: two of its parts in one load, the third ahead of them.
          uint32_t w[4];
          float sum[4];
          ldmatrix_t(w, Ws + (2 * L + ks * 16 + (mat & 1) * 8 + r8) * XROW + c0);
          mma(sum, bt, w[0], w[1], true);
          ldmatrix_t(w, Ws + ((mat >> 1) * L + ks * 16 + (mat & 1) * 8 + r8) * XROW + c0);
          mma(sum, bt, w[2], w[3], false);
          mma(sum, bt, w[0], w[1], false);
          add(S[m][0], sum);
        } else {
#pragma unroll
          for (int pair = 0; pair < NTW / 2; ++pair) {
            float sum[2][4];
#pragma unroll
            for (int p = 2; p >= 0; --p) {
              uint32_t w[4];
              ldmatrix_t(w, Ws + (p * L + ks * 16 + (mat & 1) * 8 + r8) * XROW + c0 + pair * 16 + (mat >> 1) * 8);
              mma(sum[0], bt, w[0], w[1], p == 2);
              mma(sum[1], bt, w[2], w[3], p == 2);
            }
            add(S[m][2 * pair], sum[0]);
            add(S[m][2 * pair + 1], sum[1]);
          }
        }
      }
    }
  }
#pragma unroll
  for (int m = 0; m < MPW; ++m)
#pragma unroll
    for (int nt = 0; nt < NTW; ++nt)
#pragma unroll
      for (int e = 0; e < 4; ++e) probe = fmaf(S[m][nt][e], 0.f, probe);
  if (__syncthreads_or(probe != 0.f)) {
    constexpr int SHARES = WARPS / CW;           // warps that hold rows of a column
    float* sums = reinterpret_cast<float*>(Ws);  // [2][SHARES][COLS], of alternate tokens
    const bf16 *Kc = stage0, *Qc = Kc + L * NROW, *Vc = Qc + L * NROW;
    const float d = decay[head];
    read_state();
#pragma unroll 1
    for (int t0 = begin; t0 < end; t0 += L) {
      const int n = min(L, end - t0);
      fetch(t0, n, 0);
      asm volatile("cp.async.wait_group 0;\n" ::: "memory");
      __syncthreads();
#pragma unroll 1
      for (int i = 0; i < n; ++i) {
        float* share = sums + ((i & 1) * SHARES + warp / CW) * COLS + c0 + 2 * t4;
#pragma unroll
        for (int nt = 0; nt < NTW; ++nt) {
          const float2 v = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(Vc + i * XROW + c0 + nt * 8 + 2 * t4));
          float2 o = make_float2(0.f, 0.f);
#pragma unroll
          for (int m = 0; m < MPW; ++m)
#pragma unroll
            for (int side = 0; side < 2; ++side) {
              if (m0 + m >= MT) continue;
              const int at = i * NROW + (m0 + m) * 16 + g + 8 * side;
              const float k = __bfloat162float(Kc[at]), q = __bfloat162float(Qc[at]);
              float* s = S[m][nt] + 2 * side;
              s[0] = fmaf(k, v.x, d * s[0]), s[1] = fmaf(k, v.y, d * s[1]);
              o.x = fmaf(s[0], q, o.x), o.y = fmaf(s[1], q, o.y);
            }
#pragma unroll
          for (int w = 4; w < 32; w <<= 1) {
            o.x += __shfl_xor_sync(0xffffffffu, o.x, w);
            o.y += __shfl_xor_sync(0xffffffffu, o.y, w);
          }
          if (g == 0) *reinterpret_cast<float2*>(share + nt * 8) = o;
        }
        __syncthreads();
        if (tid < COLS) {
          float o = 0.f;
#pragma unroll
          for (int w = 0; w < SHARES; ++w) o += sums[((i & 1) * SHARES + w) * COLS + tid];
          o_raw[(size_t)(t0 + i) * H * dv + head * dv + col0 + tid] = o;
        }
      }
      __syncthreads();  // the stage and the sums may be written again
    }
  }
#pragma unroll
  for (int m = 0; m < MPW; ++m)
    if (m0 + m < MT)
#pragma unroll
      for (int nt = 0; nt < NTW; ++nt)
#pragma unroll
        for (int side = 0; side < 2; ++side)
          *reinterpret_cast<float2*>(mine + (size_t)((m0 + m) * 16 + g + 8 * side) * dv + nt * 8) =
              make_float2(S[m][nt][2 * side], S[m][nt][2 * side + 1]);
}

}  // namespace

// As omnia_lightning_recurrence (lightning.cu) for bfloat16 rows, of the `count` requests that `entries` lists (null: of the
// first `count`), the longest of which brings `longest` tokens; `rows` is room for [the step's tokens, 2 H DK + H dv]
// bfloat16 on 16 bytes, dv a multiple of LIGHTNING_COLS.
extern "C" int omnia_lightning_chunk(const void* proj, int stride, int q_col, int k_col, int v_col, int H, int dv, int longest,
                                     void* rows, const float* decay, float* S_state, const int* cu_seqlens,
                                     const int* state_slots, const int* entries, int count, float* o_raw, cudaStream_t stream) {
  if (count == 0 || longest == 0) return 0;
  if (H < 1 || dv < COLS || dv % COLS || count < 0 || longest < 0 || (((uintptr_t)rows | (uintptr_t)S_state | (uintptr_t)o_raw) & 15))
    return (int)cudaErrorInvalidValue;
  int device = 0;
  static bool configured[64] = {};
  if (cudaGetDevice(&device) != cudaSuccess || device < 0 || device >= 64) return (int)cudaErrorInvalidDevice;
  if (!configured[device]) {
    const cudaError_t e =
        cudaFuncSetAttribute(lightning_chunk_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_bytes(L));
    if (e != cudaSuccess) return (int)e;
    configured[device] = true;
  }
  const int width = 2 * H * N + H * dv;
  const long long blocks = ((long long)longest * (width / 8) + 255) / 256, most = (8LL * omnia_sm_count() + count - 1) / count;
  launch_pdl(lightning_act_kernel, dim3((unsigned)(blocks < most ? blocks : most), count), dim3(256), 0, stream, (const bf16*)proj,
             stride, q_col, k_col, v_col, H * N, width, cu_seqlens, entries, (bf16*)rows);
  launch_pdl(lightning_chunk_kernel, dim3(H * (dv / COLS), count), dim3(THREADS), smem_bytes(L), stream, (const bf16*)rows, H, dv,
             decay, S_state, cu_seqlens, state_slots, entries, o_raw);
  return OMNIA_LAUNCH_RESULT();
}
