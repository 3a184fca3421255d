// CUDA-core attention (forward and backward), fp32 math for any element type.
// It is the full-precision path for fp32 tensors (tensor cores would round the
// operands) and the fallback for shapes the tensor-core kernels do not take.
//
// Bound (counters at 8x12 heads x 1024 x 64 fp32 causal): the backward by shared-memory reads, 66 and 72 % of the wavefronts an SM can
// serve; the forward by the latency of its 16 warps (36 %, issue slots 45 %, most stalls on shared memory and the FMA pipe).
// A block of 256 threads owns 64 or 128 rows (queries; keys in the dK/dV kernel) and
// walks the other sequence in tiles of 64 rows in shared memory. A thread computes TI x 4 scores: 16
// neighbouring lanes share its TI rows and hold columns 16 apart, so a 16-byte read of the rows is a
// broadcast and one of the columns conflict-free, and 4 k of both feed TI x 16 multiplications (TI = 4: 12
// shared-memory wavefronts against 64 FMA clocks of a warp). The dot products run on packed
// fma.rn.f32x2, even and odd elements in separate sums. A row's 64 scores stay within its warp: online
// softmax by shuffles over 16 lanes, probabilities through shared memory without a block barrier, and
// the second products read them back four at a time. No atomics: results are reproducible.
// Forward and backward of that case 2.1 ms (one row per warp with scalar shared-memory reads 10.6).
// Masked keys and queries have weight 0; where a causal tile that they lie in holds values that are not finite (0 * NaN), its
// products walk each row's visible part only.
// Tensors are addressed as base + b*sb + h*sh + row*ss + d; head_dim is padded with zeros to DP.
#include "common.cuh"
#include "attention.cuh"
#include <atomic>

namespace mt {

constexpr int kMaxD = 128;
constexpr int kAtThreads = 256;
constexpr int kAtCols = 64;                 // rows of the other sequence per tile
constexpr int kAtPitch = kAtCols + 4;       // pitch of a row of scores

__device__ __forceinline__ void fma2(uint64_t& d, uint64_t a, uint64_t b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}
__device__ __forceinline__ uint64_t pack2(float a, float b) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ float2 unpack2(uint64_t v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}

// dst[r][d] = mul * src row row0 + r, r < ROWS, d < DP: zero past the sequence and past D.
template <typename T, int DP, int ROWS>
__device__ __forceinline__ void load_rows(float* dst, const T* src, int64_t stride, int row0, int total, int D, float mul, bool vec) {
  constexpr int VN = Vec16<T>::N, PER = DP / VN;
  if (vec) {
#pragma unroll 4
    for (int i = threadIdx.x; i < ROWS * PER; i += kAtThreads) {
      const int r = i / PER, c = (i - r * PER) * VN;
      Vec16<T> t;
      t.u = make_uint4(0, 0, 0, 0);
      if (row0 + r < total && c < D) t.load(src + (int64_t)(row0 + r) * stride + c);
#pragma unroll
      for (int e = 0; e < VN; e += 4)
        *reinterpret_cast<float4*>(dst + r * (DP + 4) + c + e) =
            make_float4(t.get(e) * mul, t.get(e + 1) * mul, t.get(e + 2) * mul, t.get(e + 3) * mul);
    }
  } else {
    for (int i = threadIdx.x; i < ROWS * DP; i += kAtThreads) {
      const int r = i / DP, c = i - r * DP;
      dst[r * (DP + 4) + c] = row0 + r < total && c < D ? to_f(src[(int64_t)(row0 + r) * stride + c]) * mul : 0.f;
    }
  }
}

// Whether this thread's part of a 64-row tile in shared memory holds a value that is not finite.
template <int DP>
__device__ __forceinline__ bool tile_odd(const float* tile) {
  bool odd = false;
#pragma unroll 2
  for (int i = threadIdx.x; i < kAtCols * DP / 4; i += kAtThreads) {
    const float4 v = *reinterpret_cast<const float4*>(tile + i / (DP / 4) * (DP + 4) + i % (DP / 4) * 4);
    odd |= !(isfinite(v.x) && isfinite(v.y) && isfinite(v.z) && isfinite(v.w));
  }
  return odd;
}

// s[i][j] = rows[i] . cols[j]: this thread's rows start at `rows` (two apart), its columns at `cols` (16 apart).
template <int DP, int TI>
__device__ __forceinline__ void dots(float (&s)[TI][4], const float* rows, const float* cols) {
  uint64_t acc[TI][4];
#pragma unroll
  for (int i = 0; i < TI; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0;
#pragma unroll (TI == 8 ? 1 : 2)
  for (int d = 0; d < DP; d += 4) {
    ulonglong2 c[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) c[j] = *reinterpret_cast<const ulonglong2*>(cols + j * 16 * (DP + 4) + d);
#pragma unroll
    for (int i = 0; i < TI; ++i) {
      const ulonglong2 r = *reinterpret_cast<const ulonglong2*>(rows + i * 2 * (DP + 4) + d);
#pragma unroll
      for (int j = 0; j < 4; ++j) { fma2(acc[i][j], r.x, c[j].x); fma2(acc[i][j], r.y, c[j].y); }
    }
  }
#pragma unroll
  for (int i = 0; i < TI; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) { const float2 v = unpack2(acc[i][j]); s[i][j] = v.x + v.y; }
}

// acc[i][p] += sum over 64 j of w[i][j] * x[j][32 p + 2 tx .. + 1]; w = this thread's rows of scores, x shifted by 2 tx.
template <int DP, int TI>
__device__ __forceinline__ void combine(uint64_t (&acc)[TI][DP / 32], const float* w, const float* x) {
#pragma unroll (TI == 8 ? 1 : 2)
  for (int j = 0; j < kAtCols; j += 4) {
    uint64_t v[4][DP / 32];
#pragma unroll
    for (int e = 0; e < 4; ++e)
#pragma unroll
      for (int p = 0; p < DP / 32; ++p) v[e][p] = *reinterpret_cast<const uint64_t*>(x + (j + e) * (DP + 4) + 32 * p);
#pragma unroll
    for (int i = 0; i < TI; ++i) {
      const float4 q = *reinterpret_cast<const float4*>(w + i * 2 * kAtPitch + j);
      const uint64_t q4[4] = {pack2(q.x, q.x), pack2(q.y, q.y), pack2(q.z, q.z), pack2(q.w, q.w)};
#pragma unroll
      for (int e = 0; e < 4; ++e)
#pragma unroll
        for (int p = 0; p < DP / 32; ++p) fma2(acc[i][p], q4[e], v[e][p]);
    }
  }
}

// The same over row i's j in [lo + 2 i, hi + 2 i) alone: whatever stands in the other rows of x, or for them in w, is not touched.
template <int DP, int TI>
__device__ __forceinline__ void combine_visible(uint64_t (&acc)[TI][DP / 32], const float* w, const float* x, int lo, int hi) {
#pragma unroll 1
  for (int j = 0; j < kAtCols; ++j) {
#pragma unroll
    for (int i = 0; i < TI; ++i) {
      if (j < lo + 2 * i || j >= hi + 2 * i) continue;
      const float q = w[i * 2 * kAtPitch + j];
      const uint64_t q2 = pack2(q, q);
#pragma unroll
      for (int p = 0; p < DP / 32; ++p) fma2(acc[i][p], q2, *reinterpret_cast<const uint64_t*>(x + j * (DP + 4) + 32 * p));
    }
  }
}

template <typename T, int DP>
__device__ __forceinline__ void store_row(T* dst, const uint64_t (&acc)[DP / 32], float mul, int tx, int D) {
#pragma unroll
  for (int p = 0; p < DP / 32; ++p) {
    const float2 v = unpack2(acc[p]);
    const int d = 32 * p + 2 * tx;
    if (d < D) dst[d] = from_f<T>(v.x * mul);
    if (d + 1 < D) dst[d + 1] = from_f<T>(v.y * mul);
  }
}

struct SimtParams {
  const void* q; const void* k; const void* v; const void* d_o;
  void* o; void* dq; void* dk; void* dv;
  float* lse; const float* delta;
  mt_strides3 sq, sk, sv, so, sdo, sdq, sdk, sdv;
  int heads, kv_heads, group, S, D, causal, vec;
  float scale;
};

// Blocks per SM that shared memory allows: the register budget follows from it.
constexpr int at_resident(int dp, int ti) { return dp <= 64 || (dp <= 96 && ti == 4) ? 2 : 1; }
template <int DP, int TI> constexpr int fwd_smem() { return (16 * TI * (DP + 4) + 2 * kAtCols * (DP + 4) + 16 * TI * kAtPitch) * 4; }
template <int DP> constexpr int bwd_smem() { return (4 * kAtCols * (DP + 4) + kAtCols * kAtPitch + 2 * kAtCols) * 4; }

template <typename T, int DP, int TI>
__global__ void __launch_bounds__(kAtThreads, at_resident(DP, TI))
attn_fwd_simt(const SimtParams P) {
  constexpr int ROWS = 16 * TI;
  extern __shared__ __align__(16) float sm[];
  float* Qs = sm;                            // [ROWS][DP + 4], scaled
  float* Ks = Qs + ROWS * (DP + 4);          // [64][DP + 4]
  float* Vs = Ks + kAtCols * (DP + 4);       // [64][DP + 4]
  float* Ps = Vs + kAtCols * (DP + 4);       // [ROWS][68]
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, half = lane >> 4, tx = lane & 15;
  const int b = blockIdx.y / P.heads, h = blockIdx.y % P.heads, hk = h / P.group;
  const int row_base = (int)(gridDim.x - 1 - blockIdx.x) * ROWS;          // causal: a head's longest rows start first
  const int S = P.S, D = P.D;
  const T* kb = (const T*)P.k + (int64_t)b * P.sk.b + (int64_t)hk * P.sk.h;
  const T* vb = (const T*)P.v + (int64_t)b * P.sv.b + (int64_t)hk * P.sv.h;
  load_rows<T, DP, ROWS>(Qs, (const T*)P.q + (int64_t)b * P.sq.b + (int64_t)h * P.sq.h, P.sq.s, row_base, S, D, P.scale, P.vec);
  const int r0 = warp * 2 * TI + half;       // this thread's rows: r0, r0 + 2, ...
  const int warp_last = row_base + warp * 2 * TI + 2 * TI - 1;
  float m[TI], l[TI];
  uint64_t acc[TI][DP / 32];
#pragma unroll
  for (int i = 0; i < TI; ++i) {
    m[i] = -INFINITY; l[i] = 0.f;
#pragma unroll
    for (int p = 0; p < DP / 32; ++p) acc[i][p] = 0;
  }
  const int kv_end = P.causal ? min(row_base + ROWS, S) : S;
  for (int t0 = 0; t0 < kv_end; t0 += kAtCols) {
    __syncthreads();
    load_rows<T, DP, kAtCols>(Ks, kb, P.sk.s, t0, S, D, 1.f, P.vec);
    load_rows<T, DP, kAtCols>(Vs, vb, P.sv.s, t0, S, D, 1.f, P.vec);
    __syncthreads();
    bool odd = false;                                       // on the diagonal: rows that not every query sees, and not all finite
    if (P.causal && t0 + kAtCols > row_base + 1) odd = __syncthreads_or(tile_odd<DP>(Vs));
    if (P.causal && t0 > warp_last) continue;               // no row of this warp sees the tile
    float s[TI][4];
    dots<DP, TI>(s, Qs + r0 * (DP + 4), Ks + tx * (DP + 4));
    const bool edge = t0 + kAtCols > S || (P.causal && t0 + kAtCols > row_base + warp * 2 * TI + 1);
    __syncwarp();
#pragma unroll
    for (int i = 0; i < TI; ++i) {
      const int gr = row_base + r0 + 2 * i;
      if (edge) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int gj = t0 + tx + 16 * j;
          if (gj >= S || (P.causal && gj > gr)) s[i][j] = -INFINITY;
        }
      }
      float mx = fmaxf(fmaxf(s[i][0], s[i][1]), fmaxf(s[i][2], s[i][3]));
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
      const float mn = fmaxf(m[i], mx);
      const float corr = m[i] == -INFINITY ? 0.f : __expf(m[i] - mn);
      float sum = 0.f;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float p = s[i][j] == -INFINITY ? 0.f : __expf(s[i][j] - mn);
        sum += p;
        Ps[(r0 + 2 * i) * kAtPitch + tx + 16 * j] = p;
      }
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
      l[i] = l[i] * corr + sum;
      m[i] = mn;
      const uint64_t c2 = pack2(corr, corr);
#pragma unroll
      for (int p = 0; p < DP / 32; ++p) asm("mul.rn.f32x2 %0, %0, %1;" : "+l"(acc[i][p]) : "l"(c2));
    }
    __syncwarp();
    if (odd) combine_visible<DP, TI>(acc, Ps + r0 * kAtPitch, Vs + 2 * tx, -kAtCols, row_base + r0 + 1 - t0);
    else combine<DP, TI>(acc, Ps + r0 * kAtPitch, Vs + 2 * tx);
  }
  T* ob = (T*)P.o + (int64_t)b * P.so.b + (int64_t)h * P.so.h;
#pragma unroll
  for (int i = 0; i < TI; ++i) {
    const int gr = row_base + r0 + 2 * i;
    if (gr >= S) continue;
    store_row<T, DP>(ob + (int64_t)gr * P.so.s, acc[i], l[i] > 0.f ? 1.f / l[i] : 0.f, tx, D);
    if (tx == 0) P.lse[(int64_t)blockIdx.y * S + gr] = m[i] + __logf(l[i]);
  }
}

// delta[b,h,i] = sum_d dO[i,d] * O[i,d]. Eight lanes per row, 16-byte loads when
// head_dim and the strides allow (traffic: one read of O and dO).
template <typename T>
__global__ void __launch_bounds__(256)
attn_delta_kernel(const T* __restrict__ o, const T* __restrict__ d_o, float* __restrict__ delta, mt_strides3 so,
                  mt_strides3 sdo, int heads, int S, int D, int64_t total_rows, int vec) {
  constexpr int VN = Vec16<T>::N;
  const int sub = threadIdx.x & 7;
  const int64_t row = (int64_t)blockIdx.x * 32 + (threadIdx.x >> 3);
  float s = 0.f;
  if (row < total_rows) {
    const int64_t bh = row / S;
    const int i = (int)(row - bh * S);
    const int b = (int)(bh / heads), h = (int)(bh % heads);
    const T* op = o + (int64_t)b * so.b + (int64_t)h * so.h + (int64_t)i * so.s;
    const T* dp = d_o + (int64_t)b * sdo.b + (int64_t)h * sdo.h + (int64_t)i * sdo.s;
    if (vec) {
      for (int d = sub * VN; d < D; d += 8 * VN) {
        Vec16<T> a, g;
        a.load(op + d);
        g.load(dp + d);
#pragma unroll
        for (int e = 0; e < VN; ++e) s += a.get(e) * g.get(e);
      }
    } else {
      for (int d = sub; d < D; d += 8) s += to_f(op[d]) * to_f(dp[d]);
    }
  }
  s += __shfl_xor_sync(0xffffffffu, s, 1);
  s += __shfl_xor_sync(0xffffffffu, s, 2);
  s += __shfl_xor_sync(0xffffffffu, s, 4);
  if (sub == 0 && row < total_rows) delta[row] = s;
}

template <typename T, int DP>
__global__ void __launch_bounds__(kAtThreads, DP <= 64 ? 2 : 1)
attn_bwd_dq_simt(const SimtParams P) {
  constexpr int TI = 4, ROWS = 64;
  extern __shared__ __align__(16) float sm[];
  float* Qs = sm;                            // [64][DP + 4], scaled
  float* Gs = Qs + ROWS * (DP + 4);          // dO rows
  float* Ks = Gs + ROWS * (DP + 4);
  float* Vs = Ks + kAtCols * (DP + 4);
  float* Ps = Vs + kAtCols * (DP + 4);       // dS
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, half = lane >> 4, tx = lane & 15;
  const int b = blockIdx.y / P.heads, h = blockIdx.y % P.heads, hk = h / P.group;
  const int row_base = (int)(gridDim.x - 1 - blockIdx.x) * ROWS;
  const int S = P.S, D = P.D;
  const T* kb = (const T*)P.k + (int64_t)b * P.sk.b + (int64_t)hk * P.sk.h;
  const T* vb = (const T*)P.v + (int64_t)b * P.sv.b + (int64_t)hk * P.sv.h;
  load_rows<T, DP, ROWS>(Qs, (const T*)P.q + (int64_t)b * P.sq.b + (int64_t)h * P.sq.h, P.sq.s, row_base, S, D, P.scale, P.vec);
  load_rows<T, DP, ROWS>(Gs, (const T*)P.d_o + (int64_t)b * P.sdo.b + (int64_t)h * P.sdo.h, P.sdo.s, row_base, S, D, 1.f, P.vec);
  const int r0 = warp * 2 * TI + half;
  const int warp_last = row_base + warp * 2 * TI + 2 * TI - 1;
  float lrow[TI], drow[TI];
  uint64_t acc[TI][DP / 32];
#pragma unroll
  for (int i = 0; i < TI; ++i) {
    const int gr = row_base + r0 + 2 * i;
    lrow[i] = gr < S ? P.lse[(int64_t)blockIdx.y * S + gr] : 0.f;
    drow[i] = gr < S ? P.delta[(int64_t)blockIdx.y * S + gr] : 0.f;
#pragma unroll
    for (int p = 0; p < DP / 32; ++p) acc[i][p] = 0;
  }
  const int kv_end = P.causal ? min(row_base + ROWS, S) : S;
  for (int t0 = 0; t0 < kv_end; t0 += kAtCols) {
    __syncthreads();
    load_rows<T, DP, kAtCols>(Ks, kb, P.sk.s, t0, S, D, 1.f, P.vec);
    load_rows<T, DP, kAtCols>(Vs, vb, P.sv.s, t0, S, D, 1.f, P.vec);
    __syncthreads();
    bool odd = false;
    if (P.causal && t0 + kAtCols > row_base + 1) odd = __syncthreads_or(tile_odd<DP>(Ks) | tile_odd<DP>(Vs));
    if (P.causal && t0 > warp_last) continue;
    float p[TI][4], dp[TI][4];
    dots<DP, TI>(p, Qs + r0 * (DP + 4), Ks + tx * (DP + 4));
#pragma unroll
    for (int i = 0; i < TI; ++i) {
      const int gr = row_base + r0 + 2 * i;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int gj = t0 + tx + 16 * j;
        p[i][j] = gj < S && gr < S && (!P.causal || gj <= gr) ? __expf(p[i][j] - lrow[i]) : 0.f;
      }
    }
    dots<DP, TI>(dp, Gs + r0 * (DP + 4), Vs + tx * (DP + 4));
    __syncwarp();
#pragma unroll
    for (int i = 0; i < TI; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) Ps[(r0 + 2 * i) * kAtPitch + tx + 16 * j] = p[i][j] * (dp[i][j] - drow[i]) * P.scale;
    __syncwarp();
    if (odd) combine_visible<DP, TI>(acc, Ps + r0 * kAtPitch, Ks + 2 * tx, -kAtCols, row_base + r0 + 1 - t0);
    else combine<DP, TI>(acc, Ps + r0 * kAtPitch, Ks + 2 * tx);
  }
  T* dqb = (T*)P.dq + (int64_t)b * P.sdq.b + (int64_t)h * P.sdq.h;
#pragma unroll
  for (int i = 0; i < TI; ++i) {
    const int gr = row_base + r0 + 2 * i;
    if (gr < S) store_row<T, DP>(dqb + (int64_t)gr * P.sdq.s, acc[i], 1.f, tx, D);
  }
}

// The block owns rows of one key/value head and sums the contributions of the `group` query heads that read it.
template <typename T, int DP>
__global__ void __launch_bounds__(kAtThreads, DP <= 64 ? 2 : 1)
attn_bwd_dkv_simt(const SimtParams P) {
  constexpr int TI = 4, ROWS = 64;
  extern __shared__ __align__(16) float sm[];
  float* Ks = sm;                            // [64][DP + 4] this block's key rows, scaled
  float* Vs = Ks + ROWS * (DP + 4);
  float* Qs = Vs + ROWS * (DP + 4);          // query tile
  float* Gs = Qs + kAtCols * (DP + 4);       // dO tile
  float* Ps = Gs + kAtCols * (DP + 4);       // P, then dS: [key][query]
  float* Ls = Ps + ROWS * kAtPitch;          // lse and delta of the query tile
  float* Ds = Ls + kAtCols;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, half = lane >> 4, tx = lane & 15;
  const int b = blockIdx.y / P.kv_heads, h = blockIdx.y % P.kv_heads;
  const int row_base = (int)blockIdx.x * ROWS;            // causal: the first keys are read by the most queries
  const int S = P.S, D = P.D;
  load_rows<T, DP, ROWS>(Ks, (const T*)P.k + (int64_t)b * P.sk.b + (int64_t)h * P.sk.h, P.sk.s, row_base, S, D, P.scale, P.vec);
  load_rows<T, DP, ROWS>(Vs, (const T*)P.v + (int64_t)b * P.sv.b + (int64_t)h * P.sv.h, P.sv.s, row_base, S, D, 1.f, P.vec);
  const int r0 = warp * 2 * TI + half;
  uint64_t acck[TI][DP / 32], accv[TI][DP / 32];
#pragma unroll
  for (int i = 0; i < TI; ++i)
#pragma unroll
    for (int p = 0; p < DP / 32; ++p) { acck[i][p] = 0; accv[i][p] = 0; }
  const int q_begin = P.causal ? row_base : 0;            // only queries i >= j see key j (ROWS == kAtCols)
  for (int gq = 0; gq < P.group; ++gq) {
    const int hq = h * P.group + gq;
    const int64_t bhq = (int64_t)b * P.heads + hq;
    const T* qb = (const T*)P.q + (int64_t)b * P.sq.b + (int64_t)hq * P.sq.h;
    const T* gb = (const T*)P.d_o + (int64_t)b * P.sdo.b + (int64_t)hq * P.sdo.h;
    for (int t0 = q_begin; t0 < S; t0 += kAtCols) {
      __syncthreads();
      load_rows<T, DP, kAtCols>(Qs, qb, P.sq.s, t0, S, D, 1.f, P.vec);
      load_rows<T, DP, kAtCols>(Gs, gb, P.sdo.s, t0, S, D, 1.f, P.vec);
      if (threadIdx.x < kAtCols) {
        const int gi = t0 + threadIdx.x;
        Ls[threadIdx.x] = gi < S ? P.lse[bhq * S + gi] : 0.f;
        Ds[threadIdx.x] = gi < S ? P.delta[bhq * S + gi] : 0.f;
      }
      __syncthreads();
      bool odd = false;
      if (P.causal && t0 < row_base + ROWS - 1)
        odd = __syncthreads_or(tile_odd<DP>(Qs) | tile_odd<DP>(Gs) | !isfinite(Ds[threadIdx.x % kAtCols]));
      float p[TI][4], ds[TI][4];
      dots<DP, TI>(p, Ks + r0 * (DP + 4), Qs + tx * (DP + 4));
#pragma unroll
      for (int i = 0; i < TI; ++i) {
        const int gj = row_base + r0 + 2 * i;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int c = tx + 16 * j, gi = t0 + c;
          p[i][j] = gi < S && gj < S && (!P.causal || gj <= gi) ? __expf(p[i][j] - Ls[c]) : 0.f;
          Ps[(r0 + 2 * i) * kAtPitch + c] = p[i][j];
        }
      }
      __syncwarp();
      if (odd) combine_visible<DP, TI>(accv, Ps + r0 * kAtPitch, Gs + 2 * tx, row_base + r0 - t0, 3 * kAtCols);
      else combine<DP, TI>(accv, Ps + r0 * kAtPitch, Gs + 2 * tx);
      dots<DP, TI>(ds, Vs + r0 * (DP + 4), Gs + tx * (DP + 4));
      __syncwarp();
#pragma unroll
      for (int i = 0; i < TI; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int c = tx + 16 * j;
          Ps[(r0 + 2 * i) * kAtPitch + c] = p[i][j] * (ds[i][j] - Ds[c]) * P.scale;
        }
      __syncwarp();
      if (odd) combine_visible<DP, TI>(acck, Ps + r0 * kAtPitch, Qs + 2 * tx, row_base + r0 - t0, 3 * kAtCols);
      else combine<DP, TI>(acck, Ps + r0 * kAtPitch, Qs + 2 * tx);
    }
  }
  T* dkb = (T*)P.dk + (int64_t)b * P.sdk.b + (int64_t)h * P.sdk.h;
  T* dvb = (T*)P.dv + (int64_t)b * P.sdv.b + (int64_t)h * P.sdv.h;
#pragma unroll
  for (int i = 0; i < TI; ++i) {
    const int gj = row_base + r0 + 2 * i;
    if (gj >= S) continue;
    store_row<T, DP>(dkb + (int64_t)gj * P.sdk.s, acck[i], 1.f, tx, D);
    store_row<T, DP>(dvb + (int64_t)gj * P.sdv.s, accv[i], 1.f, tx, D);
  }
}

int attn_delta(const AttnArgs& a, cudaStream_t st) {
  const int64_t rows = a.batch * a.heads * a.seq;
  if (rows == 0) return MT_OK;
  MT_DISPATCH_FLOAT(a.dtype, T, {
    constexpr int VN = Vec16<T>::N;
    auto ok = [&](const mt_strides3& s) { return s.b % VN == 0 && s.h % VN == 0 && s.s % VN == 0; };
    const int vec = a.head_dim % VN == 0 && aligned16(a.o) && aligned16(a.d_o) && ok(a.so) && ok(a.sdo);
    attn_delta_kernel<T><<<(unsigned)((rows + 31) / 32), 256, 0, st>>>(
        (const T*)a.o, (const T*)a.d_o, a.delta, a.so, a.sdo, (int)a.heads, (int)a.seq, (int)a.head_dim, rows, vec);
  });
  MT_LAUNCH_CHECK();
  return MT_OK;
}

static SimtParams simt_params(const AttnArgs& a, bool bwd) {
  SimtParams p{};
  p.q = a.q; p.k = a.k; p.v = a.v; p.d_o = a.d_o; p.o = a.o_out; p.dq = a.dq; p.dk = a.dk; p.dv = a.dv;
  p.lse = a.lse; p.delta = a.delta;
  p.sq = a.sq; p.sk = a.sk; p.sv = a.sv; p.so = a.so; p.sdo = a.sdo; p.sdq = a.sdq; p.sdk = a.sdk; p.sdv = a.sdv;
  p.heads = (int)a.heads; p.kv_heads = (int)a.kv_heads; p.group = (int)(a.heads / a.kv_heads);
  p.S = (int)a.seq; p.D = (int)a.head_dim; p.causal = a.causal; p.scale = a.scale;
  const int vn = a.dtype == MT_F32 ? 4 : 8;
  auto ok = [&](const void* ptr, const mt_strides3& s) { return aligned16(ptr) && s.b % vn == 0 && s.h % vn == 0 && s.s % vn == 0; };
  p.vec = p.D % vn == 0 && ok(a.q, a.sq) && ok(a.k, a.sk) && ok(a.v, a.sv) && (!bwd || ok(a.d_o, a.sdo));
  return p;
}

static int launch_simt(void (*kern)(const SimtParams), std::atomic<bool>* ready, dim3 grid, int smem, const SimtParams& p,
                       cudaStream_t st) {
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 16 || !ready[dev].load(std::memory_order_acquire)) {    // racing first calls set the same attribute twice, harmlessly
    MT_CHECK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    if (dev >= 0 && dev < 16) ready[dev].store(true, std::memory_order_release);
  }
  kern<<<grid, kAtThreads, smem, st>>>(p);
  MT_LAUNCH_CHECK();
  return MT_OK;
}

template <typename T, int DP, int TI>
static int launch_fwd_simt(const AttnArgs& a, cudaStream_t st) {
  static std::atomic<bool> ready[16];
  const dim3 grid((unsigned)((a.seq + 16 * TI - 1) / (16 * TI)), (unsigned)(a.batch * a.heads));
  return launch_simt(attn_fwd_simt<T, DP, TI>, ready, grid, fwd_smem<DP, TI>(), simt_params(a, false), st);
}

template <typename T, int DP>
static int launch_fwd_simt(const AttnArgs& a, cudaStream_t st) {
  // 128 rows per block read K and V half as often; 64 where they would leave SMs without a block
  return a.batch * a.heads * ((a.seq + 127) / 128) >= 2 * sm_count() ? launch_fwd_simt<T, DP, 8>(a, st) : launch_fwd_simt<T, DP, 4>(a, st);
}

template <typename T, int DP>
static int launch_bwd_simt(const AttnArgs& a, cudaStream_t st) {
  static std::atomic<bool> ready_q[16], ready_kv[16];
  const unsigned tiles = (unsigned)((a.seq + 63) / 64);
  const SimtParams p = simt_params(a, true);
  const int rc = launch_simt(attn_bwd_dq_simt<T, DP>, ready_q, dim3(tiles, (unsigned)(a.batch * a.heads)), bwd_smem<DP>(), p, st);
  return rc ? rc : launch_simt(attn_bwd_dkv_simt<T, DP>, ready_kv, dim3(tiles, (unsigned)(a.batch * a.kv_heads)), bwd_smem<DP>(), p, st);
}

#define MT_SIMT_DIM(FN, T, D) \
  return (D) <= 32 ? FN<T, 32>(a, st) : (D) <= 64 ? FN<T, 64>(a, st) : (D) <= 96 ? FN<T, 96>(a, st) : FN<T, 128>(a, st)

int attn_fwd_simt_launch(const AttnArgs& a, cudaStream_t st) {
  if (a.batch * a.heads * a.seq == 0) return MT_OK;
  MT_REQUIRE(a.head_dim <= kMaxD && a.head_dim > 0, "attention: head_dim must be in [1,128]");
  MT_REQUIRE(a.batch * a.heads <= 65535, "attention: batch*heads too large for the CUDA-core kernel");
  MT_DISPATCH_FLOAT(a.dtype, T, MT_SIMT_DIM(launch_fwd_simt, T, a.head_dim));
  return MT_OK;
}

int attn_bwd_simt_launch(const AttnArgs& a, cudaStream_t st) {
  if (a.batch * a.heads * a.seq == 0) return MT_OK;
  MT_REQUIRE(a.head_dim <= kMaxD && a.head_dim > 0, "attention: head_dim must be in [1,128]");
  MT_REQUIRE(a.batch * a.heads <= 65535, "attention: batch*heads too large for the CUDA-core kernel");
  const int rc = attn_delta(a, st);
  if (rc) return rc;
  MT_DISPATCH_FLOAT(a.dtype, T, MT_SIMT_DIM(launch_bwd_simt, T, a.head_dim));
  return MT_OK;
}
#undef MT_SIMT_DIM

}  // namespace mt
