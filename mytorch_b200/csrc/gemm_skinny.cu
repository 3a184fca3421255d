// Products with few rows (M <= 64) that stream a weight matrix W[N,K] once: what a decoding step
// and a tiny batch spend their time on. HBM-bound: algorithmic traffic N*K*s (+ x and y).
//
// A 128-row tcgen05 tile would run one CTA per 128 columns - 6 to 24 of 148 SMs for the widths of a
// block - with K walked by one producer thread. Here every SM streams its share of the weight rows:
//   * A round is 1-5 groups of weight rows (8 rows per group in half types, 4 in fp32). Groups travel
//     by bulk copies into a ring of rounds in shared memory, as far ahead as the ring allows (60-200
//     KB per SM): HBM sees runs of 12 KB, where 16-byte loads in fragment order (64-byte runs)
//     reached only 3 of 6.4 TB/s.
//   * The eight warps of a block split K between them, so the work on a row has no long chain even
//     where a layer has one group per SM; their sums meet in shared memory in a fixed order. Long K
//     (the down-projections) is split further over a cluster whose blocks add their partial sums
//     through distributed shared memory: each block then reads 1/2 to 1/8 of x.
//   * The order of k in a dot product is free as long as both operands agree, so 16 consecutive
//     bytes of a row (8 k) are the B fragments of two mma.m16n8k16 (tokens as rows, weight rows as
//     columns) and the A fragments are the same pieces of x: no ldmatrix, no transposes. fp32 uses
//     FFMA, four k per lane.
//   * The first rounds are requested before griddepcontrol.wait when the caller says the weights are
//     constants: they travel while the previous kernel in the stream finishes.
//   * A LayerNorm or RMSNorm in front of the product is folded in: each block normalises the rows
//     in shared memory (a few KB out of L2) instead of a kernel of its own.
// Measured (fp16, weights cold, early): 8 x 768 -> 2304 with LayerNorm 4.1 us, 8 x 768 -> 768 2.4, 8 x 3072
// -> 768 3.3, 8 x 768 -> 50304 with LayerNorm 17.7 (12.0 at the copy rate), 32 x 5120 -> 1280 11.4; the
// tcgen05 tile 12.9 on average for the first three, the CUDA-core tile in fp32 103 us.
#include "gemm.cuh"
#include "skinny.cuh"
#include "sm100.cuh"
#include <atomic>
#include <cooperative_groups.h>

namespace mt {
namespace cg = cooperative_groups;
using namespace sm100;

constexpr int kSkWarps = 8;
constexpr int kSkThreads = 32 * kSkWarps;
constexpr int kSkRing = 8;               // most rounds of weights in the ring
constexpr int kSkAhead = 4;              // outputs per thread whose bias and residual are loaded ahead
constexpr int kSkBarBytes = 128;         // ring barriers, the barrier of x, the abort flag

struct SkinnyParams {
  const void* x; int64_t ldx;
  int M, K;
  const void* w[3]; const void* bias[3];
  int n0, n01, N;                  // cumulative ends of the segments
  int64_t ldw;
  void* out; int64_t ldo;
  const void* residual;
  int act, norm; float softcap;
  const void* gamma; const void* beta; float eps;
  int early, rounds;
  int kc;                          // K per block (a multiple of 32, or all of K)
  int its;                         // steps of 32 k per warp
  int ring;                        // rounds the ring holds
  int whole_rows;                  // the rows of W are contiguous and not split: unpadded in the ring
  int x_bytes, nb_bytes;           // shared-memory extents: rows of x; gamma and beta
  int* flag;
};

__device__ __forceinline__ float skinny_finish(const SkinnyParams& p, float v, float bias, float residual) {
  v += bias;
  switch (p.act) {
    case MT_ACT_GELU: v = 0.5f * v * (1.f + tanhf(0.7978845608f * (v + 0.044715f * v * v * v))); break;
    case MT_ACT_RELU2: { const float r = fmaxf(v, 0.f); v = r * r; break; }
    case MT_ACT_RELU: v = fmaxf(v, 0.f); break;
    default: break;
  }
  v += residual;
  if (p.softcap > 0.f) v = p.softcap * tanhf(v / p.softcap);
  return v;
}

__device__ __forceinline__ int skinny_segment(const SkinnyParams& p, int row, int& local) {
  if (row < p.n0) { local = row; return 0; }
  if (row < p.n01) { local = row - p.n0; return 1; }
  local = row - p.n01;
  return 2;
}

// Elements between two rows of x or W in shared memory. Half types: 64 bytes modulo 128, so that the 16-byte
// reads of a quarter warp (two rows of 64 bytes) touch every bank once; fp32 reads 128 bytes of one row.
template <typename T> __host__ __device__ constexpr int skinny_pitch(int k) {
  return sizeof(T) == 2 ? (k + 63) / 64 * 64 + 32 : (k + 3) / 4 * 4;
}

// Normalises the rows of x in shared memory in place: a warp takes up to RW rows side by side. Mean
// and squared deviations are merged lane by lane (one pass over the row, no cancellation).
template <typename T, int RW>
__device__ __forceinline__ void skinny_norm_rows(const SkinnyParams& p, T* xs, int pitch, int rows, const T* gamma, const T* beta) {
  constexpr int VN = Vec16<T>::N;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nvec = p.K / VN;
  for (int r0 = warp; r0 < rows; r0 += kSkWarps * RW) {
    float mu[RW] = {}, m2[RW] = {}, rstd[RW];
    if (p.norm == 2) {
      for (int vi = lane; vi < nvec; vi += 32)
#pragma unroll
        for (int j = 0; j < RW; ++j) {
          const int r = min(r0 + j * kSkWarps, rows - 1);
          Vec16<T> t;
          t.load(xs + r * pitch + vi * VN);
#pragma unroll
          for (int e = 0; e < VN; ++e) m2[j] += t.get(e) * t.get(e);
        }
#pragma unroll
      for (int j = 0; j < RW; ++j) rstd[j] = rsqrtf(warp_sum(m2[j]) / p.K + p.eps);
    } else {
      float n = 0.f;                       // values a lane has seen, the same for all its rows
      for (int vi = lane; vi < nvec; vi += 32) {
        const float n1 = n + VN, f = VN / n1, g = n * f;
#pragma unroll
        for (int j = 0; j < RW; ++j) {
          const int r = min(r0 + j * kSkWarps, rows - 1);
          Vec16<T> t;
          t.load(xs + r * pitch + vi * VN);
          float s = 0.f, q = 0.f;
#pragma unroll
          for (int e = 0; e < VN; ++e) s += t.get(e);
          s *= 1.f / VN;
#pragma unroll
          for (int e = 0; e < VN; ++e) { const float d = t.get(e) - s; q += d * d; }
          const float d = s - mu[j];
          mu[j] += d * f;
          m2[j] += q + d * d * g;
        }
        n = n1;
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        const float no = __shfl_xor_sync(0xffffffffu, n, o), n1 = n + no;
        const float f = n1 > 0.f ? no / n1 : 0.f, g = n * f;
#pragma unroll
        for (int j = 0; j < RW; ++j) {
          const float mo = __shfl_xor_sync(0xffffffffu, mu[j], o), qo = __shfl_xor_sync(0xffffffffu, m2[j], o);
          const float d = mo - mu[j];
          mu[j] += d * f;
          m2[j] += qo + d * d * g;
        }
        n = n1;
      }
      // the lanes' merged means differ in the last bits: all take lane 0's
#pragma unroll
      for (int j = 0; j < RW; ++j) {
        mu[j] = __shfl_sync(0xffffffffu, mu[j], 0);
        rstd[j] = rsqrtf(__shfl_sync(0xffffffffu, m2[j], 0) / p.K + p.eps);
      }
    }
    for (int vi = lane; vi < nvec; vi += 32) {
      Vec16<T> g, b;
      if (p.gamma) g.load(gamma + vi * VN);
      if (p.beta) b.load(beta + vi * VN);
#pragma unroll
      for (int j = 0; j < RW; ++j) {
        const int r = r0 + j * kSkWarps;
        if (r >= rows) break;
        Vec16<T> t;
        t.load(xs + r * pitch + vi * VN);
#pragma unroll
        for (int e = 0; e < VN; ++e) {
          float h = (t.get(e) - mu[j]) * rstd[j];
          if (p.gamma) h *= g.get(e);
          if (p.beta) h += b.get(e);
          t.set(e, h);
        }
        t.store(xs + r * pitch + vi * VN);
      }
    }
  }
}

template <typename T> __device__ __forceinline__ void mma_16816(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                                                uint32_t b0, uint32_t b1);
template <> __device__ __forceinline__ void mma_16816<__half>(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                                              uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
template <> __device__ __forceinline__ void mma_16816<__nv_bfloat16>(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2,
                                                                     uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// Rows of W in a group (8 in half types, 4 in fp32).
template <typename T> struct SkinnyGroup { static constexpr int rows = sizeof(T) == 2 ? 8 : 4; };

// MV = rows of x a block covers (half: 16 per MMA tile; fp32: grid.y walks chunks of MV rows), GR =
// groups per round.
template <typename T, int MV, int GR>
__global__ void __launch_bounds__(kSkThreads, 2)
skinny_kernel(const SkinnyParams p) {
  constexpr bool kHalf = sizeof(T) == 2;
  constexpr int R = SkinnyGroup<T>::rows;
  constexpr int NR = GR * R;                              // weight rows, and output columns, of a round
  constexpr int MT = kHalf ? MV / 16 : 1;
  extern __shared__ __align__(128) uint8_t sk_smem[];
  const uint32_t bars = smem_u32(sk_smem);                // full barrier per ring slot, then the barrier of x
  volatile int* abort_flag = reinterpret_cast<volatile int*>(sk_smem + 8 * (kSkRing + 1));
  T* xs = reinterpret_cast<T*>(sk_smem + kSkBarBytes);
  T* gs = reinterpret_cast<T*>(sk_smem + kSkBarBytes + p.x_bytes);         // gamma, then beta
  const int pitch = skinny_pitch<T>(p.kc);
  const int wpitch = p.whole_rows ? p.kc : pitch;
  T* ring = reinterpret_cast<T*>(sk_smem + kSkBarBytes + p.x_bytes + p.nb_bytes);
  float* red = reinterpret_cast<float*>(ring + (size_t)p.ring * NR * wpitch);   // [warp][MV][NR], two if rounds follow
  float* part = red + kSkWarps * MV * NR;                 // a cluster (one round): the block's sums
  auto cluster = cg::this_cluster();
  const int csize = (int)cluster.num_blocks(), crank = (int)cluster.block_rank();
  const int first = (int)blockIdx.x / csize, stride = (int)gridDim.x / csize;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int m0 = kHalf ? 0 : (int)blockIdx.y * MV, rows = min(MV, p.M - m0);
  const int k0 = crank * p.kc, k1 = min(p.K, k0 + p.kc);  // this block's share of K
  const uint32_t row_bytes = (uint32_t)(max(0, k1 - k0) * (int)sizeof(T));
  const uint32_t x_bar = bars + 8 * kSkRing;

  if (threadIdx.x == 0) {
    for (int i = 0; i <= kSkRing; ++i) mbar_init(bars + 8 * i, 1);
    *abort_flag = 0;
    fence_barrier_init();
    fence_proxy_async();
  }
  __syncthreads();
  // Requests the weights of a round into a ring slot. A bulk copy costs its warp about 100 cycles: rows
  // that stand together in memory (all of K) come as one copy per group, by warp 0; parts of rows
  // as one copy each, spread over the warps.
  auto request = [&](int round, int slot) {
    if (round >= p.rounds) return;
    const int n = min(NR, p.N - round * NR);
    const uint32_t bar = bars + 8 * slot;
    const uint32_t dst = smem_u32(ring + (size_t)slot * NR * wpitch);
    if (threadIdx.x == 0) mbar_expect_tx(bar, (uint32_t)n * row_bytes);
    if (p.whole_rows) {
      if (warp == 0) {
        __syncwarp();
        if (lane < GR && lane * R < n) {
          int local;
          const int seg = skinny_segment(p, round * NR + lane * R, local);
          bulk_load_1d(dst + (uint32_t)(lane * R * wpitch * (int)sizeof(T)), (const T*)p.w[seg] + (int64_t)local * p.ldw,
                       (uint32_t)min(R, n - lane * R) * row_bytes, bar);
        }
      }
    } else {
      __syncthreads();                                    // the barrier expects the bytes before they come
      const int r = lane * kSkWarps + warp;
      if (r < n && row_bytes) {
        int local;
        const int seg = skinny_segment(p, round * NR + r, local);
        bulk_load_1d(dst + (uint32_t)(r * wpitch * (int)sizeof(T)), (const T*)p.w[seg] + (int64_t)local * p.ldw + k0, row_bytes, bar);
      }
    }
  };
  auto request_first = [&] { for (int r = 0; r < p.ring; ++r) request(first + r * stride, r); };
  if (p.early) request_first();
  grid_dependency_wait();
  allow_dependents();
  if (!p.early) request_first();
  if (warp == 1) {                                        // this block's part of x; gamma and beta
    const uint32_t nb = p.norm ? (uint32_t)(p.K * (int)sizeof(T)) : 0u;
    if (lane == 0) {
      mbar_expect_tx(x_bar, (uint32_t)rows * row_bytes + (p.gamma ? nb : 0u) + (p.beta ? nb : 0u));
      if (nb && p.gamma) bulk_load_1d(smem_u32(gs), p.gamma, nb, x_bar);
      if (nb && p.beta) bulk_load_1d(smem_u32(gs + p.K), p.beta, nb, x_bar);
    }
    __syncwarp();
    if (row_bytes)
      for (int r = lane; r < rows; r += 32)
        bulk_load_1d(smem_u32(xs + r * pitch), (const T*)p.x + (int64_t)(m0 + r) * p.ldx + k0, row_bytes, x_bar);
  }
  auto load_bias = [&](int n) {
    int local;
    const int seg = skinny_segment(p, n, local);
    return p.bias[seg] ? to_f(((const T*)p.bias[seg])[local]) : 0.f;
  };
  // bias and residual of the outputs this thread will finish in its first round
  const int per = (rows * NR + csize - 1) / csize;        // outputs this block finishes in a round
  const int o0 = crank * per, o1 = min(rows * NR, o0 + per);
  float ahead_b[kSkAhead] = {}, ahead_r[kSkAhead] = {};
#pragma unroll
  for (int a = 0; a < kSkAhead; ++a) {
    const int i = o0 + threadIdx.x + a * kSkThreads;
    const int m = i / NR, n = first * NR + i % NR;
    if (i < o1 && n < p.N) {
      ahead_b[a] = load_bias(n);
      if (p.residual) ahead_r[a] = to_f(((const T*)p.residual)[(int64_t)(m0 + m) * p.ldo + n]);
    }
  }
  mbar_wait(x_bar, 0, abort_flag);
  if (p.norm) {
    if (rows <= kSkWarps) skinny_norm_rows<T, 1>(p, xs, pitch, rows, gs, gs + p.K);
    else skinny_norm_rows<T, MV <= 16 ? 2 : 4>(p, xs, pitch, rows, gs, gs + p.K);
    __syncthreads();
  }
  // half: row = lane / 4, 8 k from (lane % 4) * 8; fp32: row = lane / 8, 4 k from (lane % 8) * 4
  const int wrow = kHalf ? lane >> 2 : lane >> 3, wk = kHalf ? (lane & 3) * 8 : (lane & 7) * 4;
  const int kl = warp * p.its * 32 + wk, kn = k1 - k0;    // this lane's first k and the end, inside the block's share
  int nth = 0, slot = 0;                                  // rounds done, ring slot
  uint32_t phase = 0;
  for (int round = first; round < p.rounds; round += stride, ++nth) {
    mbar_wait(bars + 8 * slot, phase, abort_flag);
    const T* src = ring + ((size_t)slot * NR + wrow) * wpitch + kl;
    const T* xr = xs + kl;
    float* buf = red + (nth & 1) * kSkWarps * MV * NR;
    if constexpr (kHalf) {
      float acc[GR][MT][4] = {};
#pragma unroll 2
      for (int it = 0; it < p.its; ++it) {
        const int left = kn - (kl - wk + it * 32);        // warp-uniform
        if (left <= 0) break;
        // Rows past the last token read whatever follows: their sums are never stored.
        uint4 a[MT][2], w[GR];
#pragma unroll
        for (int mt = 0; mt < MT; ++mt)
#pragma unroll
          for (int h = 0; h < 2; ++h)
            a[mt][h] = *reinterpret_cast<const uint4*>(xr + (mt * 16 + h * 8 + wrow) * pitch + it * 32);
#pragma unroll
        for (int g = 0; g < GR; ++g) w[g] = *reinterpret_cast<const uint4*>(src + g * 8 * wpitch + it * 32);
        if (left < 32 && wk >= left) {                    // the end of a K that is no multiple of 32
#pragma unroll
          for (int mt = 0; mt < MT; ++mt) a[mt][0] = a[mt][1] = make_uint4(0, 0, 0, 0);
#pragma unroll
          for (int g = 0; g < GR; ++g) w[g] = make_uint4(0, 0, 0, 0);
        }
#pragma unroll
        for (int g = 0; g < GR; ++g) {
#pragma unroll
          for (int mt = 0; mt < MT; ++mt) {
            mma_16816<T>(acc[g][mt], a[mt][0].x, a[mt][1].x, a[mt][0].y, a[mt][1].y, w[g].x, w[g].y);
            mma_16816<T>(acc[g][mt], a[mt][0].z, a[mt][1].z, a[mt][0].w, a[mt][1].w, w[g].z, w[g].w);
          }
        }
      }
#pragma unroll
      for (int g = 0; g < GR; ++g)
#pragma unroll
        for (int mt = 0; mt < MT; ++mt)
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const int m = mt * 16 + h * 8 + wrow;
            if (m < rows)
              *reinterpret_cast<float2*>(buf + (warp * MV + m) * NR + g * 8 + (lane & 3) * 2) =
                  make_float2(acc[g][mt][h * 2], acc[g][mt][h * 2 + 1]);
          }
    } else {
      float acc[GR][MV] = {};
      for (int it = 0; it < p.its; ++it) {
        if (kl + it * 32 < kn) {
          float4 w[GR];
#pragma unroll
          for (int g = 0; g < GR; ++g) w[g] = *reinterpret_cast<const float4*>(src + g * 4 * wpitch + it * 32);
#pragma unroll
          for (int m = 0; m < MV; ++m) {
            if (m < rows) {
              const float4 a = *reinterpret_cast<const float4*>(xr + m * pitch + it * 32);
#pragma unroll
              for (int g = 0; g < GR; ++g)
                acc[g][m] = fmaf(w[g].x, a.x, fmaf(w[g].y, a.y, fmaf(w[g].z, a.z, fmaf(w[g].w, a.w, acc[g][m]))));
            }
          }
        }
      }
#pragma unroll
      for (int g = 0; g < GR; ++g)
#pragma unroll
        for (int m = 0; m < MV; ++m) {
          float v = acc[g][m];
          v += __shfl_xor_sync(0xffffffffu, v, 4);
          v += __shfl_xor_sync(0xffffffffu, v, 2);
          v += __shfl_xor_sync(0xffffffffu, v, 1);
          if ((lane & 7) == (m & 7) && m < rows) buf[(warp * MV + m) * NR + g * 4 + wrow] = v;
        }
    }
    __syncthreads();
    request(round + p.ring * stride, slot);               // the slot has been read by all warps
    auto block_sum = [&](int i) {
      float v = 0.f;
#pragma unroll
      for (int w = 0; w < kSkWarps; ++w) v += buf[w * MV * NR + i];
      return v;
    };
    if (csize > 1) {
      for (int i = threadIdx.x; i < rows * NR; i += kSkThreads) part[i] = block_sum(i);
      cluster.sync();
    }
#pragma unroll 1
    for (int a = 0, i = o0 + (int)threadIdx.x; i < o1; ++a, i += kSkThreads) {
      const int m = i / NR, n = round * NR + i % NR;
      if (n >= p.N) continue;
      float v = 0.f;
      if (csize > 1) for (int c = 0; c < csize; ++c) v += *cluster.map_shared_rank(part + i, c);
      else v = block_sum(i);
      const int64_t off = (int64_t)(m0 + m) * p.ldo + n;
      float b, r;
      if (nth == 0 && a < kSkAhead) {
        b = a == 0 ? ahead_b[0] : a == 1 ? ahead_b[1] : a == 2 ? ahead_b[2] : ahead_b[3];
        r = a == 0 ? ahead_r[0] : a == 1 ? ahead_r[1] : a == 2 ? ahead_r[2] : ahead_r[3];
      } else {
        b = load_bias(n);
        r = p.residual ? to_f(((const T*)p.residual)[off]) : 0.f;
      }
      ((T*)p.out)[off] = from_f<T>(skinny_finish(p, v, b, r));
    }
    if (csize > 1) cluster.sync();                        // nobody leaves while its sums are still being read
    if (++slot == p.ring) { slot = 0; phase ^= 1u; }
  }
  if (threadIdx.x == 0 && *abort_flag && p.flag) atomicMax(p.flag, 105);   // a bounded wait expired
}

constexpr size_t kSkSmemMax = 226 * 1024;

// How a product runs with gr groups per round, K split over `cluster` blocks and per_sm blocks resident
// on an SM.
template <typename T>
static SkinnyShape skinny_shape(const SkinnyArgs& a, int N, int mv, int gr, int cluster, int per_sm) {
  constexpr int R = SkinnyGroup<T>::rows;
  const int sms = sm_count();
  SkinnyShape s{};
  s.gr = gr;
  s.cluster = cluster;
  s.kc = cluster == 1 ? a.K : ((a.K + cluster - 1) / cluster + 31) / 32 * 32;
  s.its = ((s.kc + 31) / 32 + kSkWarps - 1) / kSkWarps;
  s.rounds = ((N + R - 1) / R + gr - 1) / gr;
  const int x_rows = a.M < mv ? a.M : mv;
  const size_t row = skinny_pitch<T>(s.kc) * sizeof(T);
  s.x_bytes = (int)((x_rows * row + 127) / 128 * 128);
  s.nb_bytes = a.norm ? (int)((2 * (size_t)a.K * sizeof(T) + 127) / 128 * 128) : 0;
  const size_t round_bytes = gr * R * row, sums = (size_t)mv * gr * R * 4;
  const size_t fixed = kSkBarBytes + (size_t)s.x_bytes + s.nb_bytes, budget = per_sm == 2 ? kSkSmemMax / 2 : kSkSmemMax;
  s.blocks = s.rounds;
  if (cluster == 1 && s.blocks > sms * per_sm) s.blocks = sms * per_sm;
  const int deepest = (s.rounds + s.blocks - 1) / s.blocks;           // rounds of the busiest block
  const size_t sum_bytes = (deepest > 1 ? 2 : 1) * kSkWarps * sums + (cluster > 1 ? sums : 0);
  s.ring = deepest < kSkRing ? deepest : kSkRing;
  while (s.ring > 1 && fixed + sum_bytes + s.ring * round_bytes > budget) --s.ring;
  s.smem = fixed + sum_bytes + s.ring * round_bytes;
  // (fragments of rows past the last token are read too, and must lie inside the block's memory)
  if (s.smem < kSkBarBytes + mv * row) s.smem = kSkBarBytes + mv * row;
  const int chunks_y = sizeof(T) == 2 ? 1 : (a.M + mv - 1) / mv;
  const int all = s.blocks * cluster * chunks_y, here = (all + sms - 1) / sms;     // blocks of the busiest SM
  const int waves = (all + sms * per_sm - 1) / (sms * per_sm);
  // A round is a chain of a few hundred instructions per warp (measured: about 1000 cycles and 400 per
  // group and 16 tokens; fp32 250 per group and 100 per group and token), which a second block hides.
  const double chain = sizeof(T) == 2 ? 1000.0 + 400.0 * gr * (mv / 16) : 800.0 + 250.0 * gr + 100.0 * gr * mv;
  const double round_clk = chain / (here < per_sm ? here : per_sm);
  // HBM: 22 bytes per cycle and SM, less where fewer bytes are in flight than ~2200 cycles of latency want
  const double flight = (double)(here < per_sm ? here : per_sm) * (deepest > s.ring ? s.ring - 0.5 : s.ring) * round_bytes;
  const double rate = flight / 2200.0 < 22.0 ? flight / 2200.0 : 22.0;
  const double smem_clk = here * deepest * round_clk, hbm_clk = (double)here * deepest * round_bytes / rate;
  s.cost = waves * (cluster > 1 ? 2100.0 : 1200.0) + (smem_clk > hbm_clk ? smem_clk : hbm_clk) + here * (x_rows * row / 48.0);
  if (s.smem > budget || (s.ring == 1 && deepest > 1)) s.cost = 1e30;
  return s;
}

template <typename T, int MV, int GR>
static int launch_skinny(const SkinnyArgs& a, SkinnyParams& p, const SkinnyShape& s, cudaStream_t st) {
  auto kern = skinny_kernel<T, MV, GR>;
  static std::atomic<bool> ready[16];      // per device; racing first calls set the same attributes twice, harmlessly
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 16 || !ready[dev].load(std::memory_order_acquire)) {
    MT_CHECK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSkSmemMax));
    MT_CHECK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared));
    if (dev >= 0 && dev < 16) ready[dev].store(true, std::memory_order_release);
  }
  p.kc = s.kc; p.its = s.its; p.rounds = s.rounds; p.ring = s.ring;
  p.x_bytes = s.x_bytes; p.nb_bytes = s.nb_bytes;
  p.whole_rows = s.cluster == 1 && a.ldw == a.K;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(s.blocks * s.cluster), sizeof(T) == 2 ? 1u : (unsigned)((a.M + MV - 1) / MV));
  cfg.blockDim = dim3(kSkThreads);
  cfg.dynamicSmemBytes = s.smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)s.cluster;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = overlap_launches() ? 2 : 1;
  MT_CHECK_CUDA(cudaLaunchKernelEx(&cfg, kern, p));
  count_launch();
  return MT_OK;
}

template <typename T, int MV> constexpr int skinny_most_groups() { return sizeof(T) == 2 ? (MV <= 32 ? 5 : 3) : 4; }

template <typename T, int MV>
static SkinnyShape best_shape(const SkinnyArgs& a, int N) {
  SkinnyShape best{};
  best.cost = 1e30;
  for (int cluster = 1; cluster <= 8; cluster *= 2) {
    if (cluster > 1 && (a.norm || a.K < 512 * cluster)) break;        // a norm needs whole rows
    for (int gr = 1; gr <= skinny_most_groups<T, MV>(); ++gr) {
      if (sizeof(T) == 4 && gr == 3) continue;
      for (int per_sm = 1; per_sm <= 2; ++per_sm) {
        const SkinnyShape s = skinny_shape<T>(a, N, MV, gr, cluster, per_sm);
        if (s.cost < best.cost) best = s;
      }
    }
  }
  return best;
}

template <typename T, int MV>
static int launch_skinny_shape(const SkinnyArgs& a, SkinnyParams& p, const SkinnyShape& s, cudaStream_t st) {
  constexpr bool kHalf = sizeof(T) == 2;
  constexpr int GM = skinny_most_groups<T, MV>();
  switch (s.gr) {
    case 1: return launch_skinny<T, MV, 1>(a, p, s, st);
    case 2: return launch_skinny<T, MV, 2>(a, p, s, st);
    case 3: return launch_skinny<T, MV, kHalf ? 3 : 1>(a, p, s, st);
    case 4: return launch_skinny<T, MV, GM >= 4 ? 4 : 1>(a, p, s, st);
    default: return launch_skinny<T, MV, GM >= 5 ? 5 : 1>(a, p, s, st);
  }
}

// FN<T, MV>(...) with the rows of x that a block covers.
#define MT_SKINNY_ROWS(a, FN, ...)                                                                                    \
  ((a).dtype == MT_F32   ? ((a).M == 1   ? FN<float, 1>(__VA_ARGS__)                                                  \
                            : (a).M == 2 ? FN<float, 2>(__VA_ARGS__)                                                  \
                            : (a).M <= 4 ? FN<float, 4>(__VA_ARGS__)                                                  \
                            : (a).M <= 8 ? FN<float, 8>(__VA_ARGS__) : FN<float, 16>(__VA_ARGS__))                    \
   : (a).dtype == MT_F16 ? ((a).M <= 16   ? FN<__half, 16>(__VA_ARGS__)                                               \
                            : (a).M <= 32 ? FN<__half, 32>(__VA_ARGS__) : FN<__half, 64>(__VA_ARGS__))                \
                         : ((a).M <= 16   ? FN<__nv_bfloat16, 16>(__VA_ARGS__)                                        \
                            : (a).M <= 32 ? FN<__nv_bfloat16, 32>(__VA_ARGS__) : FN<__nv_bfloat16, 64>(__VA_ARGS__)))

bool skinny_fits(const SkinnyArgs& a, SkinnyShape& shape) {
  const bool f32 = a.dtype == MT_F32;
  const int vec = f32 ? 4 : 8;
  if (a.M < 1 || a.M > kSkinnyMaxRows) return false;
  if (a.K < vec || a.K % vec || a.ldx % vec || a.ldw % vec || !aligned16(a.x)) return false;
  for (int i = 0; i < a.nseg; ++i) {
    if (!aligned16(a.w[i]) || a.n[i] < 1) return false;
    if (a.nseg > 1 && a.n[i] % 8) return false;            // a group of rows lies in one segment
  }
  if (a.norm && ((a.gamma && !aligned16(a.gamma)) || (a.beta && !aligned16(a.beta)))) return false;
  if (a.norm && !f32 && a.M > 32) return false;
  // The rows of x of one block have to fit shared memory beside a ring of weights: a quick bound here; the launch
  // shapes have the last word (a norm keeps K whole: eight rows in half types end near K = 4200).
  const int64_t rows = f32 ? (a.M < 16 ? a.M : 16) : a.M, es = f32 ? 4 : 2;
  const int64_t kc = a.norm ? a.K : (a.K + 7) / 8;
  if (rows * kc * es > 100 * 1024 || a.K > 32768) return false;
  int N = 0;
  for (int i = 0; i < a.nseg; ++i) N += a.n[i];
  shape = MT_SKINNY_ROWS(a, best_shape, a, N);
  return shape.cost < 1e30;
}

int skinny_gemm(const SkinnyArgs& a, const SkinnyShape& shape, cudaStream_t st) {
  SkinnyParams p{};
  p.x = a.x; p.ldx = a.ldx; p.M = a.M; p.K = a.K;
  for (int i = 0; i < 3; ++i) { p.w[i] = a.w[i]; p.bias[i] = a.bias[i]; }
  p.n0 = a.n[0];
  p.n01 = a.n[0] + (a.nseg > 1 ? a.n[1] : 0);
  p.N = p.n01 + (a.nseg > 2 ? a.n[2] : 0);
  if (a.nseg < 2) p.n01 = p.N;
  p.ldw = a.ldw; p.out = a.out; p.ldo = a.ldo; p.residual = a.residual;
  p.act = a.act; p.softcap = a.softcap;
  p.gamma = a.gamma; p.beta = a.beta; p.eps = a.eps;
  p.early = a.early_weights;
  p.norm = a.norm;
  p.flag = device_flag_ptr();
  return MT_SKINNY_ROWS(a, launch_skinny_shape, a, p, shape, st);
}

}  // namespace mt
