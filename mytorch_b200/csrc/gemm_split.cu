// Tensor-core GEMM for operands that gemm_tcgen05.cu does not take, with sums at least as exact as a
// chain of fp32 FMAs: fp32 matrices, and half matrices whose pointers or pitches TMA cannot address.
//
// Two launches. `prepare_kernel` rewrites the operands with a 16-byte pitch: an fp32 value x becomes three
// bf16 planes h + m + l = 2^24 x (8 significant bits each, rounded to nearest: exact; the factor keeps the planes of
// the smallest fp32 values among bf16's normal numbers, and the sums are multiplied by 2^-48), a half value is copied. `gemm_split_kernel` then multiplies plane by plane:
//   fp32: l.h + h.l + m.m + m.h + h.m + h.h, smallest first; the products left out (m.l, l.m, l.l) are below
//   2^-25 of a term. Every bf16 product is exact in the fp32 accumulator.
// The accumulator in tensor memory is not kept over all of K, for its additions cut off instead of rounding:
// after each chunk of K the epilogue warps add it to fp32 registers (round to nearest) while the next chunk goes to
// the other accumulator. The chunk is chosen so that the sum is no further from 64 bits than a chain of
// fp32 FMAs (relative error, 2-norm; in brackets the chain's):
//   fp32, every 64 of K:  K = 16 4.8e-8 (7.4e-8), 256 8.8e-8 (2.9e-7), 3072 1.2e-7 (9.9e-7), 131072 3.0e-7 (6.5e-6) of
//   normal values; of values in [0, 1) 5.2e-8 (6.2e-8), 8.7e-8 (2.2e-7), 9.7e-8 (7.8e-7), 1.3e-7 (6.9e-6).
//   fp16 in [0, 1), the worst case of the half types, every 64 of K 1.9e-7, 128 4.7e-7, 256 1.15e-6, 512 2.65e-6 whatever
//   K is; the chain 1.4e-8 sqrt(K), which is smaller below K = 200.
//
// Persistent. A slot of a CTA's ring holds 128 rows of one plane of A and of B (2 x 16 KB), a 64-deep slice of fp32
// operands three slots. A CTA pair (cta_group::2) works on a 256 x 256 tile: the 24 MMAs of a slice last 3072 tensor
// cycles while the ring's other half fills. A single CTA's 128 x 128 tile has 1536 cycles of MMAs for the same 96 KB
// and measures 3600 a slice; it is there for products with too few tiles. Where even those are few
// (weight gradients of small layers), K is split over a cluster of up to eight CTAs whose sums meet
// through distributed shared memory in a fixed order: no atomics, the same bits every time.
// Against the CUDA-core kernel, fp32: 8192 x 768 -> 3072 1417 -> 179 us (tensor pipe 60 % of its cycles; with GELU and the second
// output 27 %, for the next tile's MMAs do not hide that epilogue), its weight gradient 1547 -> 242, 4096 x 256 -> 1024 106 -> 21,
// 256 x 4096 x 256 212 -> 26; bf16 with odd pitches: 50257 x 3885 -> 768 to fp32 12390 -> 464 us, 3885 x 50257 -> 768 15420 -> 457.
//
// A sum that is not finite (an operand is, or one is above 2^103, or the result above 2^79) is computed again as a plain
// chain of fp32 FMAs, so infinities and NaNs come out as fp32 arithmetic gives them. The epilogue only leaves such 32 x 32
// pieces out and marks them; they are made up after the CTA's last tile, when no role waits for another any more.
#include "gemm.cuh"
#include "sm100.cuh"
#include "prof.cuh"
#include "tempbuf.cuh"
#include <atomic>
#include <string.h>

namespace mt {

using namespace sm100;

constexpr int kSpM = 128, kSpN = 128, kSpK = 64;
constexpr int kSpPlane = 128 * kSpK * 2;             // 16 KB: one plane of one operand's tile
constexpr int kSpSlot = 2 * kSpPlane;
constexpr int kSpSlots = 6;
constexpr int kSpEpiWarps = 8;
constexpr int kSpThreads = 64 + 32 * kSpEpiWarps;
constexpr int kSpStage = 32 * 33 * 4;                // an epilogue warp's 32 x 32 transpose buffer
constexpr int kSpSmem = kSpSlots * kSpSlot + kSpEpiWarps * kSpStage + 1024 /*align*/ + 256 /*barriers*/;
constexpr int kSpPitch = kSpN + 1;                   // row pitch (floats) of the sums a cluster exchanges
static_assert(kSpM * kSpPitch * 4 <= kSpSlots * kSpSlot, "a tile's sums fit the ring");

constexpr float kSpScale = 16777216.f, kSpUnscale = 1.f / (kSpScale * kSpScale);     // exact

struct SplitParams {
  const void* A; const void* B; void* C; void* preact; const void* bias; const void* aux;
  int64_t M, N, K, lda, ldb, ldc;
  int trans_a, trans_b, in_dtype, out_dtype, act, aux_mode, accumulate;
  float alpha;
  int tiles_m, tiles_n, n_fast, csize, kb_total, kb_per_rank, chunk;
  uint8_t* left_out;        // fp32, K not split: [tile][CTA][epilogue warp] the pieces (bit = 32 columns) that are made up at the end
  int* flag;
};

__device__ __forceinline__ float load_typed(const void* p, int64_t i, int dt) {
  return dt == MT_F32 ? ((const float*)p)[i] : dt == MT_F16 ? __half2float(((const __half*)p)[i]) : __bfloat162float(((const __nv_bfloat16*)p)[i]);
}
__device__ __forceinline__ void store_typed(void* p, int64_t i, int dt, float v) {
  if (dt == MT_F32) ((float*)p)[i] = v;
  else if (dt == MT_F16) ((__half*)p)[i] = __float2half_rn(v);
  else ((__nv_bfloat16*)p)[i] = __float2bfloat16_rn(v);
}

__device__ __forceinline__ bool split_finite(float v) { return fabsf(v) <= 3.402823466e38f; }

// Everything behind the sum of one output; aux and old are what its aux operand and C hold (0 where not read).
__device__ __forceinline__ void split_finish(const SplitParams& P, float v, float bias, float aux, float old, int64_t m, int64_t n) {
  v = P.alpha * v + bias;
  const int64_t off = m * P.ldc + n;
  if (P.preact) store_typed(P.preact, off, P.out_dtype, (P.act & kActStoreGrad) ? act_grad(v, P.act) : v);
  switch (P.act & 0xff) {
    case MT_ACT_GELU: v = 0.5f * v * (1.f + tanhf(0.7978845608f * (v + 0.044715f * v * v * v))); break;
    case MT_ACT_RELU2: { const float r = fmaxf(v, 0.f); v = r * r; break; }
    case MT_ACT_RELU: v = fmaxf(v, 0.f); break;
    default: break;
  }
  if (P.aux_mode) v = aux_apply(v, aux, P.aux_mode);
  if (P.accumulate) v += old;
  store_typed(P.C, off, P.out_dtype, v);
}

// One warp: the outputs (m0 + r, n0 + lane) whose bit r is set in the lane's `missing`, as chains of fp32 FMAs over the original operands.
// Its own function, and the parameters stay where they are (__grid_constant__): inlined, it cost the kernel 2-4 us. All of
// 8192 x 768 -> 3072: 0.66 ms with a NaN operand, which the first 32 k settle, 4.6 ms with an infinite one (the CUDA-core kernel 1.4).
constexpr int kSpRedoPitch = 36;                     // rows of A: 16-byte reads
constexpr int kSpRedo = 32 * (kSpRedoPitch + 33) * 4;        // its shared memory: 32 x 32 of A and of B
static __device__ __noinline__ void split_make_up(const SplitParams& P, int64_t m0, int64_t n0, uint32_t missing, float* s) {
  const int lane = threadIdx.x & 31;
  const float* A = (const float*)P.A;
  const float* B = (const float*)P.B;
  const int64_t M = P.M, N = P.N, K = P.K, lda = P.lda, ldb = P.ldb;
  const bool ta = P.trans_a, tb = P.trans_b;
  float* const as = s;                               // [row][k]
  float* const bs = s + 32 * kSpRedoPitch;           // [k][column]
  float acc[32];
#pragma unroll
  for (int r = 0; r < 32; ++r) acc[r] = 0.f;
  for (int64_t k0 = 0; k0 < K; k0 += 32) {
    __syncwarp();
    for (int i0 = 0; i0 < 32; i0 += 8) {             // lanes walk the contiguous direction; zeros past the edges
      float va[8], vb[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const int64_t am = m0 + (ta ? lane : i0 + u), ak = k0 + (ta ? i0 + u : lane);
        const int64_t bn = n0 + (tb ? i0 + u : lane), bk = k0 + (tb ? lane : i0 + u);
        va[u] = am < M && ak < K ? A[ta ? ak * lda + am : am * lda + ak] : 0.f;
        vb[u] = bn < N && bk < K ? B[tb ? bn * ldb + bk : bk * ldb + bn] : 0.f;
      }
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        as[ta ? lane * kSpRedoPitch + i0 + u : (i0 + u) * kSpRedoPitch + lane] = va[u];
        bs[tb ? lane * 33 + i0 + u : (i0 + u) * 33 + lane] = vb[u];
      }
    }
    __syncwarp();
    // (the zeros behind the last k leave a sum as it is)
    for (int k = 0; k < 32; k += 4) {
      const float b0 = bs[k * 33 + lane], b1 = bs[(k + 1) * 33 + lane], b2 = bs[(k + 2) * 33 + lane], b3 = bs[(k + 3) * 33 + lane];
#pragma unroll
      for (int r = 0; r < 32; ++r) {
        const float4 x = *reinterpret_cast<const float4*>(as + r * kSpRedoPitch + k);
        acc[r] = fmaf(x.w, b3, fmaf(x.z, b2, fmaf(x.y, b1, fmaf(x.x, b0, acc[r]))));
      }
    }
    bool done = true;                                // what is NaN stays NaN
#pragma unroll
    for (int r = 0; r < 32; ++r) done = done && (isnan(acc[r]) || m0 + r >= M);
    if (__all_sync(0xffffffffu, done || n0 + lane >= N)) break;
  }
  __syncwarp();
#pragma unroll
  for (int r = 0; r < 32; ++r) s[r * 33 + lane] = acc[r];
  __syncwarp();
  const int64_t n = n0 + lane;
  if (n < P.N) {
    const float bias = P.bias ? load_typed(P.bias, n, P.in_dtype) : 0.f;
#pragma unroll 1
    for (int r = 0; r < 32; ++r) {
      if (!(missing >> r & 1)) continue;
      const int64_t off = (m0 + r) * P.ldc + n;
      split_finish(P, s[r * 33 + lane], bias, P.aux_mode ? load_typed(P.aux, off, P.out_dtype) : 0.f,
                   P.accumulate ? load_typed(P.C, off, P.out_dtype) : 0.f, m0 + r, n);
    }
  }
  __syncwarp();
}

template <bool F32, bool A_MN, bool B_MN, bool PAIR>
__global__ void __launch_bounds__(kSpThreads, 1)
gemm_split_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const __grid_constant__ SplitParams P) {
  constexpr int PLANES = F32 ? 3 : 1;
  constexpr int TM = PAIR ? 256 : 128, TN = PAIR ? 256 : 128;      // tile of a CTA or a pair; either way a CTA stages 128 rows of A and of B
  constexpr int NC = TN / 2;                         // columns an epilogue warp holds
  extern __shared__ uint8_t sp_smem[];
  const uint32_t raw = smem_u32(sp_smem);
  const uint32_t base = (raw + 1023u) & ~1023u;      // the 128-byte swizzle repeats every 1024 bytes
  uint8_t* const base_ptr = sp_smem + (base - raw);
  float* const stages = reinterpret_cast<float*>(base_ptr + kSpSlots * kSpSlot);
  uint8_t* const bar_ptr = base_ptr + kSpSlots * kSpSlot + kSpEpiWarps * kSpStage;
  const uint32_t bar0 = smem_u32(bar_ptr);
  auto full_bar = [&](int s) { return bar0 + 8u * s; };
  auto empty_bar = [&](int s) { return bar0 + 8u * (kSpSlots + s); };
  auto accf_bar = [&](int b) { return bar0 + 8u * (2 * kSpSlots + b); };
  auto acce_bar = [&](int b) { return bar0 + 8u * (2 * kSpSlots + 2 + b); };
  uint32_t* const tmem_slot = reinterpret_cast<uint32_t*>(bar_ptr + 8 * (2 * kSpSlots + 4));
  volatile int* const abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  volatile int* const redo_flag = abort_flag + 1;    // this CTA has outputs to make up
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int csize = PAIR ? 1 : P.csize;              // CTAs that split K
  const int prank = PAIR ? (int)cluster_ctarank() : 0;
  const int rank = csize > 1 ? (int)cluster_ctarank() : 0;
  const int per_worker = PAIR ? 2 : csize;
  const int worker = (int)blockIdx.x / per_worker, workers = (int)gridDim.x / per_worker;
  if (threadIdx.x == 0) {
    for (int s = 0; s < kSpSlots; ++s) { mbar_init(full_bar(s), 1); mbar_init(empty_bar(s), 1); }
    for (int b = 0; b < 2; ++b) { mbar_init(accf_bar(b), 1); mbar_init(acce_bar(b), PAIR ? 2 * kSpEpiWarps : kSpEpiWarps); }
    *abort_flag = 0;
    *redo_flag = 0;
    fence_barrier_init();
    fence_proxy_async();
  }
  if (warp == 1) {
    if (PAIR) { tmem_alloc_pair(smem_u32(tmem_slot), 2 * TN); tmem_relinquish_pair(); }
    else { tmem_alloc(smem_u32(tmem_slot), 2 * TN); tmem_relinquish(); }
  }
  tc_fence_before();
  __syncthreads();
  if (PAIR) cluster_sync_all();                      // the peer's barriers exist before anything signals them
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  griddep_launch();
  griddep_wait();

  const int total = P.tiles_m * P.tiles_n;
  const int kb0 = rank * P.kb_per_rank, kb1 = min(P.kb_total, kb0 + P.kb_per_rank);
  if (warp == 0) {
    // ------------------------------------------------------------ producer --
    if (lane == 0) {
      prefetch_tmap(&tmA);
      prefetch_tmap(&tmB);
      int slot = 0;
      uint32_t phase = 0;
      long long issued = 0;
      bool ok = true;
      for (int t = worker; t < total && ok; t += workers) {
        const int m0 = (P.n_fast ? t / P.tiles_n : t % P.tiles_m) * TM + prank * 128, n0 = (P.n_fast ? t % P.tiles_n : t / P.tiles_m) * TN + prank * 128;
        for (int kb = kb0; kb < kb1 && ok; ++kb) {
          for (int pl = 0; pl < PLANES; ++pl) {
            if (!mbar_wait(empty_bar(slot), phase ^ 1u, abort_flag)) { ok = false; break; }
            const uint32_t sa = base + slot * kSpSlot, sb = sa + kSpPlane;
            const uint32_t bar = PAIR ? mapa_shared(full_bar(slot), 0) : full_bar(slot);     // rank 0 counts both CTAs' copies
            if (prank == 0) mbar_expect_tx(full_bar(slot), PAIR ? 2 * kSpSlot : kSpSlot);
            auto load = [&](uint32_t dst, const CUtensorMap* map, int x, int y) {
              if (PAIR) tma_load_3d_pair(dst, map, bar, x, y, pl);
              else tma_load_3d(dst, map, bar, x, y, pl);
            };
            if (!A_MN) load(sa, &tmA, kb * kSpK, m0);
            else for (int j = 0; j < 2; ++j) load(sa + j * (kSpK * 128), &tmA, m0 + j * 64, kb * kSpK);
            if (!B_MN) load(sb, &tmB, kb * kSpK, n0);
            else for (int j = 0; j < 2; ++j) load(sb + j * (kSpK * 128), &tmB, n0 + j * 64, kb * kSpK);
            ++issued;
            if (++slot == kSpSlots) { slot = 0; phase ^= 1u; }
          }
        }
      }
      if (!ok && prank == 0) {                         // bounded: the copies in flight land before shared memory goes away
        const long long n = issued < kSpSlots ? issued : kSpSlots;
        int s = slot;
        uint32_t ph = phase;
        for (long long i = 0; i < n; ++i) {
          if (--s < 0) { s = kSpSlots - 1; ph ^= 1u; }
          const long long t0 = clock64();
          while (!mbar_try_wait(full_bar(s), ph) && clock64() - t0 < kWaitLimitCycles) {}
        }
      }
    }
  } else if (warp == 1) {
    // ---------------------------------------------------------- MMA issuer --
    if (lane == 0 && prank == 0) {
      const uint32_t idesc = idesc_f16(F32 || P.in_dtype == MT_BF16, A_MN, B_MN, TM, TN);
      auto commit = [&](uint32_t bar) { if (PAIR) umma_commit_pair(bar); else umma_commit(bar); };
      int slot = 0, it = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int t = worker; t < total && ok; t += workers) {
        for (int kc = kb0; kc < kb1 && ok; kc += P.chunk, ++it) {
          const int buf = it & 1;
          if (!mbar_wait(acce_bar(buf), ((it >> 1) & 1) ^ 1u, abort_flag)) { ok = false; break; }
          tc_fence_after();
          const uint32_t d = tmem_base + buf * TN;
          const int ke = min(kb1, kc + P.chunk);
          for (int kb = kc; kb < ke && ok; ++kb) {
            // the slots of a slice are neighbours: kSpSlots is a multiple of PLANES
            for (int pl = 0; pl < PLANES && ok; ++pl) ok = mbar_wait(full_bar(slot + pl), phase, abort_flag);
            if (!ok) break;
            tc_fence_after();
            auto product = [&](int pa, int pb, uint32_t acc) {
              const uint32_t sa = base + (slot + pa) * kSpSlot, sb = base + (slot + pb) * kSpSlot + kSpPlane;
              uint64_t a[4], b[4];
#pragma unroll
              for (int k = 0; k < 4; ++k) {
                a[k] = A_MN ? smem_desc_sw128(sa + k * 2048, kSpK * 128, 1024) : smem_desc_sw128(sa + k * 32, 16, 1024);
                b[k] = B_MN ? smem_desc_sw128(sb + k * 2048, kSpK * 128, 1024) : smem_desc_sw128(sb + k * 32, 16, 1024);
              }
              if (PAIR) {
#pragma unroll
                for (int k = 0; k < 4; ++k) umma_f16_pair(d, a[k], b[k], idesc, k ? 1u : acc);
              } else {
                umma_f16_x4(d, a, b, idesc, acc);
              }
            };
            const uint32_t acc = kb > kc ? 1u : 0u;
            if (F32) {
              product(2, 0, acc);
              product(0, 2, 1u);
              product(1, 1, 1u);
              product(1, 0, 1u);
              product(0, 1, 1u);
              product(0, 0, 1u);
            } else {
              product(0, 0, acc);
            }
            for (int pl = 0; pl < PLANES; ++pl) commit(empty_bar(slot + pl));
            slot += PLANES;
            if (slot == kSpSlots) { slot = 0; phase ^= 1u; }
          }
          if (ok) commit(accf_bar(buf));
        }
      }
    }
  } else {
    // ------------------------------------------------------------ epilogue --
    const int quarter = warp & 3, c0 = ((warp - 2) >> 2) * NC;      // 32 rows, half of the tile's columns
    float* const stage = stages + (warp - 2) * (32 * 33);
    int it = 0;
    bool ok = true;
    for (int t = worker; t < total && ok; t += workers) {
      const int64_t m0 = (int64_t)(P.n_fast ? t / P.tiles_n : t % P.tiles_m) * TM + prank * 128 + quarter * 32;
      const int64_t n0 = (int64_t)(P.n_fast ? t % P.tiles_n : t / P.tiles_m) * TN + c0;
      float acc[NC];
#pragma unroll
      for (int e = 0; e < NC; ++e) acc[e] = 0.f;
      for (int kc = kb0; kc < kb1; kc += P.chunk, ++it) {
        const int buf = it & 1;
        if (!__all_sync(0xffffffffu, mbar_wait(accf_bar(buf), (it >> 1) & 1, abort_flag))) { ok = false; break; }
        tc_fence_after();
        const uint32_t taddr = tmem_base + ((uint32_t)(quarter * 32) << 16) + buf * TN + c0;
#pragma unroll
        for (int h = 0; h < NC; h += 32) {
          uint32_t r[32];
          tmem_ld32(taddr + h, r);
          tmem_ld_wait();
#pragma unroll
          for (int e = 0; e < 32; ++e) acc[h + e] += __uint_as_float(r[e]);
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) {
          if (PAIR) mbar_arrive_cluster(mapa_shared(acce_bar(buf), 0));
          else mbar_arrive(acce_bar(buf));
        }
      }
      if (!ok) break;
      if (csize > 1) {
        // all copies and MMAs of this CTA are done: its ring holds the sums for the cluster
        float* rows = reinterpret_cast<float*>(base_ptr) + (quarter * 32 + lane) * kSpPitch + c0;
#pragma unroll
        for (int e = 0; e < NC; ++e) rows[e] = acc[e];
      } else {
        // thread = row becomes lane = column: rows of 128 bytes to and from global memory, any pitch
        uint32_t left_out = 0;
#pragma unroll
        for (int h = 0; h < NC / 32; ++h) {
          const int64_t n = n0 + h * 32 + lane;
          __syncwarp();
          bool fine = true;
#pragma unroll
          for (int e = 0; e < 32; ++e) {
            if (F32) fine = fine && split_finite(acc[h * 32 + e]);
            stage[lane * 33 + e] = F32 ? acc[h * 32 + e] * kSpUnscale : acc[h * 32 + e];
          }
          if (F32 && __any_sync(0xffffffffu, !fine)) {
            left_out |= 1u << h;
            continue;
          }
          __syncwarp();
          if (n < P.N) {
            const float bias = P.bias ? load_typed(P.bias, n, P.in_dtype) : 0.f;
            const int rows = (int)min((int64_t)32, P.M - m0);
            const bool plain = !P.preact && !P.act && !P.aux_mode && !P.accumulate;
            for (int r0 = 0; r0 < rows; r0 += 8) {
              if (plain && r0 + 8 <= rows) {
                float v[8];
#pragma unroll
                for (int u = 0; u < 8; ++u) v[u] = stage[(r0 + u) * 33 + lane];
#pragma unroll
                for (int u = 0; u < 8; ++u) store_typed(P.C, (m0 + r0 + u) * P.ldc + n, P.out_dtype, P.alpha * v[u] + bias);
              } else {
                // (kept small: with eight copies of it in a row the kernel ran 15 % slower)
#pragma unroll 2
                for (int r = r0; r < min(r0 + 8, rows); ++r) {
                  const int64_t off = (m0 + r) * P.ldc + n;
                  split_finish(P, stage[r * 33 + lane], bias, P.aux_mode ? load_typed(P.aux, off, P.out_dtype) : 0.f,
                               P.accumulate ? load_typed(P.C, off, P.out_dtype) : 0.f, m0 + r, n);
                }
              }
            }
          }
        }
        if (F32 && lane == 0) {
          P.left_out[((int64_t)t * (PAIR ? 2 : 1) + prank) * kSpEpiWarps + warp - 2] = (uint8_t)left_out;
          if (left_out) *redo_flag = 1;
        }
      }
    }
  }

  // ------------------------------------------------- sums of a cluster, teardown --
  tc_fence_before();
  __syncthreads();
  if (PAIR) cluster_sync_all();                        // neither CTA leaves, nor frees tensor memory, while its peer still works
  auto rows_mask = [](int rows) { return 0xffffffffu >> (32 - rows); };
  if (F32 && csize == 1 && *redo_flag && !*abort_flag) {
    // the ring is idle: every copy into it was consumed by a product whose sum the epilogue has seen
    float* const scratch = reinterpret_cast<float*>(base_ptr + warp * kSpRedo);
    constexpr int kPieces = kSpEpiWarps * (NC / 32);
    static_assert((kSpThreads / 32) * kSpRedo <= kSpSlots * kSpSlot, "scratch fits the ring");
    for (int t = worker; t < total; t += workers) {
      const int64_t mt0 = (int64_t)(P.n_fast ? t / P.tiles_n : t % P.tiles_m) * TM + prank * 128, nt0 = (int64_t)(P.n_fast ? t % P.tiles_n : t / P.tiles_m) * TN;
      const uint8_t* marks = P.left_out + ((int64_t)t * (PAIR ? 2 : 1) + prank) * kSpEpiWarps;
      for (int i = warp; i < kPieces; i += kSpThreads / 32) {
        const int w = i / (NC / 32), h = i % (NC / 32);
        const int64_t m0 = mt0 + ((w + 2) & 3) * 32, n0 = nt0 + (w >> 2) * NC + h * 32;
        if ((marks[w] >> h & 1) && m0 < P.M && n0 < P.N) split_make_up(P, m0, n0, rows_mask((int)min((int64_t)32, P.M - m0)), scratch);
      }
    }
  }
  if (!PAIR && csize > 1) {
    cluster_sync_all();
    const bool have = worker < total;
    const int64_t m0 = (int64_t)(P.n_fast ? worker / P.tiles_n : worker % P.tiles_m) * kSpM;
    const int64_t n0 = (int64_t)(P.n_fast ? worker % P.tiles_n : worker / P.tiles_m) * kSpN;
    const int share = kSpM / csize;
    auto sum_at = [&](int r, int col, int c) { return mapa_shared(base + (uint32_t)(r * kSpPitch + col) * 4u, (uint32_t)c); };     // in CTA c
    auto load_sum = [&](uint32_t at) {
      float x;
      asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(x) : "r"(at) : "memory");
      return x;
    };
    if (have) {
      float bias[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int64_t n = n0 + j * 32 + lane;
        bias[j] = P.bias && n < P.N ? load_typed(P.bias, n, P.in_dtype) : 0.f;
      }
      for (int r = rank * share + warp; r < (rank + 1) * share && m0 + r < P.M; r += kSpThreads / 32) {
        float v[4] = {}, aux[4] = {}, old[4] = {};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int64_t n = n0 + j * 32 + lane, off = (m0 + r) * P.ldc + n;
          if (n < P.N && P.aux_mode) aux[j] = load_typed(P.aux, off, P.out_dtype);
          if (n < P.N && P.accumulate) old[j] = load_typed(P.C, off, P.out_dtype);
        }
        for (int c = 0; c < csize; ++c) {
          const uint32_t at = sum_at(r, lane, c);
#pragma unroll
          for (int j = 0; j < 4; ++j) v[j] += load_sum(at + 128u * j);
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int64_t n = n0 + j * 32 + lane;
          if (n >= P.N) continue;
          if (F32 && !split_finite(v[j])) *redo_flag = 1;
          else split_finish(P, F32 ? v[j] * kSpUnscale : v[j], bias[j], aux[j], old[j], m0 + r, n);
        }
      }
    }
    if (F32) {
      __syncthreads();
      if (have && *redo_flag && !*abort_flag) {        // the scratch lies behind the sums, which tell what is missing
        float* const scratch = reinterpret_cast<float*>(base_ptr + (kSpM * kSpPitch * 4 + 127) / 128 * 128 + warp * kSpRedo);
        static_assert((kSpM * kSpPitch * 4 + 127) / 128 * 128 + (kSpThreads / 32) * kSpRedo <= kSpSlots * kSpSlot, "sums and scratch fit the ring");
        for (int i = warp; i < 4 * ((share + 31) / 32); i += kSpThreads / 32) {
          const int r0 = rank * share + (i >> 2) * 32, col = (i & 3) * 32 + lane;
          const int rows = (int)min((int64_t)min(32, (rank + 1) * share - r0), P.M - m0 - r0);
          if (rows <= 0 || n0 + (i & 3) * 32 >= P.N) continue;
          uint32_t missing = 0;
          for (int r = 0; r < rows; ++r) {
            float v = 0.f;
            for (int c = 0; c < csize; ++c) v += load_sum(sum_at(r0 + r, col, c));
            if (!split_finite(v)) missing |= 1u << r;
          }
          if (__any_sync(0xffffffffu, missing)) split_make_up(P, m0 + r0, n0 + (i & 3) * 32, missing, scratch);
        }
      }
    }
    __syncwarp();
    cluster_sync_all();                                // nobody leaves while its sums are still being read
  }
  if (threadIdx.x == 0 && *abort_flag && P.flag) atomicMax(P.flag, 106);   // a bounded wait expired
  if (warp == 1) {
    tc_fence_after();
    if (PAIR) tmem_dealloc_pair(tmem_base, 2 * TN);
    else tmem_dealloc(tmem_base, 2 * TN);
  }
}

// One operand [rows, cols] (row stride ld) and where its planes go: [planes][rows][pitch], pitch a multiple of 8.
struct PrepareJob { const void* src; void* dst; int64_t rows, cols, ld, pitch, units; int vec; };

// A thread rewrites eight neighbouring values. HBM-bound: fp32 reads 4 and writes 6 bytes a value.
template <bool F32>
__global__ void __launch_bounds__(256)
prepare_kernel(const PrepareJob a, const PrepareJob b) {
  grid_dependency_wait();
  allow_dependents();
  const int64_t total = a.units + b.units;
  for (int64_t u = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; u < total; u += (int64_t)gridDim.x * blockDim.x) {
    const bool first = u < a.units;
    const PrepareJob& j = first ? a : b;
    const int64_t i = first ? u : u - a.units;
    const int64_t per_row = j.pitch / 8;
    const int64_t row = total < (1ll << 32) ? (int64_t)((uint32_t)i / (uint32_t)per_row) : i / per_row;
    const int64_t col = (i - row * per_row) * 8;
    const int64_t dst = row * j.pitch + col;
    if (F32) {
      const float* s = (const float*)j.src + row * j.ld + col;
      float x[8];
      if (j.vec && col + 8 <= j.cols) {
        const float4 p = *reinterpret_cast<const float4*>(s), q = *reinterpret_cast<const float4*>(s + 4);
        x[0] = p.x; x[1] = p.y; x[2] = p.z; x[3] = p.w;
        x[4] = q.x; x[5] = q.y; x[6] = q.z; x[7] = q.w;
      } else {
#pragma unroll
        for (int e = 0; e < 8; ++e) x[e] = col + e < j.cols ? s[e] : 0.f;
      }
      Vec16<__nv_bfloat16> h, m, l;
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const float v = x[e] * kSpScale;
        h.e[e] = __float2bfloat16_rn(v);
        const float r = v - __bfloat162float(h.e[e]);          // exact
        m.e[e] = __float2bfloat16_rn(r);
        l.e[e] = __float2bfloat16_rn(r - __bfloat162float(m.e[e]));
      }
      __nv_bfloat16* d = (__nv_bfloat16*)j.dst + dst;
      const int64_t plane = j.rows * j.pitch;
      h.store(d);
      m.store(d + plane);
      l.store(d + 2 * plane);
    } else {
      const uint16_t* s = (const uint16_t*)j.src + row * j.ld + col;
      __align__(16) uint16_t x[8];
#pragma unroll
      for (int e = 0; e < 8; ++e) x[e] = col + e < j.cols ? s[e] : (uint16_t)0;
      *reinterpret_cast<uint4*>((uint16_t*)j.dst + dst) = *reinterpret_cast<const uint4*>(x);
    }
  }
}

// The CUDA-core kernel takes about 8 us and 0.05 us per k for each 64 x 64 tile an SM has (measured in fp32: 256^3
// 21 us, 4096 x 256 x 256 29, 4096 x 256 x 65 15, 4096 x 1024 x 256 102); this path 15-23 us for small products, most of
// it the host's two launches, allocation and tensor maps (256^3 17 us, 4096 x 256 x 256 20, 4096 x 256 x 65 23).
constexpr double kSplitMinUs = 30.0;

bool gemm_split_supported(const GemmArgs& g) {
  if (g.M < 16 || g.N < 16 || g.K < (g.in_dtype == MT_F32 ? 16 : 256)) return false;   // (half, K = 91: error 1.56e-7, FMA chain 1.46e-7)
  if (g.M >= (1ll << 30) || g.N >= (1ll << 30) || g.K > (1ll << 17)) return false;   // (K: as far as the error was measured)
  const double tiles = (double)((g.M + 63) / 64) * (double)((g.N + 63) / 64) / (0.87 * sm_count());
  return 8.0 + 0.05 * (double)g.K * (tiles > 1.0 ? tiles : 1.0) >= kSplitMinUs;
}

template <bool F32, bool A_MN, bool B_MN, bool PAIR>
static int launch_split(const CUtensorMap& ta, const CUtensorMap& tb, const SplitParams& P, int grid, cudaStream_t st) {
  auto kern = gemm_split_kernel<F32, A_MN, B_MN, PAIR>;
  static std::atomic<bool> ready[16];      // per device; racing first calls set the same attribute twice, harmlessly
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 16 || !ready[dev].load(std::memory_order_acquire)) {
    MT_CHECK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kSpSmem));
    if (dev >= 0 && dev < 16) ready[dev].store(true, std::memory_order_release);
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)grid);
  cfg.blockDim = dim3(kSpThreads);
  cfg.dynamicSmemBytes = kSpSmem;
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = PAIR ? 2u : (unsigned)P.csize;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = overlap_launches() ? 2 : 1;
  MT_CHECK_CUDA(cudaLaunchKernelEx(&cfg, kern, ta, tb, P));
  count_launch();
  return MT_OK;
}

int gemm_split(const GemmArgs& g, cudaStream_t st) {
  const bool f32 = g.in_dtype == MT_F32;
  const int planes = f32 ? 3 : 1;
  PrepareJob job[2] = {};
  const void* src[2] = {g.A, g.B};
  const int64_t rows[2] = {g.trans_a ? g.K : g.M, g.trans_b ? g.N : g.K};
  const int64_t cols[2] = {g.trans_a ? g.M : g.K, g.trans_b ? g.K : g.N};
  const int64_t ld[2] = {g.lda, g.ldb};
  size_t bytes = 0, at[2] = {0, 0};
  for (int i = 0; i < 2; ++i) {
    PrepareJob& j = job[i];
    j.src = src[i]; j.rows = rows[i]; j.cols = cols[i]; j.ld = ld[i];
    j.vec = aligned16(src[i]) && ld[i] % 4 == 0;
    j.pitch = (cols[i] + 7) / 8 * 8;
    if (!f32 && aligned16(src[i]) && ld[i] % 8 == 0) continue;       // this half operand can be read where it is
    j.units = rows[i] * (j.pitch / 8);
    at[i] = bytes;
    bytes += ((size_t)planes * rows[i] * j.pitch * 2 + 255) / 256 * 256;
  }
  const size_t marks_at = bytes;
  if (f32) bytes += 2 * (size_t)((g.M + 127) / 128) * (size_t)((g.N + 127) / 128) * kSpEpiWarps;      // (no fewer than a pair's tiles have)
  TempBuf tmp(bytes, st);
  if (!tmp.ok()) {                                                   // no room for the planes
    cudaGetLastError();
    return gemm_simt(g, st);
  }
  for (int i = 0; i < 2; ++i) job[i].dst = job[i].units ? (char*)tmp.ptr + at[i] : nullptr;
  const int64_t units = job[0].units + job[1].units;
  if (units) {
    const int64_t want = (units + 255) / 256, most = (int64_t)sm_count() * 16;
    const dim3 grid((unsigned)(want < most ? want : most));
    if (f32) MT_CHECK_CUDA(launch_overlapped(prepare_kernel<true>, grid, dim3(256), 0, st, job[0], job[1]));
    else MT_CHECK_CUDA(launch_overlapped(prepare_kernel<false>, grid, dim3(256), 0, st, job[0], job[1]));
    count_launch();
  }
  CUtensorMap map[2];
  const bool mn[2] = {g.trans_a != 0, g.trans_b == 0};
  for (int i = 0; i < 2; ++i) {
    const PrepareJob& j = job[i];
    const uint64_t pitch = (uint64_t)(j.units ? j.pitch : j.ld);
    const uint64_t dims[3] = {(uint64_t)j.cols, (uint64_t)j.rows, (uint64_t)planes};
    const uint64_t strides[2] = {pitch, pitch * (uint64_t)j.rows};
    const uint32_t box[3] = {64, (uint32_t)(mn[i] ? kSpK : 128), 1};
    const int rc = make_tmap_nd(&map[i], j.units ? j.dst : j.src, f32 || g.in_dtype == MT_BF16, 3, dims, strides, box);
    if (rc) return rc;
  }
  ProfScope prof(PROF_GEMM, st, 2.0 * (double)g.M * (double)g.N * (double)g.K);
  SplitParams P{};
  P.A = g.A; P.B = g.B; P.C = g.C; P.preact = g.preact; P.bias = g.bias; P.aux = g.aux;
  P.M = g.M; P.N = g.N; P.K = g.K; P.lda = g.lda; P.ldb = g.ldb; P.ldc = g.ldc;
  P.trans_a = g.trans_a; P.trans_b = g.trans_b; P.in_dtype = g.in_dtype; P.out_dtype = g.out_dtype;
  P.act = g.act; P.aux_mode = g.aux_mode; P.accumulate = g.accumulate; P.alpha = g.alpha;
  P.kb_total = (int)((g.K + kSpK - 1) / kSpK);
  // Slices that stay in tensor memory: the error grows with them, the FMA chain's with sqrt(K), and the epilogue's additions
  // cost time (3885 x 50257 -> 768: one slice 700 us, two 585, four 515, eight 479).
  P.chunk = f32 || g.K < 2048 ? 1 : g.K < 12288 ? 2 : g.K < 49152 ? 4 : 8;
  P.left_out = f32 ? (uint8_t*)tmp.ptr + marks_at : nullptr;
  P.flag = device_flag_ptr();
  // Neighbouring tiles share the larger operand's panel unless it fits the L2 anyway.
  P.n_fast = g.M > g.N ? 1 : 0;
  const int sms = sm_count(), pairs = resident_cta_pairs();
  auto tiles_of = [&](int t) { return ((g.M + t - 1) / t) * ((g.N + t - 1) / t); };
  long long tiles = tiles_of(128);
  // K over a cluster while that leaves no CTA waiting for an SM and each at least two slices.
  P.csize = 1;
  while (P.csize < 8 && tiles * P.csize * 2 <= sms && P.kb_total >= 4 * P.csize) P.csize *= 2;
  P.kb_per_rank = (P.kb_total + P.csize - 1) / P.csize;
  while (P.csize > 1 && (P.csize - 1) * P.kb_per_rank >= P.kb_total) {        // no rank without work
    P.csize /= 2;
    P.kb_per_rank = (P.kb_total + P.csize - 1) / P.csize;
  }
  // A pair's 256 x 256 tile needs half the operand bytes per multiplication: a slice takes it about 4300
  // cycles, a single CTA's 128 x 128 tile 3600 (one plane: 1990, 1770); which one is ahead is a matter of how many rounds
  // of tiles each leaves on the chip (fp32 8192 x 768 -> 3072: pair 179 us, single 423; 3072 x 8192 x 768: 308, 260).
  const double kb_one = f32 ? 3600.0 : 1770.0, kb_pair = f32 ? 4300.0 : 1990.0;
  const double one = (double)((tiles * P.csize + sms - 1) / sms) * (P.kb_per_rank * kb_one + 4000.0);
  const double two = (double)((tiles_of(256) + pairs - 1) / pairs) * (P.kb_total * kb_pair + 6000.0);
  const bool pair = two < one;
  if (pair) {
    tiles = tiles_of(256);
    P.csize = 1;
    P.kb_per_rank = P.kb_total;
  }
  const int64_t t = pair ? 256 : 128;
  P.tiles_m = (int)((g.M + t - 1) / t);
  P.tiles_n = (int)((g.N + t - 1) / t);
  const int grid = pair ? 2 * (int)(tiles < pairs ? tiles : pairs) : P.csize > 1 ? (int)tiles * P.csize : (int)(tiles < sms ? tiles : sms);
#define MT_SPLIT_ORDER(F, A, B) \
  (pair ? launch_split<F, A, B, true>(map[0], map[1], P, grid, st) : launch_split<F, A, B, false>(map[0], map[1], P, grid, st))
#define MT_SPLIT(F)                                                                       \
  (mn[0] ? (mn[1] ? MT_SPLIT_ORDER(F, true, true) : MT_SPLIT_ORDER(F, true, false))       \
         : (mn[1] ? MT_SPLIT_ORDER(F, false, true) : MT_SPLIT_ORDER(F, false, false)))
  return f32 ? MT_SPLIT(true) : MT_SPLIT(false);
#undef MT_SPLIT
#undef MT_SPLIT_ORDER
}

}  // namespace mt
