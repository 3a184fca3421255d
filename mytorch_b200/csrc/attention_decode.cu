// Attention of a few new query rows against a key/value cache (the inference step:
// gpt2_trainer/gpt2.py:29-86 Cache and :167-215 cached attention; Sq != Skv as in
// fused_ops/flash_cross_attention.py) and the append of new K/V rows to that cache.
//
// The cache is a preallocated ring [B, H, max_len, D]: appending never moves old rows, and once
// max_len rows are held the oldest is overwritten - the "drop the oldest token" policy of the
// reference's Cache.update without its concatenate-and-slice copies. Softmax attention does not
// depend on the order of the keys, so the ring order is immaterial for the result.
//
// Decode attention is HBM bound: it reads kv_len*D*2 elements of K and V per (batch, key/value head)
// once (+ q and o rows). One block - or a cluster of up to eight that split the keys - works on one
// key/value head of one sequence and on up to five of the query heads that share it, so grouped
// heads do not read the cache again. A key row is spread over D*s/16 lanes as 16-byte vectors
// (coalesced; a warp holds four K and four V loads per lane in flight), the dot product is a
// shuffle reduction over those lanes, and each lane group keeps its own online softmax and its
// slice of O. Lane groups and warps merge through shared memory, blocks of a cluster through
// distributed shared memory: no scratch in HBM and no second kernel.
// With `fused` the same kernel also does the step's preparation: rotary embedding and QK-norm of
// the new query and key (nanochat) and the append of the new key/value row to the cache.
// 8x12 heads x 144 keys x 64 fp16, 24 caches in turn: 7.2 us (one block per query head and one key row per lane 8.5); 32x10 heads on
// 2 x 310 keys x 128 bf16 14.8 (36.0).
#include "common.cuh"
#include "attention.cuh"
#include "decode.cuh"
#include <atomic>
#include <cooperative_groups.h>

namespace mt {
namespace cg = cooperative_groups;

constexpr int kDecWarps = 4;
constexpr int kDecMaxGroup = 5;       // query heads per block
constexpr int kDecUnroll = 4;         // key rows in flight per lane

struct DecodeParams {
  const void* q; const void* k_new; const void* v_new;
  void* kc; void* vc; void* o;
  mt_strides3 sq, sk_new, sv_new, sc, so;
  int heads, kv_heads, group, chunks, q_len, kv_len, causal_offset;
  float scale_log2;
  int fused, append_slot, early;      // append_slot: cache row of the new key (fused)
  const float* cs; const float* sn;   // rotary tables' row of the new position, null = no rotary / norm
  float eps;
};

// One head vector in shared memory: x -> rmsnorm(rope(x)), rounded like the separate kernel's output.
template <typename T, int D>
__device__ __forceinline__ void rope_norm_vector(float* v, const float* cs, const float* sn, float eps, int lane) {
  float r[D / 32], ss = 0.f;
#pragma unroll
  for (int i = 0; i < D / 32; ++i) {
    const int d = lane + 32 * i;
    const float partner = v[d < D / 2 ? d + D / 2 : d - D / 2];
    r[i] = v[d] * cs[d] + (d < D / 2 ? -partner : partner) * sn[d];
    ss += r[i] * r[i];
  }
  ss = warp_sum(ss);
  const float rstd = rsqrtf(ss * (1.f / D) + eps);
  __syncwarp();
#pragma unroll
  for (int i = 0; i < D / 32; ++i) v[lane + 32 * i] = to_f(from_f<T>(r[i] * rstd));
  __syncwarp();
}

template <typename T, int D, int G>
__global__ void __launch_bounds__(kDecWarps * 32)
attn_decode_kernel(const DecodeParams p) {
  constexpr int VN = Vec16<T>::N;
  constexpr int LPK = D / VN;              // lanes per key row
  constexpr int KPI = 32 / LPK;            // key rows per load
  constexpr int U = kDecUnroll;
  __shared__ float q_s[G][D];
  __shared__ __align__(16) T new_k[D];
  __shared__ __align__(16) T new_v[D];
  __shared__ float tmp[D];
  __shared__ float red_m[kDecWarps][G], red_l[kDecWarps][G];
  __shared__ float red_o[kDecWarps][G][D];
  __shared__ float part_m[G], part_l[G];
  __shared__ float part_o[G][D];
  auto cluster = cg::this_cluster();
  const int splits = (int)cluster.num_blocks(), split = (int)cluster.block_rank();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int idx = (int)blockIdx.x / splits;
  const int qi = idx % p.q_len;
  idx /= p.q_len;
  const int chunk = idx % p.chunks;
  idx /= p.chunks;
  const int hk = idx % p.kv_heads, b = idx / p.kv_heads;
  const int h0 = hk * p.group + chunk * G;
  const int gn = min(G, p.group - chunk * G);   // query heads of this block
  const T* kbase = (const T*)p.kc + (int64_t)b * p.sc.b + (int64_t)hk * p.sc.h;
  const T* vbase = (const T*)p.vc + (int64_t)b * p.sc.b + (int64_t)hk * p.sc.h;
  const int n_keys = p.causal_offset < 0 ? p.kv_len : min(p.kv_len, p.causal_offset + qi + 1);
  const int per = (n_keys + splits - 1) / splits;
  const int j_begin = split * per, j_end = min(n_keys, j_begin + per);
  const int grp = lane / LPK, dl = (lane % LPK) * VN;
  const int slot = p.fused ? p.append_slot : -1;          // the new key: read from shared memory
  Vec16<T> kv[U], vv[U];
  auto load_pass = [&](int j0) {
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int j = j0 + u * KPI + grp;
      kv[u].u = make_uint4(0, 0, 0, 0);
      vv[u].u = make_uint4(0, 0, 0, 0);
      if (j < j_end && j != slot) {
        kv[u].load(kbase + (int64_t)j * p.sc.s + dl);
        vv[u].load(vbase + (int64_t)j * p.sc.s + dl);
      }
    }
  };
  const int j_first = j_begin + warp * (KPI * U);
  // Cached rows that no kernel of this step writes may be read before the one in front has finished.
  if (p.early) load_pass(j_first);
  grid_dependency_wait();
  allow_dependents();
  if (!p.early) load_pass(j_first);
  for (int i = threadIdx.x; i < G * D; i += kDecWarps * 32) {
    const int g = i / D, d = i % D;
    q_s[g][d] = g < gn ? to_f(((const T*)p.q)[(int64_t)b * p.sq.b + (int64_t)(h0 + g) * p.sq.h + (int64_t)qi * p.sq.s + d]) : 0.f;
  }
  if (p.fused) {
    const T* kn = (const T*)p.k_new + (int64_t)b * p.sk_new.b + (int64_t)hk * p.sk_new.h;
    const T* vn = (const T*)p.v_new + (int64_t)b * p.sv_new.b + (int64_t)hk * p.sv_new.h;
    for (int d = threadIdx.x; d < D; d += kDecWarps * 32) {
      new_k[d] = kn[d];
      new_v[d] = vn[d];
      tmp[d] = to_f(kn[d]);
    }
    __syncthreads();
    if (p.cs) {
      for (int g = warp; g <= G; g += kDecWarps)
        rope_norm_vector<T, D>(g < G ? q_s[g] : tmp, p.cs, p.sn, p.eps, lane);
      __syncthreads();
      for (int d = threadIdx.x; d < D; d += kDecWarps * 32) new_k[d] = from_f<T>(tmp[d]);
      __syncthreads();
    }
    // one block per key/value head writes the new row into the cache; every block reads it from
    // shared memory
    if (split == 0 && chunk == 0) {
      T* kd = (T*)p.kc + (int64_t)b * p.sc.b + (int64_t)hk * p.sc.h + (int64_t)p.append_slot * p.sc.s;
      T* vd = (T*)p.vc + (int64_t)b * p.sc.b + (int64_t)hk * p.sc.h + (int64_t)p.append_slot * p.sc.s;
      for (int d = threadIdx.x; d < D; d += kDecWarps * 32) { kd[d] = new_k[d]; vd[d] = new_v[d]; }
    }
  }
  __syncthreads();
  float qr[G][VN], acc[G][VN], m[G], l[G];
#pragma unroll
  for (int g = 0; g < G; ++g) {
    m[g] = -INFINITY;
    l[g] = 0.f;
#pragma unroll
    for (int e = 0; e < VN; ++e) { qr[g][e] = q_s[g][dl + e] * p.scale_log2; acc[g][e] = 0.f; }
  }
  for (int j0 = j_first; j0 < j_end; j0 += kDecWarps * KPI * U) {
    if (j0 != j_first) load_pass(j0);
    if (p.fused) {
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (j0 + u * KPI + grp == slot) { kv[u].load(new_k + dl); vv[u].load(new_v + dl); }
    }
#pragma unroll
    for (int g = 0; g < G; ++g) {
      float s[U], mx = m[g];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        float dot = 0.f;
#pragma unroll
        for (int e = 0; e < VN; ++e) dot = fmaf(kv[u].get(e), qr[g][e], dot);
#pragma unroll
        for (int o = LPK / 2; o > 0; o >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, o);
        s[u] = j0 + u * KPI + grp < j_end ? dot : -INFINITY;
        mx = fmaxf(mx, s[u]);
      }
      if (mx == -INFINITY) {               // no key of this lane group yet (per lane; no shuffles below), or only NaN scores
        bool nan = false;
#pragma unroll
        for (int u = 0; u < U; ++u) nan |= isnan(s[u]);
        if (!nan) continue;
        mx = 0.f;
      }
      const float alpha = exp2f(m[g] - mx);
      m[g] = mx;
      l[g] *= alpha;
#pragma unroll
      for (int e = 0; e < VN; ++e) acc[g][e] *= alpha;
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const float pr = exp2f(s[u] - mx);
        l[g] += pr;
#pragma unroll
        for (int e = 0; e < VN; ++e) acc[g][e] = fmaf(pr, vv[u].get(e), acc[g][e]);
      }
    }
  }
  // lane groups of a warp
#pragma unroll
  for (int g = 0; g < G; ++g) {
#pragma unroll
    for (int o = LPK; o < 32; o <<= 1) {
      const float mo = __shfl_xor_sync(0xffffffffu, m[g], o), lo = __shfl_xor_sync(0xffffffffu, l[g], o);
      const float mn = fmaxf(m[g], mo);
      const float a = m[g] == -INFINITY ? 0.f : exp2f(m[g] - mn), c = mo == -INFINITY ? 0.f : exp2f(mo - mn);
      l[g] = l[g] * a + lo * c;
#pragma unroll
      for (int e = 0; e < VN; ++e) acc[g][e] = acc[g][e] * a + __shfl_xor_sync(0xffffffffu, acc[g][e], o) * c;
      m[g] = mn;
    }
    if (grp == 0) {
#pragma unroll
      for (int e = 0; e < VN; ++e) red_o[warp][g][dl + e] = acc[g][e];
    }
    if (lane == 0) { red_m[warp][g] = m[g]; red_l[warp][g] = l[g]; }
  }
  __syncthreads();
  // warps of the block, then (through distributed shared memory) blocks of the cluster
  auto out = [&](int g, int d, float v) {
    if (g < gn) ((T*)p.o)[(int64_t)b * p.so.b + (int64_t)(h0 + g) * p.so.h + (int64_t)qi * p.so.s + d] = from_f<T>(v);
  };
  for (int i = threadIdx.x; i < G * D; i += kDecWarps * 32) {
    const int g = i / D, d = i % D;
    float mm = -INFINITY, ll = 0.f, v = 0.f;
#pragma unroll
    for (int w = 0; w < kDecWarps; ++w) mm = fmaxf(mm, red_m[w][g]);
#pragma unroll
    for (int w = 0; w < kDecWarps; ++w) {
      const float a = red_m[w][g] == -INFINITY ? 0.f : exp2f(red_m[w][g] - mm);
      ll += red_l[w][g] * a;
      v += red_o[w][g][d] * a;
    }
    if (splits == 1) out(g, d, ll == 0.f ? 0.f : v / ll);
    else {
      part_o[g][d] = v;
      if (d == 0) { part_m[g] = mm; part_l[g] = ll; }
    }
  }
  if (splits > 1) {
    cluster.sync();
    for (int i = split * kDecWarps * 32 + threadIdx.x; i < G * D; i += splits * kDecWarps * 32) {
      const int g = i / D, d = i % D;
      float mm = -INFINITY, ll = 0.f, v = 0.f;
      for (int r = 0; r < splits; ++r) mm = fmaxf(mm, *cluster.map_shared_rank(&part_m[g], r));
      for (int r = 0; r < splits; ++r) {
        const float mr = *cluster.map_shared_rank(&part_m[g], r);
        const float a = mr == -INFINITY ? 0.f : exp2f(mr - mm);
        ll += *cluster.map_shared_rank(&part_l[g], r) * a;
        v += *cluster.map_shared_rank(&part_o[g][d], r) * a;
      }
      out(g, d, ll == 0.f ? 0.f : v / ll);
    }
    cluster.sync();                        // nobody leaves while its partial is still being read
  }
}

// cache[b, h, (pos0 + i) % max_len, :] = new[b, h, i, :]
template <typename T>
__global__ void __launch_bounds__(256)
kv_append_kernel(const T* __restrict__ k_new, const T* __restrict__ v_new, T* __restrict__ k_cache, T* __restrict__ v_cache,
                 mt_strides3 sk, mt_strides3 sv, mt_strides3 sc, int heads, int n_new, int pos0, int max_len, int D,
                 int64_t total) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
    const int d = (int)(i % D);
    int64_t r = i / D;
    const int t = (int)(r % n_new);
    r /= n_new;
    const int h = (int)(r % heads), b = (int)(r / heads);
    const int64_t dst = (int64_t)b * sc.b + (int64_t)h * sc.h + (int64_t)((pos0 + t) % max_len) * sc.s + d;
    k_cache[dst] = k_new[(int64_t)b * sk.b + (int64_t)h * sk.h + (int64_t)t * sk.s + d];
    v_cache[dst] = v_new[(int64_t)b * sv.b + (int64_t)h * sv.h + (int64_t)t * sv.s + d];
  }
}

template <typename T, int D, int G>
static int launch_decode_g(const DecodeParams& p, int blocks, int splits, cudaStream_t st) {
  auto kern = attn_decode_kernel<T, D, G>;
  static std::atomic<bool> ready[16];      // per device; racing first calls set the same attribute twice, harmlessly
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 16 || !ready[dev].load(std::memory_order_acquire)) {
    // the split of L1 that the step's products use: an SM does not have to drain to change it
    MT_CHECK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared));
    if (dev >= 0 && dev < 16) ready[dev].store(true, std::memory_order_release);
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(blocks * splits));
  cfg.blockDim = dim3(kDecWarps * 32);
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)splits;
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

template <typename T, int D>
static int launch_decode(DecodeParams& p, int64_t batch, cudaStream_t st) {
  // query heads of a key/value head in equal chunks of at most kDecMaxGroup
  p.chunks = (p.group + kDecMaxGroup - 1) / kDecMaxGroup;
  const int G = (p.group + p.chunks - 1) / p.chunks;
  const int64_t blocks = batch * p.kv_heads * p.chunks * p.q_len;
  MT_REQUIRE(blocks * 8 < (1ll << 31), "attn_decode: too many query rows");
  // Split the keys until a block needs one pass over its warps' loads (a pass is a full memory latency:
  // 6.2 us for three of them at 8x12 heads x 140 keys x 64, fp16), as long as all blocks stay
  // resident (four per SM with one query head per block, two with more).
  constexpr int kPass = kDecWarps * (32 / (D / Vec16<T>::N)) * kDecUnroll;
  const int resident = sm_count() * (G == 1 ? 4 : 2);
  int splits = 1;
  while (splits < 8 && p.kv_len > splits * kPass && blocks * splits * 2 <= resident) splits *= 2;
  switch (G) {
    case 1: return launch_decode_g<T, D, 1>(p, (int)blocks, splits, st);
    case 2: return launch_decode_g<T, D, 2>(p, (int)blocks, splits, st);
    case 3: return launch_decode_g<T, D, 3>(p, (int)blocks, splits, st);
    case 4: return launch_decode_g<T, D, 4>(p, (int)blocks, splits, st);
    default: return launch_decode_g<T, D, 5>(p, (int)blocks, splits, st);
  }
}

int attn_decode_step(const DecodeStep& a, cudaStream_t st) {
  DecodeParams p{};
  p.q = a.q; p.k_new = a.k_new; p.v_new = a.v_new;
  p.kc = a.k_cache; p.vc = a.v_cache; p.o = a.o;
  p.sq = a.sq; p.sk_new = a.sk_new; p.sv_new = a.sv_new; p.sc = a.sc; p.so = a.so;
  p.heads = (int)a.heads; p.kv_heads = (int)a.kv_heads; p.group = (int)(a.heads / a.kv_heads);
  p.q_len = (int)a.q_len; p.kv_len = (int)a.kv_len; p.causal_offset = a.causal_offset;
  p.scale_log2 = a.scale * 1.4426950408889634f;
  p.fused = a.fused; p.append_slot = (int)a.append_slot; p.early = a.early_cache;
  p.cs = a.cos_row; p.sn = a.sin_row; p.eps = a.eps;
  MT_DISPATCH_FLOAT(a.dtype, T, return (a.head_dim == 64 ? launch_decode<T, 64>(p, a.batch, st) : launch_decode<T, 128>(p, a.batch, st)));
  return MT_OK;
}

int kv_append(const void* k_new, const void* v_new, void* k_cache, void* v_cache, mt_strides3 sk, mt_strides3 sv,
              mt_strides3 scache, int64_t batch, int64_t heads, int64_t n_new, int64_t pos0, int64_t max_len,
              int64_t head_dim, int dtype, cudaStream_t st) {
  const int64_t total = batch * heads * n_new * head_dim;
  if (total == 0) return MT_OK;
  int64_t blocks = (total + 255) / 256;
  if (blocks > (int64_t)sm_count() * 16) blocks = (int64_t)sm_count() * 16;
  MT_DISPATCH_FLOAT(dtype, T, (kv_append_kernel<T><<<(unsigned)blocks, 256, 0, st>>>(
      (const T*)k_new, (const T*)v_new, (T*)k_cache, (T*)v_cache, sk, sv, scache, (int)heads, (int)n_new, (int)pos0,
      (int)max_len, (int)head_dim, total)));
  MT_LAUNCH_CHECK();
  return MT_OK;
}

}  // namespace mt

using namespace mt;

extern "C" {

int mt_attn_decode_gqa(const void* q, const void* k_cache, const void* v_cache, void* o, mt_strides3 sq, mt_strides3 skv,
                       mt_strides3 so, int64_t batch, int64_t heads, int64_t kv_heads, int64_t q_len, int64_t kv_len,
                       int64_t head_dim, float scale, int causal_offset, int dtype, void* stream) {
  MT_REQUIRE(q && k_cache && v_cache && o && batch >= 0 && heads > 0 && q_len >= 0 && kv_len >= 0 && head_dim > 0,
             "attn_decode: bad arguments");
  MT_REQUIRE(kv_heads > 0 && heads % kv_heads == 0, "attn_decode: query heads must be a multiple of key/value heads");
  MT_REQUIRE(head_dim == 64 || head_dim == 128, "attn_decode: head_dim must be 64 or 128");
  MT_REQUIRE(batch * heads * q_len < (1ll << 31), "attn_decode: too many query rows");
  constexpr int64_t kAlign = 8;   // 16-byte vector loads of half rows (4 for fp32 rows is implied)
  MT_REQUIRE(skv.b % kAlign == 0 && skv.h % kAlign == 0 && skv.s % kAlign == 0 && aligned16(k_cache) && aligned16(v_cache),
             "attn_decode: cache rows must be 16-byte aligned");
  if (batch == 0 || q_len == 0) return MT_OK;
  DecodeStep d{};
  d.q = q; d.k_cache = const_cast<void*>(k_cache); d.v_cache = const_cast<void*>(v_cache); d.o = o;
  d.sq = sq; d.sc = skv; d.so = so;
  d.batch = batch; d.heads = heads; d.kv_heads = kv_heads; d.q_len = q_len; d.kv_len = kv_len; d.head_dim = head_dim;
  d.scale = scale; d.causal_offset = causal_offset; d.dtype = dtype;
  return attn_decode_step(d, as_stream(stream));
}

int mt_attn_decode(const void* q, const void* k_cache, const void* v_cache, void* o, mt_strides3 sq, mt_strides3 skv,
                   mt_strides3 so, int64_t batch, int64_t heads, int64_t q_len, int64_t kv_len, int64_t head_dim,
                   float scale, int causal_offset, int dtype, void* stream) {
  return mt_attn_decode_gqa(q, k_cache, v_cache, o, sq, skv, so, batch, heads, heads, q_len, kv_len, head_dim, scale,
                            causal_offset, dtype, stream);
}

int mt_kv_append(const void* k_new, const void* v_new, void* k_cache, void* v_cache, mt_strides3 sk, mt_strides3 sv,
                 mt_strides3 scache, int64_t batch, int64_t heads, int64_t n_new, int64_t pos0, int64_t max_len,
                 int64_t head_dim, int dtype, void* stream) {
  MT_REQUIRE(k_new && v_new && k_cache && v_cache && batch >= 0 && heads > 0 && n_new >= 0 && pos0 >= 0 && max_len > 0 &&
             head_dim > 0 && n_new <= max_len, "kv_append: bad arguments");
  return kv_append(k_new, v_new, k_cache, v_cache, sk, sv, scache, batch, heads, n_new, pos0, max_len, head_dim, dtype,
                   as_stream(stream));
}

}  // extern "C"
