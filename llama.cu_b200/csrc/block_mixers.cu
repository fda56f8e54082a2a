// Mixers of the block models: attention over a sliding window and pooled blocks, linear recurrences, and the fused
// one-token launch of all branches of a mixer.
#include <algorithm>

#include <math_constants.h>

#include "block_ops.cuh"
#include "elem.cuh"
#include "gemv.cuh"

namespace lcu {
namespace {

constexpr int MX_THREADS = 256;
constexpr int PART_FLOATS = 4096;  // partial sums of the value pass (groups x value columns)

__host__ __device__ __forceinline__ int pow2_at_least(int n) {
  int p = 1;
  while (p < n) p *= 2;
  return p;
}

// what position i sees: blocks 0 .. blocks-1 and tokens lo .. i
__host__ __device__ __forceinline__ void window_of(int i, int window, int pool, int& lo, int& blocks) {
  lo = i + 1 > window ? i + 1 - window : 0;
  const int past = i + 1 - window;  // positions that have left the window
  blocks = pool > 0 && past > 0 ? past / pool : 0;
}

__device__ __forceinline__ float block_max(float v, float* red) {
  v = warp_max(v);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  float m = red[0];
#pragma unroll
  for (int w = 1; w < MX_THREADS / 32; ++w) m = fmaxf(m, red[w]);
  return m;
}
__device__ __forceinline__ float block_sum(float v, float* red) {
  v = warp_sum(v);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  float s = 0.f;
#pragma unroll
  for (int w = 0; w < MX_THREADS / 32; ++w) s += red[w];
  return s;
}

// ------------------------------------------------------------------ attention of one query row and head
template <typename T>
__host__ __device__ __forceinline__ int query_cols(const attn_rows<T>& p) {
  return (p.dim + 7) / 8 * 8 + (p.key2 ? (p.dim2 + 7) / 8 * 8 : 0);
}
// `rank` of `C` CTAs takes a slice of the visible keys.  The row's own key and value come from `cur_k` / `cur_v` (shared
// memory copies) when given, else from the cache.  Leaves max, sum and the unnormalised value row in res[0], res[1],
// res[2 ..].  Shared memory: q [query_cols], scores [slice], part [PART_FLOATS].
template <typename T>
__device__ void attend_slice(const attn_rows<T>& p, const T* q_row, int head, int pos, int rank, int C, const T* cur_k, const T* cur_v, float* q,
                             float* sc, float* part, float* red, float* res) {
  constexpr int VEC = 16 / sizeof(T);
  const int tid = threadIdx.x;
  const int kvh = head / (p.heads / p.kv_heads);
  const int ldk = p.cache.ldk, ldv = p.cache.ldv;
  const int k_cols = (p.dim + 7) / 8 * 8, v_cols = (p.vdim + 7) / 8 * 8, q_cols = query_cols(p);
  const T* kc = p.cache.k + kvh * p.cache.k_head;
  const T* vc = p.cache.v + kvh * p.cache.v_head;
  const T* kp = p.cache.kp + (size_t)kvh * p.cache.n_blocks * ldk;
  const T* vp = p.cache.vp + (size_t)kvh * p.cache.n_blocks * ldv;
  int lo, blocks;
  window_of(pos, p.window, p.pool, lo, blocks);
  const int total = blocks + pos + 1 - lo;
  const int t0 = (int)((long long)total * rank / C), n = (int)((long long)total * (rank + 1) / C) - t0;
  for (int d = tid; d < q_cols; d += MX_THREADS) q[d] = d < p.dim || p.key2 ? to_f(q_row[head * p.q_head + d]) : 0.f;
  __syncthreads();
  auto key_at = [&](int t) -> const T* {
    if (t < blocks) return kp + (size_t)t * ldk;
    const int j = lo + t - blocks;
    return cur_k && j == pos ? cur_k : kc + (size_t)(j - p.cache.first) * ldk;
  };
  auto value_at = [&](int t) -> const T* {
    if (t < blocks) return vp + (size_t)t * ldv;
    const int j = lo + t - blocks;
    return cur_v && j == pos ? cur_v : vc + (size_t)(j - p.cache.first) * ldv;
  };
  // scores: lpk lanes per key
  {
    const int lpk = min(32, pow2_at_least((k_cols + VEC - 1) / VEC)), groups = MX_THREADS / lpk, grp = tid / lpk, sub = tid % lpk;
    constexpr int U = 4;
    const int rounds = (n + groups * U - 1) / (groups * U);  // (the same for every lane: the shuffles below are warp-wide)
    for (int rd = 0; rd < rounds; ++rd) {
      float s[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        s[u] = 0.f;
        const int t = (rd * U + u) * groups + grp;
        if (t < n) {
          const T* k = key_at(t0 + t);
          for (int d = sub * VEC; d < k_cols; d += lpk * VEC) {
            const uint4 raw = *reinterpret_cast<const uint4*>(k + d);
#pragma unroll
            for (int e = 0; e < VEC; ++e) s[u] = fmaf(q[d + e], to_f(reinterpret_cast<const T*>(&raw)[e]), s[u]);
          }
          if (p.key2) {
            const T* k2 = p.key2 + (size_t)(lo + t0 + t - blocks - p.first2) * p.ld2 - k_cols;
            for (int d = k_cols + sub * VEC; d < q_cols; d += lpk * VEC) {
              const uint4 raw = *reinterpret_cast<const uint4*>(k2 + d);
#pragma unroll
              for (int e = 0; e < VEC; ++e) s[u] = fmaf(q[d + e], to_f(reinterpret_cast<const T*>(&raw)[e]), s[u]);
            }
          }
        }
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        for (int o = lpk >> 1; o > 0; o >>= 1) s[u] += __shfl_xor_sync(0xffffffffu, s[u], o);
        const int t = (rd * U + u) * groups + grp;
        if (sub == 0 && t < n) sc[t] = s[u] * p.scale;
      }
    }
  }
  __syncthreads();
  float mx = -CUDART_INF_F;
  for (int t = tid; t < n; t += MX_THREADS) mx = fmaxf(mx, sc[t]);
  mx = block_max(mx, red);
  const float ref = mx > -CUDART_INF_F ? mx : 0.f;  // (scores of -inf alone weigh nothing; one that is no number reaches the sum either way)
  float sum = 0.f;
  for (int t = tid; t < n; t += MX_THREADS) {
    const float e = expf(sc[t] - ref);
    sc[t] = e;
    sum += e;
  }
  sum = block_sum(sum, red);  // (its barriers also publish the exponentials)
  // values: lpv lanes per row of values, groups of them walk the keys
  const int lpv = min(32, pow2_at_least((v_cols + VEC - 1) / VEC)), groups = MX_THREADS / lpv, grp = tid / lpv, sub = tid % lpv;
  for (int d0 = 0; d0 < v_cols; d0 += lpv * VEC) {
    const int d = d0 + sub * VEC;
    float acc[VEC] = {};
    if (d < v_cols) {
#pragma unroll 4
      for (int t = grp; t < n; t += groups) {
        const uint4 raw = *reinterpret_cast<const uint4*>(value_at(t0 + t) + d);
        const float w = sc[t];
#pragma unroll
        for (int e = 0; e < VEC; ++e) acc[e] = fmaf(w, to_f(reinterpret_cast<const T*>(&raw)[e]), acc[e]);
      }
    }
    __syncthreads();
#pragma unroll
    for (int e = 0; e < VEC; ++e) part[(grp * lpv + sub) * VEC + e] = acc[e];
    __syncthreads();
    for (int j = tid; j < lpv * VEC && d0 + j < p.vdim; j += MX_THREADS) {
      float v = 0.f;
      for (int g = 0; g < groups; ++g) v += part[g * lpv * VEC + j];
      res[2 + d0 + j] = v;
    }
  }
  if (tid == 0) {
    res[0] = n > 0 ? mx : -CUDART_INF_F;
    res[1] = n > 0 ? sum : 0.f;
  }
  __syncthreads();
}

// rows of a pass, one CTA per (row, head); keys and blocks are in the cache already
template <typename T>
__global__ void __launch_bounds__(MX_THREADS) window_rows_kernel(const attn_rows<T> p, int pos0, int max_keys) {
  extern __shared__ __align__(16) float sm[];
  __shared__ float red[MX_THREADS / 32];
  pdl_launch_dependents();
  pdl_wait();
  const int head = blockIdx.x, r = blockIdx.y;
  float* q = sm;
  float* part = q + query_cols(p);
  float* res = part + PART_FLOATS;
  float* sc = res + 2 + round_up_dev(p.vdim + 2, 4);
  attend_slice(p, p.q + (size_t)r * p.ld, head, pos0 + r, 0, 1, (const T*)nullptr, (const T*)nullptr, q, sc, part, red, res);
  float inv = p.out_scale / res[1];
  if (p.sink) {
    const float top = fmaxf(res[0], p.sink[head]), f = expf(res[0] - top);
    inv = p.out_scale * f / (res[1] * f + expf(p.sink[head] - top));
  }
  if (p.gate) inv *= sigmoid_f(to_f(p.gate[(size_t)r * p.ldg + head]));
  for (int d = threadIdx.x; d < p.vdim; d += MX_THREADS) p.out[(size_t)r * p.ldo + head * p.vdim + d] = from_f<T>(res[2 + d] * inv);
}

// new rows of k and v into the cache
template <typename T>
__global__ void __launch_bounds__(256) window_append_kernel(const attn_rows<T> p, int m, int pos0) {
  pdl_launch_dependents();
  pdl_wait();
  const int r = blockIdx.x;
  for (int i = threadIdx.x; i < p.kv_heads * p.dim; i += 256) {
    const int g = i / p.dim, d = i - g * p.dim;
    p.cache.k[((size_t)g * p.cache.ctx_len + pos0 + r) * p.cache.ldk + d] = p.k[(size_t)r * p.ld + i];
  }
  for (int i = threadIdx.x; i < p.kv_heads * p.vdim; i += 256) {
    const int g = i / p.vdim, d = i - g * p.vdim;
    p.cache.v[((size_t)g * p.cache.ctx_len + pos0 + r) * p.cache.ldv + d] = p.v[(size_t)r * p.ld + i];
  }
}

// mean of the cached rows of one block
template <typename T>
__device__ __forceinline__ void pool_block(const T* rows, int ld, int pool, const T* last, T* out, int dim) {
  for (int d = threadIdx.x; d < dim; d += blockDim.x) {
    float s = 0.f;
    const int stored = last ? pool - 1 : pool;
#pragma unroll 8
    for (int j = 0; j < stored; ++j) s += to_f(rows[(size_t)j * ld + d]);
    if (last) s += to_f(last[d]);
    out[d] = from_f<T>(s / (float)pool);
  }
}
template <typename T>
__global__ void __launch_bounds__(128) window_pool_kernel(const attn_rows<T> p, int first_block) {
  pdl_launch_dependents();
  pdl_wait();
  const int b = first_block + blockIdx.x, g = blockIdx.y;
  const size_t row = (size_t)g * p.cache.ctx_len + (size_t)b * p.pool, dst = (size_t)g * p.cache.n_blocks + b;
  pool_block(p.cache.k + row * p.cache.ldk, p.cache.ldk, p.pool, (const T*)nullptr, p.cache.kp + dst * p.cache.ldk, p.dim);
  pool_block(p.cache.v + row * p.cache.ldv, p.cache.ldv, p.pool, (const T*)nullptr, p.cache.vp + dst * p.cache.ldv, p.vdim);
}

// ------------------------------------------------------------------ recurrences over rows
// The first launch lays a pass's rows out for the next, in binary32: per head and row q, k (rotated and scaled),
// the decays of a wkv layer and its bonus sum_i q_i u_i k_i (the same for every value column) as one run of `stride`
// floats, and the values by blocks of `cols` columns.  The next walks the rows: a CTA owns `cols` value columns of one
// head with their whole state in registers - G lanes share NC columns, each lane holding KC channels of each - and rows
// come in SC_ROWS at a time by bulk copies into a ring of stages.  Lane `sub` of a group holds channels
// (c / 4) * 4 G + 4 sub + c % 4, so that a warp reads row vectors as contiguous 16-byte pieces.
//
// A walk is a chain of dependent rows (about 80 ns each, whatever the width), so long passes are cut into chunks of rows that
// are walked side by side: one launch (SCAN_STATE) forms what every chunk adds to the state and the product of its decays, the
// next (SCAN_CHUNK) starts every chunk from the states before it - S <- P S + local, chunk after chunk, in the CTA's registers -
// and forms the results.  Everything stays products and sums in binary32 (no quotients of decays: a product that underflows is a
// state that has faded).  2000 rows, one walk -> the two launches, in us: retention, 4 heads of 128 x 128 154 -> 15.6 + 31.5, 16 heads
// 180 -> 47 + 112 (four chunks); wkv, 16 heads of 64 x 64 159 -> 18.6 + 34.0, 64 heads 205 -> 55 + 117.
constexpr int SC_THREADS = 128;
constexpr int SC_ROWS = 16;
constexpr int SC_MAX_STAGES = 4;
enum scan_mode { SCAN_WHOLE, SCAN_STATE, SCAN_CHUNK };
// value columns per group of lanes: two keep a single walk's chain short, four halve the shared-memory reads per state entry
// once chunks supply the warps
__host__ __device__ constexpr int scan_nc(int kc, int mode) { return mode != SCAN_WHOLE && kc == 4 ? 4 : 2; }

struct scan_shape {
  int kc, G, dimp, cols, blocks, stride;
};
scan_shape scan_shape_of(int dim, int vdim, bool wkv, int mode) {
  scan_shape s;
  s.kc = dim <= 128 ? 4 : dim <= 256 ? 8 : 16;
  s.G = std::max(2, pow2_at_least((dim + s.kc - 1) / s.kc));
  s.dimp = s.G * s.kc;
  s.cols = SC_THREADS / s.G * scan_nc(s.kc, mode);
  s.blocks = (vdim + s.cols - 1) / s.cols;
  s.stride = (wkv ? 3 : 2) * s.dimp + 4;
  return s;
}
size_t scan_stage_bytes(const scan_shape& z) { return (size_t)SC_ROWS * (z.stride + z.cols) * sizeof(float); }
// Stages of a chunk's ring and CTAs of an SM: three stages where four CTAs fit an SM with them (heads up to 64, retention up to 128),
// else two (four CTAs of wkv heads of 128 or retention heads of 192, two or three up to 256, one above).
constexpr size_t SC_SM_SMEM = 228 * 1024, SC_CTA_SMEM = 1024 + 64;  // an SM's shared memory; what a CTA takes of it beside its stages
int scan_chunk_stages(const scan_shape& z) { return 4 * (3 * scan_stage_bytes(z) + SC_CTA_SMEM) <= SC_SM_SMEM ? 3 : 2; }
int scan_ctas_per_sm(const scan_shape& z) { return (int)std::min<size_t>(4, SC_SM_SMEM / (scan_chunk_stages(z) * scan_stage_bytes(z) + SC_CTA_SMEM)); }
// rows per chunk (a multiple of SC_ROWS), 0 = one walk over all rows.  The CTAs of all chunks are resident at once, four per SM where
// they fit: that keeps its arithmetic busy, and a second wave would be a second walk.  Both chunk launches walk a chunk, so fewer than
// three chunks, or chunks shorter than the launch costs, gain nothing: prompts of four-layer models, one walk / chunks, in us - wkv heads
// of 128 at width 1024 with 192, 240, 320 rows 567 / 598, 595 / 621, 652 / 629; of 64 595 / 597, 626 / 627, 667 / 622.
constexpr int SC_MAX_CHUNKS = 32, SC_MIN_ROWS = 256;
int scan_most_chunks(const scan_shape& z, int heads, int m, int sms) {
  return std::min(std::min(SC_MAX_CHUNKS, m / 64), scan_ctas_per_sm(z) * sms / std::max(1, heads * z.blocks));
}
int scan_chunk_rows(const scan_shape& z, int heads, int m, int sms) {
  const int chunks = scan_most_chunks(z, heads, m, sms);
  return m < SC_MIN_ROWS || chunks < 3 ? 0 : (m + chunks * SC_ROWS - 1) / (chunks * SC_ROWS) * SC_ROWS;
}

constexpr int SP_ROWS = 4;  // rows per warp
template <typename T, bool WKV>
__global__ void __launch_bounds__(256) scan_prepare_kernel(const scan_rows<T> p, const scan_shape z, int m, int pos0) {
  pdl_launch_dependents();
  pdl_wait();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, half = p.rot_dims >> 1;
  const int head = blockIdx.y * 8 + warp, r0 = blockIdx.x * SP_ROWS, nr = min(SP_ROWS, m - r0);
  if (head >= p.heads) return;
  float* out = p.packed + ((size_t)head * m + r0) * z.stride;
  float bonus[SP_ROWS] = {};
  for (int d = lane; d < z.dimp; d += 32) {
    const bool in = d < p.dim, turn = !WKV && d < p.rot_dims, low = d < half;
    const int pd = low ? d + half : d - half;
    const float u = WKV && in ? p.u[head * p.dim + d] : 0.f;
    float q[SP_ROWS], k[SP_ROWS], qo[SP_ROWS], ko[SP_ROWS];
    float2 cs[SP_ROWS];
#pragma unroll
    for (int r = 0; r < SP_ROWS; ++r) {
      const T* qr = p.q + (size_t)(r0 + r) * p.ldq + head * p.dim;
      const T* kr = p.k + (size_t)(r0 + r) * p.ldk + head * p.dim;
      const bool live = in && r < nr;
      q[r] = live ? to_f(qr[d]) : 0.f;
      k[r] = live ? to_f(kr[d]) : 0.f;
      if (live && turn) {
        qo[r] = to_f(qr[pd]);
        ko[r] = to_f(kr[pd]);
        cs[r] = p.rope[(size_t)(pos0 + r0 + r) * half + (low ? d : d - half)];
      }
    }
#pragma unroll
    for (int r = 0; r < SP_ROWS; ++r) {
      if (r >= nr) continue;
      if (WKV) {
        bonus[r] = fmaf(q[r] * u, k[r], bonus[r]);
      } else {
        if (turn) {
          q[r] = low ? q[r] * cs[r].x - qo[r] * cs[r].y : q[r] * cs[r].x + qo[r] * cs[r].y;
          k[r] = low ? k[r] * cs[r].x - ko[r] * cs[r].y : k[r] * cs[r].x + ko[r] * cs[r].y;
        }
        k[r] *= p.kscale;
      }
      float* o = out + (size_t)r * z.stride;
      o[d] = q[r];
      o[z.dimp + d] = k[r];
      if (WKV && !in) o[2 * z.dimp + d] = 0.f;  // (the other channels' decays are written by their own kernel)
    }
  }
#pragma unroll
  for (int r = 0; r < SP_ROWS; ++r) {
    const float b = warp_sum(bonus[r]);
    if (lane < 4 && r < nr) out[(size_t)r * z.stride + z.stride - 4 + lane] = lane == 0 && WKV ? b : 0.f;
  }
  float* v = p.packed_v + (size_t)head * z.blocks * m * z.cols;
  for (int j = lane; j < z.blocks * z.cols; j += 32) {
    const int b = j / z.cols, c = j - b * z.cols;
    float x[SP_ROWS];
#pragma unroll
    for (int r = 0; r < SP_ROWS; ++r) x[r] = j < p.vdim && r < nr ? to_f(p.v[(size_t)(r0 + r) * p.ldv + head * p.vdim + j]) : 0.f;
#pragma unroll
    for (int r = 0; r < SP_ROWS; ++r)
      if (r < nr) v[((size_t)b * m + r0 + r) * z.cols + c] = x[r];
  }
}

// The same with four channels per lane, where head sizes and strides allow: one load and one store per lane and row part instead of
// four dependent rounds, and heads below eight leave no warp idle (`per_cta` heads of a CTA's eight warps, a power of two; the other
// factor takes further rows).  Latency-bound before: 14 us at 2000 rows of 4 x 128 x 128 or 16 x 64 x 64, 16 MB written.  Filulix 1024,
// 2000 tokens (four layers of each): 1.85 -> 1.82 ms.
constexpr int SP4_ROWS = 2;
template <typename T>
__device__ __forceinline__ void load4(const T* src, bool live, float (&x)[4]) {
#pragma unroll
  for (int c = 0; c < 4; ++c) x[c] = 0.f;
  if (!live) return;
  if constexpr (sizeof(T) == 2) {
    const uint2 v = *reinterpret_cast<const uint2*>(src);
    const T* t = reinterpret_cast<const T*>(&v);
#pragma unroll
    for (int c = 0; c < 4; ++c) x[c] = to_f(t[c]);
  } else {
    *reinterpret_cast<float4*>(x) = *reinterpret_cast<const float4*>(src);
  }
}
template <typename T, bool WKV>
__global__ void __launch_bounds__(256) scan_prepare4_kernel(const scan_rows<T> p, const scan_shape z, int m, int pos0, int per_cta) {
  pdl_launch_dependents();
  pdl_wait();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, half = p.rot_dims >> 1;
  const int head = blockIdx.y * per_cta + warp % per_cta, r0 = (blockIdx.x * (8 / per_cta) + warp / per_cta) * SP4_ROWS, nr = min(SP4_ROWS, m - r0);
  if (head >= p.heads || nr <= 0) return;
  float* out = p.packed + ((size_t)head * m + r0) * z.stride;
  float* v = p.packed_v + (size_t)head * z.blocks * m * z.cols;
  // the first values are requested beside the first channels
  const int n_val = z.blocks * z.cols;
  __align__(16) float x0[SP4_ROWS][4];
  float bonus[SP4_ROWS] = {};
#pragma unroll
  for (int r = 0; r < SP4_ROWS; ++r) load4(p.v + (size_t)(r0 + r) * p.ldv + head * p.vdim + 4 * lane, 4 * lane < p.vdim && r < nr, x0[r]);
  for (int d = 4 * lane; d < z.dimp; d += 128) {
    const bool in = d < p.dim, turn = !WKV && d < p.rot_dims, low = d < half;
    const int pd = low ? d + half : d - half;
    __align__(16) float q[SP4_ROWS][4], k[SP4_ROWS][4], qo[SP4_ROWS][4], ko[SP4_ROWS][4], u[4] = {};
    __align__(16) float2 cs[SP4_ROWS][4];
    if (WKV && in) *reinterpret_cast<float4*>(u) = *reinterpret_cast<const float4*>(p.u + head * p.dim + d);
#pragma unroll
    for (int r = 0; r < SP4_ROWS; ++r) {
      const T* qr = p.q + (size_t)(r0 + r) * p.ldq + head * p.dim;
      const T* kr = p.k + (size_t)(r0 + r) * p.ldk + head * p.dim;
      const bool live = in && r < nr;
      load4(qr + d, live, q[r]);
      load4(kr + d, live, k[r]);
      if (!WKV) {
        load4(qr + pd, live && turn, qo[r]);
        load4(kr + pd, live && turn, ko[r]);
        if (live && turn) {
          const float4* t = reinterpret_cast<const float4*>(p.rope + (size_t)(pos0 + r0 + r) * half + (low ? d : d - half));
          *reinterpret_cast<float4*>(&cs[r][0]) = t[0];
          *reinterpret_cast<float4*>(&cs[r][2]) = t[1];
        }
      }
    }
#pragma unroll
    for (int r = 0; r < SP4_ROWS; ++r) {
      if (r >= nr) continue;
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        if (WKV) {
          bonus[r] = fmaf(q[r][c] * u[c], k[r][c], bonus[r]);
        } else {
          if (turn) {
            q[r][c] = low ? q[r][c] * cs[r][c].x - qo[r][c] * cs[r][c].y : q[r][c] * cs[r][c].x + qo[r][c] * cs[r][c].y;
            k[r][c] = low ? k[r][c] * cs[r][c].x - ko[r][c] * cs[r][c].y : k[r][c] * cs[r][c].x + ko[r][c] * cs[r][c].y;
          }
          k[r][c] *= p.kscale;
        }
      }
      float* o = out + (size_t)r * z.stride;
      *reinterpret_cast<float4*>(o + d) = *reinterpret_cast<const float4*>(q[r]);
      *reinterpret_cast<float4*>(o + z.dimp + d) = *reinterpret_cast<const float4*>(k[r]);
      if (WKV && !in) *reinterpret_cast<float4*>(o + 2 * z.dimp + d) = make_float4(0.f, 0.f, 0.f, 0.f);
    }
  }
#pragma unroll
  for (int r = 0; r < SP4_ROWS; ++r) {
    const float b = WKV ? warp_sum(bonus[r]) : 0.f;
    if (lane < 4 && r < nr) out[(size_t)r * z.stride + z.stride - 4 + lane] = lane == 0 ? b : 0.f;
  }
  for (int j = 4 * lane; j < n_val; j += 128) {
    const int b = j / z.cols, c = j - b * z.cols;
#pragma unroll
    for (int r = 0; r < SP4_ROWS; ++r) {
      if (j >= 128) load4(p.v + (size_t)(r0 + r) * p.ldv + head * p.vdim + j, j < p.vdim && r < nr, x0[r]);
      if (r < nr) *reinterpret_cast<float4*>(v + ((size_t)b * m + r0 + r) * z.cols + c) = *reinterpret_cast<const float4*>(x0[r]);
    }
  }
}
template <typename T>
bool scan_prepare4_suits(const scan_rows<T>& p, const scan_shape& z, bool wkv) {
  const uintptr_t rows = (uintptr_t)p.q | (uintptr_t)p.k | (uintptr_t)p.v, vec = 4 * sizeof(T) - 1;
  const uintptr_t wide = (uintptr_t)p.packed | (uintptr_t)p.packed_v | (wkv ? (uintptr_t)p.u : (uintptr_t)p.rope);
  return (p.dim | p.vdim | p.ldq | p.ldk | p.ldv | z.cols | z.dimp | z.stride) % 4 == 0 && (wkv || p.rot_dims % 8 == 0) && (rows & vec) == 0 && (wide & 15) == 0;
}

struct scan_args {  // what the walks need of scan_rows
  const float *packed, *packed_v, *decay;
  float *state, *out;
  float* part;  // chunks: [chunk][head][block] {state entries, decays} of every thread; chunk 0: the state before the pass
  int dim, vdim, ldo;
  int* err;
};

// Two binary32 values in a register pair, one instruction for both (each rounded as by itself).  The walk over a chunk is bound by
// issue: three multiply-adds per state entry and row, in pairs 24 instead of 48 of a warp's 70 instructions per row.  States of 17
// chunks of 2000 rows (16 x 64 x 64 wkv / 4 x 128 x 128 retention) 18.4 -> 17.6 / 15.5 -> 14.6 us, results 33.9 -> 33.8 / 31.8 -> 31.4;
// a Filulix 1024 prompt of 2000 tokens 1.900 -> 1.878 ms.
using pair32 = unsigned long long;
__device__ __forceinline__ pair32 pair_of(float a, float b) {
  pair32 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ float2 floats_of(pair32 a) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(a));
  return r;
}
__device__ __forceinline__ pair32 fma_pair(pair32 a, pair32 b, pair32 c) {
  pair32 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ pair32 mul_pair(pair32 a, pair32 b) {
  pair32 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}

template <int KC, int G, bool WKV, int MODE>
__global__ void __launch_bounds__(SC_THREADS) scan_kernel(const scan_args p, const scan_shape z, int m, int pos0, int n_stages, int chunk_rows) {
  constexpr int NC = scan_nc(KC, MODE);
  constexpr int RB = 4;                         // rows reduced together
  constexpr int VALUES = RB * NC;
  constexpr int SPREAD = G < VALUES ? G : VALUES;  // lanes of a group that end up with results
  constexpr int KEEP = VALUES / SPREAD;            // results per such lane
  constexpr int DIMP = G * KC, STRIDE = (WKV ? 3 : 2) * DIMP + 4, COLS = SC_THREADS / G * NC;
  constexpr int PART = NC * KC + (WKV ? KC : 0);   // floats a thread leaves of a chunk
  extern __shared__ __align__(16) float sm[];
  __shared__ uint64_t bars[SC_MAX_STAGES];
  const int tid = threadIdx.x, sub = tid % G, grp = tid / G;
  const int head = blockIdx.x, v0 = blockIdx.y * COLS, D = p.dim, DV = p.vdim;
  const int chunk = MODE == SCAN_WHOLE ? 0 : blockIdx.z, first = chunk * chunk_rows, rows_here = MODE == SCAN_WHOLE ? m : min(chunk_rows, m - first);
  constexpr int STAGE = SC_ROWS * (STRIDE + COLS);
  const int n_tiles = (rows_here + SC_ROWS - 1) / SC_ROWS;
  if (tid == 0) {
    for (int i = 0; i < n_stages; ++i) mbar_init(smem_u32(&bars[i]), 1);
    fence_mbar_init();
  }
  __syncthreads();
  pdl_launch_dependents();
  pdl_wait();
  const float* rows = p.packed + ((size_t)head * m + first) * STRIDE;
  const float* vals = p.packed_v + (((size_t)head * z.blocks + blockIdx.y) * m + first) * COLS;
  auto fetch = [&](int tile) {
    const int s = tile % n_stages, nr = min(SC_ROWS, rows_here - tile * SC_ROWS);
    const uint32_t bar = smem_u32(&bars[s]), dst = smem_u32(sm + s * STAGE);
    const uint32_t b0 = (uint32_t)(nr * STRIDE) * 4, b1 = (uint32_t)(nr * COLS) * 4;
    mbar_arrive_expect_tx(bar, b0 + b1);
    bulk_g2s(dst, rows + (size_t)tile * SC_ROWS * STRIDE, b0, bar);
    bulk_g2s(dst + SC_ROWS * STRIDE * 4, vals + (size_t)tile * SC_ROWS * COLS, b1, bar);
  };
  if (tid == 0)
    for (int t = 0; t < n_stages && t < n_tiles; ++t) fetch(t);

  float S[NC][KC], P[WKV && MODE == SCAN_STATE ? KC : 1];
  float* st = p.state + (size_t)head * D * DV;
  const int c0 = v0 + grp * NC;  // first of this group's columns
  auto part_of = [&](int slot) { return p.part + (((size_t)slot * gridDim.x + head) * z.blocks + blockIdx.y) * (PART * SC_THREADS) + tid; };
  const bool from_state = MODE == SCAN_WHOLE || (MODE == SCAN_STATE && chunk == 0);
#pragma unroll
  for (int n = 0; n < NC; ++n)
#pragma unroll
    for (int c = 0; c < KC; ++c) {
      const int i = (c >> 2) * 4 * G + 4 * sub + (c & 3);
      S[n][c] = from_state && pos0 > 0 && c0 + n < DV && i < D ? st[(size_t)i * DV + c0 + n] : 0.f;
    }
  const float dec = WKV ? 0.f : p.decay[head];
  if (MODE == SCAN_STATE && chunk == 0) {  // (the last chunk overwrites the state while others still start from it)
    float* o = part_of(0);
#pragma unroll
    for (int j = 0; j < NC * KC; ++j) o[j * SC_THREADS] = S[j / KC][j % KC];
  }
  if (MODE == SCAN_CHUNK) {
    const float through = WKV ? 0.f : powf(dec, (float)chunk_rows);  // decay over a whole chunk
    const float* o = part_of(chunk == 0 ? 0 : 1);                    // (slot 1 has the whole state behind chunk 0)
#pragma unroll
    for (int j = 0; j < NC * KC; ++j) S[j / KC][j % KC] = o[j * SC_THREADS];
#pragma unroll 4
    for (int b = 2; b <= chunk; ++b) {
      o = part_of(b);
#pragma unroll
      for (int c = 0; c < KC; ++c) {
        const float w = WKV ? o[(NC * KC + c) * SC_THREADS] : through;
#pragma unroll
        for (int n = 0; n < NC; ++n) S[n][c] = fmaf(w, S[n][c], o[(n * KC + c) * SC_THREADS]);
      }
    }
  }

  // one row: updates the state, leaves this lane's share of its columns' results in o.  Neighbouring channels go in pairs.
  pair32 S2[NC][KC / 2], P2[WKV && MODE == SCAN_STATE ? KC / 2 : 1];
#pragma unroll
  for (int c = 0; c < KC / 2; ++c) {
#pragma unroll
    for (int n = 0; n < NC; ++n) S2[n][c] = pair_of(S[n][2 * c], S[n][2 * c + 1]);
    if (WKV && MODE == SCAN_STATE) P2[c] = pair_of(1.f, 1.f);
  }
  const pair32 dec2 = pair_of(dec, dec);
  auto advance = [&](const float* row, const float* val, float (&o)[NC]) {
    float v[NC];
    if (NC == 4) *reinterpret_cast<float4*>(v) = *reinterpret_cast<const float4*>(val);
    else *reinterpret_cast<float2*>(v) = *reinterpret_cast<const float2*>(val);
    pair32 o2[NC];
#pragma unroll
    for (int c4 = 0; c4 < KC / 4; ++c4) {
      const int at = c4 * 4 * G + 4 * sub;
      const ulonglong2 k4 = *reinterpret_cast<const ulonglong2*>(row + DIMP + at);
      ulonglong2 q4 = make_ulonglong2(0, 0), w4 = make_ulonglong2(dec2, dec2);
      if (MODE != SCAN_STATE) q4 = *reinterpret_cast<const ulonglong2*>(row + at);
      if (WKV) w4 = *reinterpret_cast<const ulonglong2*>(row + 2 * DIMP + at);
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int c = c4 * 2 + e;
        const pair32 q = e ? q4.y : q4.x, k = e ? k4.y : k4.x, w = e ? w4.y : w4.x;
        if (WKV && MODE == SCAN_STATE) P2[c] = mul_pair(P2[c], w);
#pragma unroll
        for (int n = 0; n < NC; ++n) {
          if (WKV && MODE != SCAN_STATE) o2[n] = c == 0 ? mul_pair(q, S2[n][c]) : fma_pair(q, S2[n][c], o2[n]);
          S2[n][c] = fma_pair(w, S2[n][c], mul_pair(k, pair_of(v[n], v[n])));
          if (!WKV && MODE != SCAN_STATE) o2[n] = c == 0 ? mul_pair(q, S2[n][c]) : fma_pair(q, S2[n][c], o2[n]);
        }
      }
    }
#pragma unroll
    for (int n = 0; n < NC && MODE != SCAN_STATE; ++n) {
      const float2 x = floats_of(o2[n]);
      o[n] = x.x + x.y;
    }
  };
  for (int tile = 0; tile < n_tiles; ++tile) {
    const int s = tile % n_stages, nr = min(SC_ROWS, rows_here - tile * SC_ROWS);
    mbar_wait(smem_u32(&bars[s]), (uint32_t)(tile / n_stages) & 1u, p.err, DEV_ERR_FULL_WAIT);  // (expired: the error word is set, results are not used)
    const float* rs = sm + s * STAGE;
    const float* vs = rs + SC_ROWS * STRIDE + grp * NC;
    float* out = p.out + (size_t)(first + tile * SC_ROWS) * p.ldo + head * DV;
    // results of RB rows, value number row * NC + column: lanes exchange halves, bit after bit of `sub` keeps values with that
    // bit of their number, until a lane has one left (or the group has no more lanes)
    auto finish = [&](const float (&o)[RB][NC], int r) {
      float x[VALUES];
#pragma unroll
      for (int i = 0; i < VALUES; ++i) x[i] = o[i / NC][i % NC];
#pragma unroll
      for (int y = 1; y < G; y <<= 1) {
        if (y < SPREAD) {
          const bool up = sub & y;
#pragma unroll
          for (int i = 0; i < VALUES / (2 * y); ++i) x[i] = (up ? x[2 * i + 1] : x[2 * i]) + __shfl_xor_sync(0xffffffffu, up ? x[2 * i] : x[2 * i + 1], y);
        } else {
          x[0] += __shfl_xor_sync(0xffffffffu, x[0], y);
        }
      }
      if (sub < SPREAD && c0 + sub % NC < DV) {
#pragma unroll
        for (int e = 0; e < KEEP; ++e) {
          const int at = e * SPREAD + sub, b = at / NC, n = at % NC;
          if (SPREAD < NC && c0 + n >= DV) continue;
          float y = x[e];
          if (WKV) y = fmaf(rs[(r + b) * STRIDE + STRIDE - 4], vs[(r + b) * COLS + n], y);
          out[(size_t)(r + b) * p.ldo + c0 + n] = y;
        }
      }
    };
    int r = 0;
    if (nr == SC_ROWS) {  // whole tiles: the exchange of one row block runs beside the next block's arithmetic
      float o[2][RB][NC];
#pragma unroll
      for (; r < SC_ROWS; r += RB) {
        const int cur = (r / RB) & 1;
#pragma unroll
        for (int b = 0; b < RB; ++b) advance(rs + (r + b) * STRIDE, vs + (r + b) * COLS, o[cur][b]);
        if (MODE != SCAN_STATE && r > 0) finish(o[cur ^ 1], r - RB);
      }
      if (MODE != SCAN_STATE) finish(o[(SC_ROWS / RB - 1) & 1], SC_ROWS - RB);
    }
#pragma unroll 1
    for (; r < nr; ++r) {
      float o[NC];
      advance(rs + r * STRIDE, vs + r * COLS, o);
#pragma unroll
      for (int n = 0; n < NC && MODE != SCAN_STATE; ++n) {
        float y = o[n];
#pragma unroll
        for (int b = 1; b < G; b <<= 1) y += __shfl_xor_sync(0xffffffffu, y, b);
        if (sub == n % G && c0 + n < DV) {
          if (WKV) y = fmaf(rs[r * STRIDE + STRIDE - 4], vs[r * COLS + n], y);
          out[(size_t)r * p.ldo + c0 + n] = y;
        }
      }
    }
    __syncthreads();  // the stage may be overwritten
    if (tid == 0 && tile + n_stages < n_tiles) fetch(tile + n_stages);
  }
#pragma unroll
  for (int c = 0; c < KC / 2; ++c) {
#pragma unroll
    for (int n = 0; n < NC; ++n) {
      const float2 x = floats_of(S2[n][c]);
      S[n][2 * c] = x.x;
      S[n][2 * c + 1] = x.y;
    }
    if (WKV && MODE == SCAN_STATE) {
      const float2 x = floats_of(P2[c]);
      P[2 * c] = x.x;
      P[2 * c + 1] = x.y;
    }
  }
  if (MODE == SCAN_STATE) {
    float* o = part_of(chunk + 1);
#pragma unroll
    for (int j = 0; j < NC * KC; ++j) o[j * SC_THREADS] = S[j / KC][j % KC];
    if (WKV)
#pragma unroll
      for (int c = 0; c < KC; ++c) o[(NC * KC + c) * SC_THREADS] = P[c];
    return;
  }
  if (MODE == SCAN_CHUNK && first + rows_here < m) return;
#pragma unroll
  for (int n = 0; n < NC; ++n)
#pragma unroll
    for (int c = 0; c < KC; ++c) {
      const int i = (c >> 2) * 4 * G + 4 * sub + (c & 3);
      if (c0 + n < DV && i < D) st[(size_t)i * DV + c0 + n] = S[n][c];
    }
}

template <int KC, int G, bool WKV, int MODE>
int launch_scan_shape(const scan_args& a, const scan_shape& z, int heads, int m, int pos0, int chunk_rows, cudaStream_t stream) {
  const size_t stage = scan_stage_bytes(z);
  const int n_stages = (int)std::min<size_t>(MODE == SCAN_WHOLE ? SC_MAX_STAGES : scan_chunk_stages(z), (200 * 1024) / stage);
  static bool attr_done[16] = {};
  int dev = 0;
  LCU_CUDA(cudaGetDevice(&dev));
  if (dev < 16 && !attr_done[dev]) {
    LCU_CUDA(cudaFuncSetAttribute((scan_kernel<KC, G, WKV, MODE>), cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024));
    attr_done[dev] = true;
  }
  const int chunks = MODE == SCAN_WHOLE ? 1 : (m + chunk_rows - 1) / chunk_rows - (MODE == SCAN_STATE);  // (nothing follows the last chunk)
  LCU_CUDA(launch_after(scan_kernel<KC, G, WKV, MODE>, dim3(heads, z.blocks, chunks), dim3(SC_THREADS), stage * n_stages, stream, a, z, m, pos0, n_stages,
                        chunk_rows));
  return LCU_OK;
}

template <bool WKV>
int launch_scan_kernel(const scan_args& a, const scan_shape& z, int heads, int m, int pos0, int chunk_rows, cudaStream_t stream) {
#define LCU_SCAN(KC, GG)                                                                                        \
  if (z.kc == KC && z.G == GG) {                                                                                \
    if (!chunk_rows) return launch_scan_shape<KC, GG, WKV, SCAN_WHOLE>(a, z, heads, m, pos0, 0, stream);        \
    const int rc = launch_scan_shape<KC, GG, WKV, SCAN_STATE>(a, z, heads, m, pos0, chunk_rows, stream);        \
    return rc ? rc : launch_scan_shape<KC, GG, WKV, SCAN_CHUNK>(a, z, heads, m, pos0, chunk_rows, stream);      \
  }
  LCU_SCAN(4, 2);
  LCU_SCAN(4, 4);
  LCU_SCAN(4, 8);
  LCU_SCAN(4, 16);
  LCU_SCAN(4, 32);
  LCU_SCAN(8, 32);
  LCU_SCAN(16, 32);
#undef LCU_SCAN
  LCU_REQUIRE(false, "scan: head size %d", a.dim);
}

// ------------------------------------------------------------------ one token, all branches
constexpr int ST_CLUSTER = 8;

// sum over the cluster of a value every thread of a CTA holds; `slot` is a shared float that stays valid until the next
// cluster barrier
__device__ __forceinline__ float cluster_total(float v, float* slot) {
  if (threadIdx.x == 0) *slot = v;
  cluster_sync();
  float t = 0.f;
#pragma unroll
  for (int r = 0; r < ST_CLUSTER; ++r) t += ld_dsmem_f32(mapa(smem_u32(slot), r));
  return t;
}

// The keys of a slice, a running maximum, sum and output per warp: the warps of a CTA meet once (as the LLaMA family's decode
// attention does).  Heads of up to 32 vectors of 16 bytes; a key is shared by `lanes` neighbouring lanes.  Rows that earlier steps
// wrote are requested ahead of the wait.  Leaves maximum, sum and the value row in res. .
constexpr int ST_KEYS = 4;  // keys of a group of lanes requested together
template <typename T>
__device__ __forceinline__ bool step_attend_suits(const attn_rows<T>& p) {
  return (max(p.dim, p.vdim) + 7) / 8 * 8 <= 32 * (16 / (int)sizeof(T));
}
template <typename T>
__device__ void step_attend(const attn_rows<T>& p, int head, int pos, int rank, float* part, float* res) {
  constexpr int VEC = 16 / sizeof(T), WARPS = MX_THREADS / 32;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, kvh = head / (p.heads / p.kv_heads);
  const int ldk = p.cache.ldk, ldv = p.cache.ldv, k_cols = (p.dim + 7) / 8 * 8, v_cols = (p.vdim + 7) / 8 * 8;
  const int lanes = pow2_at_least((max(k_cols, v_cols) + VEC - 1) / VEC), groups = MX_THREADS / lanes, grp = tid / lanes, d = tid % lanes * VEC;
  int lo, blocks;
  window_of(pos, p.window, p.pool, lo, blocks);
  const int total = blocks + pos + 1 - lo;
  const int t0 = (int)((long long)total * rank / ST_CLUSTER), n = (int)((long long)total * (rank + 1) / ST_CLUSTER) - t0;
  const T* kc = p.cache.k + kvh * p.cache.k_head;
  const T* vc = p.cache.v + kvh * p.cache.v_head;
  const T* kp = p.cache.kp + (size_t)kvh * p.cache.n_blocks * ldk;
  const T* vp = p.cache.vp + (size_t)kvh * p.cache.n_blocks * ldv;
  uint4 kr[ST_KEYS], vr[ST_KEYS];
  const uint4 zero = make_uint4(0, 0, 0, 0);
  auto fetch = [&](int base) {  // all but the token itself, which is the last key
#pragma unroll
    for (int i = 0; i < ST_KEYS; ++i) {
      const int t = t0 + base + i * groups + grp, at = t < blocks ? t : lo + t - blocks;
      const bool there = base + i * groups + grp < n && t + 1 < total;
      kr[i] = there && d < k_cols ? __ldcg(reinterpret_cast<const uint4*>((t < blocks ? kp : kc) + (size_t)at * ldk + d)) : zero;
      vr[i] = there && d < v_cols ? __ldcg(reinterpret_cast<const uint4*>((t < blocks ? vp : vc) + (size_t)at * ldv + d)) : zero;
    }
  };
  fetch(0);
  pdl_wait();
  float q[VEC], acc[VEC] = {}, mx = -CUDART_INF_F, sum = 0.f;
#pragma unroll
  for (int e = 0; e < VEC; ++e) q[e] = d + e < p.dim ? to_f(p.q[head * p.q_head + d + e]) : 0.f;
  T ck[VEC], cv[VEC];  // the token's own key and value
#pragma unroll
  for (int e = 0; e < VEC; ++e) {
    ck[e] = d + e < p.dim ? p.k[kvh * p.dim + d + e] : from_f<T>(0.f);
    cv[e] = d + e < p.vdim ? p.v[kvh * p.vdim + d + e] : from_f<T>(0.f);
  }
  const int rounds = (n + groups * ST_KEYS - 1) / (groups * ST_KEYS);  // (the same for every lane: the shuffles are warp-wide)
  for (int rd = 0; rd < rounds; ++rd) {
    const int base = rd * groups * ST_KEYS;
    if (rd > 0) fetch(base);
    float s[ST_KEYS], top = mx;
#pragma unroll
    for (int i = 0; i < ST_KEYS; ++i) {
      const bool own = t0 + base + i * groups + grp + 1 == total;
      s[i] = 0.f;
#pragma unroll
      for (int e = 0; e < VEC; ++e) s[i] = fmaf(q[e], to_f(own ? ck[e] : reinterpret_cast<const T*>(&kr[i])[e]), s[i]);
    }
    for (int o = lanes >> 1; o > 0; o >>= 1)
#pragma unroll
      for (int i = 0; i < ST_KEYS; ++i) s[i] += __shfl_xor_sync(0xffffffffu, s[i], o);
#pragma unroll
    for (int i = 0; i < ST_KEYS; ++i) {
      s[i] = base + i * groups + grp < n ? s[i] * p.scale : -CUDART_INF_F;
      top = fmaxf(top, s[i]);
    }
    for (int o = lanes; o < 32; o <<= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, o));
    const float ref = top > -CUDART_INF_F ? top : 0.f, keep = expf(mx - ref);
    mx = top;
    sum *= keep;
#pragma unroll
    for (int e = 0; e < VEC; ++e) acc[e] *= keep;
#pragma unroll
    for (int i = 0; i < ST_KEYS; ++i) {
      const bool own = t0 + base + i * groups + grp + 1 == total;
      const float w = expf(s[i] - ref);  // (0 for keys past the slice)
      sum += w;
#pragma unroll
      for (int e = 0; e < VEC; ++e) acc[e] = fmaf(w, to_f(own ? cv[e] : reinterpret_cast<const T*>(&vr[i])[e]), acc[e]);
    }
  }
  for (int o = lanes; o < 32; o <<= 1) {
    sum += __shfl_xor_sync(0xffffffffu, sum, o);
#pragma unroll
    for (int e = 0; e < VEC; ++e) acc[e] += __shfl_xor_sync(0xffffffffu, acc[e], o);
  }
  float* warp_max = part;  // [WARPS], [WARPS], [WARPS][lanes * VEC]
  float* warp_total = part + WARPS;
  float* rows = part + 2 * WARPS;
  if (lane == 0) {
    warp_max[warp] = mx;
    warp_total[warp] = sum;
  }
  if (lane < lanes)
#pragma unroll
    for (int e = 0; e < VEC; ++e) rows[warp * lanes * VEC + d + e] = acc[e];
  __syncthreads();
  float top = warp_max[0], f[WARPS];
#pragma unroll
  for (int x = 1; x < WARPS; ++x) top = fmaxf(top, warp_max[x]);
#pragma unroll  // (a warp without keys has maximum -inf and sums 0; one whose scores are no numbers has sums that are none, whatever its factor)
  for (int x = 0; x < WARPS; ++x) f[x] = warp_max[x] > -CUDART_INF_F ? expf(warp_max[x] - top) : 0.f;
  for (int j = tid; j < p.vdim; j += MX_THREADS) {
    float v = 0.f;
#pragma unroll
    for (int x = 0; x < WARPS; ++x) v = fmaf(f[x], rows[x * lanes * VEC + j], v);
    res[2 + j] = v;
  }
  if (tid == 0) {
    float t = 0.f;
#pragma unroll
    for (int x = 0; x < WARPS; ++x) t = fmaf(f[x], warp_total[x], t);
    res[0] = top;
    res[1] = t;
  }
}

template <typename T>
__device__ void step_attention(const step_branch<T>& b, int head, int rank, int pos, float* sm, float* red) {
  const attn_rows<T>& p = b.attn;
  const int tid = threadIdx.x, per = p.heads / p.kv_heads, kvh = head / per;
  const int ldk = p.cache.ldk, ldv = p.cache.ldv;
  T* cur_k = reinterpret_cast<T*>(sm);  // [ldk], [ldv]: the token's key and value as the cache will hold them
  T* cur_v = cur_k + ldk;
  float* q = sm + ldk + ldv;
  float* part = q + ldk;
  float* res = part + PART_FLOATS;
  float* sc = res + 2 + round_up_dev(p.vdim + 2, 4);
  const bool one_pass = step_attend_suits(p);
  const bool keeps = head % per == 0 && rank == 0;
  if (one_pass) step_attend(p, head, pos, rank, part, res);
  else pdl_wait();
  if (!one_pass || keeps) {
    for (int d = tid; d < ldk; d += MX_THREADS) cur_k[d] = d < p.dim ? p.k[kvh * p.dim + d] : from_f<T>(0.f);
    for (int d = tid; d < ldv; d += MX_THREADS) cur_v[d] = d < p.vdim ? p.v[kvh * p.vdim + d] : from_f<T>(0.f);
    __syncthreads();
  }
  if (!one_pass) attend_slice(p, p.q, head, pos, rank, ST_CLUSTER, cur_k, cur_v, q, sc, part, red, res);
  // the first query head of a group keeps the token: its cache rows, and the means of the block it completes (which no
  // position sees before the next step)
  if (keeps) {
    const size_t row = (size_t)kvh * p.cache.ctx_len + pos;
    for (int d = tid; d < p.dim; d += MX_THREADS) p.cache.k[row * ldk + d] = cur_k[d];
    for (int d = tid; d < p.vdim; d += MX_THREADS) p.cache.v[row * ldv + d] = cur_v[d];
    if (p.pool > 0 && (pos + 1) % p.pool == 0) {
      const size_t first = row - (p.pool - 1), dst = (size_t)kvh * p.cache.n_blocks + pos / p.pool;
      pool_block(p.cache.k + first * ldk, ldk, p.pool, cur_k, p.cache.kp + dst * ldk, p.dim);
      pool_block(p.cache.v + first * ldv, ldv, p.pool, cur_v, p.cache.vp + dst * ldv, p.vdim);
    }
  }
  cluster_sync();
  float mx = -CUDART_INF_F, sum = 0.f, f[ST_CLUSTER];
#pragma unroll
  for (int r = 0; r < ST_CLUSTER; ++r) mx = fmaxf(mx, ld_dsmem_f32(mapa(smem_u32(res), r)));
#pragma unroll
  for (int r = 0; r < ST_CLUSTER; ++r) {
    const float m = ld_dsmem_f32(mapa(smem_u32(res), r));
    f[r] = m > -CUDART_INF_F ? expf(m - mx) : 0.f;  // (an empty slice and one whose scores are no numbers: as the warps above)
    sum += f[r] * ld_dsmem_f32(mapa(smem_u32(res + 1), r));
  }
  float inv = p.out_scale / sum;
  if (p.sink) {
    const float top = fmaxf(mx, p.sink[head]), g = expf(mx - top);
    inv = p.out_scale * g / (sum * g + expf(p.sink[head] - top));
  }
  if (p.gate) inv *= sigmoid_f(to_f(p.gate[head]));
  const int d1 = p.vdim * (rank + 1) / ST_CLUSTER;
  for (int d = p.vdim * rank / ST_CLUSTER + tid; d < d1; d += MX_THREADS) {
    float v = 0.f;
#pragma unroll
    for (int r = 0; r < ST_CLUSTER; ++r) v += f[r] * ld_dsmem_f32(mapa(smem_u32(res + 2 + d), r));
    b.out[head * p.vdim + d] = from_f<T>(v * inv);
  }
  cluster_sync();
}

// What a step reads of weights, states and caches does not depend on the kernel before it (a step begins when the one before it has
// ended), so the first of it - all of it at the usual sizes - is in registers when the wait ends.  Filulix step, four layers, attention in
// one pass and this, at 40 / 430 positions, us: 1024 wide 132 -> 127 / 137 -> 128, 2048 wide 165 -> 163 / 171 -> 164.
constexpr int ST_STATE = 8, ST_RANK = 16;  // state entries and weights of the decay's second product a thread holds
template <typename T, bool WKV>
__device__ void step_recurrence(const step_branch<T>& b, int head, int rank, int pos, float* sm, float* red) {
  const scan_rows<T>& p = b.scan;
  const int tid = threadIdx.x, D = p.dim, DV = p.vdim;
  float* q = sm;
  float* k = q + D;
  float* w = k + D;        // wkv: decays
  float* part = w + D;     // [MX_THREADS]
  float* lows = part + MX_THREADS;
  __shared__ float s_slot;
  const int half = p.rot_dims >> 1;
  // ---- ahead of the wait
  const int v0 = DV * rank / ST_CLUSTER, nv = DV * (rank + 1) / ST_CLUSTER - v0;  // (at most 64 columns)
  const int ng = nv > 0 ? MX_THREADS / nv : 0, grp = nv > 0 ? tid / nv : 0, j = tid - grp * nv;
  const bool walks = nv > 0 && grp < ng;
  float* st = p.state + (size_t)head * D * DV + v0 + j;
  const float dec = WKV ? 0.f : p.decay[head];
  const float* u = WKV ? p.u + head * D : nullptr;
  float S0[ST_STATE], u0[WKV ? ST_STATE : 1];
#pragma unroll
  for (int s = 0; s < ST_STATE; ++s) {
    const int i = grp + s * ng;
    S0[s] = walks && i < D && pos > 0 ? __ldcg(st + (size_t)i * DV) : 0.f;
    if (WKV) u0[s] = walks && i < D ? u[i] : 0.f;
  }
  const int ch_all = p.heads * D, ng2 = max(1, MX_THREADS / D), grp2 = tid / D, c2 = tid - grp2 * D;  // decays: groups of threads share the rank
  float a0[WKV ? ST_RANK : 1], w0 = 0.f;
  float2 cs = make_float2(1.f, 0.f);
  if (WKV) {
#pragma unroll
    for (int s = 0; s < ST_RANK; ++s) {
      const int r = grp2 + s * ng2;
      a0[s] = D <= MX_THREADS && grp2 < ng2 && r < b.rank ? b.w2t[(size_t)r * ch_all + head * D + c2] : 0.f;
    }
    if (tid < D) w0 = b.w0[head * D + tid];
  } else if (tid < p.rot_dims) {
    cs = p.rope[(size_t)pos * half + (tid < half ? tid : tid - half)];
  }
  const int out_c = head * DV + v0 + tid;
  const float gain = tid < nv && b.norm ? b.norm[out_c] : 1.f;
  pdl_wait();
  const float v = walks ? to_f(p.v[head * DV + v0 + j]) : 0.f;
  const float gate = tid < nv ? to_f(b.g[out_c]) : 0.f;
  for (int d = tid; d < D; d += MX_THREADS) {
    const T *qr = p.q + head * D, *kr = p.k + head * D;
    float qv = to_f(qr[d]), kv = to_f(kr[d]);
    if (!WKV) {
      if (d < p.rot_dims) {
        const bool low = d < half;
        if (d != tid) cs = p.rope[(size_t)pos * half + (low ? d : d - half)];
        const int pd = low ? d + half : d - half;
        const float qo = to_f(qr[pd]), ko = to_f(kr[pd]);
        qv = low ? qv * cs.x - qo * cs.y : qv * cs.x + qo * cs.y;
        kv = low ? kv * cs.x - ko * cs.y : kv * cs.x + ko * cs.y;
      }
      kv *= p.kscale;
    }
    q[d] = qv;
    k[d] = kv;
  }
  if (WKV) {
    for (int r = tid; r < b.rank; r += MX_THREADS) lows[r] = tanhf(b.low[r]);
    __syncthreads();
    if (ng2 > 1) {
      float a = 0.f;
      if (grp2 < ng2) {
#pragma unroll
        for (int s = 0; s < ST_RANK; ++s)
          if (grp2 + s * ng2 < b.rank) a = fmaf(a0[s], lows[grp2 + s * ng2], a);
#pragma unroll 8
        for (int r = grp2 + ST_RANK * ng2; r < b.rank; r += ng2) a = fmaf(b.w2t[(size_t)r * ch_all + head * D + c2], lows[r], a);
      }
      part[tid] = a;
      __syncthreads();
      if (tid < D) {
        float z = w0;
        for (int g = 0; g < ng2; ++g) z += part[g * D + tid];
        w[tid] = expf(-expf(z));
      }
    } else {
      for (int c = tid; c < D; c += MX_THREADS) {
        float z = b.w0[head * D + c];
        for (int r = 0; r < b.rank; ++r) z = fmaf(b.w2t[(size_t)r * ch_all + head * D + c], lows[r], z);
        w[c] = expf(-expf(z));
      }
    }
  }
  __syncthreads();
  float o = 0.f;
  if (nv > 0) {
    float acc = 0.f;
    auto take = [&](int i, float S, float ui) {
      const float kv = k[i] * v;
      if (WKV) {
        acc = fmaf(q[i], fmaf(ui, kv, S), acc);
        S = fmaf(w[i], S, kv);
      } else {
        S = fmaf(dec, S, kv);
        acc = fmaf(q[i], S, acc);
      }
      st[(size_t)i * DV] = S;
    };
    if (walks) {
#pragma unroll
      for (int s = 0; s < ST_STATE; ++s)
        if (grp + s * ng < D) take(grp + s * ng, S0[s], WKV ? u0[WKV ? s : 0] : 0.f);
#pragma unroll 4
      for (int i = grp + ST_STATE * ng; i < D; i += ng) take(i, pos > 0 ? st[(size_t)i * DV] : 0.f, WKV ? u[i] : 0.f);
    }
    part[tid] = acc;
    __syncthreads();
    if (tid < nv)
#pragma unroll 8
      for (int g = 0; g < ng; ++g) o += part[g * nv + tid];
  }
  // (up to 32 columns - heads of up to 256 values - are the first warp's)
  const float ss = cluster_total(DV <= 32 * ST_CLUSTER ? warp_sum(o * o) : block_sum(o * o, red), &s_slot);
  const float inv = 1.0f / sqrtf(ss / (float)DV + b.eps);
  if (tid < nv) b.out[out_c] = from_f<T>(o * inv * gain * silu_f(gate) * b.out_scale);
  cluster_sync();
}

// lines of the caches, states and weights this CTA will read, requested while the kernel before it ends
template <typename T>
__device__ __forceinline__ void step_lines(const step_branch<T>& b, int head, int rank, int pos) {
  const int tid = threadIdx.x;
  if (b.kind == BRANCH_WINDOW_ATTN) {
    const attn_rows<T>& p = b.attn;
    int lo, blocks;
    window_of(pos, p.window, p.pool, lo, blocks);
    const int kvh = head / (p.heads / p.kv_heads), total = blocks + pos + 1 - lo;
    const int t0 = (int)((long long)total * rank / ST_CLUSTER), n = (int)((long long)total * (rank + 1) / ST_CLUSTER) - t0;
    constexpr int LINE = 128 / sizeof(T);
    const int lk = (p.cache.ldk + LINE - 1) / LINE, lv = (p.cache.ldv + LINE - 1) / LINE;
    for (int i = tid; i < n * (lk + lv); i += MX_THREADS) {
      const int t = t0 + i / (lk + lv), l = i % (lk + lv);
      const bool pooled = t < blocks, key = l < lk;
      const size_t row = pooled ? (size_t)kvh * p.cache.n_blocks + t : (size_t)kvh * p.cache.ctx_len + lo + t - blocks;
      const T* base = key ? (pooled ? p.cache.kp : p.cache.k) : (pooled ? p.cache.vp : p.cache.v);
      l2_line(base + row * (key ? p.cache.ldk : p.cache.ldv) + (key ? l : l - lk) * LINE);
    }
  } else {
    const scan_rows<T>& p = b.scan;
    const int v0 = p.vdim * rank / ST_CLUSTER, nv = p.vdim * (rank + 1) / ST_CLUSTER - v0;
    if (nv > 0)
      for (int i = tid; i < p.dim; i += MX_THREADS) l2_line(p.state + ((size_t)head * p.dim + i) * p.vdim + v0);
    if (b.kind == BRANCH_WKV) {
      const int per = (p.dim + 31) / 32;
      for (int i = tid; i < b.rank * per; i += MX_THREADS)
        l2_line(b.w2t + (size_t)(i / per) * p.heads * p.dim + head * p.dim + min(32 * (i % per), p.dim - 1));
      if (tid < per) {
        l2_line(b.w0 + head * p.dim + 32 * tid);
        l2_line(p.u + head * p.dim + 32 * tid);
        l2_line(b.norm + head * p.dim + 32 * tid);
      }
    }
  }
}

template <typename T>
__global__ void __launch_bounds__(MX_THREADS) mixer_step_kernel(const __grid_constant__ mixer_step<T> p) {
  extern __shared__ __align__(16) float sm[];
  __shared__ float red[MX_THREADS / 32];
  pdl_launch_dependents();
  const int cl = blockIdx.x / ST_CLUSTER, rank = blockIdx.x % ST_CLUSTER;
  const int bi = p.n_branches > 1 && cl >= p.b[1].first ? 1 : 0;
  const step_branch<T>& b = p.b[bi];
  const int head = cl - b.first;
  const int pos = *p.pos;  // (settled before this step began)
  step_lines(b, head, rank, pos);
  if (b.kind == BRANCH_WINDOW_ATTN) step_attention(b, head, rank, pos, sm, red);
  else if (b.kind == BRANCH_RETENTION) step_recurrence<T, false>(b, head, rank, pos, sm, red);
  else step_recurrence<T, true>(b, head, rank, pos, sm, red);
}

template <typename T>
size_t attention_smem(const attn_rows<T>& p, int keys, bool step) {
  return ((step ? p.cache.ldk + p.cache.ldv : 0) + query_cols(p) + PART_FLOATS + 2 + round_up(p.vdim + 2, 4) + keys + 8) * sizeof(float);
}
template <typename T>
int most_keys(const attn_rows<T>& p, int last_pos) {
  int lo, blocks;
  window_of(last_pos, p.window, p.pool, lo, blocks);
  return blocks + std::min(p.window, last_pos + 1);
}

}  // namespace

int& window_mma_mode() {
  static int mode = 1;
  return mode;
}

template <typename T>
int launch_window_append(const attn_rows<T>& p, int m, int pos0, cudaStream_t stream) {
  LCU_REQUIRE(pos0 >= 0 && pos0 + m <= p.cache.ctx_len, "window attention: rows %d..%d outside the cache of %d", pos0, pos0 + m, p.cache.ctx_len);
  LCU_CUDA(launch_after(window_append_kernel<T>, dim3(m), dim3(256), 0, stream, p, m, pos0));
  if (p.pool > 0) {
    const int b0 = pos0 / p.pool, b1 = (pos0 + m) / p.pool;
    if (b1 > b0) LCU_CUDA(launch_after(window_pool_kernel<T>, dim3(b1 - b0, p.kv_heads), dim3(128), 0, stream, p, b0));
  }
  return LCU_OK;
}

template <typename T>
int launch_window_attention(const attn_rows<T>& p, int m, int pos0, cudaStream_t stream) {
  if constexpr (sizeof(T) == 2)
    if (window_mma_mode() && window_mma_supported(p.dim, p.key2 ? p.dim2 : 0, p.vdim)) return launch_window_mma(p, m, pos0, stream);
  const int keys = most_keys(p, pos0 + m - 1);
  const size_t smem = attention_smem(p, keys, false);
  LCU_REQUIRE(smem <= 220 * 1024, "window attention: %d visible keys", keys);
  static bool attr_done[16] = {};
  int dev = 0;
  LCU_CUDA(cudaGetDevice(&dev));
  if (dev < 16 && !attr_done[dev]) {
    LCU_CUDA(cudaFuncSetAttribute(window_rows_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, 220 * 1024));
    attr_done[dev] = true;
  }
  LCU_CUDA(launch_after(window_rows_kernel<T>, dim3(p.heads, m), dim3(MX_THREADS), smem, stream, p, pos0, keys));
  return LCU_OK;
}

template <typename T>
int launch_scan(const scan_rows<T>& p, bool wkv, int m, int pos0, cudaStream_t stream) {
  scan_shape z = scan_shape_of(p.dim, p.vdim, wkv, SCAN_CHUNK);
  const int chunk_rows = scan_chunk_rows(z, p.heads, m, gemv_sm_count());
  if (!chunk_rows) z = scan_shape_of(p.dim, p.vdim, wkv, SCAN_WHOLE);
  const dim3 grid((m + SP_ROWS - 1) / SP_ROWS, (p.heads + 7) / 8);
  if (scan_prepare4_suits(p, z, wkv)) {
    const int per_cta = p.heads >= 8 ? 8 : pow2_at_least(p.heads), rows = 8 / per_cta * SP4_ROWS;
    const dim3 grid4((m + rows - 1) / rows, (p.heads + per_cta - 1) / per_cta);
    if (wkv) LCU_CUDA(launch_after(scan_prepare4_kernel<T, true>, grid4, dim3(256), 0, stream, p, z, m, pos0, per_cta));
    else LCU_CUDA(launch_after(scan_prepare4_kernel<T, false>, grid4, dim3(256), 0, stream, p, z, m, pos0, per_cta));
  } else if (wkv) LCU_CUDA(launch_after(scan_prepare_kernel<T, true>, grid, dim3(256), 0, stream, p, z, m, pos0));
  else LCU_CUDA(launch_after(scan_prepare_kernel<T, false>, grid, dim3(256), 0, stream, p, z, m, pos0));
  const scan_args a{p.packed, p.packed_v, p.decay, p.state, p.out, p.part, p.dim, p.vdim, p.ldo, p.err};
  return wkv ? launch_scan_kernel<true>(a, z, p.heads, m, pos0, chunk_rows, stream) : launch_scan_kernel<false>(a, z, p.heads, m, pos0, chunk_rows, stream);
}

void scan_scratch(int heads, int dim, int vdim, bool wkv, size_t rows, size_t* packed_floats, size_t* value_floats, size_t* part_floats) {
  const scan_shape whole = scan_shape_of(dim, vdim, wkv, SCAN_WHOLE), z = scan_shape_of(dim, vdim, wkv, SCAN_CHUNK);
  *packed_floats = heads * rows * z.stride;
  *value_floats = heads * rows * std::max(whole.blocks * whole.cols, z.blocks * z.cols);
  // (passes of fewer rows have no more chunks)
  const int sms = gemv_sm_count();
  const size_t chunks = scan_chunk_rows(z, heads, (int)rows, sms) ? scan_most_chunks(z, heads, (int)rows, sms) : 0;
  *part_floats = chunks * heads * z.blocks * SC_THREADS * z.kc * (scan_nc(z.kc, SCAN_CHUNK) + (wkv ? 1 : 0));
}
void scan_plan(int heads, int dim, int vdim, bool wkv, int m, int sms, int* chunk_rows, int* ctas, int* ctas_per_sm, int* smem_per_cta) {
  const scan_shape z = scan_shape_of(dim, vdim, wkv, SCAN_CHUNK);
  *chunk_rows = scan_chunk_rows(z, heads, m, sms);
  *ctas = *chunk_rows ? heads * z.blocks * ((m + *chunk_rows - 1) / *chunk_rows) : heads * scan_shape_of(dim, vdim, wkv, SCAN_WHOLE).blocks;
  *ctas_per_sm = scan_ctas_per_sm(z);
  *smem_per_cta = (int)(scan_chunk_stages(z) * scan_stage_bytes(z));
}
void scan_decay_layout(int dim, int vdim, int m, size_t* head_stride, size_t* row_stride, size_t* offset) {
  const scan_shape z = scan_shape_of(dim, vdim, true, SCAN_WHOLE);  // (the same for chunks)
  *head_stride = (size_t)m * z.stride;
  *row_stride = z.stride;
  *offset = 2 * (size_t)z.dimp;
}

template <typename T>
int launch_mixer_step(const mixer_step<T>& p, int ctx_len, cudaStream_t stream) {
  size_t smem = 0;
  for (int i = 0; i < p.n_branches; ++i) {
    const step_branch<T>& b = p.b[i];
    if (b.kind == BRANCH_WINDOW_ATTN) smem = std::max(smem, attention_smem(b.attn, most_keys(b.attn, ctx_len - 1) / ST_CLUSTER + 2, true));
    else smem = std::max(smem, (3 * (size_t)b.scan.dim + MX_THREADS + b.rank + 8) * sizeof(float));
  }
  LCU_REQUIRE(smem <= 220 * 1024, "mixer step: %zu bytes of shared memory", smem);
  static bool attr_done[16] = {};
  int dev = 0;
  LCU_CUDA(cudaGetDevice(&dev));
  if (dev < 16 && !attr_done[dev]) {
    LCU_CUDA(cudaFuncSetAttribute(mixer_step_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, 220 * 1024));
    attr_done[dev] = true;
  }
  return launch_clustered(mixer_step_kernel<T>, p.n_clusters * ST_CLUSTER, ST_CLUSTER, MX_THREADS, smem, stream, p);
}

#define LCU_BLOCK_MIXERS(T)                                                                    \
  template int launch_window_append<T>(const attn_rows<T>&, int, int, cudaStream_t);           \
  template int launch_window_attention<T>(const attn_rows<T>&, int, int, cudaStream_t);  \
  template int launch_scan<T>(const scan_rows<T>&, bool, int, int, cudaStream_t);              \
  template int launch_mixer_step<T>(const mixer_step<T>&, int, cudaStream_t);
LCU_BLOCK_MIXERS(__nv_bfloat16)
LCU_BLOCK_MIXERS(float)

}  // namespace lcu
