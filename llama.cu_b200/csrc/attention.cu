// Fused attention over the fp16 KV cache for sm_100a.
//
// Replaces the reference's matmul_qk -> softmax_rows -> matmul_qkv chain (llama_cu.cu:400-531,
// called at 1161-1171) and its per-layer score tensor with one kernel that keeps scores on chip:
//   score  s_t = half( (sum_i q_i k_ti) / sqrtf(head_dim) )                    llama_cu.cu:420-425
//   out    o_j = half( sum_t e^(s_t - max) v_tj / sum_t e^(s_t - max) )        llama_cu.cu:443-529
// (the reference rounds each quotient e^(s_t - max) / sum to half; here exponentials and sums stay in binary32).
//
// One thread-block cluster of CS CTAs serves one (query row, head): each CTA takes a contiguous
// slice of the cached positions.  K and V are stored head-major ([head][position][head_dim], keys
// already rotated), so a slice is one contiguous run of 2*head_dim-byte rows.  A short decode step is a chain of
// dependent steps, not bytes, so the chain is kept short: every warp runs over its rows with a running maximum, sum
// and output of its own - no barrier before the end - then a CTA's warps meet once in shared memory and the
// cluster's CTAs once in rank 0's (st.shared::cluster).  Rows older than the pass's first position do not depend on
// the kernel before this one: they, and the position itself, are read before griddepcontrol.wait.
// With two passes over the slice, three block and two cluster barriers a launch took 4.6 / 5.9 us from its wait to its last
// store at 20 / 300 positions (32 heads).  Decode step of 8 layers, before -> now, at 40 / 430 positions, in us: 4096 wide with u8
// weights 472 -> 443 / 484 -> 444, 4096 wide fp16 620 -> 610 / 627 -> 616, 1024 wide 194 -> 185 / 197 -> 186.
#include "attention.cuh"

namespace lcu {
namespace {

constexpr int ATT_THREADS = 256;
constexpr int ATT_WARPS = ATT_THREADS / 32;
constexpr int AS_CH = 64;  // rows a CTA takes at a time

__device__ __forceinline__ void st_dsmem_f32(uint32_t addr, float v) {
  asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(addr), "f"(v) : "memory");
}

// Tensor-parallel decode: the CTA that wrote a head's output (into this GPU's row and, as peer stores, into the other
// GPUs' rows) counts itself behind a device-scope fence; the last one of the launch fences at system scope - cumulative
// over everything counted before it - and writes this GPU's flag into the memory of every GPU that waits for the row.
__device__ __forceinline__ void publish_when_last(const attn_params& p, int tid, int n_ctas) {
  __syncthreads();  // the storing threads' writes are ordered before thread 0's fence
  if (tid == 0) {
    __threadfence();
    if (atomicAdd(p.done_count, 1) == n_ctas - 1) {
      atomicExch(p.done_count, 0);
      fence_acq_rel_sys();
      const int stamp = *p.seq * p.exchanges_per_step + p.exchange_id;
      for (int q = 0; q < p.n_peer_flag; ++q) st_relaxed_sys(p.peer_flag[q], stamp);
    }
  }
}

// What a warp has seen so far: maximum of its scores, sum of exponentials and sum of exponentials x V relative to it.  A row
// is shared by LPR lanes (8 halves = 16 bytes each); lanes of all row groups hold the same maximum, sums per group.
template <int HD>
struct warp_rows {
  static constexpr int LPR = HD / 8;             // lanes that share one cached row
  static constexpr int RPW = 32 / LPR;           // rows a warp handles per round
  static constexpr int RPR = ATT_WARPS * RPW;    // rows per round of the whole CTA
  static constexpr int ROUNDS = AS_CH / RPR;     // rounds of one chunk
  float m, sum, acc[8], e[ROUNDS];

  __device__ __forceinline__ void clear() {
    m = -CUDART_INF_F;
    sum = 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i) acc[i] = 0.f;
  }
  // scores of one chunk, rounded to half, and their exponentials (kept for `values`); valid(j): round j's row exists
  template <class Key, class Valid>
  __device__ __forceinline__ void scores(const float (&q)[8], float scale_div, Key key, Valid valid) {
    float top = -CUDART_INF_F;
#pragma unroll
    for (int j = 0; j < ROUNDS; ++j) {
      const uint4 kv = key(j);
      const __half2* h = reinterpret_cast<const __half2*>(&kv);
      float s = 0.f;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float2 f = __half22float2(h[i]);
        s += q[2 * i] * f.x;
        s += q[2 * i + 1] * f.y;
      }
#pragma unroll
      for (int o = LPR / 2; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
      e[j] = valid(j) ? __half2float(__float2half(s / scale_div)) : -CUDART_INF_F;
      top = fmaxf(top, e[j]);
    }
#pragma unroll
    for (int o = LPR; o < 32; o <<= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, o));
    top = fmaxf(top, m);
    // (a score that is no number leaves the maximum alone but not the sum: without any maximum scores are taken as they are)
    const float ref = top > -CUDART_INF_F ? top : 0.f, keep = expf(m - ref);
    m = top;
    sum = __fmul_rn(sum, keep);  // (rounded by itself, whatever the compiler makes of the additions behind it)
#pragma unroll
    for (int i = 0; i < 8; ++i) acc[i] = __fmul_rn(acc[i], keep);
#pragma unroll
    for (int j = 0; j < ROUNDS; ++j) {
      e[j] = expf(e[j] - ref);  // (0 for rows that do not exist)
      sum += e[j];
    }
  }
  template <class Value, class Valid>
  __device__ __forceinline__ void values(Value value, Valid valid) {
#pragma unroll
    for (int j = 0; j < ROUNDS; ++j) {
      if (!valid(j)) continue;
      const uint4 vv = value(j);
      const __half2* h = reinterpret_cast<const __half2*>(&vv);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float2 f = __half22float2(h[i]);
        acc[2 * i] += e[j] * f.x;
        acc[2 * i + 1] += e[j] * f.y;
      }
    }
  }
};

// Shared memory where the warps of a CTA and the CTAs of a cluster meet.
template <int HD>
struct meeting {
  float cta_max[8], cta_sum[8];  // of all ranks (rank 0's copy is used)
  float cta_out[8][HD];
  float warp_max[ATT_WARPS], warp_sum[ATT_WARPS];
  float warp_out[ATT_WARPS][HD];
};

// combines warps, then ranks, in fixed order; `threads` consumer threads on named barrier 1; every thread of the CTA has
// arrived at the cluster's start barrier.  Threads beyond the consumers only take part in cluster_sync().
template <int HD>
__device__ __forceinline__ void meet_and_store(const attn_params& p, meeting<HD>& mt, warp_rows<HD>& w, int head, int qrow, uint32_t rank, uint32_t cs) {
  constexpr int LPR = warp_rows<HD>::LPR;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
#pragma unroll
  for (int o = LPR; o < 32; o <<= 1) {
    w.sum += __shfl_xor_sync(0xffffffffu, w.sum, o);
#pragma unroll
    for (int i = 0; i < 8; ++i) w.acc[i] += __shfl_xor_sync(0xffffffffu, w.acc[i], o);
  }
  if (lane < LPR) {
    *reinterpret_cast<float4*>(&mt.warp_out[warp][lane * 8]) = make_float4(w.acc[0], w.acc[1], w.acc[2], w.acc[3]);
    *reinterpret_cast<float4*>(&mt.warp_out[warp][lane * 8 + 4]) = make_float4(w.acc[4], w.acc[5], w.acc[6], w.acc[7]);
  }
  if (lane == 0) {
    mt.warp_max[warp] = w.m;
    mt.warp_sum[warp] = w.sum;
  }
  bar_sync(1, ATT_THREADS);
  // (a part without rows has maximum -inf and sums 0; one whose scores are no numbers has sums that are none, whatever its weight)
  auto weight = [](float m, float top) { return m > -CUDART_INF_F ? expf(m - top) : 0.f; };
  asm volatile("barrier.cluster.wait.aligned;" ::: "memory");  // remote stores need the target CTA to have started
  if (tid < HD) {
    float top = mt.warp_max[0];
#pragma unroll
    for (int i = 1; i < ATT_WARPS; ++i) top = fmaxf(top, mt.warp_max[i]);
    float o = 0.f, s = 0.f;
#pragma unroll
    for (int i = 0; i < ATT_WARPS; ++i) {
      const float f = weight(mt.warp_max[i], top);
      o += f * mt.warp_out[i][tid];
      s += f * mt.warp_sum[i];
    }
    st_dsmem_f32(mapa(smem_u32(&mt.cta_out[rank][tid]), 0), o);
    if (tid == 0) {
      st_dsmem_f32(mapa(smem_u32(&mt.cta_max[rank]), 0), top);
      st_dsmem_f32(mapa(smem_u32(&mt.cta_sum[rank]), 0), s);
    }
  }
  cluster_sync();
  if (rank == 0 && tid < HD) {
    float top = -CUDART_INF_F;
    for (uint32_t r = 0; r < cs; ++r) top = fmaxf(top, mt.cta_max[r]);
    float o = 0.f, s = 0.f;
    for (uint32_t r = 0; r < cs; ++r) {
      const float f = weight(mt.cta_max[r], top);
      o += f * mt.cta_out[r][tid];
      s += f * mt.cta_sum[r];
    }
    const __half h = __float2half(o / s);
    const size_t at = (size_t)qrow * p.ldo + head * HD + tid;
    p.out[at] = h;
    for (int q = 0; q < p.n_peer_out; ++q) p.peer_out[q][at] = h;  // tensor-parallel: into every GPU's row (peer stores)
  }
  if (rank == 0 && p.done_count != nullptr) publish_when_last(p, tid, (int)(gridDim.y * gridDim.z));
}

__device__ __forceinline__ void load_query(float (&q)[8], const __half* at) {
  const uint4 qv = __ldcg(reinterpret_cast<const uint4*>(at));
  const __half2* h = reinterpret_cast<const __half2*>(&qv);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 f = __half22float2(h[i]);
    q[2 * i] = f.x;
    q[2 * i + 1] = f.y;
  }
}

template <int HD>
__global__ void __launch_bounds__(ATT_THREADS) attn_kernel(const attn_params p) {
  using rows = warp_rows<HD>;
  __shared__ __align__(16) meeting<HD> mt;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int grp = lane / rows::LPR, gl = lane % rows::LPR;
  const uint32_t rank = cluster_ctarank(), cs = cluster_nctarank();
  const int head = blockIdx.y, qrow = blockIdx.z;

  pdl_launch_dependents();
  asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");  // (split-phase: waited for before the first remote store)

  // the position was settled before this step's first kernel began
  const int start_pos = p.pos ? *p.pos : p.pos_value;
  const int T = start_pos + qrow + 1;  // causal: row r sees positions 0 .. start_pos + r
  const int chunk = (T + (int)cs - 1) / (int)cs;
  const int t0 = min(T, (int)rank * chunk), t1 = min(T, t0 + chunk);
  const int n = t1 - t0;
  const __half* kbase = p.k_cache + ((size_t)head * p.ctx_len + t0) * HD + gl * 8;
  const __half* vbase = p.v_cache + ((size_t)head * p.ctx_len + t0) * HD + gl * 8;
  const int row0 = warp * rows::RPW + grp;
  auto row_of = [&](int base, int j) { return base + j * rows::RPR + row0; };
  auto load = [&](const __half* b, int t) { return __ldcg(reinterpret_cast<const uint4*>(b + (size_t)t * HD)); };

  uint4 kreg[rows::ROUNDS], vreg[rows::ROUNDS];
  auto fetch = [&](int base, int from, int to) {  // this thread's rows of a chunk that lie in from .. to - 1
#pragma unroll
    for (int j = 0; j < rows::ROUNDS; ++j) {
      const int t = row_of(base, j);
      if (t >= from && t < to) {
        kreg[j] = load(kbase, t);
        vreg[j] = load(vbase, t);
      }
    }
  };
#pragma unroll
  for (int j = 0; j < rows::ROUNDS; ++j) kreg[j] = vreg[j] = make_uint4(0, 0, 0, 0);
  const int old = min(n, start_pos - t0);  // rows of the slice that earlier passes wrote
  fetch(0, 0, old);
  pdl_wait();
  float q[8];
  load_query(q, p.q + (size_t)qrow * p.ldq + head * HD + gl * 8);
  fetch(0, max(old, 0), n);
  const float scale_div = sqrtf((float)HD);

  rows w;
  w.clear();
  for (int base = 0; base < n; base += AS_CH) {
    if (base > 0) fetch(base, 0, n);
    auto valid = [&](int j) { return row_of(base, j) < n; };
    w.scores(q, scale_div, [&](int j) { return kreg[j]; }, valid);
    w.values([&](int j) { return vreg[j]; }, valid);
  }
  meet_and_store(p, mt, w, head, qrow, rank, cs);
}

// ---------------------------------------------------------------------------------------------------
// Streaming variant for long slices.  Same arithmetic, same thread-to-row assignment and summation order as
// attn_kernel (the two give identical bits), but the rows come through shared memory: a producer warp brings the
// slice in as contiguous bulk copies of up to 64 rows (the cache is head-major, so a slice is one contiguous run),
// K and V chunks in turn, through a ring of buffers with full/empty mbarriers.  With per-thread
// loads a CTA has at most 4 rows per thread in flight and a 260-row slice pays a memory latency every few rounds;
// here the ring keeps 64 KB per CTA requested at all times.
constexpr int AS_NB = 4;   // ring buffers
constexpr int AS_THREADS = ATT_THREADS + 32;

template <int HD>
__global__ void __launch_bounds__(AS_THREADS, 3) attn_stream_kernel(const attn_params p) {
  using rows = warp_rows<HD>;
  constexpr int CHUNK_BYTES = AS_CH * HD * 2;
  extern __shared__ __align__(128) uint8_t ring[];
  __shared__ __align__(16) meeting<HD> mt;
  __shared__ uint64_t bars[2 * AS_NB];  // full[AS_NB], empty[AS_NB]

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int grp = lane / rows::LPR, gl = lane % rows::LPR;
  const uint32_t rank = cluster_ctarank(), cs = cluster_nctarank();
  const int head = blockIdx.y, qrow = blockIdx.z;

  pdl_launch_dependents();
  asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
  const int start_pos = p.pos ? *p.pos : p.pos_value;  // (settled before this step's first kernel began)
  const int T = start_pos + qrow + 1;
  const int chunk = (T + (int)cs - 1) / (int)cs;
  const int t0 = min(T, (int)rank * chunk), t1 = min(T, t0 + chunk);
  const int n = t1 - t0;
  const int nch = (n + AS_CH - 1) / AS_CH;
  if (tid == 0) {
    for (int i = 0; i < AS_NB; ++i) {
      mbar_init(smem_u32(&bars[i]), 1);
      mbar_init(smem_u32(&bars[AS_NB + i]), ATT_WARPS);
    }
    fence_mbar_init();
  }
  __syncthreads();

  if (warp == ATT_WARPS) {
    // ---- producer: copy i is the K (i even) or V (i odd) part of chunk i / 2; chunks of rows that earlier passes wrote are
    // requested before the kernel ahead of this one has ended
    const __half* kb = p.k_cache + ((size_t)head * p.ctx_len + t0) * HD;
    const __half* vb = p.v_cache + ((size_t)head * p.ctx_len + t0) * HD;
    if (lane == 0) {
      bool waited = false;
      for (int i = 0; i < 2 * nch; ++i) {
        const int b = i % AS_NB, use = i / AS_NB, c = i >> 1;
        const int rows_here = min(AS_CH, n - c * AS_CH);
        if (!waited && t0 + c * AS_CH + rows_here > start_pos) {
          pdl_wait();
          waited = true;
        }
        if (use > 0 && !mbar_wait(smem_u32(&bars[AS_NB + b]), (use - 1) & 1, p.err, DEV_ERR_EMPTY_WAIT)) break;
        const uint32_t bytes = (uint32_t)rows_here * (HD * 2), full = smem_u32(&bars[b]);
        mbar_arrive_expect_tx(full, bytes);
        bulk_g2s(smem_u32(ring + b * CHUNK_BYTES), ((i & 1) ? vb : kb) + (size_t)c * AS_CH * HD, bytes, full);
      }
    }
    __syncwarp();
    asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
    cluster_sync();
    if (rank == 0 && p.done_count != nullptr) __syncthreads();  // (publish_when_last)
    return;
  }

  pdl_wait();
  float q[8];
  load_query(q, p.q + (size_t)qrow * p.ldq + head * HD + gl * 8);
  const float scale_div = sqrtf((float)HD);
  bool ok = true;
  rows w;
  w.clear();
  const int row0 = warp * rows::RPW + grp;
  for (int c = 0; c < nch; ++c) {
    auto valid = [&](int j) { return ok && c * AS_CH + j * rows::RPR + row0 < n; };
    auto at = [&](const uint8_t* buf, int j) { return *reinterpret_cast<const uint4*>(buf + (size_t)(j * rows::RPR + row0) * (HD * 2) + gl * 16); };
    const int kb = (2 * c) % AS_NB, vb = (2 * c + 1) % AS_NB;
    const uint32_t parity = (uint32_t)((2 * c) / AS_NB) & 1u;
    ok = ok && mbar_wait(smem_u32(&bars[kb]), parity, p.err, DEV_ERR_FULL_WAIT);
    w.scores(q, scale_div, [&](int j) { return valid(j) ? at(ring + kb * CHUNK_BYTES, j) : make_uint4(0, 0, 0, 0); }, valid);
    __syncwarp();
    if (lane == 0) mbar_arrive(smem_u32(&bars[AS_NB + kb]));
    ok = ok && mbar_wait(smem_u32(&bars[vb]), parity, p.err, DEV_ERR_FULL_WAIT);
    w.values([&](int j) { return at(ring + vb * CHUNK_BYTES, j); }, valid);
    __syncwarp();
    if (lane == 0) mbar_arrive(smem_u32(&bars[AS_NB + vb]));
  }
  meet_and_store(p, mt, w, head, qrow, rank, cs);
}

template <int HD>
int launch_hd(const attn_params& p, int m, int cs, cudaStream_t stream, int pdl) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(cs, p.n_heads, m);
  cfg.blockDim = dim3(ATT_THREADS);
  cfg.dynamicSmemBytes = 0;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = cs;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl ? 2 : 1;
  LCU_CUDA(cudaLaunchKernelEx(&cfg, attn_kernel<HD>, p));
  return LCU_OK;
}

template <int HD>
int launch_stream_hd(const attn_params& p, int m, int cs, cudaStream_t stream, int pdl) {
  const size_t smem = (size_t)AS_NB * AS_CH * HD * 2;
  LCU_REQUIRE(p.err != nullptr, "attention: the streaming kernel needs a device error word");
  static bool attr_done[16] = {};
  int dev = 0;
  LCU_CUDA(cudaGetDevice(&dev));
  if (dev < 16 && !attr_done[dev]) {
    LCU_CUDA(cudaFuncSetAttribute(attn_stream_kernel<HD>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024));
    attr_done[dev] = true;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(cs, p.n_heads, m);
  cfg.blockDim = dim3(AS_THREADS);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = cs;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl ? 2 : 1;
  LCU_CUDA(cudaLaunchKernelEx(&cfg, attn_stream_kernel<HD>, p));
  return LCU_OK;
}

int g_attn_stream = -1;  // -1 = streaming kernel when a CTA's slice can exceed 64 rows, 0 = never, 1 = always

}  // namespace

void attention_set_stream_mode(int mode) { g_attn_stream = mode; }

// loads the decode attention kernels on the current device ahead of their first launch (see gemv_single_row_preload)
int attention_preload() {
  cudaFuncAttributes fa;
  LCU_CUDA(cudaFuncGetAttributes(&fa, attn_kernel<128>));
  LCU_CUDA(cudaFuncGetAttributes(&fa, attn_kernel<64>));
  LCU_CUDA(cudaFuncGetAttributes(&fa, attn_stream_kernel<128>));
  LCU_CUDA(cudaFuncGetAttributes(&fa, attn_stream_kernel<64>));
  return LCU_OK;
}

int launch_attention(const attn_params& p, int m, int cluster, int max_T, cudaStream_t stream, int pdl) {
  LCU_REQUIRE(m >= 1 && p.n_heads >= 1, "attention: empty problem");
  LCU_REQUIRE(cluster >= 1 && cluster <= 8 && (cluster & (cluster - 1)) == 0, "attention: cluster size %d not in {1,2,4,8}", cluster);
  LCU_REQUIRE(max_T >= 1 && max_T <= p.ctx_len, "attention: %d positions exceed the context length %d", max_T, p.ctx_len);
  const bool streaming = p.err != nullptr && (g_attn_stream == 1 || (g_attn_stream < 0 && (max_T + cluster - 1) / cluster > AS_CH));
  if (streaming) {
    if (p.head_dim == 128) return launch_stream_hd<128>(p, m, cluster, stream, pdl);
    if (p.head_dim == 64) return launch_stream_hd<64>(p, m, cluster, stream, pdl);
  }
  if (p.head_dim == 128) return launch_hd<128>(p, m, cluster, stream, pdl);
  if (p.head_dim == 64) return launch_hd<64>(p, m, cluster, stream, pdl);
  LCU_REQUIRE(false, "attention: head_dim %d not supported (64 or 128)", p.head_dim);
}

}  // namespace lcu
