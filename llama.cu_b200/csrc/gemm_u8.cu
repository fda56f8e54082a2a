// Product of several rows with a matrix of 8-bit weights on tcgen05, the weights expanded on their way into tensor memory:
// out(m,N) = x(m,K) . w(N,K)^T + beta * out, w = half((q - 127.5) * scale) as everywhere (llama_cu.cu:287-289).
//
// The weight tile is the A operand (128 weight rows = tensor-memory lanes), so a converting thread owns one weight row: it reads
// 64 bytes of it from shared memory, expands them with the row's scales and stores 32 packed columns with tcgen05.st - the
// expanded weights never pass through shared or global memory.  The activation rows (t <= 224 of them, a multiple of 16) are the
// B operand.  Warp roles: warps 0-15 convert (four per k-block of 64, two k-blocks per stage) and store the results, warp 16 issues
// the TMA loads, warp 17 the MMAs.
//
// What bounds it: per k-block 128 weight rows and 200 activation rows cost 400 cycles of MMA and 530 of shared-memory traffic, and
// expanding about 250 on every scheduler.  200 rows, 4096 x 11008, blocks of 64: 867 us through the weight-streaming GEMV in passes
// of 8 rows, each of which reads the whole matrix, 30 us here (600 TFLOP/s); 2 rows: 20 us.
// Few tiles leave SMs idle, so K is split over a cluster of up to 8 CTAs, whose partial sums meet in distributed shared memory
// and are added in rank order.  Every mbarrier wait is bounded.
#include <algorithm>

#include "gemm_tc.cuh"
#include "tc_common.cuh"

namespace lcu {
namespace {

constexpr int U8_ROWS = 128;                    // weight rows per tile
constexpr int U8_KB = 64, U8_STAGE_K = 128;     // K per k-block and per stage
constexpr int U8_CONV_WARPS = 16, U8_THREADS = (U8_CONV_WARPS + 2) * 32;
constexpr int U8_MAX_T = 224;                   // activation rows per tile: three stages fit beside each other
constexpr uint32_t U8_Q_BYTES = U8_ROWS * U8_STAGE_K;
constexpr int U8_GROUPS = U8_CONV_WARPS / 4;    // converting warpgroups, each with every fourth k-block and two buffers
constexpr int U8_BUFS = 2 * U8_GROUPS, U8_BUF_COLS = U8_KB / 2;  // expanded k-blocks in tensor memory, two halves per column
constexpr int U8_MAX_STAGES = 8;
constexpr uint32_t U8_TMEM = 512, U8_A_COL = 256;  // accumulator columns, then the expanded weights
constexpr int U8_AHEAD = 4;                     // k-blocks of a warpgroup whose scales are requested ahead

// 16 columns of K, A in tensor memory
__device__ __forceinline__ void tc_mma_f16_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(d_tmem),
      "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void tc_st_32x32(uint32_t taddr, const uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
      "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};" ::"r"(taddr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]),
      "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]),
      "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
      : "memory");
}
__device__ __forceinline__ void tc_ld_32x16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
        "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}
// bytes (q0, q1) picked by `selector` -> half((q - 127.5) * scale): 1024 + q, minus 1024, minus 127.5 (all exact), times scale
__device__ __forceinline__ uint32_t expand_pair(uint32_t word, uint32_t selector, __half2 scale) {
  const uint32_t v = __byte_perm(word, 0x64646464u, selector);
  __half2 h = *reinterpret_cast<const __half2*>(&v);
  h = __hsub2(h, __half2half2(__ushort_as_half(0x6400)));
  h = __hsub2(h, __half2half2(__ushort_as_half(0x57f8)));
  h = __hmul2(h, scale);
  return *reinterpret_cast<uint32_t*>(&h);
}

template <int BS>  // weights per scale: 32, 64, 128
__global__ void __launch_bounds__(U8_THREADS, 1) gemm_u8_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_q,
                                                                const __half* scales, __half* out, int m, int N, int K, float beta, int t, int nstages,
                                                                int splits, int* err) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* smem = smem_raw + (base - smem_u32(smem_raw));
  const uint32_t X_BLOCK = (uint32_t)t * (U8_KB * 2), STAGE = U8_Q_BYTES + 2 * X_BLOCK;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + (size_t)nstages * STAGE);
  uint64_t *full = bars, *empty = bars + 2 * U8_MAX_STAGES, *conv = empty + U8_MAX_STAGES, *freed = conv + U8_BUFS, *done = freed + U8_BUFS;
  // full: every slot has two barriers, used in turn.  A converting warpgroup looks at every other stage; with one barrier per slot and
  // an odd number of slots it looked at that barrier every other time it was filled, and where a load was overtaken by the next
  // stage's, the phase before the awaited one passed for it.
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(done + 1);
  volatile float* failed = reinterpret_cast<volatile float*>(tmem_slot + 1);  // 1: a wait of this CTA ran out

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = splits > 1 ? (int)cluster_ctarank() : 0;
  const int n0 = (blockIdx.x / splits) * U8_ROWS, m0 = blockIdx.y * t;
  const int groups = K / U8_STAGE_K, st0 = rank * groups / splits, n_st = (rank + 1) * groups / splits - st0;
  const uint32_t idesc = (1u << 4) | ((uint32_t)(t >> 3) << 17) | ((uint32_t)(U8_ROWS >> 4) << 24);

  if (threadIdx.x == 0) {
    for (int i = 0; i < 2 * nstages; ++i) mbar_init(smem_u32(&full[i]), 1);
    for (int i = 0; i < nstages; ++i) mbar_init(smem_u32(&empty[i]), 1);
    for (int i = 0; i < U8_BUFS; ++i) {
      mbar_init(smem_u32(&conv[i]), 4);
      mbar_init(smem_u32(&freed[i]), 1);
    }
    mbar_init(smem_u32(done), 1);
    *failed = 0.f;
    fence_mbar_init();
  }
  if (warp == U8_CONV_WARPS + 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(U8_TMEM) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  pdl_launch_dependents();
  pdl_wait();
  constexpr bool HEED = false;  // nobody clears the error word between stand-alone calls: what stands there may be an earlier launch's

  // rows of the tile this thread converts and stores; tiles may hang over N
  const int quad = warp & 3, group = warp >> 2, row = quad * 32 + lane, n = n0 + row;
  const uint32_t lane_base = tmem + ((uint32_t)(quad * 32) << 16);
  bool go = false;
  if (warp < U8_CONV_WARPS) {
    // k-blocks group, group + 4, ..: the half of a stage with the group's lowest bit, every other stage.  A row past N multiplies
    // zero-filled bytes by row N - 1's scales and is never stored.
    const int per_row = K / BS, half = group & 1, n_blk = 2 * n_st;
    const __half* sc = scales + (size_t)min(n, N - 1) * per_row;
    auto scales_of = [&](int blk) -> uint32_t {
      if (blk >= n_blk) return 0;
      const int at = (2 * st0 + blk) * U8_KB / BS;
      if (BS == 32) return __ldg(reinterpret_cast<const unsigned int*>(sc + at));  // two blocks
      return __ldg(reinterpret_cast<const unsigned short*>(sc) + at);
    };
    uint32_t ahead[U8_AHEAD];
#pragma unroll
    for (int i = 0; i < U8_AHEAD; ++i) ahead[i] = scales_of(group + i * U8_GROUPS);
    bool ok = true;
    int s = group >> 1, f = s;
    uint32_t phase = 0;
    for (int b0 = group; b0 < n_blk && ok; b0 += U8_AHEAD * U8_GROUPS) {
#pragma unroll
      for (int u = 0; u < U8_AHEAD; ++u) {
        const int blk = b0 + u * U8_GROUPS, buf = blk % U8_BUFS;
        if (blk >= n_blk) break;
        const uint32_t sw = ahead[u];
        ahead[u] = scales_of(blk + U8_AHEAD * U8_GROUPS);
        ok = mbar_wait(smem_u32(&full[f]), phase, err, DEV_ERR_FULL_WAIT, HEED);
        if (ok && blk >= U8_BUFS) ok = mbar_wait(smem_u32(&freed[buf]), (blk / U8_BUFS - 1) & 1, err, DEV_ERR_EMPTY_WAIT, HEED);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        tc_fence_after();
        const uint8_t* q = smem + (size_t)s * STAGE + row * U8_STAGE_K;
        uint32_t r[32];
#pragma unroll
        for (int c = 0; c < 4; ++c) {  // (rows are 128-byte swizzled: 16-byte piece j of a row lies at j ^ (row & 7))
          const uint4 v = *reinterpret_cast<const uint4*>(q + (((4 * half + c) ^ (row & 7)) << 4));
          const uint32_t w[4] = {v.x, v.y, v.z, v.w};
          const __half2 f = __half2half2(__ushort_as_half((unsigned short)(BS == 32 && c >= 2 ? sw >> 16 : sw & 0xffffu)));
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            r[8 * c + 2 * e] = expand_pair(w[e], 0x4140, f);
            r[8 * c + 2 * e + 1] = expand_pair(w[e], 0x4342, f);
          }
        }
        tc_st_32x32(lane_base + U8_A_COL + (uint32_t)(buf * U8_BUF_COLS), r);
        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&conv[buf]));
        s += U8_GROUPS / 2;
        if (s >= nstages) s -= nstages;
        f += U8_GROUPS / 2;
        if (f >= 2 * nstages) {
          f -= 2 * nstages;
          phase ^= 1;
        }
      }
    }
    ok = mbar_wait(smem_u32(done), 0, err, DEV_ERR_TMEM_WAIT, HEED) && ok;
    tc_fence_after();
    go = __all_sync(0xffffffffu, ok && *failed == 0.f);
    if (!go && lane == 0) *failed = 1.f;
  } else if (warp == U8_CONV_WARPS) {
    if (tc_elect()) {  // ---- TMA producer
      tc_ring r, f;
      for (int i = 0; i < n_st; ++i, r.step(nstages), f.step(2 * nstages)) {
        if (!mbar_wait(smem_u32(&empty[r.slot]), r.phase ^ 1u, err, DEV_ERR_EMPTY_WAIT, HEED)) break;
        const uint32_t bar = smem_u32(&full[f.slot]), dst = base + (uint32_t)r.slot * STAGE;
        mbar_arrive_expect_tx(bar, STAGE);
        tma_load_2d(dst, &map_q, (st0 + i) * (U8_STAGE_K / 2), n0, bar);
        tma_load_3d(dst + U8_Q_BYTES, &map_x, 0, m0, (st0 + i) * 2, bar);
      }
    }
    __syncwarp();
  } else {  // ---- MMA issuer
    bool ok = true;
    tc_ring r, f, e;
    for (int i = 0; i < n_st && ok; ++i, r.step(nstages), f.step(2 * nstages)) {
      ok = mbar_wait_warp(smem_u32(&full[f.slot]), f.phase, err, DEV_ERR_FULL_WAIT, HEED);
      if (!ok) break;
      const uint64_t x = smem_desc_sw128(base + (uint32_t)r.slot * STAGE + U8_Q_BYTES);
#pragma unroll
      for (int g = 0; g < 2; ++g, e.step(U8_BUFS)) {
        ok = ok && mbar_wait_warp(smem_u32(&conv[e.slot]), e.phase, err, DEV_ERR_FULL_WAIT, HEED);
        if (!ok) break;
        tc_fence_after();
        if (tc_elect()) {
          const uint64_t xb = x + (uint64_t)g * (X_BLOCK >> 4);
          const uint32_t a = tmem + U8_A_COL + (uint32_t)(e.slot * U8_BUF_COLS);
#pragma unroll
          for (int k = 0; k < U8_KB / 16; ++k) tc_mma_f16_ts(tmem, a + 8 * k, xb + 2 * k, idesc, (i | g | k) != 0);
          tc_commit(smem_u32(&freed[e.slot]));
          if (g == 1) tc_commit(smem_u32(&empty[r.slot]));
        }
        __syncwarp();
      }
    }
    if (tc_elect()) {  // (also after a failed wait: lets the other warps leave, without results)
      if (!ok) *failed = 1.f;
      __threadfence_block();
      tc_commit(smem_u32(done));
    }
    __syncwarp();
  }

  // out[token][n]: a warp writes 32 consecutive outputs of one token
  auto store = [&](int col, float v) {
    if (m0 + col >= m || n >= N) return;
    __half* o = out + (size_t)(m0 + col) * N + n;
    if (beta != 0.f) v = v + beta * __half2float(*o);
    *o = __float2half(v);
  };
  if (splits == 1) {
    if (go)
      for (int c = 16 * group; c < t; c += 16 * U8_GROUPS) {
        uint32_t r[16];
        tc_ld_32x16(lane_base + (uint32_t)c, r);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
        for (int j = 0; j < 16; ++j) store(c + j, __uint_as_float(r[j]));
      }
  } else {
    // partial sums [column][128 rows] where the stages were; CTA `rank` adds every splits-th piece of 16 columns
    float* part = reinterpret_cast<float*>(smem);
    if (go)
      for (int c = 16 * group; c < t; c += 16 * U8_GROUPS) {
        uint32_t r[16];
        tc_ld_32x16(lane_base + (uint32_t)c, r);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
        for (int j = 0; j < 16; ++j) part[(c + j) * U8_ROWS + row] = __uint_as_float(r[j]);
      }
    __syncwarp();
    cluster_sync();
    go = __all_sync(0xffffffffu, go && (lane >= splits || ld_dsmem_f32(mapa(smem_u32((const void*)failed), (uint32_t)lane)) == 0.f));
    if (go)
      for (int c = 16 * (rank + splits * group); c < t; c += 16 * U8_GROUPS * splits) {
        float sum[16];
#pragma unroll
        for (int j = 0; j < 16; ++j) sum[j] = 0.f;
        for (int q = 0; q < splits; ++q) {
          const uint32_t src = mapa(smem_u32(part + c * U8_ROWS + row), (uint32_t)q);
#pragma unroll
          for (int j = 0; j < 16; ++j) sum[j] += ld_dsmem_f32(src + (uint32_t)(j * U8_ROWS * 4));
        }
#pragma unroll
        for (int j = 0; j < 16; ++j) store(c + j, sum[j]);
      }
    __syncwarp();
    cluster_sync();  // nobody leaves while its partial sums are being read
  }
  tc_fence_before();
  __syncthreads();
  if (warp == U8_CONV_WARPS + 1) {
    __syncwarp();
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(U8_TMEM) : "memory");
  }
}

template <int BS>
int launch_u8(const CUtensorMap& map_x, const CUtensorMap& map_q, const __half* scales, __half* out, int m, int N, int K, float beta, int t, int splits,
              int* err, cudaStream_t stream) {
  const size_t stage = U8_Q_BYTES + (size_t)t * U8_KB * 4;
  const int nstages = (int)std::min<size_t>(U8_MAX_STAGES, 220 * 1024 / stage);
  const size_t smem = nstages * stage + 1024 /* alignment slack */ + 512 /* barriers, tmem slot */;
  static bool attr_done[16] = {};
  int dev = 0;
  LCU_CUDA(cudaGetDevice(&dev));
  if (dev < 16 && !attr_done[dev]) {
    LCU_CUDA(cudaFuncSetAttribute((gemm_u8_kernel<BS>), cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024));
    attr_done[dev] = true;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((N + U8_ROWS - 1) / U8_ROWS * splits, (m + t - 1) / t);
  cfg.blockDim = dim3(U8_THREADS);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  int n_attr = 0;
  if (splits > 1) {
    attr[n_attr].id = cudaLaunchAttributeClusterDimension;
    attr[n_attr].val.clusterDim.x = splits;
    attr[n_attr].val.clusterDim.y = 1;
    attr[n_attr].val.clusterDim.z = 1;
    ++n_attr;
  }
  if (prompt_pdl()) {
    attr[n_attr].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[n_attr].val.programmaticStreamSerializationAllowed = 1;
    ++n_attr;
  }
  cfg.attrs = attr;
  cfg.numAttrs = n_attr;
  LCU_CUDA(cudaLaunchKernelEx(&cfg, gemm_u8_kernel<BS>, map_x, map_q, scales, out, m, N, K, beta, t, nstages, splits, err));
  return LCU_OK;
}

}  // namespace

// Fitted to timings of 12 shapes (2 to 600 rows) over tile heights and splits: a wave of CTAs takes 5.4 us and, per k-block, what the
// longer of converting (any tile) and feeding the tensor core (tall tiles) takes; a cluster's exchange about half a microsecond per
// CTA.  Clusters of 4 and 8 leave some SMs of a GPC without a CTA.  4096 x 4096: 100 rows 12.7 us in four parts, 20.9 in one;
// 4096 x 11008: 200 rows 30.0 us as one tile of 208 rows per weight tile, 42.4 as two of 112 (a second wave).
void gemm_u8_plan(int m, int N, int K, int sms, int* tile_rows, int* splits) {
  double best = 1e30;
  const int least = (m + U8_MAX_T - 1) / U8_MAX_T;
  for (int tiles = least; tiles < least + 4; ++tiles) {
    const int t = ((m + tiles - 1) / tiles + 15) / 16 * 16;
    const double per_block = std::max(0.235, 0.06 + 0.00156 * t);
    for (int sp = 1; sp <= 8; sp *= 2) {
      if (K / U8_STAGE_K < 2 * sp) continue;
      const long at_once = std::max(1, sp <= 2 ? sms : sp == 4 ? sms - 12 : sms - 36);
      const long ctas = (long)((N + U8_ROWS - 1) / U8_ROWS) * ((m + t - 1) / t) * sp, waves = (ctas + at_once - 1) / at_once;
      const double est = waves * (5.4 + (double)K / U8_KB / sp * per_block + (sp > 1 ? 0.5 * sp : 0.0));
      if (est < best - 0.2) {  // (ties stay with fewer tiles and no split)
        best = est;
        *tile_rows = t;
        *splits = sp;
      }
    }
  }
}

bool gemm_u8_supported(int m, int N, int K, int bs, const void* lhs, const void* q, const void* scales) {
  return m >= 2 && m <= 65535 && N >= 2 && N % 2 == 0 && K > 0 && K % 256 == 0 && (bs == 32 || bs == 64 || bs == 128) && ((uintptr_t)lhs & 15) == 0 &&
         ((uintptr_t)q & 15) == 0 && ((uintptr_t)scales & 3) == 0;
}

int launch_gemm_u8(__half* out, const __half* lhs, const uint8_t* q, const __half* scales, int bs, int m, int N, int K, float beta, int* err,
                   cudaStream_t stream) {
  LCU_REQUIRE(err != nullptr, "gemm_u8: no error word");
  LCU_REQUIRE(gemm_u8_supported(m, N, K, bs, lhs, q, scales), "gemm_u8: unsupported shape m=%d N=%d K=%d blocks of %d or unaligned pointers", m, N, K, bs);
  int t = 16, splits = 1;
  gemm_u8_plan(m, N, K, gemv_sm_count(), &t, &splits);
  CUtensorMap map_x, map_q;
  {
    const uint64_t dims[3] = {(uint64_t)U8_KB, (uint64_t)m, (uint64_t)(K / U8_KB)}, strides[2] = {(uint64_t)K * 2, (uint64_t)U8_KB * 2};
    const uint32_t box[3] = {(uint32_t)U8_KB, (uint32_t)t, 2};
    const int rc = tc_encode_map(&map_x, lhs, 3, dims, strides, box);
    if (rc) return rc;
  }
  {  // (two weights per 16-bit element of the map)
    const uint64_t dims[2] = {(uint64_t)K / 2, (uint64_t)N}, strides[1] = {(uint64_t)K};
    const uint32_t box[2] = {(uint32_t)U8_STAGE_K / 2, (uint32_t)U8_ROWS};
    const int rc = tc_encode_map(&map_q, q, 2, dims, strides, box, true);
    if (rc) return rc;
  }
  if (bs == 32) return launch_u8<32>(map_x, map_q, scales, out, m, N, K, beta, t, splits, err, stream);
  if (bs == 64) return launch_u8<64>(map_x, map_q, scales, out, m, N, K, beta, t, splits, err, stream);
  return launch_u8<128>(map_x, map_q, scales, out, m, N, K, beta, t, splits, err, stream);
}

}  // namespace lcu
