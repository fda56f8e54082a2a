// Attention over a sliding window and pooled blocks for several rows on tcgen05, bfloat16 caches (block_attn.cu has the same
// function on warp-level tiles, for few rows and the shapes this kernel does not take).
//
// A CTA takes 128 query rows of one head and walks the visible keys in tiles of 128 twice - block means first, then the tokens from
// the first row's window start to the last row:
//   pass 1  S = Q K^T into tensor memory, a running maximum per row;
//   pass 2  S again, e^(s - maximum) as bfloat16 into tensor memory, where it is the A operand of the product with V; sums in
//           binary32 from the unrounded exponentials, results divided at the end.
// With the maximum known first, the output accumulator is never rescaled, and the second score product costs less than the
// hand-over a rescale needs.  Warp 0 issues the tensor copies, warp 1 the MMAs, warps 2-17 own a row and 32 of a tile's 128 keys per
// thread.  Two score accumulators and two probability tiles let exponentials run under the neighbouring tiles' MMAs.
// Keys may come in two parts (a head's own, and one that all heads share); each is padded to blocks of 64 columns by the tensor
// copies' zero fill.  Rows past the last position are filled with zeros too: a stale cache row never meets a probability of zero.
// Bound by the MMAs and by filling the ring from L2 (128 KB per tile at 192 key columns), with one CTA per SM.  Prompts of 2000
// tokens, window 1024: 16 heads of 192 x 128 (four layers) 1.66 -> 1.43 ms in all against the 64-row warp-level tiles, 122 us of
// every layer; 4 heads of 128 x 128 with block means (four layers) 2.12 -> 1.86 ms.
#include <math_constants.h>

#include <algorithm>

#include "block_ops.cuh"
#include "elem.cuh"
#include "tc_common.cuh"

namespace lcu {
namespace {

using bf16 = __nv_bfloat16;
constexpr int WT_Q = 128, WT_K = 128;     // query rows and keys per tile
constexpr int WT_EPI_WARPS = 16, WT_THREADS = 64 + 32 * WT_EPI_WARPS;
constexpr uint32_t WT_BLOCK = 128 * 64 * 2;  // 128 rows x 64 columns
constexpr uint32_t WT_V_ATOM = 64 * 64 * 2;  // 64 keys x 64 columns
constexpr float LOG2E = 1.4426950408889634f;
// tensor memory: S[2], O, P[2] (two bfloat16 per column)
constexpr uint32_t WT_S = 0, WT_O = 256, WT_P = 384, WT_TMEM = 512;
enum { B_Q, B_K_FULL, B_K_EMPTY = B_K_FULL + 2, B_V_FULL = B_K_EMPTY + 2, B_V_EMPTY = B_V_FULL + 2, B_S_FULL = B_V_EMPTY + 2, B_S_EMPTY = B_S_FULL + 2,
       B_P_FULL = B_S_EMPTY + 2, B_P_EMPTY = B_P_FULL + 2, B_O_FULL = B_P_EMPTY + 2, B_COUNT };

struct wt_params {
  bf16* out;
  const float* sink;
  const bf16* gate;
  int ldo, ldg, heads, group, vdim, window, pool, first, first2, m, pos0, own_blocks, vec_out;
  float scale2, out_scale;
  int* err;
};

__device__ __forceinline__ float wt_ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ void wt_mma_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(d_tmem),
      "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void wt_st_32x16(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};" ::"r"(taddr), "r"(r[0]),
      "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]),
      "r"(r[14]), "r"(r[15])
      : "memory");
}

// NK: 64-column blocks of a key (both parts), HV: value columns of the tile
template <int NK, int HV>
__global__ void __launch_bounds__(WT_THREADS, 1)
    window_tc_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_q2, const __grid_constant__ CUtensorMap map_k,
                     const __grid_constant__ CUtensorMap map_k2, const __grid_constant__ CUtensorMap map_v, const __grid_constant__ CUtensorMap map_kp,
                     const __grid_constant__ CUtensorMap map_vp, const wt_params p) {
  constexpr uint32_t K_BYTES = NK * WT_BLOCK, V_BYTES = (HV / 64) * 2 * WT_V_ATOM;
  constexpr uint32_t BF16 = tc_elem<bf16>::IDESC_FORMAT;
  constexpr uint32_t IDESC_QK = (1u << 4) | BF16 | ((uint32_t)(WT_K >> 3) << 17) | ((uint32_t)(WT_Q >> 4) << 24);
  constexpr uint32_t IDESC_PV = (1u << 4) | BF16 | (1u << 16) /* B: keys x columns */ | ((uint32_t)(HV >> 3) << 17) | ((uint32_t)(WT_Q >> 4) << 24);
  extern __shared__ uint8_t smem_raw[];
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* smem = smem_raw + (base - smem_u32(smem_raw));
  const uint32_t k_ring = base + K_BYTES, v_ring = k_ring + 2 * K_BYTES;
  float* stats = reinterpret_cast<float*>(smem + 3 * K_BYTES + 2 * V_BYTES);  // [128 rows][4]: maxima, then sums
  uint64_t* bars = reinterpret_cast<uint64_t*>(stats + 2 * WT_Q * 4);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + B_COUNT);
  auto bar = [&](int i) { return smem_u32(&bars[i]); };

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // row tiles in descending order (the last ones see the most keys), heads of a key/value group next to each other
  const int head = blockIdx.x, q0 = (gridDim.y - 1 - blockIdx.y) * WT_Q, kvh = head / p.group;
  const int first_pos = p.pos0 + q0, last_pos = first_pos + min(WT_Q, p.m - q0) - 1;
  auto blocks_of = [&](int pos) {
    const int past = pos + 1 - p.window;
    return p.pool > 0 && past > 0 ? past / p.pool : 0;
  };
  const int n_blocks = blocks_of(last_pos), lo = max(0, first_pos + 1 - p.window);
  const int pool_tiles = (n_blocks + WT_K - 1) / WT_K, n_tiles = pool_tiles + (last_pos - lo + WT_K) / WT_K;

  if (threadIdx.x == 0) {
    for (int i = 0; i < B_COUNT; ++i) {
      const bool many = (i >= B_S_EMPTY && i < B_S_EMPTY + 2) || (i >= B_P_FULL && i < B_P_FULL + 2);
      mbar_init(bar(i), many ? WT_EPI_WARPS : 1);
    }
    fence_mbar_init();
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(WT_TMEM) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  pdl_launch_dependents();
  pdl_wait();

  if (warp == 0) {
    if (tc_elect()) {  // ---- loads: Q; pass 1: every K; pass 2: K_0, then K_j+1 and V_j alternately, as they are consumed
      mbar_arrive_expect_tx(bar(B_Q), K_BYTES);
      for (int b = 0; b < NK; ++b)
        if (b < p.own_blocks) tma_load_3d(base + b * WT_BLOCK, &map_q, b * 64, head, q0, bar(B_Q));
        else tma_load_3d(base + b * WT_BLOCK, &map_q2, (b - p.own_blocks) * 64, head, q0, bar(B_Q));
      bool ok = true;
      tc_ring rk, rv;
      auto place = [&](int tile) { return tile < pool_tiles ? tile * WT_K : lo + (tile - pool_tiles) * WT_K; };
      auto load_k = [&](int tile) {
        ok = ok && mbar_wait(bar(B_K_EMPTY + rk.slot), rk.phase ^ 1u, p.err, DEV_ERR_EMPTY_WAIT);
        if (!ok) return;
        const uint32_t full = bar(B_K_FULL + rk.slot), dst = k_ring + (uint32_t)rk.slot * K_BYTES;
        mbar_arrive_expect_tx(full, K_BYTES);
        const int t0 = place(tile);
        for (int b = 0; b < NK; ++b) {
          if (tile < pool_tiles) tma_load_3d(dst + b * WT_BLOCK, &map_kp, b * 64, t0, kvh, full);
          else if (b < p.own_blocks) tma_load_3d(dst + b * WT_BLOCK, &map_k, b * 64, t0 - p.first, kvh, full);
          else tma_load_2d(dst + b * WT_BLOCK, &map_k2, (b - p.own_blocks) * 64, t0 - p.first2, full);
        }
        rk.step(2);
      };
      auto load_v = [&](int tile) {
        ok = ok && mbar_wait(bar(B_V_EMPTY + rv.slot), rv.phase ^ 1u, p.err, DEV_ERR_EMPTY_WAIT);
        if (!ok) return;
        const uint32_t full = bar(B_V_FULL + rv.slot), dst = v_ring + (uint32_t)rv.slot * V_BYTES;
        mbar_arrive_expect_tx(full, V_BYTES);
        const int t0 = place(tile);
        for (int h = 0; h < 2; ++h)
          for (int a = 0; a < HV / 64; ++a) {
            const uint32_t to = dst + (uint32_t)(h * (HV / 64) + a) * WT_V_ATOM;
            if (tile < pool_tiles) tma_load_3d(to, &map_vp, a * 64, t0 + h * 64, kvh, full);
            else tma_load_3d(to, &map_v, a * 64, t0 + h * 64 - p.first, kvh, full);
          }
        rv.step(2);
      };
      for (int j = 0; j < n_tiles && ok; ++j) load_k(j);
      load_k(0);
      for (int j = 0; j < n_tiles && ok; ++j) {
        if (j + 1 < n_tiles) load_k(j + 1);
        load_v(j);
      }
    }
    __syncwarp();
  } else if (warp == 1) {  // ---- MMAs
    bool ok = mbar_wait_warp(bar(B_Q), 0, p.err, DEV_ERR_FULL_WAIT);
    tc_ring rk, rs, rv;
    auto scores = [&]() {  // the next K tile into the next score accumulator
      ok = ok && mbar_wait_warp(bar(B_S_EMPTY + rs.slot), rs.phase ^ 1u, p.err, DEV_ERR_TMEM_WAIT);
      ok = ok && mbar_wait_warp(bar(B_K_FULL + rk.slot), rk.phase, p.err, DEV_ERR_FULL_WAIT);
      if (!ok) return;
      tc_fence_after();
      if (tc_elect()) {
#pragma unroll
        for (int b = 0; b < NK; ++b) {
          const uint64_t a_desc = smem_desc_sw128(base + b * WT_BLOCK), b_desc = smem_desc_sw128(k_ring + (uint32_t)rk.slot * K_BYTES + b * WT_BLOCK);
#pragma unroll
          for (int k = 0; k < 4; ++k) tc_mma_f16(tmem + WT_S + (uint32_t)(rs.slot * WT_K), a_desc + 2 * k, b_desc + 2 * k, IDESC_QK, (b | k) != 0);
        }
        tc_commit(bar(B_K_EMPTY + rk.slot));
        tc_commit(bar(B_S_FULL + rs.slot));
      }
      __syncwarp();
      rk.step(2);
      rs.step(2);
    };
    for (int j = 0; j <= n_tiles && ok; ++j) scores();  // pass 1, and the first tile of pass 2
    for (int j = 0; j < n_tiles && ok; ++j, rv.step(2)) {
      if (j + 1 < n_tiles) scores();
      ok = ok && mbar_wait_warp(bar(B_P_FULL + rv.slot), rv.phase, p.err, DEV_ERR_FULL_WAIT);
      ok = ok && mbar_wait_warp(bar(B_V_FULL + rv.slot), rv.phase, p.err, DEV_ERR_FULL_WAIT);
      if (!ok) break;
      tc_fence_after();
      if (tc_elect()) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const uint64_t b_desc = smem_desc_sw128_mn(v_ring + (uint32_t)rv.slot * V_BYTES + h * (HV / 64) * WT_V_ATOM, WT_V_ATOM);
          const uint32_t a = tmem + WT_P + (uint32_t)(rv.slot * 64 + h * 32);
#pragma unroll
          for (int k = 0; k < 4; ++k)  // 16 keys: 8 columns of probabilities, two 8-key groups (2 x 1024 bytes) of V
            wt_mma_ts(tmem + WT_O, a + 8 * k, b_desc + (uint64_t)(k * 2048 >> 4), IDESC_PV, (j | h | k) != 0);
        }
        tc_commit(bar(B_V_EMPTY + rv.slot));
        tc_commit(bar(B_P_EMPTY + rv.slot));
      }
      __syncwarp();
    }
    if (tc_elect()) {
      tc_commit(bar(B_O_FULL));  // (also after a failed wait: lets the other warps leave)
      if (!ok) {
        tc_commit(bar(B_S_FULL));
        tc_commit(bar(B_S_FULL + 1));
      }
    }
    __syncwarp();
  } else {
    const int quad = warp & 3, cq = (warp - 2) >> 2;
    const int row = quad * 32 + lane, r = q0 + row, pos = p.pos0 + r;
    const int warp_first = p.pos0 + q0 + quad * 32, warp_last = warp_first + 31;
    const uint32_t lane_base = tmem + ((uint32_t)(quad * 32) << 16);
    tc_ring rs, rp;
    bool go = true;
    // scores of this thread's 32 keys of tile j in units of log2, keys it does not see -inf; false: none of the warp's rows sees any
    auto load_scores = [&](int j, float (&s)[32]) -> bool {
      const bool ok = mbar_wait(bar(B_S_FULL + rs.slot), rs.phase, p.err, DEV_ERR_TMEM_WAIT);
      tc_fence_after();
      go = __all_sync(0xffffffffu, ok);  // (the error word is looked at once, before the results are stored)
      if (!go) return false;
      const bool pooled = j < pool_tiles;
      const int k0 = (pooled ? j * WT_K : lo + (j - pool_tiles) * WT_K) + cq * 32;
      const bool any = pooled ? k0 < blocks_of(warp_last) : k0 <= warp_last && k0 + 31 > warp_first - p.window;
      if (any) {
        uint32_t raw[32];
        tc_ld_32x32(lane_base + WT_S + (uint32_t)(rs.slot * WT_K + cq * 32), raw);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        const bool all = pooled ? k0 + 32 <= blocks_of(warp_first) : k0 + 31 <= warp_first && k0 > warp_last - p.window;
#pragma unroll
        for (int i = 0; i < 32; ++i) s[i] = __uint_as_float(raw[i]) * p.scale2;
        if (!all) {
          const int from = pooled ? 0 : pos + 1 - p.window, to = pooled ? blocks_of(pos) - 1 : pos;
#pragma unroll
          for (int i = 0; i < 32; ++i)
            if (k0 + i < from || k0 + i > to) s[i] = -CUDART_INF_F;
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar(B_S_EMPTY + rs.slot));
      rs.step(2);
      return any;
    };
    // ---- pass 1
    float mx = -CUDART_INF_F;
    for (int j = 0; j < n_tiles && go; ++j) {
      float s[32];
      if (!load_scores(j, s)) continue;
      float a = fmaxf(s[0], s[1]), b = fmaxf(s[2], s[3]);
#pragma unroll
      for (int i = 4; i < 32; i += 4) {
        a = fmaxf(a, fmaxf(s[i], s[i + 1]));
        b = fmaxf(b, fmaxf(s[i + 2], s[i + 3]));
      }
      mx = fmaxf(mx, fmaxf(a, b));
    }
    stats[row * 4 + cq] = mx;
    bar_sync(1, 32 * WT_EPI_WARPS);
    {
      const float4 q = *reinterpret_cast<const float4*>(stats + row * 4);
      mx = fmaxf(fmaxf(q.x, q.y), fmaxf(q.z, q.w));
    }
    const float ref = mx > -CUDART_INF_F ? mx : 0.f;  // (rows past the last one may see nothing)
    // ---- pass 2
    float sum = 0.f;
    for (int j = 0; j < n_tiles && go; ++j) {
      float s[32];
      const bool any = load_scores(j, s);
      if (!go) break;
      uint32_t e[16];
      if (any) {
        float s0 = 0.f, s1 = 0.f;
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          const float a = wt_ex2(s[2 * i] - ref), b = wt_ex2(s[2 * i + 1] - ref);
          s0 += a;
          s1 += b;
          e[i] = tc_elem<bf16>::pack(a, b);
        }
        sum += s0 + s1;
      } else {
#pragma unroll
        for (int i = 0; i < 16; ++i) e[i] = 0;
      }
      const bool ok = mbar_wait(bar(B_P_EMPTY + rp.slot), rp.phase ^ 1u, p.err, DEV_ERR_TMEM_WAIT);
      go = __all_sync(0xffffffffu, ok);
      if (!go) break;
      tc_fence_after();
      wt_st_32x16(lane_base + WT_P + (uint32_t)(rp.slot * 64 + cq * 16), e);
      asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar(B_P_FULL + rp.slot));
      rp.step(2);
    }
    float* sums = stats + WT_Q * 4;
    sums[row * 4 + cq] = sum;
    bar_sync(1, 32 * WT_EPI_WARPS);
    {
      const float4 q = *reinterpret_cast<const float4*>(sums + row * 4);
      sum = (q.x + q.y) + (q.z + q.w);
    }
    float inv = p.out_scale / sum;
    if (p.sink) {  // one more term of the denominator, against the larger of it and the row's maximum
      const float s2 = p.sink[head] * LOG2E, top = fmaxf(mx, s2), f = wt_ex2(mx - top);
      inv = p.out_scale * f / (sum * f + wt_ex2(s2 - top));
    }
    if (p.gate && r < p.m) inv *= sigmoid_f(to_f(p.gate[(size_t)r * p.ldg + head]));
    const bool ok = mbar_wait(bar(B_O_FULL), 0, p.err, DEV_ERR_TMEM_WAIT);
    tc_fence_after();
    if (__all_sync(0xffffffffu, ok && go && *(volatile int*)p.err == 0) && cq * 32 < HV) {
      uint32_t o[32];
      tc_ld_32x32(lane_base + WT_O + (uint32_t)(cq * 32), o);
      asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
      if (r < p.m) {
        bf16* dst = p.out + (size_t)r * p.ldo + head * p.vdim + cq * 32;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int d = cq * 32 + 8 * i;
          uint32_t w[4];
#pragma unroll
          for (int e = 0; e < 4; ++e) w[e] = tc_elem<bf16>::pack(__uint_as_float(o[8 * i + 2 * e]) * inv, __uint_as_float(o[8 * i + 2 * e + 1]) * inv);
          if (p.vec_out) {
            if (d < p.vdim) *reinterpret_cast<uint4*>(dst + 8 * i) = make_uint4(w[0], w[1], w[2], w[3]);
          } else {
#pragma unroll
            for (int e = 0; e < 8; ++e)
              if (d + e < p.vdim) dst[8 * i + e] = __ushort_as_bfloat16((unsigned short)(w[e >> 1] >> (16 * (e & 1))));
          }
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    __syncwarp();
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(WT_TMEM) : "memory");
  }
}

template <int NK, int HV>
int launch_blocks(const CUtensorMap (&maps)[7], const wt_params& q, cudaStream_t stream) {
  constexpr size_t SMEM = 3 * (size_t)NK * WT_BLOCK + 2 * (size_t)(HV / 64) * 2 * WT_V_ATOM + 2 * WT_Q * 4 * 4 + B_COUNT * 8 + 16 + 1024 /* alignment slack */;
  static bool attr_done[16] = {};
  int dev = 0;
  LCU_CUDA(cudaGetDevice(&dev));
  if (dev < 16 && !attr_done[dev]) {
    LCU_CUDA(cudaFuncSetAttribute((window_tc_kernel<NK, HV>), cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM));
    attr_done[dev] = true;
  }
  LCU_CUDA(launch_after(window_tc_kernel<NK, HV>, dim3(q.heads, (q.m + WT_Q - 1) / WT_Q), dim3(WT_THREADS), SMEM, stream, maps[0], maps[1], maps[2], maps[3],
                        maps[4], maps[5], maps[6], q));
  return LCU_OK;
}

int own_key_blocks(int dim) { return (dim + 63) / 64; }

}  // namespace

// heads of up to 192 key columns (each part counted in blocks of 64) and 128 value columns; rows, heads and strides in whole 16-byte
// vectors, as tensor copies need them; a shared key part has no block means
bool window_tc_supported(const attn_rows<bf16>& p) {
  const int blocks = own_key_blocks(p.dim) + (p.key2 ? own_key_blocks(p.dim2) : 0);
  auto whole = [](const void* ptr, size_t a, size_t b) { return (((uintptr_t)ptr & 15) | (a & 7) | (b & 7)) == 0; };
  return p.err && blocks <= 3 && p.vdim <= 128 && !(p.key2 && p.pool > 0) && whole(p.q, p.ld, p.q_head) && whole(p.cache.k, p.cache.ldk, p.cache.k_head) &&
         whole(p.cache.v, p.cache.ldv, p.cache.v_head) && (!p.key2 || whole(p.key2, p.ld2, 0)) &&
         (p.pool == 0 || p.cache.n_blocks == 0 || (whole(p.cache.kp, 0, 0) && whole(p.cache.vp, 0, 0)));
}

int launch_window_tc(const attn_rows<bf16>& p, int m, int pos0, cudaStream_t stream) {
  LCU_REQUIRE(window_tc_supported(p), "window attention: head size %d + %d x %d", p.dim, p.key2 ? p.dim2 : 0, p.vdim);
  const uint64_t end = (uint64_t)(pos0 + m), k_cols = round_up(p.dim, 8), v_cols = round_up(p.vdim, 8);
  const uint64_t n_blocks = p.pool > 0 ? std::min<uint64_t>(p.cache.n_blocks, end / p.pool) : 0;
  CUtensorMap maps[7];
  auto encode = [&](int i, const bf16* ptr, uint64_t cols, uint64_t n1, size_t s1, uint64_t n2, size_t s2, uint32_t b1, uint32_t b2) {
    const uint64_t dims[3] = {cols, n1, n2}, strides[2] = {s1 * 2, s2 * 2};
    const uint32_t box[3] = {64, b1, b2};
    return tc_encode_map(&maps[i], ptr, n2 ? 3 : 2, dims, strides, box);
  };
  // queries [row][head][columns]; the queries of the shared part follow a head's own
  int rc = encode(0, p.q, p.key2 ? k_cols : p.dim, p.heads, p.q_head, m, p.ld, 1, WT_Q);
  if (!rc) rc = encode(2, p.cache.k, k_cols, end - p.cache.first, p.cache.ldk, p.kv_heads, p.cache.k_head, WT_K, 1);
  if (!rc) rc = encode(4, p.cache.v, v_cols, end - p.cache.first, p.cache.ldv, p.kv_heads, p.cache.v_head, 64, 1);
  if (rc) return rc;
  maps[1] = maps[0];
  maps[3] = maps[5] = maps[2];
  maps[6] = maps[4];
  if (p.key2) {
    rc = encode(1, p.q + k_cols, round_up(p.dim2, 8), p.heads, p.q_head, m, p.ld, 1, WT_Q);
    if (!rc) rc = encode(3, p.key2, round_up(p.dim2, 8), end - p.first2, p.ld2, 0, 0, WT_K, 1);
  }
  if (!rc && n_blocks > 0) {
    rc = encode(5, p.cache.kp, k_cols, n_blocks, p.cache.ldk, p.kv_heads, (size_t)p.cache.n_blocks * p.cache.ldk, WT_K, 1);
    if (!rc) rc = encode(6, p.cache.vp, v_cols, n_blocks, p.cache.ldv, p.kv_heads, (size_t)p.cache.n_blocks * p.cache.ldv, 64, 1);
  }
  if (rc) return rc;
  wt_params q{};
  q.out = p.out;
  q.sink = p.sink;
  q.gate = p.gate;
  q.ldo = p.ldo;
  q.ldg = p.ldg;
  q.heads = p.heads;
  q.group = p.heads / p.kv_heads;
  q.vdim = p.vdim;
  q.window = p.window;
  q.pool = p.pool;
  q.first = p.cache.first;
  q.first2 = p.first2;
  q.m = m;
  q.pos0 = pos0;
  q.own_blocks = own_key_blocks(p.dim);
  q.vec_out = p.vdim % 8 == 0 && p.ldo % 8 == 0 && ((uintptr_t)p.out & 15) == 0;
  q.scale2 = p.scale * LOG2E;
  q.out_scale = p.out_scale;
  q.err = p.err;
  const int blocks = q.own_blocks + (p.key2 ? own_key_blocks(p.dim2) : 0);
  if (p.vdim <= 64) return blocks == 1 ? launch_blocks<1, 64>(maps, q, stream) : blocks == 2 ? launch_blocks<2, 64>(maps, q, stream) : launch_blocks<3, 64>(maps, q, stream);
  return blocks == 1 ? launch_blocks<1, 128>(maps, q, stream) : blocks == 2 ? launch_blocks<2, 128>(maps, q, stream) : launch_blocks<3, 128>(maps, q, stream);
}

}  // namespace lcu
