// Single-row (batch-1) weight-streaming GEMV: every consumer warp is an independent streaming
// dot-product engine with a private shared-memory ring; no block-wide synchronisation in the loop.
//
// Measured on B200 with this library's read probe (bench_read_ceiling): a 16 KiB ring stage
// fetched as sixteen 1 KiB bulk copies tops out near 4.4 TB/s with one CTA per SM, while copies
// of 4 KiB or more reach the read ceiling of ~7.2 TB/s.  So a stage here is TWO bulk copies: one
// contiguous 4 KiB chunk (2048 fp16 / 4096 u8 weights) from each row of a row pair, and the chunk
// is mapped onto the tensor-core tile like this:
//
//   m16n8k16 tile row  m = 8*rr + seg : segment `seg` (1/8 of the chunk, 512 B) of row `rr` of the pair
//   tile column        n = seg        : the activation values of that same segment
//
// D[m][n] is wanted only on the "diagonal" n == seg(m): lane (g, c = g/2) ends up with the partial
// dot products of segment g for both rows.  All 16 tile rows still consume distinct weight bytes.
// Odd segments walk their 64-byte steps in swapped order (step ^ 1) on both operands, so the eight
// lanes of a quarter warp hit eight distinct 16-byte bank groups without padding the staged rows.
//
// A row pair (the unit RoPE and the SiLU gate need) belongs to ONE warp from its first chunk to its
// epilogue: the warp waits on its own mbarriers, accumulates in registers, reduces with shuffles and
// writes the result.  The producer warp deals chunks to the warps' rings round-robin.  As in the
// multi-row kernel (gemv.cu) the producer does not depend on the activations, so under programmatic
// dependent launch the rings of kernel n+1 fill while kernel n drains; every wait is bounded; int8
// weights are de-quantised in registers bit-identically to half((q - 127.5f) * scale)
// (reference llama_cu.cu:287-289); the RMSNorm prologue rounds where the reference does (llama_cu.cu:72-106) and sums in an order of its own.
#include <cuda_bf16.h>

#include <algorithm>

#include "gemv.cuh"

namespace lcu {
namespace {

template <int WT>
constexpr bool is16 = WT == 0 || WT == 3;  // two-byte weights: halves (0) or bfloat16 (3)

// Consumer warps per CTA (template parameter of the kernel): 4, or 5 for u8 kernels whose activation row leaves room
// for two CTAs per SM only - ten consumer warps per SM instead of eight, the u8 kernels being latency-bound.
constexpr int NW_MAX = 5;
// Stage geometry per weight type: 4 KiB of each row per stage (measured: 2 KiB stages in a ring twice as deep lose a
// third of the u8 throughput - the per-stage cost of the producer counts).
template <int WT>
struct geom {
  static constexpr int ROWB = 4096;                    // bytes of one row per stage (one bulk copy)
  static constexpr int SEG = ROWB / 8;                 // the chunk is cut into 8 segments, one per tile column
  static constexpr int NSTEPS = SEG / 64;              // 64-byte steps per segment
  static constexpr int SC_ROW = WT == 2 ? ROWB / 64 * 2 : 256;  // scale bytes reserved per row per stage (block size >= 64 / >= 32)
  static constexpr int SEG_SHIFT = 9;                  // log2(SEG)
};
constexpr int MAX_SW = 4;                   // ring depth per warp
constexpr int NACC = 4;                     // independent accumulator sets (no chain on one result)
constexpr int EMPTY_BASE = NW_MAX * MAX_SW;  // barriers: full[w * MAX_SW + s], empty[EMPTY_BASE + w * MAX_SW + s]
constexpr int BAR_BYTES = 2 * EMPTY_BASE * 8;
constexpr int SMEM_FIXED = BAR_BYTES + 64;  // barriers; the activation row's barrier and the CTA's count (tensor-parallel)

// u8 kernels read 32 activation bytes per 16 weight bytes; with the row stored flat, the two segments of a
// quarter warp would meet on the same banks.  The activations of every segment are therefore shifted by 16 more
// bytes than those of the one before (vector i of eight halves lives at byte 16 * (i + i / (SEG / 8))).
template <int WT>
__host__ __device__ __forceinline__ int row_offset(int vec_index) {
  return is16<WT> ? vec_index * 16 : (vec_index + (vec_index >> (geom<WT>::SEG_SHIFT - 3))) * 16;
}
// the activation row in shared memory: the row itself, sums over aligned groups of 64 (factored u8), sums of squares over
// aligned blocks of 256 (RMSNorm)
struct row_layout {
  int sums, squares, total;  // byte offsets
};
template <int WT>
__host__ __device__ __forceinline__ row_layout row_layout_of(int K, bool norm) {
  row_layout r;
  const int xbytes = is16<WT> ? K * 2 : K * 2 + (K >> geom<WT>::SEG_SHIFT) * 16 + 16;
  r.sums = (xbytes + 127) & ~127;
  r.squares = r.sums + (WT == 2 ? (K / 64 * 4 + 127) & ~127 : 0);
  r.total = r.squares + (norm ? (K / 256 * 4 + 127) & ~127 : 0);
  return r;
}

template <int EPI>
__device__ __forceinline__ void map_row(const gemv_params& p, int vrow, int& mat, int& row) {
  if (EPI == EPI_SILU) {
    mat = vrow & 1;
    row = vrow >> 1;
  } else if (EPI == EPI_ROPE_KV) {  // three matrices: two comparisons instead of a division
    mat = (vrow >= p.rows_per_mat) + (vrow >= 2 * p.rows_per_mat);
    row = vrow - mat * p.rows_per_mat;
  } else {
    mat = 0;
    row = vrow;
  }
}

__device__ __forceinline__ uint32_t dequant_pair(uint32_t word, uint32_t selector, __half2 scale2) {
  uint32_t v = __byte_perm(word, 0x64646464u, selector);  // bytes -> halves 1024 + q
  __half2 h = *reinterpret_cast<__half2*>(&v);
  h = __hsub2(h, __half2half2(__ushort_as_half(0x6400)));  // - 1024   (exact)
  h = __hsub2(h, __half2half2(__ushort_as_half(0x57f8)));  // - 127.5  (exact)
  h = __hmul2(h, scale2);                                  // one rounding, as the reference
  return *reinterpret_cast<uint32_t*>(&h);
}

// One 64-byte step of every segment: 16 tile rows x 32 (fp16) or 64 (u8) weights per lane group.  lo / hi: 16 bytes of the pair's
// rows; x0, x1: the activations they meet; sc_lo / sc_hi: their scales; xsum: sum of the activations of the step (factored u8).
template <int WT>
__device__ __forceinline__ void step(float (&accs)[NACC][4], const int s, const uint4& lo, const uint4& hi, const uint4& x0, const uint4& x1, __half sc_lo,
                                     __half sc_hi, float xsum) {
  float* acc = accs[(2 * s) % NACC];
  float* acc_b = accs[(2 * s + 1) % NACC];
  if (WT == 3) {
    mma_16816_bf16(acc, lo.x, hi.x, lo.y, hi.y, x0.x, x0.y);
    mma_16816_bf16(acc_b, lo.z, hi.z, lo.w, hi.w, x0.z, x0.w);
  } else if (WT == 0) {
    mma_16816(acc, lo.x, hi.x, lo.y, hi.y, x0.x, x0.y);
    mma_16816(acc_b, lo.z, hi.z, lo.w, hi.w, x0.z, x0.w);
  } else if (WT == 2) {
    const float corr = 1151.5f * xsum;
    float ta[4] = {0.f, 0.f, 0.f, 0.f}, tb[4] = {0.f, 0.f, 0.f, 0.f};
    const uint32_t M = 0x64646464u;  // bytes -> halves 1024 + q
    mma_16816(ta, __byte_perm(lo.x, M, 0x4140), __byte_perm(hi.x, M, 0x4140), __byte_perm(lo.x, M, 0x4342), __byte_perm(hi.x, M, 0x4342), x0.x, x0.y);
    mma_16816(tb, __byte_perm(lo.y, M, 0x4140), __byte_perm(hi.y, M, 0x4140), __byte_perm(lo.y, M, 0x4342), __byte_perm(hi.y, M, 0x4342), x0.z, x0.w);
    mma_16816(ta, __byte_perm(lo.z, M, 0x4140), __byte_perm(hi.z, M, 0x4140), __byte_perm(lo.z, M, 0x4342), __byte_perm(hi.z, M, 0x4342), x1.x, x1.y);
    mma_16816(tb, __byte_perm(lo.w, M, 0x4140), __byte_perm(hi.w, M, 0x4140), __byte_perm(lo.w, M, 0x4342), __byte_perm(hi.w, M, 0x4342), x1.z, x1.w);
    // only the diagonal entries (column == this lane's segment) are meaningful, and they share `corr`
    const float sl = __half2float(sc_lo), sh = __half2float(sc_hi);
    acc[0] += sl * ((ta[0] + tb[0]) - corr);
    acc[1] += sl * ((ta[1] + tb[1]) - corr);
    acc[2] += sh * ((ta[2] + tb[2]) - corr);
    acc[3] += sh * ((ta[3] + tb[3]) - corr);
  } else {
    const __half2 s_lo = __half2half2(sc_lo), s_hi = __half2half2(sc_hi);
    mma_16816(acc, dequant_pair(lo.x, 0x4140, s_lo), dequant_pair(hi.x, 0x4140, s_hi), dequant_pair(lo.x, 0x4342, s_lo),
              dequant_pair(hi.x, 0x4342, s_hi), x0.x, x0.y);
    mma_16816(acc_b, dequant_pair(lo.y, 0x4140, s_lo), dequant_pair(hi.y, 0x4140, s_hi), dequant_pair(lo.y, 0x4342, s_lo),
              dequant_pair(hi.y, 0x4342, s_hi), x0.z, x0.w);
    mma_16816(acc, dequant_pair(lo.z, 0x4140, s_lo), dequant_pair(hi.z, 0x4140, s_hi), dequant_pair(lo.z, 0x4342, s_lo),
              dequant_pair(hi.z, 0x4342, s_hi), x1.x, x1.y);
    mma_16816(acc_b, dequant_pair(lo.w, 0x4140, s_lo), dequant_pair(hi.w, 0x4140, s_hi), dequant_pair(lo.w, 0x4342, s_lo),
              dequant_pair(hi.w, 0x4342, s_hi), x1.z, x1.w);
  }
}

// Factored u8, block size >= 128: the two 64-byte steps of a 128-weight block share their scale, so the eight
// tensor-core products of both steps are summed before the one multiplication by the scale.
struct factored_pair {
  float ta[4], tb[4];
  // the correction term is the start value of one accumulator chain: sum - 1151.5 * sum(x) costs no instruction of its own
  __device__ __forceinline__ void half_step(int h, const uint4& lo, const uint4& hi, const uint4& x0, const uint4& x1, float negcorr) {
    const uint32_t M = 0x64646464u;  // bytes -> halves 1024 + q
    if (h == 0) {  // the block's first products start the two chains
      mma_16816_from(ta, __byte_perm(lo.x, M, 0x4140), __byte_perm(hi.x, M, 0x4140), __byte_perm(lo.x, M, 0x4342), __byte_perm(hi.x, M, 0x4342), x0.x, x0.y, negcorr);
      mma_16816_from(tb, __byte_perm(lo.y, M, 0x4140), __byte_perm(hi.y, M, 0x4140), __byte_perm(lo.y, M, 0x4342), __byte_perm(hi.y, M, 0x4342), x0.z, x0.w, 0.f);
    } else {
      mma_16816(ta, __byte_perm(lo.x, M, 0x4140), __byte_perm(hi.x, M, 0x4140), __byte_perm(lo.x, M, 0x4342), __byte_perm(hi.x, M, 0x4342), x0.x, x0.y);
      mma_16816(tb, __byte_perm(lo.y, M, 0x4140), __byte_perm(hi.y, M, 0x4140), __byte_perm(lo.y, M, 0x4342), __byte_perm(hi.y, M, 0x4342), x0.z, x0.w);
    }
    mma_16816(ta, __byte_perm(lo.z, M, 0x4140), __byte_perm(hi.z, M, 0x4140), __byte_perm(lo.z, M, 0x4342), __byte_perm(hi.z, M, 0x4342), x1.x, x1.y);
    mma_16816(tb, __byte_perm(lo.w, M, 0x4140), __byte_perm(hi.w, M, 0x4140), __byte_perm(lo.w, M, 0x4342), __byte_perm(hi.w, M, 0x4342), x1.z, x1.w);
  }
  __device__ __forceinline__ void add_to(float* acc, __half sc_lo, __half sc_hi) const {
    const float sl = __half2float(sc_lo), sh = __half2float(sc_hi);
    acc[0] += sl * (ta[0] + tb[0]);
    acc[1] += sl * (ta[1] + tb[1]);
    acc[2] += sh * (ta[2] + tb[2]);
    acc[3] += sh * (ta[3] + tb[3]);
  }
};

// The segment's sums of both rows, to all lanes of its quad: row 0 is in d0/d1, row 1 in d2/d3 of the quad's diagonal lane.
__device__ __forceinline__ void segment_sums(const float (&accs)[NACC][4], int lane, float& s0, float& s1) {
  const float a0 = (accs[0][0] + accs[1][0]) + (accs[2][0] + accs[3][0]), a1 = (accs[0][1] + accs[1][1]) + (accs[2][1] + accs[3][1]);
  const float a2 = (accs[0][2] + accs[1][2]) + (accs[2][2] + accs[3][2]), a3 = (accs[0][3] + accs[1][3]) + (accs[2][3] + accs[3][3]);
  const int g = lane >> 2, diag_lane = 4 * g + (g >> 1);
  s0 = __shfl_sync(0xffffffffu, (g & 1) ? a1 : a0, diag_lane);
  s1 = __shfl_sync(0xffffffffu, (g & 1) ? a3 : a2, diag_lane);
}

// The steps of a staged chunk.  Lanes of an odd segment take the steps of a pair in swapped order (bank spread); every place
// that forms a row's sum takes them in this order, so the sum's bits do not depend on the kernel.
template <int WT, bool FULL>
__device__ __forceinline__ void staged_step(float (&accs)[NACC][4], const int s, const int flip, const int c, const int g, const int vb, const uint8_t* seg0,
                                            const uint8_t* xseg, const uint8_t* st, const float* xs64, const int ci, const int bs) {
  constexpr int ROWB = geom<WT>::ROWB, SEG = geom<WT>::SEG, NSTEPS = geom<WT>::NSTEPS, CHUNK_K = ROWB / (is16<WT> ? 2 : 1);
  const int off = ((s ^ flip) << 6) + c * 16;  // byte offset inside the segment
  uint4 lo = make_uint4(0, 0, 0, 0), hi = lo, x0 = lo, x1 = lo;
  __half sc_lo = __ushort_as_half(0), sc_hi = sc_lo;
  float xsum = 0.f;
  if (FULL || off < vb) {
    lo = *reinterpret_cast<const uint4*>(seg0 + off);
    hi = *reinterpret_cast<const uint4*>(seg0 + ROWB + off);
    if (is16<WT>) {
      x0 = *reinterpret_cast<const uint4*>(xseg + off);
    } else {
      x0 = *reinterpret_cast<const uint4*>(xseg + 2 * off);
      x1 = *reinterpret_cast<const uint4*>(xseg + 2 * off + 16);
      const __half* scs = reinterpret_cast<const __half*>(st + 2 * ROWB);
      const int si = (g * SEG + off) >> bs;  // k offset inside the chunk / block size (bs is log2 of it here)
      sc_lo = scs[si];
      sc_hi = scs[geom<WT>::SC_ROW / 2 + si];
      // WT 2: sum of x over this lane's segment and step (the diagonal column of the tile)
      if (WT == 2) xsum = xs64[ci * (CHUNK_K / 64) + g * NSTEPS + (s ^ flip)];
    }
  }
  step<WT>(accs, s, lo, hi, x0, x1, sc_lo, sc_hi, xsum);
}
template <bool FULL>
__device__ __forceinline__ void staged_step_pair(float (&accs)[NACC][4], const int sp, const int flip, const int c, const int g, const int vb,
                                                 const uint8_t* seg0, const uint8_t* xseg, const uint8_t* st, const float* xs64, const int ci, const int bs) {
  constexpr int ROWB = geom<2>::ROWB, SEG = geom<2>::SEG, NSTEPS = geom<2>::NSTEPS;
  // a row's last chunk may be short; its length is a multiple of the block size, so a 128-byte pair is valid or not as a whole
  const bool ok = FULL || (sp << 7) < vb;
  float negcorr = 0.f;
  if (ok) {
    const float2 xs2 = *reinterpret_cast<const float2*>(xs64 + ci * (ROWB / 64) + g * NSTEPS + 2 * sp);
    negcorr = -1151.5f * (xs2.x + xs2.y);
  }
  factored_pair f;
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int off = (((2 * sp + h) ^ flip) << 6) + c * 16;
    uint4 lo = make_uint4(0, 0, 0, 0), hi = lo, x0 = lo, x1 = lo;
    if (ok) {
      lo = *reinterpret_cast<const uint4*>(seg0 + off);
      hi = *reinterpret_cast<const uint4*>(seg0 + ROWB + off);
      x0 = *reinterpret_cast<const uint4*>(xseg + 2 * off);
      x1 = *reinterpret_cast<const uint4*>(xseg + 2 * off + 16);
    }
    f.half_step(h, lo, hi, x0, x1, negcorr);
  }
  if (!ok) return;  // (after the warp-wide tensor-core instructions)
  const __half* scs = reinterpret_cast<const __half*>(st + 2 * ROWB);
  const int si = (g * SEG + (sp << 7)) >> bs;
  f.add_to(accs[sp % NACC], scs[si], scs[geom<2>::SC_ROW / 2 + si]);
}

// ---- the activation row: global -> shared memory, normalised, with the group sums of the factored u8 kernels.
// This is what a launch does between its predecessor's end and its first product, with nothing to hide it behind, and most of
// its instructions run once: their fetch counts as much as their latency, so loops that need no register array stay rolled.
// Squares are added per vector, by shuffles over aligned blocks of 256 and over the blocks (an order that does not depend on the
// number of threads); group sums come from the same pass as the normalised values.  Decode step, 8 layers, with the epilogue by
// batches below, in us: 1024 wide fp16 219 -> 196, 2048 wide 274 -> 253, 4096 wide 630 -> 620, with u8 weights 480 -> 468.
constexpr int ROW_VEC = 4;  // vectors of eight halves a thread requests at once

__device__ __forceinline__ float square_sum8(const uint4& q) {
  const __half2* h = reinterpret_cast<const __half2*>(&q);
  float s = 0.f;
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const float2 f = __half22float2(h[e]);
    s = fmaf(f.x, f.x, s);
    s = fmaf(f.y, f.y, s);
  }
  return s;
}
// x_i <- norm_w_i *h half(x_i * rinv)
__device__ __forceinline__ uint4 norm8(uint4 xq, const uint4& wq, float rinv) {
  __half2* x2 = reinterpret_cast<__half2*>(&xq);
  const __half2* w2 = reinterpret_cast<const __half2*>(&wq);
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const float2 f = __half22float2(x2[e]);
    x2[e] = __hmul2(w2[e], __floats2half2_rn(f.x * rinv, f.y * rinv));
  }
  return xq;
}
// vector i of the row is final: the sum of its group of 64 (eight neighbouring lanes)
__device__ __forceinline__ void row_sums8(const uint4& q, int i, int lane, float* xs64) {
  const __half2* h = reinterpret_cast<const __half2*>(&q);
  float s = 0.f;
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const float2 f = __half22float2(h[e]);
    s += f.x + f.y;
  }
  s += __shfl_xor_sync(0xffffffffu, s, 1);
  s += __shfl_xor_sync(0xffffffffu, s, 2);
  s += __shfl_xor_sync(0xffffffffu, s, 4);
  if ((lane & 7) == 0) xs64[i >> 3] = s;
}
// The row is in shared memory (each thread reads back the vectors it wrote itself, or all of them are visible): normalise
// it and form its group sums.  K is a multiple of 256, so a warp's 32 vectors are all inside the row or all outside.
// nw: norm weights of the thread's first NV vectors.
template <int WT, int NV>
__device__ __forceinline__ void row_finish(const gemv_params& p, bool norm, uint8_t* xs, float* xs64, float* squares, int tid, int threads,
                                           const uint4 (&nw)[NV], float inv_k) {
  const int vec = p.K >> 3, lane = tid & 31;
  float rinv = 1.f;
  if (norm) {
#pragma unroll 2
    for (int i = tid; i < vec; i += threads) {
      const float s = warp_sum(square_sum8(*reinterpret_cast<const uint4*>(xs + row_offset<WT>(i))));
      if (lane == 0) squares[i >> 5] = s;
    }
    bar_sync(1, threads);
    // over the blocks: every run of `span` lanes adds up all of them, so every lane ends with the whole sum
    const int blocks = vec >> 5, span = blocks >= 32 ? 32 : 1 << (32 - __clz(blocks - 1));
    float t = 0.f;
    for (int b = lane & (span - 1); b < blocks; b += 32) t += squares[b];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
      if (o < span) t += __shfl_xor_sync(0xffffffffu, t, o);
    rinv = rsqrtf(t * inv_k + p.eps);
  }
  auto finish = [&](int i, const uint4& w) {
    uint4 q = *reinterpret_cast<const uint4*>(xs + row_offset<WT>(i));
    if (norm) {
      q = norm8(q, w, rinv);
      *reinterpret_cast<uint4*>(xs + row_offset<WT>(i)) = q;
    }
    if (WT == 2) row_sums8(q, i, lane, xs64);
  };
  if (norm && vec <= threads) {  // (a path of its own: skipping code costs its fetch)
    if (tid < vec) finish(tid, nw[0]);
  } else if (norm) {
#pragma unroll
    for (int j = 0; j < NV; ++j)
      if (tid + j * threads < vec) finish(tid + j * threads, nw[j]);
#pragma unroll 1
    for (int i = tid + NV * threads; i < vec; i += threads) finish(i, *reinterpret_cast<const uint4*>(p.norm_w + i * 8));
  } else if (WT == 2) {
#pragma unroll 4
    for (int i = tid; i < vec; i += threads) finish(i, nw[0]);
  }
  bar_sync(1, threads);
}

__device__ __forceinline__ uint4 ld_stream(const void* at) {
  uint4 v;
  asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(at));
  return v;
}

// ---- what becomes of a row pair's two sums
struct pair_operands {  // what the epilogue reads from global memory, and where its results go
  __half2 prev;
  float2 cs;
  int mat, row, head, j;
  template <int WT, int EPI>
  __device__ __forceinline__ void fetch(const gemv_params& p, int pr, int pos) {
    prev = __half2half2(__ushort_as_half(0));
    cs = make_float2(1.f, 0.f);
    if (EPI == EPI_PLAIN) {
      if (WT != 3 && p.beta != 0.f) prev = *reinterpret_cast<const __half2*>(p.out + 2 * pr);
    } else if (EPI == EPI_ROPE_KV) {
      map_row<EPI_ROPE_KV>(p, 2 * pr, mat, row);
      head = row / p.head_dim;
      j = row - head * p.head_dim;
      if (mat < 2) cs = p.rope[(size_t)pos * (p.head_dim >> 1) + (j >> 1)];
    }
  }
};
template <int WT, int EPI>
__device__ __forceinline__ void store_pair(const gemv_params& p, const gemv_batch& bt, int bi, const pair_operands& po, int pr, float v0, float v1, int pos,
                                           float gate_scale) {
  const int vrow = 2 * pr;
  if (WT == 3) {
    if (EPI == EPI_PLAIN) {
      if (bt.f32[bi]) *reinterpret_cast<float2*>(reinterpret_cast<float*>(bt.out[bi]) + vrow) = make_float2(v0, v1);
      else *reinterpret_cast<__nv_bfloat162*>(reinterpret_cast<__nv_bfloat16*>(bt.out[bi]) + vrow) = __floats2bfloat162_rn(v0, v1);
    } else {  // the gate on the binary32 sums
      __nv_bfloat16* o = reinterpret_cast<__nv_bfloat16*>(bt.n > 0 ? bt.out[bi] : p.out);
      const float z = gate_scale * v0;
      o[pr] = __float2bfloat16(z / (1.0f + expf(-z)) * (gate_scale * v1));
    }
  } else if (EPI == EPI_PLAIN) {
    float a0 = v0, a1 = v1;
    __half* o = p.out + vrow;
    if (p.beta != 0.f) {
      a0 = a0 + p.beta * __low2float(po.prev);
      a1 = a1 + p.beta * __high2float(po.prev);
    }
    const __half2 r2 = __halves2half2(__float2half(a0), __float2half(a1));
    *reinterpret_cast<__half2*>(o) = r2;
    if (p.out_peer) *reinterpret_cast<__half2*>(p.out_peer + vrow) = r2;  // peer store over NVLink
    for (int q = 0; q < p.n_peer_out; ++q) *reinterpret_cast<__half2*>(p.peer_out[q] + vrow) = r2;  // tensor-parallel: into every GPU's row
  } else {
    const __half a = __float2half(v0), bq = __float2half(v1);  // the matmul's own output rounding
    if (EPI == EPI_SILU) {
      const float val = __half2float(a);  // llama_cu.cu:536-537 on the half-rounded w1 / w3 outputs
      const __half gated = __float2half(val / (1.0f + expf(-val)) * __half2float(bq));
      p.out[pr] = gated;
      for (int q = 0; q < p.n_peer_out; ++q) p.peer_out[q][pr] = gated;
    } else {
      __half o0 = a, o1 = bq;
      if (po.mat < 2) {  // llama_cu.cu:381-387, cos/sin from the context's table
        const float real = __half2float(a), imag = __half2float(bq);
        const float a_cos = po.cs.x, a_sin = po.cs.y;
        o0 = __float2half(real * a_cos - imag * a_sin);
        o1 = __float2half(real * a_sin + imag * a_cos);
      }
      const __half2 pr2 = __halves2half2(o0, o1);
      if (po.mat == 0) {
        *reinterpret_cast<__half2*>(p.q_out + po.row) = pr2;
      } else {
        __half* cache = po.mat == 1 ? p.k_cache : p.v_cache;
        *reinterpret_cast<__half2*>(cache + ((size_t)po.head * p.ctx_len + pos) * p.head_dim + po.j) = pr2;
      }
    }
  }
}

// Weight types (WT): 0 = fp16; 1 = u8, every weight rounded to half((q - 127.5) * scale) before the
// product exactly as the reference's tensor-core kernel does (llama_cu.cu:287-289, 332-341); 2 = u8
// with the scale factored out of each 64-weight group: sum_k x_k (q_k - 127.5) s = s * (sum_k x_k
// (1024 + q_k) - 1151.5 * sum_k x_k), the bytes going to the tensor core as the exact halves
// 1024 + q (one PRMT per two weights) and the group sums of x coming from the prologue.  Mode 2 has
// no per-weight rounding: it is closer to the exact product but is not the reference's rounding.  3 = bfloat16 weights and
// activations: no fused norm or cache write; EPI_PLAIN runs the matrices of `bt`, each with its own vector, on runs of CTAs.
//
// LONG: normalised fp16 rows of more than ROW_VEC vectors per thread (4096 values; the 13B and 65B models).  Their norm weights are requested
// ahead of the wait as a whole, up to 8192 values; requested behind the row's sum, one after the other, every vector past the
// fourth cost 0.25 to 0.3 us (wq|wk|wv of 6144 35.25 -> 34.74, of 8192 62.2 -> 61.0).  Code of its own, because the other launches pay for the fetch of instructions that they skip (with it in
// their kernel a step of 2048 columns took 219.0 us for 215.6, u8 with blocks of 32 252 for 238 at 1024).
template <int WT, int EPI, int NW, bool LONG = false>
__global__ void __launch_bounds__((NW + 1) * 32, NW == 4 ? 3 : 2) gemv1_kernel(const gemv_params p, const int sw, const int pf_bytes,
                                                                                        const __grid_constant__ gemv_batch bt) {
  constexpr int NCONS = NW * 32;
  static_assert(NW <= NW_MAX, "barriers");
  constexpr int ESZ = is16<WT> ? 2 : 1;
  constexpr int ROWB = geom<WT>::ROWB, SEG = geom<WT>::SEG, NSTEPS = geom<WT>::NSTEPS;
  constexpr int CHUNK_K = ROWB / ESZ;        // weights of one row per stage
  constexpr int STAGE_BYTES = 2 * ROWB + (is16<WT> ? 0 : 2 * geom<WT>::SC_ROW);

  extern __shared__ __align__(128) uint8_t smem[];
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem);  // full: [w * MAX_SW + s], empty: [EMPTY_BASE + w * MAX_SW + s]
  const uint32_t xbar = smem_u32(smem + BAR_BYTES + 32);
  int* cta_done = reinterpret_cast<int*>(smem + BAR_BYTES + 40);  // consumer warps of this CTA that are through (tensor-parallel)
  uint8_t* xs = smem + SMEM_FIXED;                     // activation row, K halves (row_offset)
  const row_layout rl = row_layout_of<WT>(p.K, WT != 3 && p.norm_w != nullptr);
  float* xs64 = reinterpret_cast<float*>(xs + rl.sums);
  float* squares = reinterpret_cast<float*>(xs + rl.squares);
  uint8_t* stages = xs + rl.total;                     // [NW][sw][STAGE_BYTES]
  auto xoff = [](int vec_index) { return row_offset<WT>(vec_index); };

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (WT != 3 || !bt.hold) pdl_launch_dependents();

  int pairs = (p.n_mats * p.rows_per_mat) >> 1, cta = blockIdx.x, n_ctas = gridDim.x, bi = 0;
  if (WT == 3 && bt.n > 0) {  // which of the batch's matrices this CTA works on
    while (bi + 1 < bt.n && (int)blockIdx.x >= bt.first_cta[bi + 1]) ++bi;
    cta = blockIdx.x - bt.first_cta[bi];
    n_ctas = bt.first_cta[bi + 1] - bt.first_cta[bi];
    pairs = bt.rows[bi] >> 1;
  }
  // (picked matrices: the producer warp reads the choice once it is there, see below)
  size_t picked = 0;
  auto weights_of = [&](int mat) { return reinterpret_cast<const uint8_t*>(WT == 3 && bt.n > 0 ? bt.w[bi] : p.w[mat]) + (WT == 3 ? picked : 0); };
  // row of a matrix in memory: gate and up rows of picked matrices alternate in blocks
  auto place_of = [&](int mat, int row) {
    if (WT == 3 && EPI == EPI_SILU && bt.n > 0) return ((row >> bt.gate_shift) << (bt.gate_shift + 1)) + (mat << bt.gate_shift) + (row & ((1 << bt.gate_shift) - 1));
    return row;
  };
  const __half* x_row = WT == 3 && EPI == EPI_PLAIN ? reinterpret_cast<const __half*>(bt.x[bi]) : p.x;
  // first pair of a CTA: floor(pairs * cta / n_ctas), without the 64-bit division
  const int per_cta = pairs / n_ctas, more = pairs - per_cta * n_ctas;
  const int pr0 = per_cta * cta + more * cta / n_ctas;
  const int npairs = per_cta * (cta + 1) + more * (cta + 1) / n_ctas - pr0;
  const int rowbytes = p.K * ESZ;
  const int nchunks = (rowbytes + ROWB - 1) / ROWB;

  // Scales of a row chunk are one contiguous run; when rows start 16-byte aligned they travel as one more bulk copy
  // per row on the same barrier, otherwise as 4-byte cp.async pieces issued by all lanes (32 more barrier arrivals).
  const bool sc_bulk = !is16<WT> && ((p.K / p.bs) & 7) == 0 && ((ROWB / p.bs) & 7) == 0;
  if (warp == NW && lane < NW * MAX_SW) {
    static_assert(NW * MAX_SW <= 32, "a barrier of each kind per lane");
    mbar_init(smem_u32(&bars[lane]), (is16<WT> || sc_bulk) ? 1 : 33);
    mbar_init(smem_u32(&bars[EMPTY_BASE + lane]), 1);
    if (lane == 0) {
      mbar_init(xbar, 1);
      *cta_done = 0;
    }
    fence_mbar_init();
  }
  __syncthreads();

  const int bs_shift = p.bs > 0 ? 31 - __clz(p.bs) : 0;  // block size is a power of two (32, 64, 128, ...)
  if (warp == NW) {
    // ------------------------------------------------------------ producer
    // (this warp's instruction chain per stage bounds the u8 kernels: shifts, no divisions)
    const uint64_t pol = policy_evict_first();
    if (WT == 3 && bt.choice != nullptr) {
      if (!bt.choice_settled) pdl_wait();
      picked = (size_t)bt.choice[bi] * bt.choice_bytes;
    }
    if (pf_bytes > 0) {  // L2 look-ahead over the first rows of this CTA
      const int rows_pf = max(1, min(pf_bytes / rowbytes, 2 * npairs));
      for (int r = lane; r < rows_pf; r += 32) {
        int mat, row;
        map_row<EPI>(p, 2 * pr0 + r, mat, row);
        l2_prefetch(weights_of(mat) + (size_t)place_of(mat, row) * rowbytes, (uint32_t)rowbytes);
      }
    }
    int slot[NW];
    uint32_t par[NW];
#pragma unroll
    for (int w = 0; w < NW; ++w) {
      slot[w] = 0;
      par[w] = 0;
    }
    const int full_rounds = npairs / NW, r_tail = npairs - full_rounds * NW;
    // one stage for consumer warp w: `cbytes` bytes of both rows of a pair (lanes 0 and 1 hold the row addresses,
    // the half warps the scale addresses) and their scales
    // Copies of a stage are issued by one predicated instruction: lanes 0 and 1 copy the two rows, lanes 2 and 16 the
    // scale runs of rows 0 and 1 when those travel as bulk copies (scale addresses are held per half warp).
    const uint32_t bars_u32 = smem_u32(bars), stages_u32 = smem_u32(stages);
    const bool lane_sc = lane >= 2;
    const bool lane_copies = lane < 2 || (sc_bulk && (lane == 2 || lane == 16));
    const uint32_t lane_dst = lane_sc ? 2 * ROWB + (lane >> 4) * (is16<WT> ? 0 : geom<WT>::SC_ROW) : lane * ROWB;
    auto issue = [&](const int w, const uint8_t* row_src, const __half* sc_src, const int cbytes) {
      const uint32_t full = bars_u32 + (uint32_t)(w * MAX_SW + slot[w]) * 8;
      mbar_wait(full + EMPTY_BASE * 8, par[w] ^ 1, p.err, DEV_ERR_EMPTY_WAIT);
      const uint32_t st = stages_u32 + (uint32_t)(w * sw + slot[w]) * STAGE_BYTES;
      const uint32_t scbytes = !is16<WT> ? (uint32_t)(cbytes >> bs_shift) * 2 : 0;  // scale bytes per row of this chunk
      if (lane == 0) mbar_arrive_expect_tx(full, (uint32_t)(2 * cbytes) + (sc_bulk ? 2 * scbytes : 0));
      __syncwarp();
      if (lane_copies)
        bulk_g2s_hint(st + lane_dst, lane_sc ? (const void*)sc_src : (const void*)row_src, lane_sc ? scbytes : (uint32_t)cbytes, full, pol);
      if (!is16<WT> && !sc_bulk) {
        const int ppr = (cbytes >> bs_shift) >> 1;  // 4-byte pieces per row
        for (int j = lane & 15; j < ppr; j += 16) cp_async4(st + 2 * ROWB + (lane >> 4) * geom<WT>::SC_ROW + j * 4, sc_src + 2 * j);
        cp_async_mbar_arrive_noinc(full);
      }
      if (++slot[w] == sw) {
        slot[w] = 0;
        par[w] ^= 1;
      }
    };
    auto pair_sources = [&](const int pr, const uint8_t*& row_src, const __half*& sc_src) {
      int mat, row;
      map_row<EPI>(p, 2 * pr + (lane & 1), mat, row);
      row_src = weights_of(mat) + (size_t)place_of(mat, row) * rowbytes;
      sc_src = nullptr;
      if (!is16<WT>) {
        int m2, r2;
        map_row<EPI>(p, 2 * pr + (lane >> 4), m2, r2);
        sc_src = p.sc[m2] + (size_t)r2 * (p.K >> bs_shift);
      }
    };
    // full rounds: chunk ci of the pairs base .. base+NW-1 goes to warps 0 .. NW-1 in turn
    for (int rd = 0; rd < full_rounds; ++rd) {
      const uint8_t* src_row[NW];
      const __half* src_sc[NW];
#pragma unroll
      for (int w = 0; w < NW; ++w) pair_sources(pr0 + rd * NW + w, src_row[w], src_sc[w]);
      for (int ci = 0; ci < nchunks; ++ci) {
        const int cbytes = min(ROWB, rowbytes - ci * ROWB);
#pragma unroll
        for (int w = 0; w < NW; ++w) issue(w, src_row[w] + (size_t)ci * ROWB, !is16<WT> ? src_sc[w] + ((ci * CHUNK_K) >> bs_shift) : nullptr, cbytes);
      }
    }
    // tail round: the pairs left over go to warps 0 .. r_tail-1
    if (r_tail > 0) {
      const uint8_t* src_row[NW];
      const __half* src_sc[NW];
#pragma unroll
      for (int w = 0; w < NW; ++w)
        if (w < r_tail) pair_sources(pr0 + full_rounds * NW + w, src_row[w], src_sc[w]);
      for (int ci = 0; ci < nchunks; ++ci) {
        const int cbytes = min(ROWB, rowbytes - ci * ROWB);
#pragma unroll
        for (int w = 0; w < NW; ++w)
          if (w < r_tail) issue(w, src_row[w] + (size_t)ci * ROWB, !is16<WT> ? src_sc[w] + ((ci * CHUNK_K) >> bs_shift) : nullptr, cbytes);
      }
    }
    if (!is16<WT>) cp_async_wait<0>();
    return;
  }

  // -------------------------------------------------------------- consumers
  // The norm weights do not depend on the previous kernel: they are brought close while this one waits for it.
  const int vec = p.K >> 3;
  const bool norm = WT != 3 && p.norm_w != nullptr;
  constexpr int NORM_VEC = LONG ? 2 * ROW_VEC : ROW_VEC;
  uint4 nw[NORM_VEC];
  const float inv_k = 1.0f / p.K;
  if (norm) {
#pragma unroll
    for (int j = 0; j < NORM_VEC; ++j)
      if (tid + j * NCONS < vec) nw[j] = *reinterpret_cast<const uint4*>(p.norm_w + (tid + j * NCONS) * 8);
  }
  pdl_wait();
  if (WT == 3 && bt.hold) pdl_launch_dependents();
  const float gate_scale = WT == 3 && EPI == EPI_SILU && bt.n > 0 ? bt.gate_scale[bi] : 1.0f;
  const int pos = EPI == EPI_ROPE_KV ? *p.pos : 0;
  if (npairs > 0) {
    // Rows of up to ROW_VEC vectors per thread are loaded by the threads themselves.  Longer rows come in as bulk copies of one
    // 512-element segment each: one trip to L2 whatever the row length, where per-thread loads would pay a round trip per
    // batch of vectors.  Both read past L1 (L2 is where another GPU's peer stores land).
    if (!LONG && vec <= ROW_VEC * NCONS) {
      if (p.n_wait > 0) {
        // tensor-parallel: parts of the row come from other GPUs; wait for their flags first
        if (tid < p.n_wait) flag_wait_at_least(p.wait_flags + tid, *p.seq * TP_EXCHANGES_PER_STEP + p.wait_id, p.err);
        bar_sync(1, NCONS);
      }
      uint4 xv[ROW_VEC];
#pragma unroll
      for (int j = 0; j < ROW_VEC; ++j)
        if (tid + j * NCONS < vec) xv[j] = __ldcg(reinterpret_cast<const uint4*>(x_row + (tid + j * NCONS) * 8));
#pragma unroll
      for (int j = 0; j < ROW_VEC; ++j)
        if (tid + j * NCONS < vec) *reinterpret_cast<uint4*>(xs + xoff(tid + j * NCONS)) = xv[j];
    } else {
      if (warp == 0) {
        if (p.n_wait > 0) {
          if (lane < p.n_wait) flag_wait_at_least(p.wait_flags + lane, *p.seq * TP_EXCHANGES_PER_STEP + p.wait_id, p.err);
          __syncwarp();
        }
        if (lane == 0) mbar_arrive_expect_tx(xbar, (uint32_t)p.K * 2);
        __syncwarp();
        const int nseg = (p.K + 511) >> 9;
        for (int sg = lane; sg < nseg; sg += 32)
          bulk_g2s(smem_u32(xs + xoff(sg * 64)), x_row + sg * 512, (uint32_t)min(1024, (p.K - sg * 512) * 2), xbar);
      }
      mbar_wait(xbar, 0, p.err, DEV_ERR_FULL_WAIT);
    }
    row_finish<WT>(p, norm, xs, xs64, squares, tid, NCONS, nw, inv_k);
  }

  const int g = lane >> 2, c = lane & 3;
  const int flip = g & 1;

  // A warp's row pairs are taken BATCH at a time: of each pair the diagonal lane of every quad holds its segment's sums, and the
  // quad's lane c keeps those of the batch's pair c, so that one tree over the segments and one epilogue (lanes 0 .. 3, a
  // pair each) serve four pairs.  A tree and an epilogue per pair were 900 of the 2900 cycles a pair of 4096 u8 weights took.
  constexpr int BATCH = 4;
  int slot = 0;
  uint32_t par = 0;
  for (int i0 = warp; i0 < npairs; i0 += BATCH * NW) {
    const int i = i0 + c * NW;
    const bool mine = g == 0 && i < npairs;
    pair_operands po;  // requested ahead of the products
    if (mine) po.fetch<WT, EPI>(p, pr0 + i, pos);
    float v0 = 0.f, v1 = 0.f;
#pragma unroll 1
    for (int k = 0; k < BATCH && i0 + k * NW < npairs; ++k) {
      float accs[NACC][4];
#pragma unroll
      for (int a = 0; a < NACC; ++a) accs[a][0] = accs[a][1] = accs[a][2] = accs[a][3] = 0.f;
      for (int ci = 0; ci < nchunks; ++ci) {
        mbar_wait(smem_u32(&bars[warp * MAX_SW + slot]), par, p.err, DEV_ERR_FULL_WAIT);
        const int cbytes = min(ROWB, rowbytes - ci * ROWB);
        const int vb = min(max(cbytes - g * SEG, 0), SEG);  // valid bytes of this lane's segment
        const uint8_t* st = stages + (size_t)(warp * sw + slot) * STAGE_BYTES;
        const uint8_t* seg0 = st + g * SEG;
        const uint8_t* xseg = xs + xoff((ci * CHUNK_K + g * (SEG / ESZ)) >> 3);
        // A full chunk (every chunk but possibly the last of a row) takes the branch-free path, so that the
        // shared loads of all eight steps can be issued ahead of the tensor-core instructions.
        if (WT == 2 && cbytes == ROWB && bs_shift >= 7) {
#pragma unroll
          for (int sp = 0; sp < NSTEPS / 2; ++sp) staged_step_pair<true>(accs, sp, flip, c, g, SEG, seg0, xseg, st, xs64, ci, bs_shift);
        } else if (WT == 2 && bs_shift >= 7) {
#pragma unroll
          for (int sp = 0; sp < NSTEPS / 2; ++sp) staged_step_pair<false>(accs, sp, flip, c, g, vb, seg0, xseg, st, xs64, ci, bs_shift);
        } else if (cbytes == ROWB) {
#pragma unroll
          for (int s = 0; s < NSTEPS; ++s) staged_step<WT, true>(accs, s, flip, c, g, SEG, seg0, xseg, st, xs64, ci, bs_shift);
        } else {
#pragma unroll
          for (int s = 0; s < NSTEPS; ++s) staged_step<WT, false>(accs, s, flip, c, g, vb, seg0, xseg, st, xs64, ci, bs_shift);
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&bars[EMPTY_BASE + warp * MAX_SW + slot]));
        if (++slot == sw) {
          slot = 0;
          par ^= 1;
        }
      }
      float s0, s1;
      segment_sums(accs, lane, s0, s1);
      if (c == k) {
        v0 = s0;
        v1 = s1;
      }
    }
#pragma unroll
    for (int o = 16; o >= 4; o >>= 1) {  // fixed-order tree over the segments
      v0 += __shfl_xor_sync(0xffffffffu, v0, o);
      v1 += __shfl_xor_sync(0xffffffffu, v1, o);
    }
    if (mine) store_pair<WT, EPI>(p, bt, bi, po, pr0 + i, v0, v1, pos, gate_scale);
  }
  // tensor-parallel: the last consumer warp of the launch to get here publishes this GPU's slice (every result went into
  // the other GPUs' rows as a peer store in the epilogue above, made by the warp's first lanes).  The fences widen with the
  // counting: a warp counts itself inside its CTA behind a CTA-scope fence (shared memory), the last warp of a CTA
  // counts the CTA behind a device-scope fence (global memory), and only the last warp of the launch pays for the
  // system-scope fence - cumulative over everything counted before it - ahead of the flags it writes into the waiting
  // GPUs' memory.  (A system-scope fence in every warp serialises for more than 10 us per launch.)
  if (p.done_count != nullptr) __syncwarp();  // (lanes 0 .. 3 made the stores)
  if (p.done_count != nullptr && lane == 0) {
    __threadfence_block();
    if (atomicAdd_block(cta_done, 1) == NW - 1) {
      __threadfence();
      if (atomicAdd(p.done_count, 1) == (int)gridDim.x - 1) {
        atomicExch(p.done_count, 0);  // (the next launch counts from zero; its warps arrive after this kernel has ended)
        fence_acq_rel_sys();
        const int stamp = *p.seq * TP_EXCHANGES_PER_STEP + p.exchange_id;
        for (int q = 0; q < p.n_peer_flag; ++q) st_relaxed_sys(p.peer_flag[q], stamp);
      }
    }
  }
}

// ---- small matrices: a launch's whole share of the weights is held in registers.
//
// A launch over a few megabytes is as long as its chain of dependent steps, not as its bytes: with a ring, CTAs start when the
// kernel before them gives its shared memory back, set barriers up, wait for their first stage and run two or three row pairs one
// after the other.  Here a warp requests the one row pair it owns (two pairs where rows fit half a chunk: DUAL) straight into
// registers as its first act; a CTA needs shared memory for the activation row only, so CTAs start while the kernels before them
// run, and what follows the wait is the row, one pass of products, one tree, one store: 1.0 us without a norm, 1.6 with one (1024
// wide).  Rows of NCH chunks of 4 KiB.  Sums are formed in the order of the ring's kernel: the same bits.  Decode step, ring ->
// held, us: 512 wide, 4 layers, 95 -> 72; 1024 wide, 8 layers, 184 -> 143, with u8 weights 232 -> 176; 2048 wide, 8 layers, 245 -> 235,
// u8 294 -> 286; Zibovik 1024 wide, 8 layers, 304 -> 278.
template <int NCH>
constexpr int held_warps = NCH == 1 ? 8 : 4;  // most warps of a CTA (64 NCH registers of weights per thread)

template <int WT, int EPI, int NCH, bool DUAL>
__global__ void __launch_bounds__(held_warps<NCH> * 32, NCH == 1 ? 2 : 3) gemv_held_kernel(const gemv_params p, const __grid_constant__ gemv_batch bt) {
  constexpr int ESZ = is16<WT> ? 2 : 1, ROWB = geom<WT>::ROWB, SEG = geom<WT>::SEG, NSTEPS = geom<WT>::NSTEPS, CHUNK_K = ROWB / ESZ;
  static_assert(!DUAL || NCH == 1, "two pairs share one chunk");
  extern __shared__ __align__(128) uint8_t xs[];  // activation row (row_layout)
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, threads = blockDim.x;
  const int g = lane >> 2, c = lane & 3, flip = g & 1, seg = DUAL ? g & 3 : g;
  if (WT != 3 || !bt.hold) pdl_launch_dependents();

  int pairs = (p.n_mats * p.rows_per_mat) >> 1, cta = blockIdx.x, bi = 0;
  if (WT == 3 && bt.n > 0) {  // which of the batch's matrices this CTA works on
    while (bi + 1 < bt.n && (int)blockIdx.x >= bt.first_cta[bi + 1]) ++bi;
    cta = blockIdx.x - bt.first_cta[bi];
    pairs = bt.rows[bi] >> 1;
  }
  const int unit = cta * (threads >> 5) + warp, pr = DUAL ? 2 * unit + (g >> 2) : unit;
  const bool live = pr < pairs;
  size_t picked = 0;
  if (WT == 3 && bt.choice != nullptr) {
    if (!bt.choice_settled) pdl_wait();
    picked = (size_t)bt.choice[bi] * bt.choice_bytes;
  }
  const int rowbytes = p.K * ESZ, shift = is16<WT> ? 0 : 31 - __clz(p.bs);
  uint4 lo[NCH][NSTEPS], hi[NCH][NSTEPS];  // zero past the row's end
  uint32_t sc[WT == 2 ? NCH : 1][2][4];    // scales of the lane's segment: with blocks of 64 eight per chunk and row, of 128 four
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    int mat, row;
    map_row<EPI>(p, 2 * (live ? pr : pairs - 1) + r, mat, row);
    int place = row;
    if (WT == 3 && EPI == EPI_SILU && bt.n > 0) place = ((row >> bt.gate_shift) << (bt.gate_shift + 1)) + (mat << bt.gate_shift) + (row & ((1 << bt.gate_shift) - 1));
    const uint8_t* w = reinterpret_cast<const uint8_t*>(WT == 3 && bt.n > 0 ? bt.w[bi] : p.w[mat]) + (WT == 3 ? picked : 0) + (size_t)place * rowbytes + c * 16;
#pragma unroll
    for (int ci = 0; ci < NCH; ++ci) {
      const uint8_t* at = w + ci * ROWB + seg * SEG;
      const int vb = rowbytes - ci * ROWB - seg * SEG - c * 16;  // valid bytes from the lane's first on
#pragma unroll
      for (int s = 0; s < NSTEPS; ++s) {
        const int off = (s ^ flip) << 6;
        (r ? hi : lo)[ci][s] = make_uint4(0, 0, 0, 0);
        if (off < vb) (r ? hi : lo)[ci][s] = ld_stream(at + off);
      }
      if (WT == 2) {  // (rows are multiples of 256 weights: two scales travel together)
        const int per = SEG >> shift, first = (ci * ROWB + seg * SEG) >> shift;
        const __half* scs = p.sc[mat] + (size_t)row * (p.K >> shift) + first;
#pragma unroll
        for (int h = 0; h < 4; ++h) sc[ci][r][h] = 2 * h < per && first + 2 * h < (p.K >> shift) ? *reinterpret_cast<const uint32_t*>(scs + 2 * h) : 0;
      }
    }
  }
  const bool norm = WT != 3 && p.norm_w != nullptr;
  const row_layout rl = row_layout_of<WT>(p.K, norm);
  float* xs64 = reinterpret_cast<float*>(xs + rl.sums);
  const int vec = p.K >> 3;
  const float inv_k = 1.0f / p.K;
  uint4 nw[ROW_VEC];
  if (norm) {
#pragma unroll
    for (int j = 0; j < ROW_VEC; ++j)
      if (tid + j * threads < vec) nw[j] = *reinterpret_cast<const uint4*>(p.norm_w + (tid + j * threads) * 8);
  }
  pdl_wait();
  if (WT == 3 && bt.hold) pdl_launch_dependents();
  const float gate_scale = WT == 3 && EPI == EPI_SILU && bt.n > 0 ? bt.gate_scale[bi] : 1.0f;
  const int pos = EPI == EPI_ROPE_KV ? *p.pos : 0;
  const __half* x_row = WT == 3 && EPI == EPI_PLAIN ? reinterpret_cast<const __half*>(bt.x[bi]) : p.x;
  auto x_at = [&](int i) { return __ldcg(reinterpret_cast<const uint4*>(x_row + i * 8)); };
  auto x_put = [&](int i, const uint4& v) { *reinterpret_cast<uint4*>(xs + row_offset<WT>(i)) = v; };
  if (vec <= threads) {
    if (tid < vec) x_put(tid, x_at(tid));
  } else {
    uint4 xv[ROW_VEC];
#pragma unroll
    for (int j = 0; j < ROW_VEC; ++j)
      if (tid + j * threads < vec) xv[j] = x_at(tid + j * threads);
#pragma unroll
    for (int j = 0; j < ROW_VEC; ++j)
      if (tid + j * threads < vec) x_put(tid + j * threads, xv[j]);
  }
  const bool mine = live && (DUAL ? (lane & 15) == 0 : lane == 0);
  pair_operands po;
  if (mine) po.fetch<WT, EPI>(p, pr, pos);
  row_finish<WT>(p, norm, xs, xs64, reinterpret_cast<float*>(xs + rl.squares), tid, threads, nw, inv_k);

  float accs[NACC][4];
#pragma unroll
  for (int a = 0; a < NACC; ++a) accs[a][0] = accs[a][1] = accs[a][2] = accs[a][3] = 0.f;
#pragma unroll
  for (int ci = 0; ci < NCH; ++ci) {
    const uint8_t* xseg = xs + row_offset<WT>((ci * CHUNK_K + seg * (SEG / ESZ)) >> 3);
    const int vb = rowbytes - ci * ROWB - seg * SEG;
    auto x_of = [&](int s, uint4& x0, uint4& x1) {
      const int off = ((s ^ flip) << 6) + c * 16;
      x0 = x1 = make_uint4(0, 0, 0, 0);
      if (ci + 1 < NCH || off < vb) {
        x0 = *reinterpret_cast<const uint4*>(xseg + (is16<WT> ? off : 2 * off));
        if (!is16<WT>) x1 = *reinterpret_cast<const uint4*>(xseg + 2 * off + 16);
      }
    };
    const float* sums = xs64 + ci * (CHUNK_K / 64) + seg * NSTEPS;
    if (WT == 2 && shift >= 7) {
#pragma unroll
      for (int sp = 0; sp < NSTEPS / 2; ++sp) {
        const bool ok = ci + 1 < NCH || (sp << 7) < vb;
        const float negcorr = ok ? -1151.5f * (sums[2 * sp] + sums[2 * sp + 1]) : 0.f;
        factored_pair f;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          uint4 x0, x1;
          x_of(2 * sp + h, x0, x1);
          f.half_step(h, lo[ci][2 * sp + h], hi[ci][2 * sp + h], x0, x1, negcorr);
        }
        auto pick = [&](int r) { return __ushort_as_half((unsigned short)(sc[ci][r][sp >> 1] >> (16 * (sp & 1)))); };
        if (ok) f.add_to(accs[sp % NACC], pick(0), pick(1));
      }
    } else {
#pragma unroll
      for (int s = 0; s < NSTEPS; ++s) {
        uint4 x0, x1;
        x_of(s, x0, x1);
        const bool ok = ci + 1 < NCH || ((s ^ flip) << 6) < vb;
        auto pick = [&](int r) { return __ushort_as_half((unsigned short)(WT == 2 ? sc[ci][r][s >> 1] >> (16 * ((s ^ flip) & 1)) : 0)); };
        step<WT>(accs, s, lo[ci][s], hi[ci][s], x0, x1, pick(0), pick(1), WT == 2 && ok ? sums[s ^ flip] : 0.f);
      }
    }
  }
  float v0, v1;
  segment_sums(accs, lane, v0, v1);
#pragma unroll
  for (int o = DUAL ? 8 : 16; o >= 4; o >>= 1) {  // (DUAL: a row's upper four segments are empty)
    v0 += __shfl_xor_sync(0xffffffffu, v0, o);
    v1 += __shfl_xor_sync(0xffffffffu, v1, o);
  }
  if (mine) store_pair<WT, EPI>(p, bt, bi, po, pr, v0, v1, pos, gate_scale);
}

template <int WT, int EPI, int NW, bool LONG = false>
int launch_one(const gemv_params& p, cudaStream_t stream, int pdl, size_t smem, int grid, int sw, int pf_bytes, const gemv_batch& bt = gemv_batch{}) {
  static bool attr_done[16] = {};
  int dev = 0;
  LCU_CUDA(cudaGetDevice(&dev));
  if (dev < 16 && !attr_done[dev]) {
    LCU_CUDA(cudaFuncSetAttribute(gemv1_kernel<WT, EPI, NW, LONG>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024));
    attr_done[dev] = true;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3((NW + 1) * 32);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl ? 1 : 0;
  LCU_CUDA(cudaLaunchKernelEx(&cfg, gemv1_kernel<WT, EPI, NW, LONG>, p, sw, pf_bytes, bt));
  return LCU_OK;
}

template <int WT, int EPI, int NCH, bool DUAL>
int launch_held_shape(const gemv_params& p, cudaStream_t stream, int pdl, int warps, int grid, const gemv_batch& bt) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(warps * 32);
  cfg.dynamicSmemBytes = row_layout_of<WT>(p.K, WT != 3 && p.norm_w != nullptr).total;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl ? 1 : 0;
  LCU_CUDA(cudaLaunchKernelEx(&cfg, gemv_held_kernel<WT, EPI, NCH, DUAL>, p, bt));
  return LCU_OK;
}

// Whether a launch's weights are held in registers, and its shape.
struct held_plan {
  int chunks = 0, warps = 0, grid = 0;  // chunks 0: no
  bool dual = false;
};
int g_held_mode = -1;  // -1 = by the rule, 0 = never
// At most twelve warps per SM, one wave beside the kernels around it (4096 wide u8, 13.8 for wo: 2 % slower held).  Rows: a launch
// between ring kernels gains nothing, so lengths stop where a model's other launches are too large - bfloat16 rows of 4 KiB
// (Filulix, 2048 wide) 185 -> 188 us, rows of two chunks of 1536 wide fp16 (8 KiB) 152 -> 173, where 1024 wide ones (5.5 KiB), whose
// step is held as a whole, gain 156 -> 143.  In between, two-byte weights are held in small launches only.  Steps in us, ring / held
// (every multiple of 256 columns, 10 layers fp16, 4 bfloat16):
//   two chunks, wo of fp16:   2304 wide 370 / 377, 2560 423 / 434, 3072 491 / 511: four warps per SM (w2 of 1024 columns has 3.5)
//   rows of 2.5 and 3 KiB:    wo of 1280 239.1 / 241.7, of 1536 246.4 / 254.4 (but 3.5 and 4 KiB: 1792 281 / 274, 2048 298 / 290);
//                             Filulix 1280 121 / 123, 1408 122 / 127, 1536 128 / 132, Zibovik 1280 154 / 156, 1408 159 / 162, 1536 168 / 170
//                             (1152: 116.4 / 116.4 and 149.9 / 148.7): three, but for picked experts (Zibovik 768 140 / 125, 1024 145 / 131)
// 8-bit weights gain or are level at every width.  Every launch of a tensor-parallel step (its step number is set) stays on the ring, the one
// that neither waits for other GPUs nor publishes to them - layer 0's wq|wk|wv - too: ring kernels are loaded ahead of the first step, in
// which other GPUs' bounded waits run while a launch stalls in loading its kernel.
constexpr int HELD_WARPS_PER_SM = 12, HELD_WARPS_TWO_CHUNKS = 4, HELD_WARPS_LONG_CHUNK = 3;
template <class PairsOf>
held_plan plan_held(int wt, int epi, const gemv_params& p, int n, PairsOf pairs_of, int sms, bool picked = false) {
  held_plan h;
  if (g_held_mode == 0 || wt == 1 || (wt == 2 && p.bs != 64 && p.bs != 128) || p.seq != nullptr) return h;
  const int rowbytes = p.K * (wt == 2 ? 1 : 2), chunks = (rowbytes + 4095) / 4096;
  if (rowbytes > (wt == 3 ? 3072 : epi == EPI_PLAIN ? 6144 : 4096)) return h;
  long long single = 0, two = 0;
  for (int i = 0; i < n; ++i) {
    single += pairs_of(i);
    two += (pairs_of(i) + 1) / 2;
  }
  h.dual = rowbytes <= 2048 && single > 4 * sms;
  const long long units = h.dual ? two : single;
  int most = HELD_WARPS_PER_SM;
  if (wt != 2 && chunks == 2) most = HELD_WARPS_TWO_CHUNKS;
  else if (wt != 2 && !picked && rowbytes > 2304 && rowbytes <= 3072) most = HELD_WARPS_LONG_CHUNK;
  if (units > most * sms) return h;
  h.warps = std::max(((int)units + sms - 1) / sms, p.norm_w ? 4 : 2);
  h.warps = std::max(std::min(h.warps, chunks == 1 ? held_warps<1> : held_warps<2>), (p.K / 8 + ROW_VEC * 32 - 1) / (ROW_VEC * 32));
  if (h.warps > (chunks == 1 ? held_warps<1> : held_warps<2>)) return h;  // (a thread holds ROW_VEC vectors of the row)
  for (int i = 0; i < n; ++i) h.grid += ((h.dual ? (pairs_of(i) + 1) / 2 : pairs_of(i)) + h.warps - 1) / h.warps;
  h.chunks = chunks;
  return h;
}
template <int WT, int EPI>
int launch_held(const held_plan& h, const gemv_params& p, cudaStream_t stream, int pdl, const gemv_batch& bt = gemv_batch{}) {
  if (h.dual) return launch_held_shape<WT, EPI, 1, true>(p, stream, pdl, h.warps, h.grid, bt);
  if constexpr (EPI == EPI_PLAIN && WT != 3)
    if (h.chunks == 2) return launch_held_shape<WT, EPI, 2, false>(p, stream, pdl, h.warps, h.grid, bt);
  return launch_held_shape<WT, EPI, 1, false>(p, stream, pdl, h.warps, h.grid, bt);
}

}  // namespace

namespace {
struct gemv1_config {
  int wt, nw, sw, grid, pf;
  bool long_norm;  // a normalised fp16 row of more than ROW_VEC vectors per thread
  size_t smem;
};
int configure(const gemv_params& p, int sms, gemv1_config& c) {
  const gemv_tuning& t = gemv_tuning_ref();
  const bool q = p.bs != 0;
  // weight type of the kernel: fp16; u8 with the reference's per-weight rounding; u8 with factored scales
  const int wt = !q ? 0 : ((t.int8_factored && p.bs >= 64) ? 2 : 1);
  const size_t stage_bytes = wt == 2 ? 2 * geom<2>::ROWB + 2 * geom<2>::SC_ROW : wt == 1 ? 2 * geom<1>::ROWB + 2 * geom<1>::SC_ROW : 2 * geom<0>::ROWB;
  const bool norm = p.norm_w != nullptr;
  const size_t fixed = SMEM_FIXED + (wt == 0 ? row_layout_of<0>(p.K, norm) : wt == 1 ? row_layout_of<1>(p.K, norm) : row_layout_of<2>(p.K, norm)).total;
  // CTAs per SM: as many as asked for that still fit with a two-deep ring per warp (the factored u8 kernel is
  // latency-bound and compiled for three); then the deepest ring that keeps them resident
  int cps = wt == 2 ? t.ctas_per_sm_int8 : t.ctas_per_sm;
  if (cps < 1) cps = 1;
  if (cps > 3) cps = 3;
  auto fits = [&](int warps, int stages, int ctas) { return fixed + (size_t)warps * stages * stage_bytes <= (size_t)(228 * 1024) / ctas - 1024; };
  while (cps > 1 && !fits(4, 2, cps)) --cps;
  // factored u8 kernels that cannot have three CTAs of four consumer warps per SM take five consumer warps per CTA
  // when those fit (a long activation row: w2 of every model, every matrix of the larger models)
  int nw = 4;
  if (wt == 2 && cps < 3 && t.consumer_warps_int8 != 4 && fits(5, 2, cps)) nw = 5;
  const bool long_norm = wt == 0 && norm && p.K > ROW_VEC * 8 * 4 * 32;
  int want_sw = wt == 2 ? t.warp_stages_int8 : t.warp_stages;
  // Normalised fp16 rows of more than 6144 values: two stages are enough, and with three the CTAs of an SM take all of its shared memory.
  // Three / two, us: w1|w3 7168 wide 84.3 / 82.3, 8192 106.9 / 102.7, output matrix 78.4 / 75.5, a step of 4 layers 1114 / 1080; but 5120
  // wide 44.9 / 46.8.
  if (long_norm && p.K > 6144) want_sw = std::min(want_sw, 2);
  int sw = want_sw < 2 ? 2 : (want_sw > MAX_SW ? MAX_SW : want_sw);
  while (sw > 2 && !fits(nw, sw, cps)) --sw;
  const size_t smem = fixed + (size_t)nw * sw * stage_bytes;
  LCU_REQUIRE(smem <= 227 * 1024, "gemv: a row of K=%d does not fit in shared memory", p.K);
  const int pairs = p.n_mats * p.rows_per_mat / 2;
  c.wt = wt;
  c.long_norm = long_norm;
  c.nw = nw;
  c.sw = sw;
  c.grid = sms * cps > pairs ? pairs : sms * cps;
  c.pf = t.prefetch_kb_per_cta * 1024;
  c.smem = smem;
  return LCU_OK;
}
}  // namespace

void gemv_held_mode(int mode) { g_held_mode = mode; }

// Loads every single-row kernel on the current device (the CUDA runtime loads a kernel at its first use; a first decode
// step whose launches stall one after the other in that loading would leave the other GPUs of a tensor-parallel step
// waiting far longer than their bounded waits allow).
int gemv_single_row_preload() {
  cudaFuncAttributes fa;
#define LCU_PRELOAD(WTV, E, NWV) LCU_CUDA(cudaFuncGetAttributes(&fa, gemv1_kernel<WTV, E, NWV>));
#define LCU_PRELOAD_E(E) LCU_PRELOAD(0, E, 4) LCU_PRELOAD(1, E, 4) LCU_PRELOAD(2, E, 4) LCU_PRELOAD(2, E, 5)
  LCU_PRELOAD_E(EPI_PLAIN)
  LCU_PRELOAD_E(EPI_ROPE_KV)
  LCU_PRELOAD_E(EPI_SILU)
#undef LCU_PRELOAD_E
#undef LCU_PRELOAD
#define LCU_PRELOAD_LONG(E) LCU_CUDA(cudaFuncGetAttributes(&fa, gemv1_kernel<0, E, 4, true>));
  LCU_PRELOAD_LONG(EPI_PLAIN)
  LCU_PRELOAD_LONG(EPI_ROPE_KV)
  LCU_PRELOAD_LONG(EPI_SILU)
#undef LCU_PRELOAD_LONG
  return LCU_OK;
}

int gemv_plan_single_row(const gemv_params& p, int epilogue, int sms, int* chunks, int* warps, int* grid) {
  gemv1_config c;
  const int rc = configure(p, sms, c);
  if (rc) return rc;
  const held_plan h = plan_held(c.wt, epilogue, p, 1, [&](int) { return p.n_mats * p.rows_per_mat / 2; }, sms);
  *chunks = h.chunks;
  *warps = h.chunks ? h.warps : c.nw;
  *grid = h.chunks ? h.grid : c.grid;
  return LCU_OK;
}

// m == 1 entry used by launch_gemv (argument checks are done there)
int launch_gemv_single_row(const gemv_params& p, int epilogue, cudaStream_t stream, int pdl, int sms) {
  gemv1_config c;
  int rc = configure(p, sms, c);
  if (rc) return rc;
  const int wt = c.wt, nw = c.nw, sw = c.sw, grid = c.grid, pf = c.pf;
  const size_t smem = c.smem;
  const held_plan h = plan_held(wt, epilogue, p, 1, [&](int) { return p.n_mats * p.rows_per_mat / 2; }, sms);
  if (h.chunks) {
#define LCU_HELD_CASE(E) \
  case E: return wt == 0 ? launch_held<0, E>(h, p, stream, pdl) : launch_held<2, E>(h, p, stream, pdl);
    switch (epilogue) {
      LCU_HELD_CASE(EPI_PLAIN)
      LCU_HELD_CASE(EPI_ROPE_KV)
      LCU_HELD_CASE(EPI_SILU)
    }
#undef LCU_HELD_CASE
  }
#define LCU_GEMV1_CASE(E)                                                                  \
  case E:                                                                                  \
    if (c.long_norm) return launch_one<0, E, 4, true>(p, stream, pdl, smem, grid, sw, pf); \
    if (wt == 0) return launch_one<0, E, 4>(p, stream, pdl, smem, grid, sw, pf);           \
    if (wt == 1) return launch_one<1, E, 4>(p, stream, pdl, smem, grid, sw, pf);           \
    if (nw == 5) return launch_one<2, E, 5>(p, stream, pdl, smem, grid, sw, pf);           \
    return launch_one<2, E, 4>(p, stream, pdl, smem, grid, sw, pf);
  switch (epilogue) {
    LCU_GEMV1_CASE(EPI_PLAIN)
    LCU_GEMV1_CASE(EPI_ROPE_KV)
    LCU_GEMV1_CASE(EPI_SILU)
  }
#undef LCU_GEMV1_CASE
  LCU_REQUIRE(false, "gemv: unknown epilogue %d", epilogue);
}

int launch_gemv_bf16(const gemv_batch& b, int K, int* err, cudaStream_t stream, int pdl) {
  LCU_REQUIRE(b.n >= 1 && b.n <= GEMV_MAX_BATCH, "gemv: %d matrices outside 1..%d", b.n, GEMV_MAX_BATCH);
  LCU_REQUIRE(K > 0 && K % 256 == 0, "gemv: K=%d must be a positive multiple of 256", K);
  long long total = 0;
  for (int i = 0; i < b.n; ++i) {
    LCU_REQUIRE(b.rows[i] > 0 && b.rows[i] % 2 == 0, "gemv: row count %d must be even", b.rows[i]);
    LCU_REQUIRE((((uintptr_t)b.w[i] | (uintptr_t)b.x[i]) & 15) == 0 && ((uintptr_t)b.out[i] & 7) == 0, "gemv: unaligned operand of matrix %d", i);
    total += b.rows[i] / 2;
  }
  gemv_params p{};
  p.n_mats = 1;
  p.rows_per_mat = (int)(2 * total);
  p.K = K;
  p.m = 1;
  p.err = err;
  gemv_batch bt = b;
  const held_plan h = plan_held(3, EPI_PLAIN, p, b.n, [&](int i) { return b.rows[i] / 2; }, gemv_sm_count(), b.choice != nullptr);
  if (h.chunks) {
    bt.first_cta[0] = 0;
    for (int i = 0; i < b.n; ++i) bt.first_cta[i + 1] = bt.first_cta[i] + ((h.dual ? (b.rows[i] / 2 + 1) / 2 : b.rows[i] / 2) + h.warps - 1) / h.warps;
    return launch_held<3, EPI_PLAIN>(h, p, stream, pdl, bt);
  }
  gemv1_config c;
  int rc = configure(p, gemv_sm_count(), c);
  if (rc) return rc;
  // CTAs are dealt to the matrices in proportion to their rows, at least one each
  const int spare = c.grid > b.n ? c.grid - b.n : 0;
  long long seen = 0;
  for (int i = 0; i < b.n; ++i) {
    bt.first_cta[i] = i + (int)(spare * seen / total);
    seen += b.rows[i] / 2;
  }
  bt.first_cta[b.n] = b.n + spare;
  return launch_one<3, EPI_PLAIN, 4>(p, stream, pdl, c.smem, b.n + spare, c.sw, c.pf, bt);
}

int launch_gemv_bf16_gated(void* out, const void* x, const void* w13, int f, int K, int* err, cudaStream_t stream, int pdl) {
  LCU_REQUIRE(K > 0 && K % 256 == 0 && f > 0, "gemv: K=%d must be a positive multiple of 256", K);
  LCU_REQUIRE((((uintptr_t)w13 | (uintptr_t)x) & 15) == 0, "gemv: unaligned operand");
  gemv_params p{};
  p.w[0] = w13;
  p.w[1] = reinterpret_cast<const uint8_t*>(w13) + (size_t)f * K * 2;
  p.n_mats = 2;
  p.rows_per_mat = f;
  p.K = K;
  p.m = 1;
  p.x = reinterpret_cast<const __half*>(x);
  p.out = reinterpret_cast<__half*>(out);
  p.err = err;
  const held_plan h = plan_held(3, EPI_SILU, p, 1, [&](int) { return f; }, gemv_sm_count());
  if (h.chunks) return launch_held<3, EPI_SILU>(h, p, stream, pdl);
  gemv1_config c;
  int rc = configure(p, gemv_sm_count(), c);
  if (rc) return rc;
  return launch_one<3, EPI_SILU, 4>(p, stream, pdl, c.smem, c.grid, c.sw, c.pf);
}

int launch_gemv_bf16_gated_picked(const gemv_batch& b, int f, int K, int* err, cudaStream_t stream, int pdl) {
  LCU_REQUIRE(b.n >= 1 && b.n <= GEMV_MAX_BATCH && b.choice && b.gate_scale, "gemv: %d picked matrices outside 1..%d", b.n, GEMV_MAX_BATCH);
  LCU_REQUIRE(K > 0 && K % 256 == 0 && f > 0, "gemv: K=%d must be a positive multiple of 256", K);
  LCU_REQUIRE(f % (1 << b.gate_shift) == 0, "gemv: %d rows in blocks of %d", f, 1 << b.gate_shift);
  LCU_REQUIRE((((uintptr_t)b.w[0] | (uintptr_t)b.x[0] | b.choice_bytes) & 15) == 0, "gemv: unaligned operand");
  gemv_params p{};
  p.n_mats = 2;
  p.rows_per_mat = f * b.n;
  p.K = K;
  p.m = 1;
  p.x = reinterpret_cast<const __half*>(b.x[0]);
  p.err = err;
  gemv_batch bt = b;
  for (int i = 0; i < b.n; ++i) {
    bt.w[i] = b.w[0];
    bt.rows[i] = 2 * f;
  }
  const held_plan h = plan_held(3, EPI_SILU, p, b.n, [&](int) { return f; }, gemv_sm_count(), true);
  if (h.chunks) {
    for (int i = 0; i <= b.n; ++i) bt.first_cta[i] = i * (h.grid / b.n);
    return launch_held<3, EPI_SILU>(h, p, stream, pdl, bt);
  }
  gemv1_config c;
  int rc = configure(p, gemv_sm_count(), c);
  if (rc) return rc;
  const int per = std::max(1, c.grid / b.n);  // every matrix the same share of the CTAs
  for (int i = 0; i <= b.n; ++i) bt.first_cta[i] = i * per;
  return launch_one<3, EPI_SILU, 4>(p, stream, pdl, c.smem, per * b.n, c.sw, c.pf, bt);
}

}  // namespace lcu
