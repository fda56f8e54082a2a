// Device-side building blocks shared by the tcgen05 kernels (prompt GEMM, prompt attention): TMA tile loads,
// tcgen05 fences / commit / MMA / tensor-memory loads, shared-memory matrix descriptors.
#pragma once
#include <cuda.h>
#include <cuda_bf16.h>

#include "common.cuh"

namespace lcu {

// 16-bit operand formats of the tcgen05 kind::f16 products: conversions, and the operand-format bits of the instruction
// descriptor (A at bit 7, B at bit 10; both operands always have the same format)
template <typename T>
struct tc_elem;
template <>
struct tc_elem<__half> {
  static constexpr uint32_t IDESC_FORMAT = 0;
  __device__ static __forceinline__ uint32_t pack(float a, float b) {
    const __half2 h = __floats2half2_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&h);
  }
  __device__ static __forceinline__ float2 unpack(uint32_t w) { return __half22float2(*reinterpret_cast<const __half2*>(&w)); }
};
template <>
struct tc_elem<__nv_bfloat16> {
  static constexpr uint32_t IDESC_FORMAT = (1u << 7) | (1u << 10);
  __device__ static __forceinline__ uint32_t pack(float a, float b) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&h);
  }
  __device__ static __forceinline__ float2 unpack(uint32_t w) { return __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&w)); }
};

__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t bar) {
  asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(dst),
               "l"(map), "r"(x), "r"(y), "r"(bar)
               : "memory");
}
// Single-thread instructions (tcgen05.mma, commit, tensor copies) take their operands from uniform registers.  Under
// `if (lane == 0)` the compiler cannot see that one thread runs and moves every operand over, for each instruction; issuing
// warps therefore keep their loops, waits and addresses common to the warp and elect a lane around the instructions alone.
// Tiles whose MMAs are short gain most - 509 rows of 4096 x 4096 on 256 x 128 pair tiles: 24.5 -> 19.1 us, 2000 of 2816 x 1024:
// 18.8 -> 14.5 - 256-wide pair tiles 1 to 2 %.
__device__ __forceinline__ bool tc_elect() {  // true for one lane (always the same) of a converged warp
  uint32_t one;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(one));
  return one != 0;
}
// mbar_wait by a whole warp with one outcome for all lanes
__device__ __forceinline__ bool mbar_wait_warp(uint32_t bar, uint32_t parity, int* err, int code, bool heed = true) {
  constexpr uint32_t ALL = 0xffffffffu;
  if (__all_sync(ALL, mbar_try_wait(bar, parity))) return true;
  const long long t0 = clock64();
  long long next_check = 400000;
  for (;;) {
    if (__all_sync(ALL, mbar_try_wait(bar, parity))) return true;
    const long long dt = clock64() - t0;
    if (__any_sync(ALL, dt > next_check)) {
      if (heed && __any_sync(ALL, *(volatile int*)err != 0)) return false;
      if (__any_sync(ALL, dt > 2000000000ll)) {
        atomicCAS(err, 0, code);
        return false;
      }
      next_check += 400000;
    }
  }
}
// place in a ring of n slots and the parity of its barriers on this lap
struct tc_ring {
  int slot = 0;
  uint32_t phase = 0;
  __device__ __forceinline__ void step(int n) {
    if (++slot == n) {
      slot = 0;
      phase ^= 1u;
    }
  }
};
// Tensor memory beside programmatic launches: tcgen05.alloc waits, without a limit, for the columns it asks for.  Kernels therefore
// allocate before griddepcontrol.launch_dependents (with a __syncthreads between): a CTA of a later kernel that already holds columns
// then never stands before an earlier kernel's CTA that still needs some.
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void tc_mma_f16(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
      "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// 32 lanes x 32 columns of fp32: thread t of the warp gets row (quadrant base + t), 32 consecutive columns
__device__ __forceinline__ void tc_ld_32x32(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
        "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]),
        "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]),
        "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
}

// shared-memory matrix descriptor of a K-major tile stored as 128-byte swizzled rows:
// start address (16-byte units), leading byte offset 1 (unused for swizzled K-major), stride byte offset
// 1024 (eight 128-byte rows form one swizzle atom), descriptor version 1, layout type 2 = 128-byte swizzle
__device__ __forceinline__ uint64_t smem_desc_sw128(uint32_t smem_addr) {
  uint64_t d = 0;
  d |= (uint64_t)((smem_addr & 0x3ffff) >> 4);
  d |= (uint64_t)1 << 16;
  d |= (uint64_t)(1024 >> 4) << 32;
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)2 << 61;
  return d;
}

// same for an MN-major operand (the N index is the contiguous one in memory: a [k][n] tile): rows of 64 n-elements
// (128 bytes, swizzled), 8 k-rows per 1024-byte atom (stride byte offset), `n_atom_stride` bytes between the atoms
// of successive 64-element n-blocks (leading byte offset)
__device__ __forceinline__ uint64_t smem_desc_sw128_mn(uint32_t smem_addr, uint32_t n_atom_stride) {
  uint64_t d = 0;
  d |= (uint64_t)((smem_addr & 0x3ffff) >> 4);
  d |= (uint64_t)((n_atom_stride >> 4) & 0x3fff) << 16;
  d |= (uint64_t)(1024 >> 4) << 32;
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)2 << 61;
  return d;
}
__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap* map, int x, int y, int z, uint32_t bar) {
  asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(dst),
               "l"(map), "r"(x), "r"(y), "r"(z), "r"(bar)
               : "memory");
}

// host: cuTensorMapEncodeTiled for fp16 tensors of rank 2 or 3 with 128-byte swizzle (gemm_tc.cu); dims / box innermost
// first, strides in bytes for dimensions 1 .. rank-1
// streamed: the tensor is read once from HBM (weights): L2 sector promotion 256 bytes instead of 128
int tc_encode_map(CUtensorMap* map, const void* ptr, int rank, const uint64_t* dims, const uint64_t* strides_bytes, const uint32_t* box,
                  bool streamed = false);

}  // namespace lcu
