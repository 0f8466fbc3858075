// Device helpers of the tensor-core kernels (gemm_tc.cu, mlp_tc.cu): tcgen05
// descriptors, mbarriers, TMA loads, the swizzled tile layout, SiLU.  Internal.
#pragma once

#include <cuda.h>
#include <cuda_bf16.h>
#include <stdint.h>

namespace op2b {

// gemm_tc.cu: the current device's flag that a kernel sets when a bounded wait
// ran out (op2b_gemm_error reads it); null, with the error set, on failure
int *tc_error_flag(const char *what, int *device = nullptr);
// gemm_tc.cu: a K-major BF16 operand (rows x K, row stride ld elements) as a
// tensor map of 64 x 128 boxes with the 128-byte swizzle
bool tc_operand_map(CUtensorMap *m, const void *base, int rows, int K, long ld);
// gemm_tc.cu: an MN-major one (K rows of mn values) in boxes of 64 x 64
bool tc_operand_map_mn(CUtensorMap *m, const void *base, int mn, int K, long ld);
// gemm_tc.cu: a row-major BF16 or FP32 matrix as a tensor map of boxes of 64
// bytes x 32 rows with the 64-byte swizzle (what one warp stores at a time);
// false if it cannot be encoded
bool tc_store_map(CUtensorMap *m, void *base, bool f32, int cols, int rows, long ld,
                  int bytes = 64);


namespace {

constexpr int kTileM = 128;
constexpr int kTileN = 128;
constexpr int kTileK = 64;
constexpr int kStageBytes = kTileM * kTileK * 2;  // one operand tile (16 KiB)
constexpr unsigned long long kWaitNs = 2000000000ull;  // 2 s per mbarrier wait

__device__ __forceinline__ uint32_t smem_u32(const void *p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}

__device__ __forceinline__ unsigned long long globaltimer() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// shared-memory matrix descriptor, version 1 (sm_100), K-major with the
// 128-byte swizzle (layout type 2 in bits 61-63): start address >> 4 in bits
// 0-13, leading byte offset >> 4 in 16-29 (unused by a swizzled K-major
// operand whose K step fits in the 128-byte row; 1 by convention), stride
// byte offset >> 4 in 32-45 (1024: the distance between 8-row groups)
__device__ __forceinline__ uint64_t umma_desc(uint32_t saddr) {
  uint64_t d = 0;
  d |= (uint64_t)((saddr >> 4) & 0x3FFFu);
  d |= (uint64_t)1 << 16;
  d |= (uint64_t)(1024 >> 4) << 32;
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)2 << 61;
  return d;
}

// The same descriptor for an MN-major operand tile (128 MN x 64 K) as TMA
// writes it with the 128-byte swizzle: two boxes of 64 MN x 64 K, 8 KiB
// apart, each 64 rows of 128 bytes (64 MN values of one k) in 1024-byte
// groups of 8 rows.  In the canonical MN-major layout ((8,n),(8,k)) :
// ((1,LBO),(8,SBO)) in 16-byte units the leading byte offset is the 8 KiB
// between the two 64-wide MN blocks and the stride byte offset the 1024 bytes
// between groups of 8 k; a K step of 16 starts 2048 bytes further on.
__device__ __forceinline__ uint64_t umma_desc_mn(uint32_t saddr) {
  uint64_t d = 0;
  d |= (uint64_t)((saddr >> 4) & 0x3FFFu);
  d |= (uint64_t)(8192 >> 4) << 16;
  d |= (uint64_t)(1024 >> 4) << 32;
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)2 << 61;
  return d;
}

// instruction descriptor, kind::f16: FP32 accumulator (bits 4-5 = 1), A and B
// bf16 (bits 7-9 = 1, 10-12 = 1), both K-major (bits 15, 16 = 0), N >> 3 in
// bits 17-22, M >> 4 in bits 24-28
__device__ __forceinline__ uint32_t umma_idesc(int nt) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(nt >> 3) << 17) |
         ((uint32_t)(kTileM >> 4) << 24);
}

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count));
}

__device__ __forceinline__ bool mbar_try(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}

__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity) {
  if (mbar_try(bar, parity)) return true;
  const unsigned long long t0 = globaltimer();
  while (!mbar_try(bar, parity))
    if (globaltimer() - t0 > kWaitNs) return false;
  return true;
}

// SiLU and its derivative, z s and s (1 + z (1 - s)) with the sigmoid
// s = 1 / (1 + 2^(-z log2 e)): two special-function operations and two
// multiply-adds.  The flushing (.ftz) forms need no range checks around them and
// change nothing: a power small enough to be flushed vanishes in the sum with
// 1, and beyond z = -87, where the reciprocal is flushed, the value is 0 as
// it is for the library's fast division.  The last product is an ordinary
// one, so small z and small results keep their subnormal values.
__device__ __forceinline__ float sigmoid_approx(float z) {
  float e, s;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e) : "f"(z * -1.4426950408889634f));
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(s) : "f"(1.0f + e));
  return s;
}
__device__ __forceinline__ float silu(float z) { return z * sigmoid_approx(z); }
__device__ __forceinline__ float silu_grad(float z) {
  const float s = sigmoid_approx(z);
  return s * (1.0f + z * (1.0f - s));
}

// Shared-memory tile layout: K-major with the 128-byte swizzle.  Row r of the
// 128 x 64 tile is 128 bytes (64 bf16) at (r / 8) * 1024 + (r % 8) * 128; its
// 16-byte chunk j (k = 8j .. 8j+7) sits at chunk position j ^ (r % 8).  The
// XOR spreads both the k-contiguous and the transposed staging stores over
// all 32 banks; the tensor core undoes it from the descriptor's swizzle mode.
__device__ __forceinline__ uint32_t sw128(int row, int kc) {
  return (uint32_t)((row >> 3) * 1024 + (row & 7) * 128 + ((kc ^ (row & 7)) << 4));
}

__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes)
               : "memory");
}

__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap *map, int x, int y,
                                            uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes "
      "[%0], [%1, {%2, %3}], [%4];" ::"r"(dst),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(bar)
      : "memory");
}

__device__ __forceinline__ bool mbar_wait_or_fail(uint32_t bar, uint32_t parity,
                                                  const volatile int *fail) {
  if (mbar_try(bar, parity)) return true;
  const unsigned long long t0 = globaltimer();
  while (!mbar_try(bar, parity)) {
    if (*fail) return false;
    if (globaltimer() - t0 > kWaitNs) return false;
  }
  return true;
}

// 32 columns of the lane's row
__device__ __forceinline__ void tmem_ld32(uint32_t addr, float *v) {
  uint32_t r[32];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
      "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]),
        "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]),
        "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(addr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 32; i++) v[i] = __uint_as_float(r[i]);
}

// 16 floats to 16 BF16 (element 2i in the low half of word i)
__device__ __forceinline__ void pack16(const float *v, uint32_t *r) {
#pragma unroll
  for (int i = 0; i < 8; i++) {
    const __nv_bfloat162 t = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
    r[i] = *reinterpret_cast<const uint32_t *>(&t);
  }
}

// A warp's 32 rows x 64 bytes out to global memory by TMA: 16 words of each
// lane's row, to column x (in elements of the map) of the rows from y on.  `out`:
// the warp's 2 KiB of shared memory, in the 64-byte swizzle; rows past the
// matrix are clipped.  `add`: an FP32 reduction instead of a store.
// CH: 16-byte pieces of a row; 2 take half of that, 32 bytes a row, in the 32-byte
// swizzle.
constexpr int kOutBytes = 32 * 64;
template <int CH = 4>
__device__ __forceinline__ void put_rows(uint8_t *out, int lane, const CUtensorMap *m, int x, int y,
                                         bool inside, const uint32_t *v, bool add) {
  if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
  __syncwarp();
#pragma unroll
  for (int i = 0; i < CH; i++)
    *reinterpret_cast<uint4 *>(
        out + lane * (16 * CH) + ((i ^ (CH == 4 ? (lane >> 1) & 3 : (lane >> 2) & 1)) << 4)) =
        make_uint4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  __syncwarp();
  if (lane == 0 && inside) {
    if (add)
      asm volatile(
          "cp.reduce.async.bulk.tensor.2d.global.shared::cta.add.tile.bulk_group "
          "[%0, {%1, %2}], [%3];" ::"l"(reinterpret_cast<uint64_t>(m)),
          "r"(x), "r"(y), "r"(smem_u32(out))
          : "memory");
    else
      asm volatile(
          "cp.async.bulk.tensor.2d.global.shared::cta.tile.bulk_group "
          "[%0, {%1, %2}], [%3];" ::"l"(reinterpret_cast<uint64_t>(m)),
          "r"(x), "r"(y), "r"(smem_u32(out))
          : "memory");
    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
  }
}

}  // namespace
}  // namespace op2b
