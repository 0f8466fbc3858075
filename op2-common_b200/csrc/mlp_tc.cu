// The graph network's three-layer MLPs (Linear-SiLU-Linear-SiLU-Linear, hidden
// width 128) as ONE persistent tensor-core kernel a pass over the rows, forward
// (k_mlp_fwd).  A layer by layer product writes each hidden activation to
// memory and reads it back, and the edge MLP's input [e, h_src, h_dst] had to
// be gathered into a 384-wide array first; here
//   * the three weight matrices stay in shared memory (K-major, 128-byte
//     swizzle) for the whole kernel: 160 KiB for the edge MLP (K = 384);
//   * warps 0-2 load the 128-row input tile in 64-column blocks into a ring of
//     16 KiB stages: direct rows by TMA, rows of h that an index names by
//     cp.async, each from its own address, so no gathered copy exists;
//   * warp 3 issues the MMAs: layer 0 of a tile runs two tiles ahead, layers 1
//     and 2 as their operands appear, so the tensor core and the activations
//     of two tiles overlap;
//   * warps 4-19 are the epilogues, eight for even and eight for odd tiles (two
//     a TMEM lane quarter, 64 columns each): bias and SiLU on the FP32
//     accumulator, rounded to BF16 and put back into TENSOR MEMORY as the next
//     layer's A operand -- the hidden activations never leave the SM (in
//     training they are also stored);
//   * tensor memory: three 128-column accumulators taken in turn and two
//     64-column BF16 operands, all 512 columns.
// The MMAs run over K in the order of k_gemm_ws and every value is rounded
// where the layer-by-layer products rounded it, so the results are the same
// bits.  Every wait is bounded and also ends when another role has recorded a
// failure; the CTA then stops, waits (bounded) for the MMAs it issued, frees
// tensor memory and returns.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

#include "op2b_gnn.h"
#include "op2b_runtime.h"
#include "ring.h"
#include "tc.cuh"

namespace op2b {
namespace {

constexpr int kW = 128;                 // hidden width
constexpr int kProducerWarps = 3, kMmaWarp = 3, kEpiWarp0 = 4, kEpiWarps = 16;
// 20 warps: five a scheduler, whose 16K registers allow 96 a thread (k_mlp_fwd keeps 64
// to 96 bytes a thread on the stack for it, k_mlp_bwd 8 to 20)
constexpr int kMlpThreads = 32 * (kEpiWarp0 + kEpiWarps);

struct MlpPart {
  const __nv_bfloat16 *p;
  const int *rows;  // null: row r is row r
  long ld;
  int cols;
};

struct MlpArgs {
  int M, k0, nout;
  MlpPart part[3];
  const __nv_bfloat16 *W[3];
  const float *b[3];
  CUtensorMap mx[3];                 // the parts without rows
  CUtensorMap mz[2], ma[2], my;      // training: Z0, Z1, A0, A1 (rows of 128) and Y
  const __nv_bfloat16 *R;            // residual added to the result, or null
  long ldr;
  void *Y;
  long ldy;
  int *err;
};

__device__ __forceinline__ void cp_async16(uint32_t dst, const void *src, bool in) {
  const int n = in ? 16 : 0;  // 0 source bytes: the chunk is zero-filled
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(n)
               : "memory");
}

__device__ __forceinline__ void cp_async16(uint32_t dst, const void *src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}

__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}

__device__ __forceinline__ bool mbar_test(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}

__device__ __forceinline__ void umma_commit(uint32_t bar) {
  asm volatile(
      "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar)
      : "memory");
}

// D (+)= A B with A in shared memory / in tensor memory
__device__ __forceinline__ void umma_ss(uint32_t d, uint64_t da, uint64_t db, uint32_t idesc,
                                        uint32_t acc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d),
      "l"(da), "l"(db), "r"(idesc), "r"(acc));
}
__device__ __forceinline__ void umma_ts(uint32_t d, uint32_t a, uint64_t db, uint32_t idesc,
                                        uint32_t acc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(d),
      "r"(a), "l"(db), "r"(idesc), "r"(acc));
}

__device__ __forceinline__ void tmem_st8(uint32_t addr, const uint32_t *r) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"r"(addr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
      : "memory");
}

// one 32-byte sector of a lane's row
__device__ __forceinline__ void ld_sector(const void *p, uint32_t *r) {
  asm volatile("ld.global.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]),
                 "=r"(r[6]), "=r"(r[7])
               : "l"(p)
               : "memory");
}

// add 16 floats of shared memory (the same address in every lane)
__device__ __forceinline__ void add_smem16(float *v, const float *b) {
#pragma unroll
  for (int i = 0; i < 4; i++) {
    const float4 t = reinterpret_cast<const float4 *>(b)[i];
    v[4 * i] += t.x, v[4 * i + 1] += t.y, v[4 * i + 2] += t.z, v[4 * i + 3] += t.w;
  }
}

// a weight matrix [nrows][k] into K-major tiles of 128 rows x 64 columns,
// zeros past its rows and columns (asynchronous: wait for the cp.async group)
__device__ __forceinline__ void load_weights(uint32_t dst, const __nv_bfloat16 *w, int nrows,
                                             int k, int tiles) {
  for (int i = threadIdx.x; i < tiles * 1024; i += kMlpThreads) {
    const int t = i >> 10, row = (i >> 3) & 127, kc = i & 7, col = t * 64 + kc * 8;
    const bool in = row < nrows && col < k;
    cp_async16(dst + t * kStageBytes + sw128(row, kc), in ? w + (long)row * k + col : w, in);
  }
}

// Input stages of 128 rows x 64 columns: as many of four as the weights and the
// epilogue warps' staging leave room for.  The results leave by TMA from 2 KiB a
// warp, blocks of 32 columns (a lane's own row segments cost an L1 cycle a row and
// instruction), or from 1 KiB, blocks of 16, where only y is written and a third
// stage is to be had that way: 458,396 rows of the edge MLP took 172 us with four
// stages and y stored by the lanes, 162 with two and 2 KiB, 158 with three and 1 KiB.
// (The row gathers as TMA gathers of four rows: 222 us, 2.4K cycles a stage.)
__host__ __device__ constexpr bool mlp_narrow(int nc, bool store) { return nc == 6 && !store; }
__host__ __device__ constexpr int mlp_ring(int nc, bool store) {
  return nc < 6 ? 4 : mlp_narrow(nc, store) ? 3 : 2;
}
__host__ __device__ constexpr int mlp_out(int nc, bool store) {
  return mlp_narrow(nc, store) ? kOutBytes / 2 : kOutBytes;
}

// NC: 64-column blocks of the input (1, 2, 4 or 6); STORE: keep Z0, A0, Z1, A1
template <int NC, bool STORE>
__global__ void __launch_bounds__(kMlpThreads, 1) k_mlp_fwd(const __grid_constant__ MlpArgs g,
                                                            int ntiles) {
  constexpr int kRing = mlp_ring(NC, STORE);
  constexpr int kOut = mlp_out(NC, STORE);
  constexpr bool kNarrow = mlp_narrow(NC, STORE);
  constexpr int kTurns = kProducerWarps < kRing ? kProducerWarps : kRing;  // loading warps
  extern __shared__ uint8_t smem_raw[];
  uint8_t *smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  uint8_t *s_w0 = smem, *s_w1 = s_w0 + NC * kStageBytes, *s_w2 = s_w1 + 2 * kStageBytes;
  uint8_t *s_ring = s_w2 + 2 * kStageBytes;
  uint8_t *s_out = s_ring + kRing * kStageBytes;  // kOut a warp
  float *s_bias = reinterpret_cast<float *>(s_out + kEpiWarps * kOut);  // 3 x 128
  // full[kRing], empty[kRing], first_full[2], acc_full[2], h_full[2], d_free[3], done
  uint64_t *bars = reinterpret_cast<uint64_t *>(s_bias + 3 * kW);
  uint32_t &s_taddr = *reinterpret_cast<uint32_t *>(bars + 2 * kRing + 10);
  int &s_fail = *reinterpret_cast<int *>(&s_taddr + 1), *s_last = &s_fail + 1;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  auto full = [&](int s) { return smem_u32(&bars[s]); };
  auto empty = [&](int s) { return smem_u32(&bars[kRing + s]); };
  auto first_full = [&](int s) { return smem_u32(&bars[2 * kRing + s]); };  // layer 0 done
  auto acc_full = [&](int s) { return smem_u32(&bars[2 * kRing + 2 + s]); };  // layer 1, 2 done
  auto h_full = [&](int s) { return smem_u32(&bars[2 * kRing + 4 + s]); };
  auto d_free = [&](int d) { return smem_u32(&bars[2 * kRing + 6 + d]); };
  const uint32_t done = smem_u32(&bars[2 * kRing + 9]);
  volatile int *fail = &s_fail;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kRing; s++) {
      mbar_init(full(s), 1);
      mbar_init(empty(s), 1);
    }
    for (int s = 0; s < 2; s++) {
      mbar_init(first_full(s), 1);
      mbar_init(acc_full(s), 1);
      mbar_init(h_full(s), kEpiWarps / 2);
    }
    for (int d = 0; d < 3; d++) mbar_init(d_free(d), kEpiWarps / 2);
    mbar_init(done, 1);
    s_fail = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == kMmaWarp) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(&s_taddr)),
                 "r"(512u));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::);
  }
  load_weights(smem_u32(s_w0), g.W[0], kW, g.k0, NC);
  load_weights(smem_u32(s_w1), g.W[1], kW, kW, 2);
  load_weights(smem_u32(s_w2), g.W[2], g.nout, kW, 2);
  asm volatile("cp.async.commit_group;" ::: "memory");
  for (int i = threadIdx.x; i < 3 * kW; i += kMlpThreads) {
    const int l = i / kW, c = i - l * kW;
    s_bias[i] = l < 2 || c < g.nout ? g.b[l][c] : 0.0f;
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = s_taddr;
  const int nloc = ntiles > (int)blockIdx.x
                       ? (ntiles - 1 - (int)blockIdx.x) / (int)gridDim.x + 1
                       : 0;  // this CTA's tiles
  // the accumulator of local tile j, the BF16 operand of slot j & 1
  const auto acc_of = [&](int j) { return tmem + (uint32_t)(j % 3) * kW; };
  const auto hid_of = [&](int s) { return tmem + 3u * kW + (uint32_t)(s * 64); };

  if (warp < kProducerWarps) {
    // stage n is one warp's (n % kTurns): the warps' latencies overlap, and each
    // waits only for its own copies.  No more warps than stages: the wait for a
    // stage's last use then follows, in the same warp, one that implies the use
    // before.
    // Direct rows (zeros outside the rows and columns) come by TMA; of indexed ones
    // lane l copies chunk l % 8 of rows l / 8 + 4 i, eight lanes a row, each lane
    // holding four rows' indices.
    const int kc = lane & 7, r0 = lane >> 3;
    const uint32_t place0 = sw128(r0, kc), place1 = sw128(r0 + 4, kc);  // even, odd i
    const int total = warp < kTurns ? nloc * NC : 0;
    int n = warp, j = warp / NC, c = warp % NC;  // stage, local tile, block
    int idx[4] = {0, 0, 0, 0}, next[4] = {0, 0, 0, 0};
    auto load_rows = [&](int jn, int cn, int *to) {
      const int *rows = NC == 1 ? nullptr : g.part[cn >> 1].rows;
      if (!rows) return;
      const int m = (int)(blockIdx.x + (unsigned)jn * gridDim.x) * kTileM + lane;
#pragma unroll
      for (int i = 0; i < 4; i++) to[i] = m + 32 * i < g.M ? __ldg(rows + m + 32 * i) : 0;
    };
    if (n < total) load_rows(j, c, idx);
    for (; n < total; n += kTurns) {
      const int st = n % kRing;
      const int jn = c + kTurns >= NC ? j + (c + kTurns) / NC : j;
      const int cn = (c + kTurns) % NC;
      if (n + kTurns < total) load_rows(jn, cn, next);
      if (n >= kRing &&
          !__all_sync(0xffffffffu, mbar_wait_or_fail(empty(st), (uint32_t)((n / kRing - 1) & 1),
                                                     fail))) {
        if (lane == 0) atomicExch(&s_fail, 1);
        break;
      }
      const int m0 = (int)(blockIdx.x + (unsigned)j * gridDim.x) * kTileM;
      const MlpPart &P = g.part[NC == 1 ? 0 : c >> 1];
      const int cb = NC == 1 ? 0 : (c & 1) * 64;
      const uint32_t dst = smem_u32(s_ring + (size_t)st * kStageBytes);
      if (!P.rows) {
        if (lane == 0) {
          mbar_expect_tx(full(st), kStageBytes);
          tma_load_2d(dst, &g.mx[NC == 1 ? 0 : c >> 1], cb, m0, full(st));
        }
      } else {
        const char *base = reinterpret_cast<const char *>(P.p + cb + kc * 8);
        const long ld = 2 * P.ld;
        const bool whole = m0 + kTileM <= g.M;
#pragma unroll
        for (int i = 0; i < 32; i++) {
          const int r = __shfl_sync(0xffffffffu, idx[i >> 3], (4 * i & 31) + r0);
          const uint32_t to = dst + (i & 1 ? place1 : place0) + (i >> 1) * 1024;
          if (whole) cp_async16(to, base + r * ld);
          else cp_async16(to, base + r * ld, m0 + 4 * i + r0 < g.M);
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncwarp();
        if (lane == 0) mbar_arrive(full(st));
      }
#pragma unroll
      for (int i = 0; i < 4; i++) idx[i] = next[i];
      j = jn;
      c = cn;
    }
    if (lane == 0) s_last[warp] = n - kTurns;
  } else if (warp == kMmaWarp) {
    if (lane == 0) {  // MMA issuer: whatever has its operands next
      const uint32_t idesc = umma_idesc(kW), idesc2 = umma_idesc((g.nout + 15) & ~15);
      const uint32_t w0 = smem_u32(s_w0), w1 = smem_u32(s_w1), w2 = smem_u32(s_w2);
      int jf = 0, cf = 0, it = 0;            // layer 0: next tile and block; stages used
      int jn[2] = {0, 1}, layer[2] = {1, 1};  // per slot: next tile and layer (1 or 2)
      unsigned long long t0 = 0;
      while (jf < nloc || jn[0] < nloc || jn[1] < nloc) {
        bool moved = false;
#pragma unroll
        for (int s = 0; s < 2; s++) {
          const int j = jn[s];
          if (j >= nloc || !mbar_test(h_full(s), (uint32_t)((layer[s] - 1) & 1))) continue;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint32_t b = layer[s] == 1 ? w1 : w2;
#pragma unroll
          for (int k = 0; k < 8; k++)
            umma_ts(acc_of(j), hid_of(s) + k * 8,
                    umma_desc(b + (uint32_t)(k >> 2) * kStageBytes + (k & 3) * 32),
                    layer[s] == 1 ? idesc : idesc2, k > 0);
          umma_commit(acc_full(s));
          if (++layer[s] == 3) layer[s] = 1, jn[s] = j + 2;
          moved = true;
        }
        // the tile's accumulator must have been read, and the slot's tile
        // before it must be past layer 0 (one completion of first_full ahead)
        const int sf = jf & 1;
        if (jf < nloc && (jn[sf] == jf || (jn[sf] == jf - 2 && layer[sf] == 2)) &&
            (cf > 0 || jf < 3 || mbar_test(d_free(jf % 3), (uint32_t)((jf / 3 - 1) & 1)))) {
          const int st = it % kRing;
          if (mbar_test(full(st), (uint32_t)((it / kRing) & 1))) {
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t a = smem_u32(s_ring + (size_t)st * kStageBytes);
            const uint32_t b = w0 + (uint32_t)cf * kStageBytes;
#pragma unroll
            for (int k = 0; k < 4; k++)
              umma_ss(acc_of(jf), umma_desc(a + k * 32), umma_desc(b + k * 32), idesc,
                      cf + k > 0);
            umma_commit(empty(st));
            it++;
            if (++cf == NC) {
              umma_commit(first_full(sf));
              cf = 0;
              jf++;
            }
            moved = true;
          }
        }
        if (moved) {
          t0 = 0;
        } else {
          if (*fail) break;
          const unsigned long long t = globaltimer();
          if (t0 == 0) t0 = t;
          if (t - t0 > kWaitNs) {
            atomicExch(&s_fail, 1);
            break;
          }
        }
      }
      umma_commit(done);
    }
  } else if (warp >= kEpiWarp0) {  // epilogue
    const int s = (warp - kEpiWarp0) >> 3, quarter = warp & 3;
    const int c0 = (((warp - kEpiWarp0) >> 2) & 1) * 64;
    const uint32_t lanes = (uint32_t)(quarter * 32) << 16;
    const uint32_t hid = hid_of(s) + lanes + (uint32_t)(c0 / 2);
    uint8_t *out = s_out + (warp - kEpiWarp0) * kOut;
    bool ok = true;
    auto wait_for = [&](uint32_t bar, int n) {  // the n-th completion (from 0) of bar
      ok = __all_sync(0xffffffffu, mbar_wait_or_fail(bar, (uint32_t)(n & 1), fail));
      if (!ok && lane == 0) atomicExch(&s_fail, 1);
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      return ok;
    };
    auto signal = [&](uint32_t bar) {
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(bar);
    };
    for (int j = s, jj = 0; j < nloc; j += 2, jj++) {
      const long row = (long)(blockIdx.x + (unsigned)j * gridDim.x) * kTileM + quarter * 32 + lane;
      const bool live = row < g.M;
      const uint32_t acc = acc_of(j) + lanes + (uint32_t)c0;
      const int y0 = (int)row - lane;
#pragma unroll 1
      for (int l = 0; l < 2; l++) {
        if (!(l == 0 ? wait_for(first_full(s), jj) : wait_for(acc_full(s), 2 * jj))) break;
#pragma unroll
        for (int k = 0; k < 2; k++) {
          float v[32];
          tmem_ld32(acc + k * 32, v);
          uint32_t p[16];
#pragma unroll
          for (int m = 0; m < 2; m++) {
            float *u = v + 16 * m;
            add_smem16(u, s_bias + l * kW + c0 + k * 32 + m * 16);
            if (STORE) pack16(u, p + 8 * m);
          }
          if (STORE) put_rows(out, lane, &g.mz[l], c0 + k * 32, y0, y0 < g.M, p, false);
#pragma unroll
          for (int m = 0; m < 2; m++) {
            float *u = v + 16 * m;
#pragma unroll
            for (int i = 0; i < 16; i++) u[i] = silu(u[i]);
            pack16(u, p + 8 * m);
            tmem_st8(hid + k * 16 + m * 8, p + 8 * m);
          }
          if (STORE) put_rows(out, lane, &g.ma[l], c0 + k * 32, y0, y0 < g.M, p, false);
        }
        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
        signal(h_full(s));
      }
      if (!ok) break;
      if (g.nout == kW) {
        uint32_t res[4][8];
        if (g.R && live) {  // in flight while the last layer's MMAs run
#pragma unroll
          for (int k = 0; k < 4; k++) ld_sector(g.R + row * g.ldr + c0 + k * 16, res[k]);
        }
        if (!wait_for(acc_full(s), 2 * jj + 1)) break;
#pragma unroll
        for (int k = 0; k < 2; k++) {
          float v[32];
          tmem_ld32(acc + k * 32, v);
          if (k == 1) signal(d_free(j % 3));  // the accumulator has been read
          uint32_t p[16];
#pragma unroll
          for (int m = 0; m < 2; m++) {
            float *u = v + 16 * m;
            add_smem16(u, s_bias + 2 * kW + c0 + k * 32 + m * 16);
            if (g.R && live) {
#pragma unroll
              for (int i = 0; i < 8; i++) {
                const float2 t = __bfloat1622float2(
                    *reinterpret_cast<__nv_bfloat162 *>(&res[2 * k + m][i]));
                u[2 * i] += t.x;
                u[2 * i + 1] += t.y;
              }
            }
            pack16(u, p + 8 * m);
            if (kNarrow)
              put_rows<2>(out, lane, &g.my, c0 + k * 32 + m * 16, y0, y0 < g.M, p + 8 * m, false);
          }
          if (!kNarrow) put_rows(out, lane, &g.my, c0 + k * 32, y0, y0 < g.M, p, false);
        }
      } else {  // the decoder: nout <= 16 FP32 columns
        if (!wait_for(acc_full(s), 2 * jj + 1)) break;
        float v[32];
        if (c0 == 0) tmem_ld32(acc, v);
        signal(d_free(j % 3));
        if (c0 == 0 && live) {
          add_smem16(v, s_bias + 2 * kW);
          float *y = reinterpret_cast<float *>(g.Y) + row * g.ldy;
#pragma unroll
          for (int i = 0; i < 16; i += 4)
            if (i < g.nout)
              *reinterpret_cast<float4 *>(y + i) = make_float4(v[i], v[i + 1], v[i + 2], v[i + 3]);
        }
      }
    }
    if (lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
  }
  __syncthreads();
  // every issued MMA has finished once "done" has arrived
  if (threadIdx.x == 0 && !mbar_wait(done, 0u)) s_fail = 1;
  if (threadIdx.x == 0 && s_fail) {  // the loads that nobody waits for any more
#pragma unroll 1
    for (int st = 0; st < kRing; st++) {
      const int n = newest_in_flight(st, kRing, s_last, kTurns);
      if (n >= 0 && !g.part[NC == 1 ? 0 : n % NC >> 1].rows)
        mbar_wait(full(st), (uint32_t)((n / kRing) & 1));
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == kMmaWarp) {
    __syncwarp();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u));
  }
  if (threadIdx.x == 0 && s_fail) atomicExch(g.err, 1);
}

int sm_count(int dev) {
  int nsm = 0;
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  return nsm > 0 ? nsm : 148;
}

constexpr size_t mlp_smem(int nc, bool store) {
  return (size_t)(nc + 4 + mlp_ring(nc, store)) * kStageBytes + kEpiWarps * mlp_out(nc, store) +
         3 * kW * sizeof(float) + (2 * mlp_ring(nc, store) + 13) * sizeof(uint64_t) + 1024;
}

template <int NC, bool STORE>
cudaError_t launch_mlp(const MlpArgs &g, cudaStream_t s, int dev) {
  static bool attr[16] = {};  // per device, once
  if (!attr[dev]) {
    const cudaError_t e = cudaFuncSetAttribute(
        k_mlp_fwd<NC, STORE>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)mlp_smem(NC, STORE));
    if (e != cudaSuccess) return e;
    attr[dev] = true;
  }
  const int ntiles = (g.M + kTileM - 1) / kTileM;
  k_mlp_fwd<NC, STORE><<<std::min(ntiles, sm_count(dev)), kMlpThreads, mlp_smem(NC, STORE), s>>>(g,
                                                                                         ntiles);
  return cudaGetLastError();
}

template <bool STORE> cudaError_t launch_mlp(const MlpArgs &g, int nc, cudaStream_t s, int dev) {
  switch (nc) {
    case 1: return launch_mlp<1, STORE>(g, s, dev);
    case 2: return launch_mlp<2, STORE>(g, s, dev);
    case 4: return launch_mlp<4, STORE>(g, s, dev);
    default: return launch_mlp<6, STORE>(g, s, dev);
  }
}

// ---------------------------------------------------------------------------
// Backward through one MLP (k_mlp_bwd): from the gradient dy of its output,
//   dZ1 = (dy W2) silu'(Z1), dZ0 = (dZ1 W1) silu'(Z0), dx = dZ0 W0
// in one pass over the row tiles, organised as k_mlp_fwd: the weights stay in
// shared memory (here as MN-major B operands, so no transposed copy is made),
// dZ1 and dZ0 go from one product to the next through tensor memory and are
// also stored, as k_mlp_dw needs them.  dx leaves as FP32 column blocks of 128,
// each stored or added to what is there, so the sums that follow (dE, dH)
// need no pass of their own.  The results leave by TMA from 2 KiB a warp of
// shared memory (stores, and reductions for what is added): a lane's own row
// segments cost a shared-memory/L1 cycle a row and instruction, and the stores'
// bursts were what the kernel waited for (edge MLP of 635,000 rows 610 -> 408 us, about
// 5 TB/s of dy, Z, dZ and FP32 dx).  The products' and roundings' order is that of the
// layer-by-layer products.
struct MlpBwdArgs {
  int M, nout, kin, nparts;
  CUtensorMap mdy;
  const __nv_bfloat16 *W[3];
  const __nv_bfloat16 *Z0, *Z1;
  CUtensorMap md[2];   // dZ0, dZ1 (rows of 128)
  CUtensorMap mdx[3];  // dx
  int add[3];          // 1: dx += , 0: dx =
  int *err;
};
constexpr int kBwdRing = 2;            // stages of dy

// rows [0, nrows) of a weight matrix [nrows][ld], columns col0 .. col0 + 127, as
// MN-major tiles: for every 64 rows two boxes of 64 columns x 64 rows
__device__ __forceinline__ void load_weights_mn(uint32_t dst, const __nv_bfloat16 *w, int nrows,
                                                int ld, int col0, int tiles) {
  for (int i = threadIdx.x; i < tiles * 1024; i += kMlpThreads) {
    const int t = i >> 10, row = (i >> 4) & 63, c = i & 15, k = t * 64 + row, col = col0 + c * 8;
    const bool in = k < nrows && col < ld;
    cp_async16(dst + t * kStageBytes + (c >> 3) * (kStageBytes / 2) + sw128(row, c & 7),
               in ? w + (long)k * ld + col : w, in);
  }
}

// NP: 128-column blocks of dx (0 to 3)
template <int NP>
__global__ void __launch_bounds__(kMlpThreads, 1) k_mlp_bwd(const __grid_constant__ MlpBwdArgs g,
                                                            int ntiles) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t *smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  uint8_t *s_w2 = smem, *s_w1 = s_w2 + 2 * kStageBytes, *s_w0 = s_w1 + 2 * kStageBytes;
  uint8_t *s_ring = s_w0 + 2 * NP * kStageBytes;
  uint8_t *s_out = s_ring + kBwdRing * kStageBytes;
  // full[kBwdRing], empty[kBwdRing], acc_full[2], h_full[2], d_free[2], done
  uint64_t *bars = reinterpret_cast<uint64_t *>(s_out + kEpiWarps * kOutBytes);
  uint32_t &s_taddr = *reinterpret_cast<uint32_t *>(bars + 2 * kBwdRing + 7);
  int &s_fail = *reinterpret_cast<int *>(&s_taddr + 1), &s_loaded = *(&s_fail + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  auto full = [&](int s) { return smem_u32(&bars[s]); };
  auto empty = [&](int s) { return smem_u32(&bars[kBwdRing + s]); };
  auto acc_full = [&](int s) { return smem_u32(&bars[2 * kBwdRing + s]); };
  auto h_full = [&](int s) { return smem_u32(&bars[2 * kBwdRing + 2 + s]); };
  auto d_free = [&](int s) { return smem_u32(&bars[2 * kBwdRing + 4 + s]); };
  const uint32_t done = smem_u32(&bars[2 * kBwdRing + 6]);
  volatile int *fail = &s_fail;
  const int nkb = g.nout > 64 ? 2 : 1;  // 64-column blocks of dy

  if (threadIdx.x == 0) {
    for (int s = 0; s < kBwdRing; s++) {
      mbar_init(full(s), 1);
      mbar_init(empty(s), 1);
    }
    for (int s = 0; s < 2; s++) {
      mbar_init(acc_full(s), 1);
      mbar_init(h_full(s), kEpiWarps / 2);
      mbar_init(d_free(s), kEpiWarps / 2);
    }
    mbar_init(done, 1);
    s_fail = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == kMmaWarp) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(&s_taddr)),
                 "r"(512u));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::);
  }
  load_weights_mn(smem_u32(s_w2), g.W[2], g.nout, kW, 0, nkb);
  load_weights_mn(smem_u32(s_w1), g.W[1], kW, kW, 0, 2);
  for (int p = 0; p < NP; p++)
    load_weights_mn(smem_u32(s_w0 + 2 * p * kStageBytes), g.W[0], kW, g.kin, p * kW, 2);
  asm volatile("cp.async.commit_group;" ::: "memory");
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = s_taddr;
  const int nloc = ntiles > (int)blockIdx.x
                       ? (ntiles - 1 - (int)blockIdx.x) / (int)gridDim.x + 1
                       : 0;
  const auto acc_of = [&](int s) { return tmem + (uint32_t)s * kW; };
  const auto hid_of = [&](int s) { return tmem + 3u * kW + (uint32_t)(s * 64); };

  if (warp < kProducerWarps) {
    if (threadIdx.x == 0) {  // dy's blocks, zeros outside its rows and columns
      const int total = nloc * nkb;
      int n = 0;
      for (; n < total; n++) {
        const int st = n % kBwdRing;
        if (n >= kBwdRing &&
            !mbar_wait_or_fail(empty(st), (uint32_t)((n / kBwdRing - 1) & 1), fail)) {
          atomicExch(&s_fail, 1);
          break;
        }
        const int m0 = (int)(blockIdx.x + (unsigned)(n / nkb) * gridDim.x) * kTileM;
        mbar_expect_tx(full(st), kStageBytes);
        tma_load_2d(smem_u32(s_ring + (size_t)st * kStageBytes), &g.mdy, n % nkb * 64, m0,
                    full(st));
      }
      s_loaded = n;
    }
  } else if (warp == kMmaWarp) {
    if (lane == 0) {
      const uint32_t idesc = umma_idesc(kW) | 1u << 16;  // B MN-major
      const uint32_t w2 = smem_u32(s_w2), w1 = smem_u32(s_w1), w0 = smem_u32(s_w0);
      // a slot's phases: 0 dy W2 (block by block, in tile order over the slots),
      // 1 dZ1 W1, 2 .. NP + 1 the blocks of dZ0 W0
      int jn[2] = {0, 1}, ph[2] = {0, 0}, nh[2] = {0, 0}, nd[2] = {0, 0};
      int jf = 0, cf = 0, it = 0;
      unsigned long long t0 = 0;
      while (jn[0] < nloc || jn[1] < nloc) {
        bool moved = false;
#pragma unroll
        for (int s = 0; s < 2; s++) {
          if (jn[s] >= nloc) continue;
          if (ph[s] == 0) {
            if (jf != jn[s]) continue;  // dy's stages arrive in tile order
            // the accumulator has been read (the NP or one read of the tile before)
            if (cf == 0 && jf >= 2 && !mbar_test(d_free(s), (uint32_t)((nd[s] - 1) & 1))) continue;
            const int st = it % kBwdRing;
            if (!mbar_test(full(st), (uint32_t)((it / kBwdRing) & 1))) continue;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t a = smem_u32(s_ring + (size_t)st * kStageBytes);
            const uint32_t b = w2 + (uint32_t)cf * kStageBytes;
#pragma unroll
            for (int k = 0; k < 4; k++)
              umma_ss(acc_of(s), umma_desc(a + k * 32), umma_desc_mn(b + k * 2048), idesc,
                      cf + k > 0);
            umma_commit(empty(st));
            it++;
            if (++cf == nkb) {
              umma_commit(acc_full(s));
              cf = 0;
              jf++;
              ph[s] = 1;
            }
          } else {
            if (ph[s] <= 2) {
              if (!mbar_test(h_full(s), (uint32_t)(nh[s] & 1))) continue;
              nh[s]++;
            } else if (!mbar_test(d_free(s), (uint32_t)((nd[s] - 1) & 1))) {
              continue;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t b = ph[s] == 1 ? w1 : w0 + (uint32_t)(2 * (ph[s] - 2)) * kStageBytes;
#pragma unroll
            for (int k = 0; k < 8; k++)
              umma_ts(acc_of(s), hid_of(s) + k * 8,
                      umma_desc_mn(b + (uint32_t)(k >> 2) * kStageBytes + (k & 3) * 2048), idesc,
                      k > 0);
            umma_commit(acc_full(s));
            if (ph[s] >= 2 || NP == 0) nd[s]++;  // this product's accumulator is read to d_free
            if (++ph[s] == NP + 2) {
              ph[s] = 0;
              jn[s] += 2;
            }
          }
          moved = true;
        }
        if (moved) {
          t0 = 0;
        } else {
          if (*fail) break;
          const unsigned long long t = globaltimer();
          if (t0 == 0) t0 = t;
          if (t - t0 > kWaitNs) {
            atomicExch(&s_fail, 1);
            break;
          }
        }
      }
      umma_commit(done);
    }
  } else if (warp >= kEpiWarp0) {
    const int s = (warp - kEpiWarp0) >> 3, quarter = warp & 3;
    const int c0 = (((warp - kEpiWarp0) >> 2) & 1) * 64;
    const uint32_t lanes = (uint32_t)(quarter * 32) << 16;
    const uint32_t acc = acc_of(s) + lanes + (uint32_t)c0;
    const uint32_t hid = hid_of(s) + lanes + (uint32_t)(c0 / 2);
    uint8_t *out = s_out + (warp - kEpiWarp0) * kOutBytes;
    auto put = [&](const CUtensorMap *m, int x, int y, const uint32_t *v, bool add) {
      put_rows(out, lane, m, x, y, y < g.M, v, add);
    };
    bool ok = true;
    int na = 0;
    auto wait_acc = [&]() {
      ok = __all_sync(0xffffffffu, mbar_wait_or_fail(acc_full(s), (uint32_t)(na & 1), fail));
      if (!ok && lane == 0) atomicExch(&s_fail, 1);
      na++;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      return ok;
    };
    auto signal = [&](uint32_t bar) {
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(bar);
    };
    for (int j = s; j < nloc && ok; j += 2) {
      const long row = (long)(blockIdx.x + (unsigned)j * gridDim.x) * kTileM + quarter * 32 + lane;
      const bool live = row < g.M;
      const int y = (int)row - lane;
#pragma unroll 1
      for (int l = 1; l >= 0; l--) {  // dZ1, then dZ0
        const __nv_bfloat16 *Z = (l ? g.Z1 : g.Z0) + row * kW + c0;
        uint32_t z[4][8];
        if (live) {
#pragma unroll
          for (int k = 0; k < 4; k++) ld_sector(Z + k * 16, z[k]);
        }
        if (!wait_acc()) break;
#pragma unroll
        for (int k = 0; k < 2; k++) {
          float v[32];
          tmem_ld32(acc + k * 32, v);
          uint32_t p[16];
#pragma unroll
          for (int m = 0; m < 2; m++) {
            float *u = v + 16 * m;
            if (live) {
#pragma unroll
              for (int i = 0; i < 8; i++) {
                const float2 t =
                    __bfloat1622float2(*reinterpret_cast<__nv_bfloat162 *>(&z[2 * k + m][i]));
                u[2 * i] *= silu_grad(t.x);
                u[2 * i + 1] *= silu_grad(t.y);
              }
            }
            pack16(u, p + 8 * m);
            if (NP > 0 || l == 1) tmem_st8(hid + k * 16 + m * 8, p + 8 * m);
          }
          put(&g.md[l], c0 + k * 32, y, p, false);
        }
        if (NP > 0 || l == 1) {
          asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
          signal(h_full(s));
        } else {
          signal(d_free(s));
        }
      }
      if (!ok) break;
#pragma unroll 1
      for (int p = 0; p < NP; p++) {
        if (!wait_acc()) break;
#pragma unroll
        for (int k = 0; k < 2; k++) {
          float v[32];
          tmem_ld32(acc + k * 32, v);
          if (k == 1) signal(d_free(s));
#pragma unroll
          for (int m = 0; m < 2; m++)
            put(&g.mdx[p], c0 + k * 32 + m * 16, y, reinterpret_cast<const uint32_t *>(v + 16 * m),
                g.add[p] != 0);
        }
      }
    }
    if (lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
  }
  __syncthreads();
  if (threadIdx.x == 0 && !mbar_wait(done, 0u)) s_fail = 1;
  if (threadIdx.x == 0 && s_fail)  // the loads that nobody waits for any more
    for (int i = max(0, s_loaded - kBwdRing); i < s_loaded; i++)
      mbar_wait(full(i % kBwdRing), (uint32_t)((i / kBwdRing) & 1));
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == kMmaWarp) {
    __syncwarp();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u));
  }
  if (threadIdx.x == 0 && s_fail) atomicExch(g.err, 1);
}

// ---------------------------------------------------------------------------
// The weight and bias gradients of one MLP's three layers in one launch
// (k_mlp_dw): dW_l += d_l^T X_l and db_l += column sums of d_l, over all rows.
// The CTAs are shared out among the layers by the bytes each reads, and a CTA
// keeps its layer's whole 128 x (up to 384) gradient in tensor memory while it
// walks its share of the rows, 64 at a time: d is read once for all column
// blocks of X (the tiled product read it once a block), and X's indexed blocks come
// from their own rows (no gathered copy).  Operand tiles (64 rows x 128 columns, MN-major)
// arrive in a ring of 12 x 16 KiB: direct rows of a line or more by TMA, two boxes
// of 64 columns, from a warp of its own (a proxy fence between them had TMA's loads
// wait for one another), the others by cp.async (narrow rows: TMA takes as long for
// 16 bytes as for 128).  With all of them by cp.async, at most eight stages in
// flight, the edge MLP's 635,000 rows took 276 us, so 209.
// Four more warps hold the sums' rounding to that of the layer by layer products, whose
// CTAs add up a few thousand rows each: the tensor core's accumulation drifts with its
// length.  An accumulator is left after J.flush blocks of rows, each at blocks of its
// own.  Of one or two (128 x 128 each) the warps add it to a running sum in tensor
// memory, of three there is room for none and they add it to the gradient; the MMAs
// go on meanwhile in the free 128 columns (two: after the warps, the ring filling).
// And the warps add d's columns up, as products with ones of four blocks (mma.sync on
// ldmatrix's fragments: a tenth of the instructions of adding values one by one, which
// held up the producers, 8 us), those by FP32 additions with compensation.  Error against
// FP64 sums of the same operands at 635,000 rows, as a part of the norm, for one
// accumulator a CTA, now and layer by layer: dW1 2.3e-5, 2.2e-6, 2.3e-6; with a mean of one
// standard deviation 4.9e-5, 2.5e-6, 2.6e-6 and db1 1.3e-5, 9e-8, 2.5e-7.  In a training
// step the edge MLP's 635,000 rows take 215 us for 208 with one accumulator, the node MLP's
// 160,000 53 for 53, the edge encoder's 158 for 182.
struct MlpDwJob {
  const __nv_bfloat16 *d;  // [M][ldd], nout columns
  long ldd;
  int nout, kin, nparts;
  MlpPart part[3];
  float *gw, *gb;
  int cta0, ctas;  // the CTAs of the job
  int flush;       // blocks of 64 rows an accumulator
  int tma;         // bit t: operand t (d, then X's parts) by TMA
  CUtensorMap map[4];
};
struct MlpDwArgs {
  int M, njobs;
  MlpDwJob job[3];
  int *err;
};
constexpr int kDwRing = 12, kDwLag = 8;  // (12: every stage is always the same operand's)
constexpr int kDwProducers = 4, kDwSumWarp0 = 6, kDwSumWarps = 4;  // warps; 4: MMA, 5: TMA
constexpr int kDwThreads = 32 * (kDwSumWarp0 + kDwSumWarps);
constexpr int kDwStage = 4096;  // what a warp adds to the gradient at a time
constexpr size_t kDwSmem =
    (size_t)kDwRing * kStageBytes + kDwSumWarps * kDwStage + kW * 4 + (2 * kDwRing + 7) * 8 + 1024;

__device__ __forceinline__ void red_add4(float *p, float a, float b, float c, float d) {
  asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p), "f"(a), "f"(b), "f"(c),
               "f"(d)
               : "memory");
}

// four 8 x 8 blocks of BF16 from the rows that lanes 0-7, 8-15, .. point to, transposed
__device__ __forceinline__ void ld_blocks(uint32_t addr, uint32_t *r) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr)
               : "memory");
}

// c[0], c[1] += the sums of the lane's two columns (2 (lane % 4) and the next one of eight)
// over 16 rows: a product with ones, all of whose rows are the same
__device__ __forceinline__ void add_columns(float (&c)[4], uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%4,%4,%4}, "
      "{%5,%6}, {%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(0x3f803f80u), "r"(b0), "r"(b1));
}

// 32 rows n .. x 32 columns cc .. of an accumulator (plus the sum of the ones before it, if
// any), added to the gradient.  Through 4 KiB of shared memory, in the 128-byte swizzle,
// so that a reduction of the warp covers whole lines of four rows: by the lanes' own rows,
// 32 lines each, the reductions held up the producers' copies (edge MLP 226 us)
__device__ __forceinline__ void dw_add(const MlpDwJob &J, uint32_t acc, bool two, uint32_t sum, int n,
                                       int cc, uint8_t *stage, int lane) {
  float v[32];
  tmem_ld32(acc, v);
  if (two) {
    float u[32];
    tmem_ld32(sum, u);
#pragma unroll
    for (int i = 0; i < 32; i++) v[i] += u[i];
  }
  __syncwarp();
#pragma unroll
  for (int i = 0; i < 8; i++)
    *reinterpret_cast<float4 *>(stage + sw128(lane, i)) =
        make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
  __syncwarp();
  const int c = lane & 7;
  float *w = J.gw + (long)n * J.kin + cc + 4 * c;
#pragma unroll
  for (int i = 0; i < 8; i++) {
    const int r = 4 * i + (lane >> 3);
    const float4 t = *reinterpret_cast<const float4 *>(stage + sw128(r, c));
    if (n + r < J.nout && cc + 4 * c < J.kin) red_add4(w + (long)r * J.kin, t.x, t.y, t.z, t.w);
  }
}

// 32 columns of an accumulator into the sum of the ones before it (`first`: none)
__device__ __forceinline__ void dw_keep(uint32_t acc, uint32_t sum, bool first) {
  float v[32];
  tmem_ld32(acc, v);
  if (!first) {
    float u[32];
    tmem_ld32(sum, u);
#pragma unroll
    for (int i = 0; i < 32; i++) v[i] += u[i];
  }
#pragma unroll
  for (int i = 0; i < 32; i += 8) tmem_st8(sum + i, reinterpret_cast<const uint32_t *>(v + i));
}

__global__ void __launch_bounds__(kDwThreads, 1) k_mlp_dw(const __grid_constant__ MlpDwArgs g) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t *smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  uint8_t *s_ring = smem;
  uint8_t *s_stage = smem + (size_t)kDwRing * kStageBytes;
  float *s_sum = reinterpret_cast<float *>(s_stage + kDwSumWarps * kDwStage);
  uint64_t *bars = reinterpret_cast<uint64_t *>(s_sum + kW);
  uint32_t &s_taddr = *reinterpret_cast<uint32_t *>(bars + 2 * kDwRing + 3);
  // s_place[0-2]: the accumulators' places at the end, [3]: bit p: there is a sum of
  // earlier ones, [4]: stages that the TMA warp went past
  int &s_fail = *reinterpret_cast<int *>(&s_taddr + 1), *s_place = &s_fail + 1;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  auto full = [&](int s) { return smem_u32(&bars[s]); };
  auto empty = [&](int s) { return smem_u32(&bars[kDwRing + s]); };
  const uint32_t done = smem_u32(&bars[2 * kDwRing]);
  const uint32_t acc_full = smem_u32(&bars[2 * kDwRing + 1]);   // one to be added and left
  const uint32_t acc_empty = smem_u32(&bars[2 * kDwRing + 2]);  // it has been
  volatile int *fail = &s_fail;
  int q = 0;
  while (q + 1 < g.njobs && (int)blockIdx.x >= g.job[q + 1].cta0) q++;
  const MlpDwJob &J = g.job[q];
  const int P = J.nparts;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kDwRing; s++) {
      mbar_init(full(s), J.tma >> s % (P + 1) & 1 ? 1 : kDwProducers);
      mbar_init(empty(s), s % (P + 1) == 0 ? 1 + kDwSumWarps : 1);  // (d: and its sums)
    }
    mbar_init(done, 1);
    mbar_init(acc_full, 1);
    mbar_init(acc_empty, kDwSumWarps);
    s_fail = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == kDwProducers) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(&s_taddr)),
                 "r"(512u));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::);
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = s_taddr;
  // the CTA's blocks of 64 rows
  const long nblk = ((long)g.M + 63) / 64, me = (int)blockIdx.x - J.cta0;
  const int b0 = (int)(nblk * me / J.ctas), b1 = (int)(nblk * (me + 1) / J.ctas), nb = b1 - b0;
  // accumulator p's place (128 columns) in tensor memory.  Of one or three the MMAs go
  // on in the free place (one: 0 and 3 in turn), which the MMA and the sum warps
  // exchange alike; of one or two there is room for the sums of those left before
  int acc_at[3] = {0, 1, 2}, spare = 3;
  const bool sums = P < 3;
  auto sum_at = [&](int p) { return P == 1 ? 1 : 2 + p; };
  // the block after which accumulator p is left, each at blocks of its own (after the
  // last block all warps read them)
  int leave[3];
#pragma unroll
  for (int p = 0; p < 3; p++) leave[p] = J.flush - p * (J.flush / P) - 1;
  auto is_full = [&](int p, int b) {
    if (b != leave[p] || b + 1 == nb) return false;
    leave[p] += J.flush;
    return true;
  };
  auto exchange = [&](int p) {  // (p is a constant of an unrolled loop)
    const int t = acc_at[p];
    if (P != 2) {
      acc_at[p] = spare;
      spare = t;
    }
    return t;
  };

  const int tma = J.tma;
  if (warp < kDwProducers && tma != (2 << P) - 1) {
    // 16 lanes a row of 256 bytes: thread t copies chunk t % 16 of the rows
    // t / 16 + 8 i, so its place moves by 1024 bytes with i
    const int c = threadIdx.x & 15, r0 = threadIdx.x >> 4;
    const uint32_t place = smem_u32(s_ring) + (c >> 3) * (kStageBytes / 2) + sw128(r0, c & 7);
    int it = 0, handed = 0;
    bool ok = true;
    auto hand_on = [&](int upto) {
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (lane == 0)
        for (int s = handed; s < upto; s++)
          if (!(tma >> s % (P + 1) & 1)) mbar_arrive(full(s % kDwRing));
      handed = upto;
    };
    // the four operands' first chunk, row stride in bytes and whether the
    // thread's chunk lies inside the columns, in registers for the whole loop
    const char *x[4];
    long ld[4];
    bool incol[4];
    const int *idx[2];
#pragma unroll
    for (int t = 0; t < 4; t++) {
      const MlpPart &X = J.part[t > 0 ? t - 1 : 0];
      x[t] = reinterpret_cast<const char *>(t ? X.p : J.d);
      ld[t] = 2 * (t ? X.ld : J.ldd);
      incol[t] = t <= P && c * 8 < (t ? X.cols : J.nout);
      if (t >= 2) idx[t - 2] = X.rows;
    }
    const int M = g.M;
    int rows[2][8];
    auto load_rows = [&](int q, int b) {
#pragma unroll
      for (int i = 0; i < 8; i++) {
        const int r = b * 64 + r0 + 8 * i;
        rows[q][i] = idx[q] && r < M ? __ldg(idx[q] + r) : r;
      }
    };
    if (P > 1 && b0 < b1) load_rows(0, b0);
    if (P > 2 && b0 < b1) load_rows(1, b0);
    for (int b = b0; b < b1 && ok; b++) {
      const int m0 = b * 64 + r0;
      const bool whole = b * 64 + 64 <= M;
#pragma unroll
      for (int t = 0; t < 4; t++) {  // d, then X's blocks
        if (t > P) break;
        if (tma >> t & 1) {  // (an empty group: stages and groups count alike)
          asm volatile("cp.async.commit_group;" ::: "memory");
          it++;
          continue;
        }
        const int st = it % kDwRing;
        if (it >= kDwRing) {
          const uint32_t par = (uint32_t)((it / kDwRing - 1) & 1);
          if (!__all_sync(0xffffffffu, mbar_try(empty(st), par))) {
            if (handed < it) {
              asm volatile("cp.async.wait_group 0;" ::: "memory");
              hand_on(it);
            }
            ok = __all_sync(0xffffffffu, mbar_wait_or_fail(empty(st), par, fail));
            if (!ok) {
              if (lane == 0) atomicExch(&s_fail, 1);
              break;
            }
          }
        }
        const uint32_t dst = place + (uint32_t)st * kStageBytes;
        const char *src = x[t] + c * 16;
        if (whole && incol[t]) {
#pragma unroll
          for (int i = 0; i < 8; i++)
            cp_async16(dst + i * 1024, src + (t >= 2 ? rows[t >= 2 ? t - 2 : 0][i] : m0 + 8 * i) * ld[t]);
        } else {
#pragma unroll
          for (int i = 0; i < 8; i++) {
            const bool in = incol[t] && m0 + 8 * i < M;
            cp_async16(dst + i * 1024,
                       in ? src + (t >= 2 ? rows[t >= 2 ? t - 2 : 0][i] : m0 + 8 * i) * ld[t] : x[t],
                       in);
          }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
        if (t >= 2 && b + 1 < b1) load_rows(t - 2, b + 1);
        it++;
        if (it - handed > kDwLag) {
          asm volatile("cp.async.wait_group %0;" ::"n"(kDwLag) : "memory");
          hand_on(it - kDwLag);
        }
      }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    hand_on(it);
  } else if (warp == kDwProducers + 1 && lane == 0) {
    int it = 0;
    bool ok = true;
    for (int b = b0; b < b1 && ok; b++)
      for (int t = 0; t <= P; t++, it++) {
        if (!(tma >> t & 1)) continue;
        const int st = it % kDwRing;
        if (it >= kDwRing &&
            !mbar_wait_or_fail(empty(st), (uint32_t)((it / kDwRing - 1) & 1), fail)) {
          atomicExch(&s_fail, 1);
          ok = false;
          break;
        }
        const uint32_t to = smem_u32(s_ring + (size_t)st * kStageBytes);
        mbar_expect_tx(full(st), kStageBytes);  // (rows and columns outside: zeros)
        tma_load_2d(to, &J.map[t], 0, b * 64, full(st));
        tma_load_2d(to + kStageBytes / 2, &J.map[t], 64, b * 64, full(st));
      }
    s_place[4] = it;
  } else if (warp == kDwProducers && lane == 0) {
    const uint32_t idesc = umma_idesc(kW) | 1u << 15 | 1u << 16;  // A and B MN-major
    int it = 0, left = 0, kept = 0;
    bool ok = true, fresh[3] = {true, true, true};
    auto wait = [&](uint32_t bar, int n) {
      ok = ok && mbar_wait_or_fail(bar, (uint32_t)(n & 1), fail);
      if (!ok) atomicExch(&s_fail, 1);
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    };
    for (int b = 0; b < nb && ok; b++) {
      const int sd = it % kDwRing;
      wait(full(sd), it / kDwRing);
      it++;
      const uint32_t a = smem_u32(s_ring + (size_t)sd * kStageBytes);
      if (P == 2 && left > 0) wait(acc_empty, left - 1);  // (the ring fills meanwhile)
#pragma unroll
      for (int p = 0; p < 3; p++) {
        if (p >= P || !ok) break;
        const int st = it % kDwRing;
        wait(full(st), it / kDwRing);
        it++;
        if (!ok) break;
        const uint32_t x = smem_u32(s_ring + (size_t)st * kStageBytes);
#pragma unroll
        for (int k = 0; k < 4; k++)
          umma_ss(tmem + (uint32_t)(acc_at[p] * kW), umma_desc_mn(a + k * 2048),
                  umma_desc_mn(x + k * 2048), idesc, !fresh[p] || k > 0);
        fresh[p] = false;
        umma_commit(empty(st));
        if (is_full(p, b)) {
          if (left > 0) wait(acc_empty, left - 1);  // the place it goes on in has been read
          left++;
          umma_commit(acc_full);
          exchange(p);
          fresh[p] = true;
          kept |= 1 << p;
        }
      }
      if (!ok) break;
      umma_commit(empty(sd));
    }
    umma_commit(done);
#pragma unroll
    for (int p = 0; p < 3; p++) s_place[p] = acc_at[p];
    s_place[3] = sums ? kept : 0;
  } else if (warp >= kDwSumWarp0) {
    // a warp adds up 32 columns of d, a lane two of each eight; of an accumulator that is
    // left it takes its lane quarter
    const int w = warp - kDwSumWarp0;
    uint32_t place[2];  // of the lane's row in the blocks of 16 columns
#pragma unroll
    for (int u = 0; u < 2; u++) {
      const int c8 = 4 * w + 2 * u + (lane >> 4);
      place[u] = (uint32_t)((c8 >> 3) * (kStageBytes / 2)) + sw128((lane >> 3 & 1) * 8 + (lane & 7), c8 & 7);
    }
    float part[4][4] = {}, sum[4][2] = {}, rest[4][2] = {};
    int left = 0, kept = 0;
    bool ok = true;
    auto wait = [&](uint32_t bar, int n) {
      ok = __all_sync(0xffffffffu, mbar_wait_or_fail(bar, (uint32_t)(n & 1), fail));
      if (!ok && lane == 0) atomicExch(&s_fail, 1);
      return ok;
    };
    auto fold = [&]() {  // four blocks' part into the sum, with the last addition's
#pragma unroll           // rounding error made good, if there is one: infinities stay
      for (int i = 0; i < 4; i++)
#pragma unroll
        for (int k = 0; k < 2; k++) {
          const float y = part[i][k] - rest[i][k], t = sum[i][k] + y, e = (t - sum[i][k]) - y;
          rest[i][k] = fabsf(e) < INFINITY ? e : 0.0f;
          sum[i][k] = t;
          part[i][k] = 0.0f;
        }
    };
    for (int b = 0; b < nb && ok; b++) {
      const int it = b * (P + 1), st = it % kDwRing;
      if (!wait(full(st), it / kDwRing)) break;
      const uint32_t d = smem_u32(s_ring + (size_t)st * kStageBytes);
      uint32_t r[8][4];  // read at once, so that the stage is free again soon
#pragma unroll
      for (int k = 0; k < 4; k++)
#pragma unroll
        for (int u = 0; u < 2; u++) ld_blocks(d + place[u] + k * 2048, r[2 * k + u]);
      __syncwarp();
      if (lane == 0) mbar_arrive(empty(st));
#pragma unroll
      for (int k = 0; k < 8; k++) {
        add_columns(part[2 * (k & 1)], r[k][0], r[k][1]);
        add_columns(part[2 * (k & 1) + 1], r[k][2], r[k][3]);
      }
      if (b % 4 == 3 || b + 1 == nb) fold();
      int which = -1, at = 0;  // the accumulator left after this block: at most one, and its
                               // code once (unrolled, cold launches took 3 us longer)
#pragma unroll
      for (int p = 0; p < 3; p++)
        if (p < P && is_full(p, b)) which = p, at = exchange(p);
      if (which < 0) continue;
      if (!wait(acc_full, left)) break;
      left++;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t lanes = tmem + ((uint32_t)((warp & 3) * 32) << 16);
#pragma unroll 1
      for (int cc = 0; cc < kW; cc += 32) {
        const uint32_t acc = lanes + (uint32_t)(at * kW + cc);
        if (sums)
          dw_keep(acc, lanes + (uint32_t)(sum_at(which) * kW + cc), !(kept >> which & 1));
        else
          dw_add(J, acc, false, 0, (warp & 3) * 32, which * kW + cc, s_stage + w * kDwStage, lane);
      }
      kept |= 1 << which;
      if (sums) asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(acc_empty);
    }
    if (lane < 4)
#pragma unroll
      for (int i = 0; i < 4; i++)
        *reinterpret_cast<float2 *>(s_sum + 32 * w + 8 * i + 2 * lane) = make_float2(sum[i][0], sum[i][1]);
  }
  __syncthreads();
  if (threadIdx.x == 0 && !mbar_wait(done, 0u)) s_fail = 1;
  if (threadIdx.x == 0 && s_fail)  // the loads that nobody waits for any more
    for (int s = max(0, s_place[4] - kDwRing); s < s_place[4]; s++)
      if (tma >> s % (P + 1) & 1) mbar_wait(full(s % kDwRing), (uint32_t)((s / kDwRing) & 1));
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  if (!s_fail && nb > 0 && warp < 8) {
    // warps w and w + 4 share a lane quarter: row n of the gradient is a lane
    const uint32_t lanes = tmem + ((uint32_t)((warp & 3) * 32) << 16);
#pragma unroll 1
    for (int cc = (warp >> 2) * 32; cc < P * kW; cc += 64) {
      const int p = cc / kW;
      dw_add(J, lanes + (uint32_t)(s_place[p] * kW + cc % kW), s_place[3] >> p & 1,
             lanes + (uint32_t)(sum_at(p) * kW + cc % kW), (warp & 3) * 32, cc,
             s_ring + warp * kDwStage, lane);  // (the ring's stages have all been used)
    }
  } else if (!s_fail && nb > 0 && warp == 8) {
    for (int c = lane; c < J.nout; c += 32) atomicAdd(J.gb + c, s_sum[c]);
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == kDwProducers) {
    __syncwarp();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u));
  }
  if (threadIdx.x == 0 && s_fail) atomicExch(g.err, 1);
}

constexpr size_t mlp_bwd_smem(int np) {
  return (size_t)(4 + 2 * np + kBwdRing) * kStageBytes + kEpiWarps * kOutBytes +
         (2 * kBwdRing + 9) * sizeof(uint64_t) + 1024;
}

template <int NP> cudaError_t launch_mlp_bwd(const MlpBwdArgs &g, cudaStream_t s, int dev) {
  static bool attr[16] = {};  // per device, once
  if (!attr[dev]) {
    const cudaError_t e = cudaFuncSetAttribute(
        k_mlp_bwd<NP>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)mlp_bwd_smem(NP));
    if (e != cudaSuccess) return e;
    attr[dev] = true;
  }
  const int ntiles = (g.M + kTileM - 1) / kTileM;
  k_mlp_bwd<NP><<<std::min(ntiles, sm_count(dev)), kMlpThreads, mlp_bwd_smem(NP), s>>>(g, ntiles);
  return cudaGetLastError();
}

bool aligned(const void *p, uintptr_t n) { return (reinterpret_cast<uintptr_t>(p) & (n - 1)) == 0; }

}  // namespace
}  // namespace op2b

using namespace op2b;

extern "C" int op2b_gnn_mlp(int M, int nparts, const op2b_mlp_part *parts, const void *const *w,
                            const float *const *b, int nout, const void *R, long ldr, void *y,
                            long ldy, void *z0, void *a0, void *z1, void *a1, void *stream) {
  const char *what = "op2b_gnn_mlp";
  if (M < 0 || nparts < 1 || nparts > 3 || !parts || !w || !b || !y) {
    set_error("%s: bad sizes or null arguments", what);
    return -1;
  }
  MlpArgs g{};
  g.M = M;
  g.nout = nout;
  for (int i = 0; i < nparts; i++) {
    const op2b_mlp_part &p = parts[i];
    if (!p.x || !aligned(p.x, 16) || p.ld % 8 || p.cols % 8 || p.cols < 8 || p.ld < p.cols ||
        (nparts > 1 ? p.cols != kW : p.cols > 64 && p.cols != kW) || (i == 0 && p.rows)) {
      set_error("%s: input part %d: 128 columns (8 to 64, or 128, of a single part), 16-byte "
                "aligned rows; the first part is direct", what, i);
      return -1;
    }
    g.part[i] = MlpPart{(const __nv_bfloat16 *)p.x, p.rows, p.ld, p.cols};
    g.k0 += p.cols;
  }
  if (nout != kW && (nout > 16 || nout < 8 || nout % 8)) {
    set_error("%s: 128 BF16 outputs, or 8 or 16 FP32 outputs", what);
    return -1;
  }
  for (int l = 0; l < 3; l++) {
    if (!w[l] || !b[l] || !aligned(w[l], 16)) {
      set_error("%s: layer %d: null or unaligned weights", what, l);
      return -1;
    }
    g.W[l] = (const __nv_bfloat16 *)w[l];
    g.b[l] = b[l];
  }
  const bool store = z0 != nullptr;
  if ((a0 != nullptr) != store || (z1 != nullptr) != store || (a1 != nullptr) != store ||
      !aligned(z0, 32) || !aligned(a0, 32) || !aligned(z1, 32) || !aligned(a1, 32)) {
    set_error("%s: z0, a0, z1, a1: all or none, 32-byte aligned", what);
    return -1;
  }
  if (nout == kW ? !aligned(y, 32) || ldy % 16 || (R && (!aligned(R, 32) || ldr % 16))
                 : !aligned(y, 16) || ldy % 4 || R != nullptr) {
    set_error("%s: rows of the result (and the residual) need 32-byte alignment, FP32 rows 16-byte",
              what);
    return -1;
  }
  g.R = (const __nv_bfloat16 *)R;
  g.ldr = ldr;
  g.Y = y;
  g.ldy = ldy;
  if (M == 0) return 0;
  int dev = 0;
  g.err = tc_error_flag(what, &dev);
  if (!g.err) return -1;
  for (int i = 0; i < nparts; i++)
    if (!parts[i].rows &&
        !tc_operand_map(&g.mx[i], parts[i].x, M, parts[i].cols, parts[i].ld)) {
      set_error("%s: input part %d cannot be described as a tensor map", what, i);
      return -1;
    }
  const int nc = nparts == 1 ? (g.k0 <= 64 ? 1 : 2) : 2 * nparts;
  if ((store && !(tc_store_map(&g.mz[0], z0, false, kW, M, kW) &&
                  tc_store_map(&g.mz[1], z1, false, kW, M, kW) &&
                  tc_store_map(&g.ma[0], a0, false, kW, M, kW) &&
                  tc_store_map(&g.ma[1], a1, false, kW, M, kW))) ||
      (nout == kW &&
       !tc_store_map(&g.my, y, false, kW, M, ldy, mlp_narrow(nc, store) ? 32 : 64))) {
    set_error("%s: the results cannot be described as tensor maps", what);
    return -1;
  }
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const cudaError_t e = store ? launch_mlp<true>(g, nc, s, dev) : launch_mlp<false>(g, nc, s, dev);
  if (rt().initialised) rt().launches++;
  return cuda_ok(e, what) ? 0 : -1;
}

extern "C" int op2b_gnn_mlp_backward(int M, const void *dy, long ldy, int nout,
                                     const void *const *w, int kin, const void *z0,
                                     const void *z1, void *d0, void *d1, int nparts,
                                     float *const *dx, const long *lddx, const int *add,
                                     void *stream) {
  const char *what = "op2b_gnn_mlp_backward";
  if (M < 0 || !dy || !w || !z0 || !z1 || !d0 || !d1 || nparts < 0 || nparts > 3 ||
      (nparts > 0 && (!dx || !lddx || !add))) {
    set_error("%s: bad sizes or null arguments", what);
    return -1;
  }
  if ((nout != kW && (nout < 8 || nout > 16 || nout % 8)) || ldy % 8 || ldy < nout ||
      !aligned(dy, 16) || kin % 8 || kin < 8 || (nparts > 0 && kin != nparts * kW)) {
    set_error("%s: 128 (or 8 or 16) output columns in 16-byte aligned rows, 128 input columns a "
              "part", what);
    return -1;
  }
  if (!aligned(z0, 32) || !aligned(z1, 32) || !aligned(d0, 32) || !aligned(d1, 32)) {
    set_error("%s: z0, z1, d0, d1 need 32-byte alignment", what);
    return -1;
  }
  MlpBwdArgs g{};
  g.M = M;
  g.nout = nout;
  g.kin = kin;
  g.nparts = nparts;
  for (int l = 0; l < 3; l++) {
    if (!w[l] || !aligned(w[l], 16)) {
      set_error("%s: layer %d: null or unaligned weights", what, l);
      return -1;
    }
    g.W[l] = (const __nv_bfloat16 *)w[l];
  }
  g.Z0 = (const __nv_bfloat16 *)z0, g.Z1 = (const __nv_bfloat16 *)z1;
  for (int p = 0; p < nparts; p++) {
    if (!dx[p] || !aligned(dx[p], 32) || lddx[p] % 8 || lddx[p] < kW) {
      set_error("%s: dx part %d: 32-byte aligned rows of at least 128 floats", what, p);
      return -1;
    }
    g.add[p] = add[p];
  }
  if (M == 0) return 0;
  int dev = 0;
  g.err = tc_error_flag(what, &dev);
  if (!g.err) return -1;
  bool mapped = tc_operand_map(&g.mdy, dy, M, nout, ldy) && tc_store_map(&g.md[0], d0, false, kW, M, kW) &&
                tc_store_map(&g.md[1], d1, false, kW, M, kW);
  for (int p = 0; p < nparts; p++) mapped = mapped && tc_store_map(&g.mdx[p], dx[p], true, kW, M, lddx[p]);
  if (!mapped) {
    set_error("%s: dy or the results cannot be described as tensor maps", what);
    return -1;
  }
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const cudaError_t e = nparts == 0   ? launch_mlp_bwd<0>(g, s, dev)
                        : nparts == 1 ? launch_mlp_bwd<1>(g, s, dev)
                        : nparts == 2 ? launch_mlp_bwd<2>(g, s, dev)
                                      : launch_mlp_bwd<3>(g, s, dev);
  if (rt().initialised) rt().launches++;
  return cuda_ok(e, what) ? 0 : -1;
}

extern "C" int op2b_gnn_mlp_dw(int M, const void *const *d, const long *ldd, int nout,
                               int nparts, const op2b_mlp_part *parts, const void *a0,
                               const void *a1, float *const *gw, float *const *gb,
                               void *stream) {
  const char *what = "op2b_gnn_mlp_dw";
  if (M < 0 || !d || !ldd || nparts < 1 || nparts > 3 || !parts || !a0 || !a1 || !gw || !gb ||
      (nout != kW && (nout < 8 || nout > 16 || nout % 8))) {
    set_error("%s: bad sizes or null arguments", what);
    return -1;
  }
  MlpDwArgs g{};
  g.M = M;
  g.njobs = 3;
  const void *act[3] = {nullptr, a0, a1};
  for (int l = 0; l < 3; l++) {
    MlpDwJob &J = g.job[l];
    if (!d[l] || !gw[l] || !gb[l] || !aligned(d[l], 16) || !aligned(gw[l], 16) || ldd[l] % 8 ||
        (l && !aligned(act[l], 16))) {
      set_error("%s: layer %d: null or unaligned operands", what, l);
      return -1;
    }
    J.d = (const __nv_bfloat16 *)d[l];
    J.ldd = ldd[l];
    J.nout = l == 2 ? nout : kW;
    J.gw = gw[l];
    J.gb = gb[l];
    J.nparts = l ? 1 : nparts;
    if (l) {
      J.part[0] = MlpPart{(const __nv_bfloat16 *)act[l], nullptr, kW, kW};
      J.kin = kW;
      continue;
    }
    for (int i = 0; i < nparts; i++) {
      const op2b_mlp_part &p = parts[i];
      if (!p.x || !aligned(p.x, 16) || p.ld % 8 || p.cols % 8 || p.cols < 8 || p.cols > kW ||
          p.ld < p.cols || (nparts > 1 && p.cols != kW) || (i == 0 && p.rows)) {
        set_error("%s: input part %d: 128 columns (8 to 128 of a single part), 16-byte aligned "
                  "rows; the first part is direct", what, i);
        return -1;
      }
      J.part[i] = MlpPart{(const __nv_bfloat16 *)p.x, p.rows, p.ld, p.cols};
      J.kin += p.cols;
    }
  }
  if (M == 0) return 0;
  int dev = 0;
  g.err = tc_error_flag(what, &dev);
  if (!g.err) return -1;
  // CTAs by the operands a job reads, those that come by 16-byte copies (indexed or narrow
  // rows) counting twice, at least four blocks of rows each.  635,000 rows, graph
  // network's indices and 8-column encoder: 207 and 157 us; at one and a half 213 and 177,
  // alike 241 and 243
  const int nsm = sm_count(dev), most = std::max(1, ((M + 63) / 64 + 3) / 4);
  int total = 0, at = 0, cost[3];
  for (int l = 0; l < 3; l++) {
    const MlpDwJob &J = g.job[l];
    cost[l] = J.nout < 64 ? 2 : 1;
    for (int i = 0; i < J.nparts; i++) cost[l] += J.part[i].rows || J.part[i].cols < 64 ? 2 : 1;
    total += cost[l];
  }
  for (int l = 0; l < 3; l++) {
    MlpDwJob &J = g.job[l];
    J.cta0 = at;
    J.ctas = std::max(1, std::min(most, nsm * cost[l] / total));
    at += J.ctas;
    // an accumulator's rows: those of a split of the layer by layer product
    const int pieces = std::max(1, std::min(2 * nsm / J.nparts, M / 256));
    J.flush = ((M + pieces - 1) / pieces + 63) / 64;
    for (int t = 0; t <= J.nparts; t++) {
      const MlpPart &X = J.part[t ? t - 1 : 0];
      const int cols = t ? X.cols : J.nout;
      if (cols < 64 || (t && X.rows)) continue;
      if (!tc_operand_map_mn(&J.map[t], t ? X.p : J.d, cols, M, t ? X.ld : J.ldd)) {
        set_error("%s: an operand cannot be described as a tensor map", what);
        return -1;
      }
      J.tma |= 1 << t;
    }
  }
  static bool attr[16] = {};
  if (!attr[dev]) {
    if (!cuda_ok(cudaFuncSetAttribute(k_mlp_dw, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)kDwSmem), what))
      return -1;
    attr[dev] = true;
  }
  k_mlp_dw<<<at, kDwThreads, kDwSmem, static_cast<cudaStream_t>(stream)>>>(g);
  if (rt().initialised) rt().launches++;
  return cuda_ok(cudaGetLastError(), what) ? 0 : -1;
}
