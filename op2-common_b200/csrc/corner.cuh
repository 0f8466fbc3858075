// A cell's operands and sums over corner records (gather.h): res_calc and the
// bres_calc fused with it, shared by the Airfoil loops (airfoil_pipe.cu) and
// the batches (batch.cu).  Compiled without FMA contraction.  Internal.
#pragma once

#include <cuda_runtime.h>

#include "airfoil_math.cuh"
#include "vec.cuh"

namespace op2b {
namespace {

struct CornerRec {
  int4 o, cn;
  unsigned meta;
};

__device__ __forceinline__ CornerRec load_crec(const int4 *ro, const int4 *rcn,
                                               const unsigned *rmeta, int c, int ncell) {
  CornerRec r;
  if (c < ncell) {
    r.o = __ldg(ro + c);
    r.cn = __ldg(rcn + c);
    r.meta = __ldg(rmeta + c);
  } else {
    r.o = r.cn = make_int4(0, 0, 0, 0);
    r.meta = 0u;
  }
  return r;
}

template <typename T> struct CornerOps {
  T qc[4], rs[4], qo[4][4], ao[4], xn[4][2], ac;
  unsigned meta;
  int bnd[4];  // fused bres_calc: boundary flag of each boundary slot
};

// The fused res_calc + bres_calc keeps a boundary cell's boundary edges in the
// unused slots of its corner record (after its interior slots, in edge order):
// meta bit 6 marks such a slot, bits 2-5 give the edge's nodes as corners and
// o holds the boundary edge, whose flag is read from the bound dat.
struct BresLink {
  const int *bound;
};

template <typename T, bool BRES = false, bool ZERO = false>
__device__ __forceinline__ void load_corner_cell(CornerOps<T> &d, int c, const CornerRec &r,
                                                 const T *__restrict__ x,
                                                 const T *__restrict__ q,
                                                 const T *__restrict__ adt,
                                                 const T *__restrict__ res,
                                                 const BresLink &bl = BresLink{}) {
  Vec<T>::ld4(q + 4 * (size_t)c, d.qc);
  if constexpr (ZERO) {  // res known to be zero: the sums start from +0, as from the array
#pragma unroll
    for (int j = 0; j < 4; j++) d.rs[j] = (T)0;
  } else {
    Vec<T>::ld4_rw(res + 4 * (size_t)c, d.rs);
  }
  d.ac = __ldg(adt + c);
  const int nd[4] = {r.cn.x, r.cn.y, r.cn.z, r.cn.w};
#pragma unroll
  for (int j = 0; j < 4; j++) Vec<T>::ld2(x + 2 * (size_t)nd[j], d.xn[j][0], d.xn[j][1]);
  const int o[4] = {r.o.x, r.o.y, r.o.z, r.o.w};
#pragma unroll
  for (int s = 0; s < 4; s++) {
    const int oo = ((r.meta >> (8 * s)) & 1u) ? o[s] : c;
    Vec<T>::ld4(q + 4 * (size_t)oo, d.qo[s]);
    d.ao[s] = __ldg(adt + oo);
  }
  d.meta = r.meta;
  if constexpr (BRES) {
    if (r.meta & 0x40404040u) {  // a boundary cell: its boundary edges' flags
#pragma unroll
      for (int s = 0; s < 4; s++)
        d.bnd[s] = ((r.meta >> (8 * s + 6)) & 1u) ? __ldg(bl.bound + o[s]) : 0;
    }
  }
}

// coordinate `comp` of corner i (0..3), by selects (no local-memory indexing)
template <typename T>
__device__ __forceinline__ T corner(const T (&xn)[4][2], unsigned i, int comp) {
  const T lo = (i & 1u) ? xn[1][comp] : xn[0][comp];
  const T hi = (i & 1u) ? xn[3][comp] : xn[2][comp];
  return (i & 2u) ? hi : lo;
}

template <typename T, bool BRES = false>
__device__ __forceinline__ void compute_corner(const CornerOps<T> &d, int c, T *__restrict__ res,
                                               const AirConst<T> &k) {
  T acc[4] = {d.rs[0], d.rs[1], d.rs[2], d.rs[3]};
  T ric, pc;  // the cell's own terms, once for its <= 4 edges
  air_prim<T>(d.qc, k, ric, pc);
#pragma unroll
  for (int s = 0; s < 4; s++) {
    const unsigned m = (d.meta >> (8 * s)) & 0xffu;
    if (!(m & 1u)) continue;
    const unsigned a = (m >> 2) & 3u, b = (m >> 4) & 3u;
    const T x1x = corner<T>(d.xn, a, 0), x1y = corner<T>(d.xn, a, 1);
    const T x2x = corner<T>(d.xn, b, 0), x2y = corner<T>(d.xn, b, 1);
    T f[4], rio, po;
    air_prim<T>(d.qo[s], k, rio, po);
    if (m & 2u) {
      air_flux_prim<T>(x1x, x1y, x2x, x2y, d.qo[s], d.qc, rio, po, ric, pc, d.ao[s], d.ac, k, f);
#pragma unroll
      for (int j = 0; j < 4; j++) acc[j] -= f[j];
    } else {
      air_flux_prim<T>(x1x, x1y, x2x, x2y, d.qc, d.qo[s], ric, pc, rio, po, d.ac, d.ao[s], k, f);
#pragma unroll
      for (int j = 0; j < 4; j++) acc[j] += f[j];
    }
  }
  if constexpr (BRES) {
    // then bres_calc's increments: the boundary slots follow every interior
    // slot, in boundary-edge order (the two loops' order)
    if (d.meta & 0x40404040u) {
#pragma unroll
      for (int s = 0; s < 4; s++) {
        const unsigned m = (d.meta >> (8 * s)) & 0xffu;
        if (!(m & 0x40u)) continue;
        const unsigned a = (m >> 2) & 3u, b = (m >> 4) & 3u;
        T rr[4];
        air_bflux_prim<T>(corner<T>(d.xn, a, 0), corner<T>(d.xn, a, 1), corner<T>(d.xn, b, 0),
                          corner<T>(d.xn, b, 1), d.qc, ric, pc, d.ac, d.bnd[s], k, rr);
        if (d.bnd[s] == 1) {  // a wall edge leaves components 0 and 3 untouched
          acc[1] += rr[1];
          acc[2] += rr[2];
        } else {
#pragma unroll
          for (int j = 0; j < 4; j++) acc[j] += rr[j];
        }
      }
    }
  }
  Vec<T>::st4(res + 4 * (size_t)c, acc);
}

}  // namespace
}  // namespace op2b
