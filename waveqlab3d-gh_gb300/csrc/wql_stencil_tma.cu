// TMA-pipelined stencil kernel for FP32 fields (the FP32-compensated mode):
// the same per-point update as the other stencil kernels,
//   DF <- A*DF + L(F),   F_out <- F + B*dt*DF   (Kahan-compensated),
// (scale_rates + set_rates + update_fields, src/fields.f90:49-171,
// src/JU_xJU_yJU_z6.f90:12-812 and 16141-16449, src/RHS_Interior.f90:133-274)
// on every plane of the block.
//
// The boundary and fault penalties of the face points (src/RHS_Interior.f90:
// 1516-1703, 1757-1772) and the PML damping of the slab points (:1782-2201)
// are folded into DF beforehand by the pre-kernels, so this kernel has no
// face- or slab-dependent work.
//
// A tile is 32 x 12 (q, r) points over a chunk of s planes; a CTA takes a
// tile (or, launched persistently, tiles in turn) and marches along its
// planes.  One
// producer thread streams each plane into shared memory with
// cp.async.bulk.tensor (TMA) through an NS-deep ring of stages guarded by
// mbarriers ("full" completes on the transaction bytes, "empty" when all
// consumer warps have read the stage):
//   main (plane s)   : the 9 field components on the tile plus a q halo of
//                      8 points each side (so every box starts on a 16-byte
//                      boundary and every q closure row of a tile is inside
//                      the box) and an r halo of 3 rows; J*metric_q on the
//                      q-extended rows, J*metric_r on the r-extended columns,
//                      the remaining 7 coefficients, the rates DF and the
//                      compensation C on the tile;
//   lead (plane s+3) : the 9 field components and J*metric_s on the tile.
// Two roles of consumer threads cover the tile, each thread two neighbouring q
// points with packed FP32 instructions: the stress threads difference the
// velocities and update the six stresses, the velocity threads form and
// difference the momentum fluxes and update the three velocities.  They share
// only the stage's data.  What bounded the kernel was a warp's own instruction
// chain, about 3000 cycles a plane whether four or six warps took the tile
// (one point a thread: 900 issue slots; two: 1100), longer than a plane's
// loads at the rate of HBM; with the roles each chain is half as long and an
// SM has twelve of them (three a scheduler).  2 x 201^3 curvilinear, per
// launch: 0.779 ms one point a thread, 0.756 two, 0.727 with the roles = 76 %
// of the measured HBM rate; 2 x 101/93x107x113 150, 150, 140 us.  32 x 8 tiles
// with three stages ran 0.757 ms there (more halo).
// A role keeps its three quantities of planes s-3..s+3 (velocities, or s-face
// fluxes) in registers (the first six read directly at the start of a chunk,
// then one pushed per step from the lead tile), so the s derivative of a
// central row needs no shared memory (lead planes outside 0..ns-1 load as
// zeros and are never used: the 12 s closure rows take the planes of their
// stencil that the window holds from it and read the at most three others
// from global memory); the q and r derivatives read the main box, the
// curvilinear q and r fluxes formed once per box point into the stage, over
// the metrics they come from, after the stress threads have taken theirs (one
// mbarrier phase from them, one among the velocity threads per step).  The r
// tiles follow the ownership rule of tile_span (the last tile is shifted to
// end on the last point), which keeps every r closure row inside tile + halo.
// DF, F_out and C are stored directly from registers.
//
// Every mbarrier wait is bounded; a wait that runs out sets *err and the
// thread leaves its loop (the producer first waits, again bounded, for the
// copies it issued).
#include <cuda.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <functional>
#include <utility>
#include <vector>

#include "wql_internal.h"
#include "wql_stencil.cuh"

namespace wql {
namespace {

template <bool CURV, int FD, int TQ_ = kTmaTQ>
struct TmaTile {
  static constexpr int TQ = TQ_, TR = tma_rows(TQ_), NC = TQ * TR;
  static constexpr int NS = CURV ? kTmaStages : 3;  // ring depth: what fits in shared memory
  static constexpr int NT = (NC / 2 + 31) / 32 * 32;  // consumer threads of a role: one per two q points, whole warps
  // r halo: 3 rows for the central operator, 4 for the upwind pair
  static constexpr int HR = FD ? 4 : 3;
  static constexpr int BQ = TQ + 16, BR = TR + 2 * HR;  // field box: q from q0-8, r from r0-HR
  static constexpr int NCC = CURV ? 7 : 3;         // tile coefficients: 6..12 or lambda, mu, 1/rho
  static constexpr int F_BOX = 9 * BR * BQ;          // words the field box copy delivers
  static constexpr int F_W = (F_BOX + 31) / 32 * 32;  // its slot, padded to 128 bytes
  static constexpr int CA_W = CURV ? 3 * TR * BQ : 0;
  static constexpr int CB_W = CURV ? 3 * BR * TQ : 0;
  static constexpr int CC_W = NCC * NC;
  static constexpr int LF_W = 9 * NC;  // lead fields (FD 1: velocities of s+4, then stresses of s+2)
  static constexpr int LC_W = CURV ? 3 * NC : 0;
  static constexpr int DF_W = 9 * NC;            // rates of the main plane
  // compensation of the main plane: 9 x NC bfloat16 in a slot of whole
  // 128-byte lines
  static constexpr int CK_BOX = 9 * NC * 2;  // bytes the copy delivers
  static constexpr int CK_W = (CK_BOX / 4 + 31) / 32 * 32;
  static constexpr int OFF_F = 0;
  static constexpr int OFF_CA = OFF_F + F_W;
  static constexpr int OFF_CB = OFF_CA + CA_W;
  static constexpr int OFF_CC = OFF_CB + CB_W;
  static constexpr int OFF_LF = OFF_CC + CC_W;
  static constexpr int OFF_LC = OFF_LF + LF_W;
  static constexpr int OFF_DF = OFF_LC + LC_W;
  static constexpr int OFF_CK = OFF_DF + DF_W;
  static constexpr int STAGE_W = OFF_CK + CK_W;
  static constexpr unsigned MAIN_BYTES = 4u * (F_BOX + CA_W + CB_W + CC_W + DF_W) + CK_BOX;
  static constexpr unsigned LEAD_BYTES = 4u * (LF_W + LC_W);
  // every sub-buffer starts on a 128-byte boundary
  static_assert(F_W % 32 == 0 && CA_W % 32 == 0 && CB_W % 32 == 0 && CC_W % 32 == 0 && LF_W % 32 == 0 &&
                    LC_W % 32 == 0 && DF_W % 32 == 0 && CK_W % 32 == 0,
                "stage sub-buffers must be multiples of 128 bytes");
};

__device__ __forceinline__ unsigned smem_u32(const void* p) {
  return (unsigned)__cvta_generic_to_shared(p);
}

__device__ __forceinline__ void mbar_init(uint64_t* b, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(b)), "r"(count) : "memory");
}

__device__ __forceinline__ void mbar_expect_tx(uint64_t* b, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(b)), "r"(bytes)
               : "memory");
}

__device__ __forceinline__ void mbar_arrive(uint64_t* b) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(b)) : "memory");
}

// One potentially blocking test of the phase with parity `parity`; the
// thread sleeps in hardware for at most about 0.5 ms before it returns false.
__device__ __forceinline__ bool mbar_try(uint64_t* b, unsigned parity) {
  unsigned ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n selp.u32 %0, 1, 0, p;\n}"
      : "=r"(ok)
      : "r"(smem_u32(b)), "r"(parity), "r"(500000u)
      : "memory");
  return ok != 0;
}

// Bounded wait for the phase of parity `parity` to complete: at most 8192
// blocking tests (a few seconds).
__device__ __forceinline__ bool mbar_wait(uint64_t* b, unsigned parity) {
  for (unsigned i = 0; i < 8192u; ++i)
    if (mbar_try(b, parity)) return true;
  return false;
}

__device__ __forceinline__ void tma_load_4d(void* dst, const CUtensorMap* map, uint64_t* bar, int c0, int c1,
                                            int c2, int c3) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, "
      "%5}], [%6];" ::"r"(smem_u32(dst)),
      "l"(map), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(smem_u32(bar))
      : "memory");
}

// Two FP32 values of neighbouring q points in one 64-bit register (the low
// word is the even point): Blackwell's packed FP32 instructions do both in
// one issue slot, each half rounded as the scalar instruction rounds it.
typedef unsigned long long f2;
__device__ __forceinline__ f2 pack(float a, float b) {
  f2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void unpack(f2 v, float& a, float& b) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ f2 add2(f2 a, f2 b) {
  f2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f2 sub2(f2 a, f2 b) {
  f2 r;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f2 mul2(f2 a, f2 b) {
  f2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c) {
  f2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ f2 dot3(f2 a0, f2 x0, f2 a1, f2 x1, f2 a2, f2 x2) {
  return fma2(a2, x2, fma2(a1, x1, mul2(a0, x0)));
}
// Two values rounded to the nearest bfloat16 (lo in the low half).
__device__ __forceinline__ unsigned bf16_pair(float lo, float hi) {
  unsigned r;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
  return r;
}

__device__ __forceinline__ f2 g2(const float* p) { return *reinterpret_cast<const f2*>(p); }

// s derivative of the three velocities (VEL) or momentum fluxes on a closure
// row (planes 0..5 and ns-6..ns-1).  The s window already holds most of the
// planes a closure row reads (planes s-3..s+3 for the central operator;
// velocities of s-2..s+4 and fluxes of s-4..s+2 for the upwind pair); the at
// most three planes of a row outside it are read from global memory.  Each row
// is a separate instantiation (the weights, offsets and window positions are
// compile-time constants, so the window stays in registers); the columns are
// summed in the order of the operator table, zero weights skipped.
template <bool CURV, int FD, bool VEL, int ROW, bool RIGHT, int T>
__device__ __forceinline__ void s_close_col(const VolumeArgs<float>& a, long long p, const f2 (&qv)[7][3],
                                            f2 (&acc)[3]) {
  constexpr float w = (float)s_close_w(FD, RIGHT, !VEL, ROW, T);
  constexpr int off = s_close_off(RIGHT, ROW, T);  // plane offset from s
  constexpr int iw = VEL ? s_close_vpos(FD, RIGHT, ROW, T) : s_close_fpos(FD, RIGHT, ROW, T);
  if constexpr (w != 0.0f) {
    f2 x[3];
    if constexpr (iw >= 0 && iw <= 6) {
#pragma unroll
      for (int c = 0; c < 3; ++c) x[c] = qv[iw][c];
    } else {
      const long long np = a.np, pp = p + off * ((long long)a.pq * a.nr);
      const float* F = a.Fin + pp;
      if constexpr (VEL) {
#pragma unroll
        for (int c = 0; c < 3; ++c) x[c] = g2(F + c * np);
      } else if constexpr (CURV) {
        const float* M = a.coef + pp;
        const f2 a0 = g2(M + 6 * np), a1 = g2(M + 7 * np), a2 = g2(M + 8 * np);
#pragma unroll
        for (int c = 0; c < 3; ++c)
          x[c] = dot3(a0, g2(F + sig(c, 0) * np), a1, g2(F + sig(c, 1) * np), a2, g2(F + sig(c, 2) * np));
      } else {
#pragma unroll
        for (int c = 0; c < 3; ++c) x[c] = g2(F + sig(c, 2) * np);
      }
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) acc[c] = fma2(pack(w, w), x[c], acc[c]);
  }
}

template <bool CURV, int FD, bool VEL, int ROW, bool RIGHT, int... T>
__device__ __forceinline__ void s_close_row(const VolumeArgs<float>& a, long long p, const f2 (&qv)[7][3], f2 (&o)[3],
                                            std::integer_sequence<int, T...>) {
#pragma unroll
  for (int c = 0; c < 3; ++c) o[c] = 0;
  (s_close_col<CURV, FD, VEL, ROW, RIGHT, T>(a, p, qv, o), ...);
}

// ks = sbp_kind(s, ns), nonzero: -1..-6 left rows 0..5, 1..6 right rows 0..5.
template <bool CURV, int FD, bool VEL>
__device__ __forceinline__ void s_closure(const VolumeArgs<float>& a, long long p, int ks, const f2 (&qv)[7][3],
                                          f2 (&o)[3]) {
  using Cols = std::make_integer_sequence<int, FD ? 10 : 9>;
  switch (ks) {
    case -1: s_close_row<CURV, FD, VEL, 0, false>(a, p, qv, o, Cols{}); break;
    case -2: s_close_row<CURV, FD, VEL, 1, false>(a, p, qv, o, Cols{}); break;
    case -3: s_close_row<CURV, FD, VEL, 2, false>(a, p, qv, o, Cols{}); break;
    case -4: s_close_row<CURV, FD, VEL, 3, false>(a, p, qv, o, Cols{}); break;
    case -5: s_close_row<CURV, FD, VEL, 4, false>(a, p, qv, o, Cols{}); break;
    case -6: s_close_row<CURV, FD, VEL, 5, false>(a, p, qv, o, Cols{}); break;
    case 1: s_close_row<CURV, FD, VEL, 0, true>(a, p, qv, o, Cols{}); break;
    case 2: s_close_row<CURV, FD, VEL, 1, true>(a, p, qv, o, Cols{}); break;
    case 3: s_close_row<CURV, FD, VEL, 2, true>(a, p, qv, o, Cols{}); break;
    case 4: s_close_row<CURV, FD, VEL, 3, true>(a, p, qv, o, Cols{}); break;
    case 5: s_close_row<CURV, FD, VEL, 4, true>(a, p, qv, o, Cols{}); break;
    default: s_close_row<CURV, FD, VEL, 5, true>(a, p, qv, o, Cols{}); break;
  }
}

// q derivative (index spacing) of three quantities of a pair of points: row(c)
// is the start of quantity c's row in the box, lq the box column of the even
// point; box columns lq-4 .. lq+5, five aligned pairs, serve both points.
// VEL: the velocities (the upwind pair's D+), else the fluxes (its D-).
template <int FD, bool VEL, typename Row>
__device__ __forceinline__ void deriv_q(Row&& row, int lq, int kq0, int kq1, int lleft, int lright, const float* tab,
                                        f2 (&o)[3]) {
  const float c1 = float(kC1), c2 = float(kC2), c3 = float(kC3);
  const float cf[7] = WQL_UP_CF;
  if (kq0 == 0 || kq1 == 0) {
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const float* x = row(c) + lq;
      const f2 m4 = g2(x - 4), m2 = g2(x - 2), z = g2(x), p2 = g2(x + 2), p4 = g2(x + 4);
      float x0, x1, a1, a2, a3, a4, b2, b3, b4, b5, u0, u1;  // a_k at -k, b_k at +k
      unpack(z, x0, x1);
      unpack(m2, a2, a1);
      unpack(m4, a4, a3);
      unpack(p2, b2, b3);
      unpack(p4, b4, b5);
      if (FD) {
        // offset by offset in ascending order, as the other axes: every order
        // that packs the even offsets rounds worse (errors of 60 steps 0.4 to
        // 2.5 % larger) and saves 1 % of the kernel at most
        const float x[10] = {a4, a3, a2, a1, x0, x1, b2, b3, b4, b5};  // -4 .. 5
#pragma unroll
        for (int i = 0; i < 7; ++i) {
          const float w = VEL ? cf[i] : -cf[6 - i];
          const int l = VEL ? i + 2 : i;
          u0 = i ? fmaf(w, x[l], u0) : w * x[l];
          u1 = i ? fmaf(w, x[l + 1], u1) : w * x[l + 1];
        }
      } else {
        // the nearest pair first, as in the other axes: the errors of 60 steps
        // are 3 % smaller than with the farthest first
        unpack(fma2(pack(c2, c2), sub2(p2, m2), pack(c1 * (x1 - a1), c1 * (b2 - x0))), u0, u1);
        u0 = fmaf(c3, b3 - a3, u0);
        u1 = fmaf(c3, b4 - a2, u1);
      }
      o[c] = pack(u0, u1);
    }
  }
  if (kq0 != 0 || kq1 != 0) {
    // one or both points on a closure row: both rows of a pair read the same
    // columns (points 0.. or n-1.., at box columns lleft.. or lright..) with
    // their own weights; the upwind pair's right rows swap its two tables
    const bool left = kq0 < 0;
    constexpr int NCOL = FD ? 10 : 9;
    const int r0 = kq0 ? (left ? -kq0 : kq0) - 1 : 0, r1 = kq1 ? (left ? -kq1 : kq1) - 1 : 0;
    const float sg0 = kq0 ? (left ? 1.0f : -1.0f) : 0.0f, sg1 = kq1 ? (left ? 1.0f : -1.0f) : 0.0f;
    const float* w = tab + (FD && (left != VEL) ? 60 : 0);
    const int l0 = left ? lleft : lright, dl = left ? 1 : -1;
    float u0[3], u1[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) u0[c] = u1[c] = 0.0f;
#pragma unroll 3
    for (int e = 0; e < NCOL; ++e) {
      const float v0 = sg0 * w[r0 * NCOL + e], v1 = sg1 * w[r1 * NCOL + e];
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        const float x = row(c)[l0 + e * dl];
        u0[c] += v0 * x;
        u1[c] += v1 * x;
      }
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      float i0 = 0.0f, i1 = 0.0f;
      if (kq0 == 0 || kq1 == 0) unpack(o[c], i0, i1);
      o[c] = pack(kq0 ? u0[c] : i0, kq1 ? u1[c] : i1);
    }
  }
}

// r derivative: val(l, c) is quantity c at box row l.
template <int FD, bool VEL, typename Val>
__device__ __forceinline__ void deriv_r(Val&& val, int lr, int kr, const float* tab, f2 (&o)[3]) {
  const float c1 = float(kC1), c2 = float(kC2), c3 = float(kC3);
  const float cf[7] = WQL_UP_CF;
  if (kr == 0 && FD) {
#pragma unroll
    for (int c = 0; c < 3; ++c) o[c] = 0;
#pragma unroll
    for (int i = 0; i < 7; ++i)
#pragma unroll
      for (int c = 0; c < 3; ++c)
        o[c] = VEL ? fma2(pack(cf[i], cf[i]), val(lr + i - 2, c), o[c])
                   : fma2(pack(-cf[6 - i], -cf[6 - i]), val(lr + i - 4, c), o[c]);
  } else if (kr == 0) {
#pragma unroll
    for (int c = 0; c < 3; ++c)
      o[c] = fma2(pack(c3, c3), sub2(val(lr + 3, c), val(lr - 3, c)),
                  fma2(pack(c2, c2), sub2(val(lr + 2, c), val(lr - 2, c)),
                       mul2(pack(c1, c1), sub2(val(lr + 1, c), val(lr - 1, c)))));
  } else {
    const bool left = kr < 0;
    constexpr int NCOL = FD ? 10 : 9;
    const int rw = (left ? -kr : kr) - 1;
    const float sgn = left ? 1.0f : -1.0f;
    const float* w = tab + (FD && (left != VEL) ? 60 : 0) + rw * NCOL;
    const int l0 = lr + (left ? -rw : rw), dl = left ? 1 : -1;
#pragma unroll
    for (int c = 0; c < 3; ++c) o[c] = 0;
#pragma unroll 3
    for (int e = 0; e < NCOL; ++e) {
      const float v = sgn * w[e];
#pragma unroll
      for (int c = 0; c < 3; ++c) o[c] = fma2(pack(v, v), val(l0 + e * dl, c), o[c]);
    }
  }
}

// s derivative of the window's three quantities.
template <bool CURV, int FD, bool VEL>
__device__ __forceinline__ void deriv_s(const VolumeArgs<float>& a, long long p, int ks, const f2 (&qv)[7][3],
                                        f2 (&o)[3]) {
  const float c1 = float(kC1), c2 = float(kC2), c3 = float(kC3);
  const float cf[7] = WQL_UP_CF;
  if (ks == 0 && FD) {
#pragma unroll
    for (int c = 0; c < 3; ++c) o[c] = 0;
#pragma unroll
    for (int i = 0; i < 7; ++i)
#pragma unroll
      for (int c = 0; c < 3; ++c)
        o[c] = VEL ? fma2(pack(cf[i], cf[i]), qv[i][c], o[c]) : fma2(pack(-cf[6 - i], -cf[6 - i]), qv[i][c], o[c]);
  } else if (ks == 0) {
#pragma unroll
    for (int c = 0; c < 3; ++c)
      o[c] = fma2(pack(c3, c3), sub2(qv[6][c], qv[0][c]),
                  fma2(pack(c2, c2), sub2(qv[5][c], qv[1][c]), mul2(pack(c1, c1), sub2(qv[4][c], qv[2][c]))));
  } else {
    s_closure<CURV, FD, VEL>(a, p, ks, qv, o);
  }
}

// The work of the consumer threads of one role on a tile's chunk.  VEL: the
// threads that difference the velocities and update the six stresses; else
// those that form and difference the momentum fluxes and update the three
// velocities.  Both roles cover every pair of points of the tile; they share
// nothing but the stage's data.
template <bool CURV, int FD, int TQW, bool VEL>
__device__ __forceinline__ bool tma_consume(const VolumeArgs<float>& a, float* sm, uint64_t* full, uint64_t* empty,
                                            uint64_t* fluxbar, uint64_t* metbar, int q0, const TileSpan& spr,
                                            int s_begin, int nstep, int tid, const float* tab, int tb) {
  using TL = TmaTile<CURV, FD, TQW>;
  constexpr int TQ = TL::TQ, TR = TL::TR, NC = TL::NC, NT = TL::NT, BQ = TL::BQ, BR = TL::BR, HR = TL::HR, NS = TL::NS;
  const int nq = a.nq, nr = a.nr, ns = a.ns, r0 = spr.origin;
  const int tx = 2 * (tid % (TQ / 2));
  static_assert(NT == NC / 2, "every thread of a role has a pair of points");
  const int ty = tid / (TQ / 2);
  const int q = q0 + tx, r = r0 + ty;
  // q = nq - 1 of an odd nq shares its pair with the pad column, which is
  // inside the row pitch: its values are computed from zeros and stored
  const bool own = q < nq && r >= spr.own_lo && r < spr.own_hi;
  const int kq0 = sbp_kind(q, nq), kq1 = q + 1 < nq ? sbp_kind(q + 1, nq) : 0, kr = sbp_kind(r, nr);
  // points whose DF the pre-kernels have set on a stage with A = 0: the
  // block's faces and the PML slabs (here the q and r sides, true for the
  // whole column)
  const int npml = a.npml;
  const bool fold_r = r == 0 || r == nr - 1 || (a.pml[2] && r < npml) || (a.pml[3] && r >= nr - npml);
  auto fold_q = [&](int i) {
    return i == 0 || i == nq - 1 || (a.pml[0] && i < npml) || (a.pml[1] && i >= nq - npml);
  };
  const bool fold0 = fold_r || fold_q(q), fold1 = fold_r || fold_q(q + 1);
  const long long np = a.np;
  const long long sts = (long long)a.pq * nr;
  const long long col = q + (long long)a.pq * r;
  const int lq = tx + 8, lr = ty + HR, li = ty * TQ + tx;
  const int lleft = 8 - q0, lright = nq - 1 - q0 + 8;  // box columns of points 0 and nq-1
  constexpr int W0 = FD ? (VEL ? -2 : -4) : -3;        // plane of the window's first entry, from s

  // s window: the three velocities, or the three s-face fluxes, of the seven
  // planes the operator reads.  Its first six entries come straight from
  // global memory, all loads in flight at once; planes outside the block stay
  // zero (only central rows read the window).
  f2 qv[7][3];
#pragma unroll
  for (int i = 0; i < 7; ++i) {
#pragma unroll
    for (int c = 0; c < 3; ++c) qv[i][c] = 0;
    const int pl = s_begin + W0 + i;
    if (i < 6 && pl >= 0 && pl < ns && q < nq && r < nr) {
      const long long pp = col + sts * pl;
      const float* F = a.Fin;
      if (VEL) {
#pragma unroll
        for (int c = 0; c < 3; ++c) qv[i][c] = g2(F + c * np + pp);
      } else if (CURV) {
        const f2 a0 = g2(a.coef + 6 * np + pp), a1 = g2(a.coef + 7 * np + pp), a2 = g2(a.coef + 8 * np + pp);
        f2 sg[6];
#pragma unroll
        for (int c = 0; c < 6; ++c) sg[c] = g2(F + (3 + c) * np + pp);
#pragma unroll
        for (int c = 0; c < 3; ++c) qv[i][c] = dot3(a0, sg[sig(c, 0) - 3], a1, sg[sig(c, 1) - 3], a2, sg[sig(c, 2) - 3]);
      } else {
#pragma unroll
        for (int c = 0; c < 3; ++c) qv[i][c] = g2(F + sig(c, 2) * np + pp);
      }
    }
  }

  for (int t = 0; t < nstep; ++t) {
    const int T = tb + t;
    const int st = T % NS;
    const int s = s_begin + t;  // output plane
    const int ks = sbp_kind(s, ns);
    const long long p = col + sts * s;
    if (!mbar_wait(&full[st], (T / NS) & 1)) {
      atomicExch(a.err, 2);
      return false;
    }
    float* S = sm + st * TL::STAGE_W;
    float* FB = S + TL::OFF_F;
    float* CA = S + TL::OFF_CA;
    float* CB = S + TL::OFF_CB;
    const float* CC = S + TL::OFF_CC;
    const float* LF = S + TL::OFF_LF;
    auto fb2 = [&](int c, int rr, int qq) -> f2 { return g2(FB + (c * BR + rr) * BQ + qq); };
    const bool fold_s = s == 0 || s == ns - 1 || (a.pml[4] && s < npml) || (a.pml[5] && s >= ns - npml);
    const comp_t* CKs = reinterpret_cast<const comp_t*>(S + TL::OFF_CK);
    // DF <- A*DF + du and the compensated update of component c.  The
    // pre-kernels have folded the boundary and fault penalties and the PML
    // damping into DF of their points: DF + term/A, or the term itself on the
    // first stage (A = 0, where DF holds nothing else).
    auto update = [&](int c, f2 du) {
      const f2 f0 = fb2(c, lr, lq);
      const f2 dfs = g2(S + TL::OFF_DF + c * NC + li);
      f2 df;
      if (a.A != 0.0f) {
        df = fma2(pack(a.A, a.A), dfs, du);
      } else {
        float d0, d1;
        unpack(dfs, d0, d1);
        df = add2(pack(fold_s || fold0 ? d0 : 0.0f, fold_s || fold1 ? d1 : 0.0f), du);
      }
      *reinterpret_cast<f2*>(a.DF + c * np + p) = df;
      // -C of the pair: two bfloat16 (low half the even point), widened
      const unsigned ck = *reinterpret_cast<const unsigned*>(CKs + c * NC + li) ^ 0x80008000u;
      const f2 y = fma2(pack(a.Bdt, a.Bdt), df, pack(__uint_as_float(ck << 16), __uint_as_float(ck & 0xffff0000u)));
      const f2 tt = add2(f0, y);
      float e0, e1;
      unpack(sub2(sub2(tt, f0), y), e0, e1);
      *reinterpret_cast<unsigned*>(a.C + c * np + p) = bf16_pair(e0, e1);
      *reinterpret_cast<f2*>(a.Fout + c * np + p) = tt;
    };

    if constexpr (VEL) {
      // own J*metric_q and J*metric_r, before the flux threads write over them
      f2 mq[3], mr[3];
      if (CURV) {
#pragma unroll
        for (int j = 0; j < 3; ++j) {
          mq[j] = g2(CA + (j * TR + ty) * BQ + lq);
          mr[j] = g2(CB + (j * BR + lr) * TQ + tx);
        }
        mbar_arrive(&metbar[st]);
      }
#pragma unroll
      for (int c = 0; c < 3; ++c) qv[6][c] = g2(LF + c * NC + li);
      if (own) {
        f2 g[3][3];
        const f2 Jinv = CURV ? g2(CC + 3 * NC + li) : 0;
#pragma unroll
        for (int d = 0; d < 3; ++d) {
          f2 o[3];
          if (d == 0)
            deriv_q<FD, true>([&](int c) -> const float* { return FB + (c * BR + lr) * BQ; }, lq, kq0, kq1, lleft,
                              lright, tab, o);
          else if (d == 1) deriv_r<FD, true>([&](int l, int c) { return fb2(c, l, lq); }, lr, kr, tab, o);
          else deriv_s<CURV, FD, true>(a, p, ks, qv, o);
          const float rh = a.rh[d];
          if (CURV) {
            // 1/h goes to the differences: taken into 1/J, its rounding is the
            // same at every point of a regular grid and adds up
#pragma unroll
            for (int c = 0; c < 3; ++c) o[c] = mul2(pack(rh, rh), o[c]);
#pragma unroll
            for (int jj = 0; jj < 3; ++jj) {
              const f2 mt = mul2(d == 0 ? mq[jj] : (d == 1 ? mr[jj] : g2(CC + jj * NC + li)), Jinv);
#pragma unroll
              for (int c = 0; c < 3; ++c) g[c][jj] = d == 0 ? mul2(mt, o[c]) : fma2(mt, o[c], g[c][jj]);
            }
          } else {
            const float sc = a.cart_metric[d] * rh;
#pragma unroll
            for (int c = 0; c < 3; ++c) g[c][d] = mul2(pack(sc, sc), o[c]);
          }
        }
        if (a.G != nullptr) {  // anelastic: every point hands its velocity gradient over
#pragma unroll
          for (int c = 0; c < 3; ++c)
#pragma unroll
            for (int jj = 0; jj < 3; ++jj) *reinterpret_cast<f2*>(a.G + (c * 3 + jj) * np + p) = g[c][jj];
        }
        const f2 lam = g2(CC + (CURV ? 4 : 0) * NC + li);
        const f2 mu = g2(CC + (CURV ? 5 : 1) * NC + li);
        const f2 l2m = fma2(pack(2.0f, 2.0f), mu, lam);
        update(3, fma2(l2m, g[0][0], mul2(lam, add2(g[1][1], g[2][2]))));
        update(4, fma2(l2m, g[1][1], mul2(lam, add2(g[0][0], g[2][2]))));
        update(5, fma2(l2m, g[2][2], mul2(lam, add2(g[0][0], g[1][1]))));
        update(6, mul2(mu, add2(g[0][1], g[1][0])));
        update(7, mul2(mu, add2(g[0][2], g[2][0])));
        update(8, mul2(mu, add2(g[1][2], g[2][1])));
      }
    } else {
      {
        f2 f[6];
#pragma unroll
        for (int c = 0; c < 6; ++c) f[c] = g2(LF + (3 + c) * NC + li);
        if (CURV) {
          const float* LC = S + TL::OFF_LC;
          const f2 a0 = g2(LC + li), a1 = g2(LC + NC + li), a2 = g2(LC + 2 * NC + li);
#pragma unroll
          for (int c = 0; c < 3; ++c) qv[6][c] = dot3(a0, f[sig(c, 0) - 3], a1, f[sig(c, 1) - 3], a2, f[sig(c, 2) - 3]);
        } else {
#pragma unroll
          for (int c = 0; c < 3; ++c) qv[6][c] = f[sig(c, 2) - 3];
        }
      }
      // curvilinear: the q- and r-face momentum fluxes J*metric*sigma of the
      // main plane, formed once per box point and written over the
      // coefficients they come from (CA becomes the q flux on the q-extended
      // rows, CB the r flux on the r-extended columns), once the other role
      // has taken its metrics; each position is handled by one thread
      if (CURV) {
        // x: the first coefficient of the position, xs: words from one to the next
        auto flux = [&](float* x, int xs, const f2 (&sg)[6]) {
          f2 m[3];
#pragma unroll
          for (int j = 0; j < 3; ++j) m[j] = g2(x + j * xs);
#pragma unroll
          for (int c = 0; c < 3; ++c)
            *reinterpret_cast<f2*>(x + c * xs) =
                dot3(m[0], sg[sig(c, 0) - 3], m[1], sg[sig(c, 1) - 3], m[2], sg[sig(c, 2) - 3]);
        };
        f2 sg[6];
#pragma unroll
        for (int c = 0; c < 6; ++c) sg[c] = fb2(3 + c, lr, lq);
        if (!mbar_wait(&metbar[st], (T / NS) & 1)) {
          atomicExch(a.err, 4);
          return false;
        }
        flux(CA + ty * BQ + lq, TR * BQ, sg);
        flux(CB + lr * TQ + tx, BR * TQ, sg);
        // the halos: lanes 0..15 take the q halo of the warp's own two rows (4
        // pairs each side), lanes 16..31 of all warps together the r halo (HR
        // rows each side, TQ/2 pairs each)
        const int lane = tid & 31, warp = tid >> 5;
        constexpr int kRHalo = 2 * HR * (TQ / 2), kRPass = NT / 2;
#pragma unroll
        for (int e0 = 0; e0 < kRHalo; e0 += kRPass) {
          const bool isq = lane < 16;
          const int e = e0 + warp * 16 + (lane - 16);
          if (isq ? e0 == 0 : e < kRHalo) {
            const int h = lane & 7, rw = e / (TQ / 2);
            const int row = isq ? 2 * warp + (lane >> 3) : (rw < HR ? rw : rw + TR);
            const int qq = isq ? (h < 4 ? 2 * h : TQ + 2 * h) : 2 * (e % (TQ / 2)) + 8;
            const int rr = isq ? row + HR : row;
#pragma unroll
            for (int c = 0; c < 6; ++c) sg[c] = fb2(3 + c, rr, qq);
            flux(isq ? CA + row * BQ + qq : CB + row * TQ + (qq - 8), isq ? TR * BQ : BR * TQ, sg);
          }
        }
        // a warp forms every q flux of its own rows (the q derivative needs
        // only those: warp sync); the r fluxes of other rows come from other
        // warps: every thread of the role arrives here and waits (bounded)
        // just before the r derivative
        __syncwarp();
        mbar_arrive(fluxbar);
      }
      if (own) {
        f2 dv[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          const int d = k == 0 ? 0 : (k == 1 ? 2 : 1);  // q, s, then r
          if (CURV && k == 2 && !mbar_wait(fluxbar, T & 1)) {
            atomicExch(a.err, 3);
            return false;
          }
          f2 o[3];
          if (d == 0)
            deriv_q<FD, false>([&](int c) -> const float* {
              return CURV ? CA + (c * TR + ty) * BQ : FB + (sig(c, 0) * BR + lr) * BQ;
            }, lq, kq0, kq1, lleft, lright, tab, o);
          else if (d == 1)
            deriv_r<FD, false>([&](int l, int c) {
              return CURV ? g2(CB + (c * BR + l) * TQ + tx) : fb2(sig(c, 1), l, lq);
            }, lr, kr, tab, o);
          else deriv_s<CURV, FD, false>(a, p, ks, qv, o);
          const float sc = CURV ? a.rh[d] : a.cart_metric[d] * a.rh[d];
#pragma unroll
          for (int c = 0; c < 3; ++c) dv[c] = k == 0 ? mul2(pack(sc, sc), o[c]) : fma2(pack(sc, sc), o[c], dv[c]);
        }
        const f2 rinv = g2(CC + (CURV ? 6 : 2) * NC + li);
#pragma unroll
        for (int c = 0; c < 3; ++c) update(c, mul2(rinv, dv[c]));
      } else if (CURV && !mbar_wait(fluxbar, T & 1)) {  // the same phase for threads without a point
        atomicExch(a.err, 3);
        return false;
      }
      // order this thread's shared-memory writes (the fluxes) before the
      // producer's next bulk copy into the stage
      if (CURV) asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    __syncwarp();
    if ((tid & 31) == 0) mbar_arrive(&empty[st]);
#pragma unroll
    for (int i = 0; i < 6; ++i)
#pragma unroll
      for (int c = 0; c < 3; ++c) qv[i][c] = qv[i + 1][c];
  }
  return true;
}

struct MapArgs {
  CUtensorMap fbox, flead, ca, cb, cc, cl, df, ck, flead2;
};

// The work of one CTA: tile (bx, by) of the block, s chunk bz.
// Ring positions continue from one tile to the next: tb counts the stages
// the CTA has used before this tile (the same count in every thread), so a
// persistent CTA keeps its mbarriers and the producer runs ahead into the
// next tile.  Returns false after a wait ran out (the error word is set).
template <bool CURV, int FD, int TQW = kTmaTQ>
__device__ __forceinline__ bool tma_body(const VolumeArgs<float>& a, const MapArgs& m, int schunk, int bx, int by,
                                         int bz, const float* tab, int& tb) {
  using TL = TmaTile<CURV, FD, TQW>;
  constexpr int TQ = TL::TQ, TR = TL::TR, NC = TL::NC, NT = TL::NT, BQ = TL::BQ, BR = TL::BR, HR = TL::HR, NS = TL::NS;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  // 128-byte aligned start, derived from the shared array itself so the
  // compiler keeps every access in the shared address space
  float* sm = reinterpret_cast<float*>(smem_raw + ((128u - (smem_u32(smem_raw) & 127u)) & 127u));
  uint64_t* full = reinterpret_cast<uint64_t*>(sm + NS * TL::STAGE_W);
  uint64_t* empty = full + NS;
  uint64_t* fluxbar = empty + NS;   // flux threads: fluxes of the step written
  // stress threads: metrics of the stage read.  One per stage: those threads
  // can be a step ahead of the flux threads that wait here, and a stage is
  // filled again only after both roles have left it
  uint64_t* metbar = fluxbar + 1;

  const int tid = threadIdx.x;
  const int nq = a.nq, nr = a.nr, ns = a.ns;
  const int q0 = bx * TQ;
  const TileSpan spr = tile_span(by, nr, TR);
  const int r0 = spr.origin;
  const int s_begin = bz * schunk;
  const int s_end = min(ns, s_begin + schunk);
  const int nstep = s_end - s_begin;

  if (tid >= 2 * NT) {  // producer warp: one thread issues every copy
    if (tid == 2 * NT) {
      for (int t = 0; t < nstep; ++t) {
        const int T = tb + t;
        const int st = T % NS;
        if (T >= NS && !mbar_wait(&empty[st], ((T / NS) & 1) ^ 1)) {
          atomicExch(a.err, 1);
          tb = T;  // stages issued so far, for the final wait on copies in flight
          return false;
        }
        const int sp = s_begin + t;  // main plane
        mbar_expect_tx(&full[st], TL::LEAD_BYTES + TL::MAIN_BYTES);
        float* S = sm + st * TL::STAGE_W;
        if (FD) {  // velocities of plane s+4, stresses and J*metric_s of plane s+2
          tma_load_4d(S + TL::OFF_LF, &m.flead, &full[st], q0, r0, sp + 4, 0);
          tma_load_4d(S + TL::OFF_LF + 3 * NC, &m.flead2, &full[st], q0, r0, sp + 2, 3);
          if (CURV) tma_load_4d(S + TL::OFF_LC, &m.cl, &full[st], q0, r0, sp + 2, 6);
        } else {
          tma_load_4d(S + TL::OFF_LF, &m.flead, &full[st], q0, r0, sp + 3, 0);
          if (CURV) tma_load_4d(S + TL::OFF_LC, &m.cl, &full[st], q0, r0, sp + 3, 6);
        }
        tma_load_4d(S + TL::OFF_F, &m.fbox, &full[st], q0 - 8, r0 - HR, sp, 0);
        tma_load_4d(S + TL::OFF_DF, &m.df, &full[st], q0, r0, sp, 0);
        tma_load_4d(S + TL::OFF_CK, &m.ck, &full[st], q0, r0, sp, 0);
        if (CURV) {
          tma_load_4d(S + TL::OFF_CA, &m.ca, &full[st], q0 - 8, r0, sp, 0);
          tma_load_4d(S + TL::OFF_CB, &m.cb, &full[st], q0, r0 - HR, sp, 3);
          tma_load_4d(S + TL::OFF_CC, &m.cc, &full[st], q0, r0, sp, 6);
        } else {
          tma_load_4d(S + TL::OFF_CC, &m.cc, &full[st], q0, r0, sp, 0);
        }
      }
    }
    tb += nstep;
    return true;
  }

  // ---- consumers: two warps' worth of threads for every pair of points, one per role
  const bool ok = tid < NT ? tma_consume<CURV, FD, TQW, true>(a, sm, full, empty, fluxbar, metbar, q0, spr, s_begin,
                                                                  nstep, tid, tab, tb)
                           : tma_consume<CURV, FD, TQW, false>(a, sm, full, empty, fluxbar, metbar, q0, spr,
                                                                   s_begin, nstep, tid - NT, tab, tb);
  tb += nstep;
  return ok;
}

// Shared-memory ring of a persistent CTA: NS stages then the mbarriers.
template <bool CURV, int FD, int TQW = kTmaTQ>
struct Ring {
  static constexpr int NS = TmaTile<CURV, FD, TQW>::NS;
  float* sm;
  uint64_t *full, *empty, *fluxbar;
  float* tab;  // closure weights
  __device__ Ring() {
    using TL = TmaTile<CURV, FD, TQW>;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    sm = reinterpret_cast<float*>(smem_raw + ((128u - (smem_u32(smem_raw) & 127u)) & 127u));
    full = reinterpret_cast<uint64_t*>(sm + NS * TL::STAGE_W);
    empty = full + NS;
    fluxbar = empty + NS;
    tab = reinterpret_cast<float*>(fluxbar + 1 + NS);
  }
  // one thread initialises the barriers once per CTA
  __device__ void init() {
    using TL = TmaTile<CURV, FD, TQW>;
    // the closure weights: the q rows differ from lane to lane, which
    // constant memory would serve one row at a time
    if (FD) {
      if (threadIdx.x < 120) tab[threadIdx.x] = (&c_up_f[0][0][0])[threadIdx.x];
    } else if (threadIdx.x < 54) {
      tab[threadIdx.x] = (&c_sbp_f[0][0])[threadIdx.x];
    }
    if (threadIdx.x == 0) {
      for (int i = 0; i < NS; ++i) {
        mbar_init(&full[i], 1);
        mbar_init(&empty[i], 2 * TL::NT / 32);
      }
      mbar_init(fluxbar, TL::NT);
      for (int i = 0; i < NS; ++i) mbar_init(fluxbar + 1 + i, TL::NT);
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
  }
  // the producer's copies of the last stages land before the CTA leaves
  // (tb = stages issued)
  __device__ void drain(int tb) {
    if (threadIdx.x == 2 * TmaTile<CURV, FD, TQW>::NT)
      for (int T = max(0, tb - NS); T < tb; ++T) mbar_wait(&full[T % NS], (T / NS) & 1);
  }
};

// Each CTA takes tiles w = blockIdx.x, blockIdx.x + gridDim.x, ... of the
// tq x tr x nchunk tiles of the block (q fastest, so neighbouring CTAs share
// halos in L2); with one CTA per tile that is one tile each.
template <bool CURV, int FD, int TQW>
__global__ void __launch_bounds__(2 * TmaTile<CURV, FD, TQW>::NT + 32, 1)
    stencil_kernel_tma(const __grid_constant__ VolumeArgs<float> a, const __grid_constant__ MapArgs m, int schunk,
                       int tq, int tr, int ntile) {
  Ring<CURV, FD, TQW> ring;
  ring.init();
  int tb = 0;
  for (int w = blockIdx.x; w < ntile; w += gridDim.x)
    if (!tma_body<CURV, FD, TQW>(a, m, schunk, w % tq, (w / tq) % tr, w / (tq * tr), ring.tab, tb)) break;
  ring.drain(tb);
}

// One launch over many blocks (of one or many scenarios): CTA i works on the
// descriptor whose CTA range holds i, found by binary search in the packed
// table (descriptors sorted by cta0).
template <bool CURV>
__global__ void __launch_bounds__(2 * TmaTile<CURV, 0>::NT + 32, 1)
    stencil_kernel_tma_batch(const TmaBatchDesc* __restrict__ d, int nd, long long total) {
  // the entry's arguments are copied to shared memory: read from there they
  // cost no registers across the plane loop (held in registers they spill)
  __shared__ VolumeArgs<float> sa;
  Ring<CURV, 0> ring;
  const long long cta = blockIdx.x;
  int lo = 0, hi = nd - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) / 2;
    if (d[mid].cta0 <= cta) lo = mid;
    else hi = mid - 1;
  }
  const TmaBatchDesc& D = d[lo];
  {
    const int* src = reinterpret_cast<const int*>(&D.a);
    int* dst = reinterpret_cast<int*>(&sa);
    for (int i = threadIdx.x; i < (int)(sizeof(VolumeArgs<float>) / sizeof(int)); i += blockDim.x) dst[i] = src[i];
  }
  // the table was written by a host copy: order that write before the
  // tensor-map proxy reads the entry's maps (in the thread that issues copies)
  if (threadIdx.x == 2 * TmaTile<CURV, 0>::NT)
    for (int i = 0; i < 9; ++i)
      asm volatile("fence.proxy.tensormap::generic.acquire.sys [%0], 128;" ::"l"(&D.m[i]) : "memory");
  ring.init();  // its barrier also publishes sa
  int tb = 0;
  const long long l = cta - D.cta0;
  tma_body<CURV, 0>(sa, *reinterpret_cast<const MapArgs*>(&D.m), D.schunk, (int)(l % D.tq),
                            (int)((l / D.tq) % D.tr), (int)(l / ((long long)D.tq * D.tr)), ring.tab, tb);
  ring.drain(tb);
}

// Both blocks of a scenario in one launch: CTAs [0, ntile0) take block 0's
// tiles, the rest block 1's.  The arguments stay kernel parameters (two
// inlined copies of the tile code, each with its own constant offsets), so
// the block pair costs what two single launches cost minus one launch tail.
struct TwoBlocks {
  VolumeArgs<float> a[2];
  MapArgs m[2];
  int schunk[2], tq[2], tr[2];
  int ntile0;
};

template <bool CURV, int FD, int TQW>
__global__ void __launch_bounds__(2 * TmaTile<CURV, FD, TQW>::NT + 32, 1)
    stencil_kernel_tma2(const __grid_constant__ TwoBlocks P) {
  Ring<CURV, FD, TQW> ring;
  ring.init();
  int tb = 0;
  const int w = blockIdx.x;
  if (w < P.ntile0) {
    tma_body<CURV, FD, TQW>(P.a[0], P.m[0], P.schunk[0], w % P.tq[0], (w / P.tq[0]) % P.tr[0],
                              w / (P.tq[0] * P.tr[0]), ring.tab, tb);
  } else {
    const int l = w - P.ntile0;
    tma_body<CURV, FD, TQW>(P.a[1], P.m[1], P.schunk[1], l % P.tq[1], (l / P.tq[1]) % P.tr[1],
                              l / (P.tq[1] * P.tr[1]), ring.tab, tb);
  }
  ring.drain(tb);
}

// Planes per s chunk of a single-block launch: the tuned value, else 32.
int chunk_planes(const VolumeArgs<float>& a) {
  if (a.schunk > 0) return a.schunk;
  return 32;
}

int sm_count() {
  static int n[64] = {0};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) return 152;
  if (!n[dev] && cudaDeviceGetAttribute(&n[dev], cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) n[dev] = 152;
  return n[dev];
}

}  // namespace

// Planes per s chunk of a launch over nb blocks of tiles[b] (q, r) tiles and
// ns[b] planes.  With 8 or more waves of one CTA per SM at 32 planes, 32: the
// scheduler evens out what is left (2 x 201^3, 11 waves: 4.43 ms a step at 32,
// 1 to 3 % more at 12 to 29 and at 41 and more).  With fewer, the length that
// ends soonest when the CTAs go to the SMs in launch order, as they become
// free; a chunk costs its planes plus 2 for its start (the six window planes)
// plus 0.5 for each plane with an s closure row.  Measured ms a step at the
// chosen length and at 12 planes: 2 x 41^3 5: 0.185, 0.236; 76/75 x 150^2 39:
// 1.05, 1.11; 101/93 x 107x113 26: 0.90, 0.93; upwind 2 x 76x101x151 26: 1.30,
// 1.35 (correlation of the rule with the measured times over 19 lengths: 0.91
// to 1.00).
// The time at which it ends, in planes, goes to *end.
int choose_chunk(const int* tiles, const int* ns, int nb, float* end_out) {
  const int sms = sm_count();
  auto ctas = [&](int c) {
    long long n = 0;
    for (int b = 0; b < nb; ++b) n += (long long)tiles[b] * ((ns[b] + c - 1) / c);
    return n;
  };
  std::vector<float> heap;
  // costs are multiples of a half plane: sums of them are exact
  auto cost = [&](int b, int z, int c) {
    const int pl = std::min(c, ns[b] - z);
    const int left = std::max(0, std::min(z + pl, 6) - z), right = std::max(0, z + pl - std::max(z, ns[b] - 6));
    return 2.0f + pl + 0.5f * std::min(pl, left + right);
  };
  // no schedule of chunks of c ends before this
  auto bound = [&](int c) {
    double total = 0.0;
    for (int b = 0; b < nb; ++b)
      for (int z = 0; z < ns[b]; z += c) total += (double)tiles[b] * cost(b, z, c);
    return total / sms;
  };
  // its end, or any later time once it is later than `most`
  auto schedule = [&](int c, float most) {
    heap.assign(sms, 0.0f);  // a min-heap of the times at which the SMs are free
    float end = 0.0f;
    for (int b = 0; b < nb; ++b)
      for (int z = 0; z < ns[b]; z += c) {
        const float t1 = cost(b, z, c);
        for (int t = 0; t < tiles[b]; ++t) {
          std::pop_heap(heap.begin(), heap.end(), std::greater<float>());
          heap.back() += t1;
          end = std::max(end, heap.back());
          if (end > most) return end;
          std::push_heap(heap.begin(), heap.end(), std::greater<float>());
        }
      }
    return end;
  };
  int best = 32;
  float best_t = 1e30f;
  if (ctas(32) >= 8LL * sms) {
    if (end_out) best_t = schedule(32, best_t);
  } else {
    // the most promising length first; the shortest of equals
    std::vector<std::pair<double, int>> order;
    for (int c = 4; c <= 48; ++c)
      if (ctas(c) <= 8LL * sms) order.push_back({bound(c), c});
    std::sort(order.begin(), order.end());
    for (const auto& [least, c] : order) {
      if (least > best_t) break;
      const float end = schedule(c, best_t);
      if (end < best_t || (end == best_t && c < best)) {
        best_t = end;
        best = c;
      }
    }
  }
  if (end_out) *end_out = best_t;
  return best;
}

int pair_chunk(const int nq[2], int nr, const int ns[2], int tq, float* end) {
  const int rows = (nr + tma_rows(tq) - 1) / tma_rows(tq);
  const int tiles[2] = {(nq[0] + tq - 1) / tq * rows, (nq[1] + tq - 1) / tq * rows};
  return choose_chunk(tiles, ns, 2, end);
}

namespace {

MapArgs stage_maps(const StencilMaps& sm) {
  MapArgs m;
  m.fbox = sm.fbox[sm.cur];
  m.flead = sm.flead[sm.cur];
  m.ca = sm.ca;
  m.cb = sm.cb;
  m.cc = sm.cc;
  m.cl = sm.cl;
  m.df = sm.df;
  m.ck = sm.ck;
  m.flead2 = sm.flead2[sm.cur];
  return m;
}

template <bool CURV, int FD, int TQW = kTmaTQ>
constexpr size_t tma_smem_bytes() {
  constexpr int NS = TmaTile<CURV, FD, TQW>::NS;
  return sizeof(float) * (size_t)NS * TmaTile<CURV, FD, TQW>::STAGE_W + (3 * NS + 1) * sizeof(uint64_t) + 120 * sizeof(float) + 128;
}
static_assert(tma_smem_bytes<true, 0>() <= 227 * 1024 &&
                  tma_smem_bytes<false, 0>() <= 227 * 1024 &&
                  tma_smem_bytes<true, 1>() <= 227 * 1024 &&
                  tma_smem_bytes<false, 1>() <= 227 * 1024,
              "the stage ring must fit in the shared memory of one CTA");
static_assert(tma_smem_bytes<false, 0, kTmaTQWide>() <= 227 * 1024 &&
                  tma_smem_bytes<false, 1, kTmaTQWide>() <= 227 * 1024,
              "the wide Cartesian stage ring must fit in the shared memory of one CTA");

template <typename K>
size_t prepare(K kern, size_t smem) {
  cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  return smem;
}

// Grid: one CTA per tile.  The kernels also run persistently (fewer CTAs,
// each taking tiles in turn with its ring and barriers kept), but with the
// tiles statically interleaved that measured slower on 2 x 201^3 blocks
// (0.54 ms against 0.50 ms per launch): the chunks holding the s closure
// rows take longer, and the hardware's dynamic CTA scheduling balances them.
template <bool CURV, int FD, int TQW = kTmaTQ>
void launch_tma(const VolumeArgs<float>& a, const StencilMaps& sm, cudaStream_t s) {
  using TL = TmaTile<CURV, FD, TQW>;
  auto kern = stencil_kernel_tma<CURV, FD, TQW>;
  static const size_t smem = prepare(kern, tma_smem_bytes<CURV, FD, TQW>());
  const int tq = (a.nq + TL::TQ - 1) / TL::TQ, tr = (a.nr + TL::TR - 1) / TL::TR;
  const int schunk = chunk_planes(a);
  const int ntile = tq * tr * ((a.ns + schunk - 1) / schunk);
  kern<<<ntile, 2 * TL::NT + 32, smem, s>>>(a, stage_maps(sm), schunk, tq, tr, ntile);
}

template <bool CURV, int FD, int TQW = kTmaTQ>
void launch_tma2(const VolumeArgs<float>& a0, const VolumeArgs<float>& a1, cudaStream_t s) {
  using TL = TmaTile<CURV, FD, TQW>;
  auto kern = stencil_kernel_tma2<CURV, FD, TQW>;
  static const size_t smem = prepare(kern, tma_smem_bytes<CURV, FD, TQW>());
  TwoBlocks P;
  const VolumeArgs<float>* a[2] = {&a0, &a1};
  int ntile[2];
  for (int b = 0; b < 2; ++b) {
    const StencilMaps& sm = *static_cast<const StencilMaps*>(a[b]->tma);
    P.a[b] = *a[b];
    P.m[b] = stage_maps(sm);
    P.tq[b] = (a[b]->nq + TL::TQ - 1) / TL::TQ;
    P.tr[b] = (a[b]->nr + TL::TR - 1) / TL::TR;
    P.schunk[b] = a[b]->schunk > 0 ? a[b]->schunk : sm.chunk2;
    ntile[b] = P.tq[b] * P.tr[b] * ((a[b]->ns + P.schunk[b] - 1) / P.schunk[b]);
  }
  P.ntile0 = ntile[0];
  kern<<<ntile[0] + ntile[1], 2 * TL::NT + 32, smem, s>>>(P);
}

template <bool CURV>
void launch_tma_batch(const TmaBatchDesc* d, int nd, long long total, cudaStream_t s) {
  using TL = TmaTile<CURV, 0>;
  auto kern = stencil_kernel_tma_batch<CURV>;
  static const size_t smem = prepare(kern, tma_smem_bytes<CURV, 0>());
  if (total <= 0) return;
  kern<<<(unsigned)total, 2 * TL::NT + 32, smem, s>>>(d, nd, total);
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_fn() {
  static EncodeTiledFn fn = nullptr;
  if (!fn) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) ==
            cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = (EncodeTiledFn)p;
  }
  return fn;
}

// 4-D map over (q, r, s, component) of an FP32 array (bf16: of a bfloat16
// array) with row pitch pq.
int encode4(CUtensorMap* map, void* base, int nq, int nr, int ns, int ncomp, int pq, int bq, int br, int bc,
            bool bf16 = false) {
  EncodeTiledFn fn = encode_fn();
  if (!fn) return 1;
  const long long np = (long long)pq * nr * ns;
  const cuuint64_t es = bf16 ? 2 : 4;
  cuuint64_t dims[4] = {(cuuint64_t)nq, (cuuint64_t)nr, (cuuint64_t)ns, (cuuint64_t)ncomp};
  cuuint64_t strides[3] = {(cuuint64_t)pq * es, (cuuint64_t)pq * nr * es, (cuuint64_t)np * es};
  cuuint32_t box[4] = {(cuuint32_t)bq, (cuuint32_t)br, 1, (cuuint32_t)bc};
  cuuint32_t estr[4] = {1, 1, 1, 1};
  CUresult r = fn(map, bf16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, base, dims,
                  strides, box, estr,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return (int)r;
}

}  // namespace

int make_stencil_maps(StencilMaps& m, void* const F[2], void* coef, void* DF, void* C, int nq, int nr, int ns, int pq,
                      bool curv, int fd, int tq) {
  const int TQ = (tq == kTmaTQWide && !curv) ? kTmaTQWide : kTmaTQ, TR = tma_rows(TQ);
  const int hr = fd ? 4 : 3;  // r halo rows
  int rc = 0;
  m.ok = 0;
  m.cur = 0;
  m.fd = fd;
  m.tq = TQ;
  m.chunk2 = 32;
  for (int i = 0; i < 2 && !rc; ++i) {
    rc = encode4(&m.fbox[i], F[i], nq, nr, ns, 9, pq, TQ + 16, TR + 2 * hr, 9);
    // lead tiles: all 9 components of one plane, or (upwind) the 3
    // velocities and, from another plane, the 6 stresses
    if (!rc) rc = encode4(&m.flead[i], F[i], nq, nr, ns, 9, pq, TQ, TR, fd ? 3 : 9);
    if (!rc && fd) rc = encode4(&m.flead2[i], F[i], nq, nr, ns, 9, pq, TQ, TR, 6);
    if (!fd) m.flead2[i] = m.flead[i];
  }
  if (!rc) rc = encode4(&m.df, DF, nq, nr, ns, 9, pq, TQ, TR, 9);
  // the compensation is bfloat16 (without one the map is never read)
  if (!rc) rc = encode4(&m.ck, C ? C : DF, nq, nr, ns, 9, pq, TQ, TR, 9, true);
  if (curv) {
    if (!rc) rc = encode4(&m.ca, coef, nq, nr, ns, kCurvCoef, pq, TQ + 16, TR, 3);
    if (!rc) rc = encode4(&m.cb, coef, nq, nr, ns, kCurvCoef, pq, TQ, TR + 2 * hr, 3);
    if (!rc) rc = encode4(&m.cc, coef, nq, nr, ns, kCurvCoef, pq, TQ, TR, 7);
    if (!rc) rc = encode4(&m.cl, coef, nq, nr, ns, kCurvCoef, pq, TQ, TR, 3);
  } else {
    if (!rc) rc = encode4(&m.cc, coef, nq, nr, ns, kCartCoef, pq, TQ, TR, 3);
    m.ca = m.cb = m.cl = m.cc;
  }
  m.ok = rc == 0;
  return rc;
}

long long fill_tma_desc(const VolumeArgs<float>& a, int chunk, TmaBatchDesc& d) {
  static_assert(sizeof(MapArgs) == sizeof(d.m), "map set layout");
  const StencilMaps& sm = *static_cast<const StencilMaps*>(a.tma);
  const MapArgs m = stage_maps(sm);
  std::memcpy(d.m, &m, sizeof(m));
  d.a = a;
  d.schunk = a.schunk > 0 ? a.schunk : chunk;
  d.tq = (a.nq + kTmaTQ - 1) / kTmaTQ;
  d.tr = (a.nr + kTmaTR - 1) / kTmaTR;
  d.nchunk = (a.ns + d.schunk - 1) / d.schunk;
  d.cta0 = 0;
  return (long long)d.tq * d.tr * d.nchunk;
}

bool tma_eligible(const VolumeArgs<float>& a) {
  // the packed launch runs the central operator on 32-wide tiles; tile_span
  // keeps every r closure row inside tile + halo for the sizes of tiles_ok
  return a.tma != nullptr && a.fd == 0 && static_cast<const StencilMaps*>(a.tma)->tq == kTmaTQ &&
         tiles_ok(a.nr, kTmaTR);
}

// A plane of a 40 x 8 tile takes about as long as one of 32 x 12 (both are a
// warp's chain of instructions), so what counts is the number of planes that
// the fullest SM walks: 40 where its schedule ends 5 % sooner.  Over 168 pairs
// (2 x 41 to 400 points in q, 14 to 150 in r) and both operators that is 0.1 %
// slower than the better width on average and 5 % at worst; by the share of
// the columns in use alone, 5.5 % and 28 % (2 x 280x41x41: 63.9 us a launch
// with 40, 50.2 with 32; 76/75 x 150^2: 141.6 with 40, 156.6 with 32).
int tma_tile_width(const int nq[2], int nr, const int ns[2], bool curv, int fd) {
  if (curv || fd > 1) return kTmaTQ;  // the other operators run per point
  auto ok = [&](int rows) { return fd ? tiles_ok_up(nr, rows) : tiles_ok(nr, rows); };
  if (!ok(tma_rows(kTmaTQWide))) return kTmaTQ;
  if (!ok(kTmaTR)) return kTmaTQWide;
  float wide = 0.0f, narrow = 0.0f;
  pair_chunk(nq, nr, ns, kTmaTQWide, &wide);
  pair_chunk(nq, nr, ns, kTmaTQ, &narrow);
  return 1.05f * wide < narrow ? kTmaTQWide : kTmaTQ;
}

void launch_stencil_tma_batch(const TmaBatchDesc* d, int nd, long long total, bool curv, void* stream) {
  cudaStream_t s = (cudaStream_t)stream;
  if (curv) launch_tma_batch<true>(d, nd, total, s);
  else launch_tma_batch<false>(d, nd, total, s);
}

void launch_stencil_tma2(const VolumeArgs<float>& a0, const VolumeArgs<float>& a1, bool curv, void* stream) {
  cudaStream_t s = (cudaStream_t)stream;
  if (!curv && static_cast<const StencilMaps*>(a0.tma)->tq == kTmaTQWide) {
    if (a0.fd) launch_tma2<false, 1, kTmaTQWide>(a0, a1, s);
    else launch_tma2<false, 0, kTmaTQWide>(a0, a1, s);
  } else if (a0.fd) {
    if (curv) launch_tma2<true, 1>(a0, a1, s);
    else launch_tma2<false, 1>(a0, a1, s);
  } else {
    if (curv) launch_tma2<true, 0>(a0, a1, s);
    else launch_tma2<false, 0>(a0, a1, s);
  }
}

void launch_stencil_tma(const VolumeArgs<float>& a, bool curv, void* stream) {
  const StencilMaps& sm = *static_cast<const StencilMaps*>(a.tma);
  cudaStream_t s = (cudaStream_t)stream;
  if (!curv && sm.tq == kTmaTQWide) {
    if (a.fd) launch_tma<false, 1, kTmaTQWide>(a, sm, s);
    else launch_tma<false, 0, kTmaTQWide>(a, sm, s);
  } else if (a.fd) {
    if (curv) launch_tma<true, 1>(a, sm, s);
    else launch_tma<false, 1>(a, sm, s);
  } else {
    if (curv) launch_tma<true, 0>(a, sm, s);
    else launch_tma<false, 0>(a, sm, s);
  }
}

}  // namespace wql
