// FP64 stencil kernel of the central operator: the same per-point update as
// the other stencil kernels,
//   DF <- A*DF + L(F),   F_out <- F + B*dt*DF
// (scale_rates + set_rates + update_fields, src/fields.f90:49-171,
// src/JU_xJU_yJU_z6.f90:12-812 and 16141-16449, src/RHS_Interior.f90:133-274).
//
// Bound: the FP64 unit.  An SM retires two FP64 multiply-adds a cycle, so a
// warp instruction holds the unit for 16 cycles, while a point's loads cost
// about a tenth of that: the design saves FP64 instructions and idle lanes
// and lets memory be read as it comes.
//   * A CTA takes a tile of w x h points whose extents follow from the block's
//     (split evenly), not from powers of two, and numbers the tile's points
//     through: lanes are idle only in its last warp.  Each tile is at least 6
//     points wide, so every closure row of a tile reads columns that the tile
//     plus a 3-point halo holds.
//   * It marches along a chunk of s planes.  Velocities and s-face fluxes of
//     planes s-3..s+3 stay in registers; the q- and r-face fluxes of the plane
//     are formed once per point of the tile and its halo into shared memory
//     (the halo's points dealt out over all threads); the velocities are read
//     through L1.
//   * A central row is (x1-x-1) + (c2/c1)(x2-x-2) + (c3/c1)(x3-x-3): five
//     instructions, its factor c1/h folded into the metric it is multiplied by.
//   * The q closure rows sit at the ends of the rows of points, where almost
//     every warp holds a few: their 6 x h points x 6 quantities are dealt out
//     over all threads of the CTA and handed back through shared memory,
//     instead of being run by every warp for a few lanes.
// Both blocks of a scenario share a launch.
#include <cuda_runtime.h>

#include <algorithm>
#include <utility>

#include "wql_internal.h"
#include "wql_stencil.cuh"

namespace wql {
namespace {

// Two CTAs per SM at 168 registers: one computes while the other waits at its
// plane's barrier (one CTA of 384 threads: 455 against 424 us a stage on 2 x
// 75x81x77 Cartesian, the same on curvilinear 67/59x71x73; three of 128 the
// same as two).
constexpr int kF64Threads = 192;
constexpr size_t kF64Smem = 110 * 1024;  // most shared memory of a CTA

struct F64Pair {
  VolumeArgs<double> a[2];
  StencilPlan64 p[2];
  int n0;  // CTAs of block 0
};

// Closure weights over c1, so that closure and central rows share the factor
// c1/h.
__constant__ double c_close[6][9] = WQL_SBP_TABLE;

template <bool CURV>
__device__ __forceinline__ void sflux(const VolumeArgs<double>& a, long long pp, double o[6]) {
  const long long np = a.np;
  const double* __restrict__ F = a.Fin + pp;
#pragma unroll
  for (int c = 0; c < 3; ++c) o[c] = F[c * np];
  if (CURV) {
    const double a0 = a.coef[6 * np + pp], a1 = a.coef[7 * np + pp], a2 = a.coef[8 * np + pp];
#pragma unroll
    for (int c = 0; c < 3; ++c) o[3 + c] = a0 * F[sig(c, 0) * np] + a1 * F[sig(c, 1) * np] + a2 * F[sig(c, 2) * np];
  } else {
#pragma unroll
    for (int c = 0; c < 3; ++c) o[3 + c] = F[sig(c, 2) * np];
  }
}

// One column of an s-closure row (see s_close_w in the operator header): from
// the register window where it holds the plane, else from memory.
template <bool CURV, int ROW, bool RIGHT, int T>
__device__ __forceinline__ void s_col(const VolumeArgs<double>& a, long long p, const double (&qv)[7][6],
                                      double (&acc)[6]) {
  constexpr double w = s_close_w(0, RIGHT, false, ROW, T) / kC1;
  constexpr int off = s_close_off(RIGHT, ROW, T), iv = off + 3;
  if constexpr (w != 0.0) {
    double x[6];
    if constexpr (iv >= 0 && iv <= 6) {
#pragma unroll
      for (int c = 0; c < 6; ++c) x[c] = qv[iv][c];
    } else {
      sflux<CURV>(a, p + off * ((long long)a.pq * a.nr), x);
    }
#pragma unroll
    for (int c = 0; c < 6; ++c) acc[c] += w * x[c];
  }
}

template <bool CURV, int ROW, bool RIGHT, int... T>
__device__ __forceinline__ void s_row(const VolumeArgs<double>& a, long long p, const double (&qv)[7][6],
                                      double (&o)[6], std::integer_sequence<int, T...>) {
#pragma unroll
  for (int c = 0; c < 6; ++c) o[c] = 0.0;
  (s_col<CURV, ROW, RIGHT, T>(a, p, qv, o), ...);
}

template <bool CURV>
__device__ __forceinline__ void s_closure64(const VolumeArgs<double>& a, long long p, int ks,
                                            const double (&qv)[7][6], double (&o)[6]) {
  using Cols = std::make_integer_sequence<int, 9>;
  switch (ks) {
    case -1: s_row<CURV, 0, false>(a, p, qv, o, Cols{}); break;
    case -2: s_row<CURV, 1, false>(a, p, qv, o, Cols{}); break;
    case -3: s_row<CURV, 2, false>(a, p, qv, o, Cols{}); break;
    case -4: s_row<CURV, 3, false>(a, p, qv, o, Cols{}); break;
    case -5: s_row<CURV, 4, false>(a, p, qv, o, Cols{}); break;
    case -6: s_row<CURV, 5, false>(a, p, qv, o, Cols{}); break;
    case 1: s_row<CURV, 0, true>(a, p, qv, o, Cols{}); break;
    case 2: s_row<CURV, 1, true>(a, p, qv, o, Cols{}); break;
    case 3: s_row<CURV, 2, true>(a, p, qv, o, Cols{}); break;
    case 4: s_row<CURV, 3, true>(a, p, qv, o, Cols{}); break;
    case 5: s_row<CURV, 4, true>(a, p, qv, o, Cols{}); break;
    default: s_row<CURV, 5, true>(a, p, qv, o, Cols{}); break;
  }
}

template <bool CURV>
__device__ __forceinline__ void fp64_tile(const VolumeArgs<double>& a, const StencilPlan64& P, int l) {
  extern __shared__ __align__(16) double sm64[];
  const int nq = a.nq, nr = a.nr, ns = a.ns;
  const int bx = l % P.kq, by = (l / P.kq) % P.kr, bz = l / (P.kq * P.kr);
  const int q0 = (int)((long long)bx * nq / P.kq), w = (int)((long long)(bx + 1) * nq / P.kq) - q0;
  const int r0 = (int)((long long)by * nr / P.kr), h = (int)((long long)(by + 1) * nr / P.kr) - r0;
  const int s_begin = bz * P.chunk, s_end = min(ns, s_begin + P.chunk);
  // shared memory: closure table, q-closure results, then two buffers of
  // fluxes (q: h rows of w+6, r: h+6 rows of w; 3 components)
  double* tab = sm64;
  double* qd = tab + 54;
  const int nqd = 6 * P.th * 12, nfq = P.th * (P.tw + 6), nfr = (P.th + 6) * P.tw;
  double* fbuf = qd + nqd;
  const int tid = threadIdx.x, nt = blockDim.x;
  for (int e = tid; e < 54; e += nt) tab[e] = (&c_close[0][0])[e] / kC1;
  const int tx = tid % w, ty = tid / w;
  const bool valid = ty < h;
  const int q = q0 + tx, r = r0 + (valid ? ty : 0);
  const int kq = sbp_kind(q, nq), kr = sbp_kind(r, nr);
  const bool hasl = q0 < 6, hasr = q0 + w > nq - 6;  // the tile holds left / right q closure points
  const int nside = (hasl ? 1 : 0) + (hasr ? 1 : 0);
  const long long np = a.np;
  const long long str = a.pq, sts = (long long)a.pq * nr;
  const long long col = q + str * r;
  const double k2 = kC2 / kC1, k3 = kC3 / kC1;

  double qv[7][6];
#pragma unroll
  for (int i = 0; i < 7; ++i) {
    const int pl = s_begin - 3 + i;
    if (i < 6 && valid && pl >= 0 && pl < ns) {
      sflux<CURV>(a, col + sts * pl, qv[i]);
    } else {
#pragma unroll
      for (int c = 0; c < 6; ++c) qv[i][c] = 0.0;
    }
  }

  int buf = 0;
  for (int s = s_begin; s < s_end; ++s, buf ^= 1) {
    const long long p = col + sts * s;
    const double* __restrict__ F = a.Fin + p;
    const int ks = sbp_kind(s, ns);
    if (valid && s + 3 < ns) sflux<CURV>(a, p + 3 * sts, qv[6]);
    double* fq = fbuf + buf * 3 * (nfq + nfr);
    double* fr = fq + 3 * nfq;
    const int wq = w + 6;
    if (CURV) {
      // d-face flux of the point at `pp` into x[0], x[n], x[2n]
      auto flux = [&](int d, long long pp, double* x, int n) {
        const double* M = a.coef + (long long)(d * 3) * np + pp;
        const double* f = a.Fin + pp;
        const double m0 = M[0], m1 = M[np], m2 = M[2 * np];
#pragma unroll
        for (int c = 0; c < 3; ++c) x[c * n] = m0 * f[sig(c, 0) * np] + m1 * f[sig(c, 1) * np] + m2 * f[sig(c, 2) * np];
      };
      if (valid) {
        flux(0, p, fq + ty * wq + tx + 3, nfq);
        flux(1, p, fr + (ty + 3) * w + tx, nfr);
      }
      for (int e = tid; e < 6 * h + 6 * w; e += nt) {
        if (e < 6 * h) {
          const int y = e / 6, x = e % 6, lx = x < 3 ? x : w + x, gq = q0 + lx - 3;
          if (gq >= 0 && gq < nq) flux(0, gq + str * (r0 + y) + sts * s, fq + y * wq + lx, nfq);
        } else {
          const int e2 = e - 6 * h, y = e2 / w, x = e2 % w, ly = y < 3 ? y : h + y, gr = r0 + ly - 3;
          if (gr >= 0 && gr < nr) flux(1, q0 + x + str * gr + sts * s, fr + ly * w + x, nfr);
        }
      }
    }
    __syncthreads();
    if (nside) {
      const int per = nside * 6 * h;
      for (int e = tid; e < 6 * per; e += nt) {
        const int c = e / per, rem = e % per, y = rem / (6 * nside), i = rem % (6 * nside);
        const bool left = hasl && i < 6;
        const int row = i % 6, gq = left ? row : nq - 1 - row;
        double acc = 0.0;
        if (gq >= q0 && gq < q0 + w) {
          const int b = left ? 0 : nq - 1, st = left ? 1 : -1;
          if (c < 3 || !CURV) {
            const double* x = a.Fin + (c < 3 ? c : sig(c - 3, 0)) * np + b + str * (r0 + y) + sts * s;
#pragma unroll
            for (int t = 0; t < 9; ++t) acc += tab[row * 9 + t] * x[t * st];
          } else {
            const double* x = fq + (c - 3) * nfq + y * wq + (b - q0 + 3);
#pragma unroll
            for (int t = 0; t < 9; ++t) acc += tab[row * 9 + t] * x[t * st];
          }
        }
        qd[(c * P.th + y) * 12 + i] = left ? acc : -acc;
      }
      __syncthreads();
    }
    if (valid) {
      double g[3][3], dv[3];
      const double Jinv = CURV ? a.coef[9 * np + p] : 1.0;
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        double o[6];
        const int kind = d == 0 ? kq : (d == 1 ? kr : ks);
        if (d == 2) {
          if (ks == 0) {
#pragma unroll
            for (int c = 0; c < 6; ++c)
              o[c] = (qv[4][c] - qv[2][c]) + k2 * (qv[5][c] - qv[1][c]) + k3 * (qv[6][c] - qv[0][c]);
          } else {
            s_closure64<CURV>(a, p, ks, qv, o);
          }
        } else if (d == 0 && kind != 0) {
          const int i = kind < 0 ? -kind - 1 : (hasl ? 6 : 0) + kind - 1;
#pragma unroll
          for (int c = 0; c < 6; ++c) o[c] = qd[(c * P.th + ty) * 12 + i];
        } else {
          const long long st = d == 0 ? 1 : str;
          // quantity c at n points along the axis
          auto X = [&](int c, int n) -> double {
            if (c < 3) return F[c * np + n * st];
            if (!CURV) return F[sig(c - 3, d) * np + n * st];
            return d == 0 ? fq[(c - 3) * nfq + ty * wq + tx + 3 + n] : fr[(c - 3) * nfr + (ty + 3 + n) * w + tx];
          };
          if (kind == 0) {
#pragma unroll
            for (int c = 0; c < 6; ++c)
              o[c] = (X(c, 1) - X(c, -1)) + k2 * (X(c, 2) - X(c, -2)) + k3 * (X(c, 3) - X(c, -3));
          } else {
            const int row = kind < 0 ? -kind - 1 : kind - 1, dir = kind < 0 ? 1 : -1;
            const double sgn = kind < 0 ? 1.0 : -1.0;
#pragma unroll
            for (int c = 0; c < 6; ++c) o[c] = 0.0;
#pragma unroll 3
            for (int t = 0; t < 9; ++t) {
              const double wt = tab[row * 9 + t];
#pragma unroll
              for (int c = 0; c < 6; ++c) o[c] += wt * X(c, (t - row) * dir);
            }
#pragma unroll
            for (int c = 0; c < 6; ++c) o[c] *= sgn;
          }
        }
        const double rh = a.rh[d] * kC1;
        if (CURV) {
#pragma unroll
          for (int jj = 0; jj < 3; ++jj) {
            const double m = rh * a.coef[(d * 3 + jj) * np + p];
#pragma unroll
            for (int c = 0; c < 3; ++c) g[c][jj] = d == 0 ? m * o[c] : g[c][jj] + m * o[c];
          }
#pragma unroll
          for (int c = 0; c < 3; ++c) dv[c] = d == 0 ? rh * o[3 + c] : dv[c] + rh * o[3 + c];
        } else {
          const double sc = a.cart_metric[d] * rh;
#pragma unroll
          for (int c = 0; c < 3; ++c) {
            dv[c] = d == 0 ? sc * o[3 + c] : dv[c] + sc * o[3 + c];
            g[c][d] = sc * o[c];
          }
        }
      }
      // 1/J of the velocity gradient goes into the moduli
      const double lam = a.coef[(CURV ? 10 : 0) * np + p] * (CURV ? Jinv : 1.0);
      const double mu = a.coef[(CURV ? 11 : 1) * np + p] * (CURV ? Jinv : 1.0);
      const double rinv = a.coef[(CURV ? 12 : 2) * np + p];
      const double lt = lam * (g[0][0] + g[1][1] + g[2][2]), m2 = mu + mu;
      double x[9];
      x[0] = dv[0]; x[1] = dv[1]; x[2] = dv[2];
      x[3] = m2 * g[0][0] + lt;
      x[4] = m2 * g[1][1] + lt;
      x[5] = m2 * g[2][2] + lt;
      x[6] = g[0][1] + g[1][0];
      x[7] = g[0][2] + g[2][0];
      x[8] = g[1][2] + g[2][1];
      // on a stage with A = 0 only the points of the pre-kernels have rates
      const int wl = a.npml;
      const bool keep = a.A != 0.0;
      const bool set = !keep && (q == 0 || q == nq - 1 || r == 0 || r == nr - 1 || s == 0 || s == ns - 1 ||
                                 (a.pml[0] && q < wl) || (a.pml[1] && q >= nq - wl) || (a.pml[2] && r < wl) ||
                                 (a.pml[3] && r >= nr - wl) || (a.pml[4] && s < wl) || (a.pml[5] && s >= ns - wl));
#pragma unroll
      for (int c = 0; c < 9; ++c) {
        const double ad = keep ? a.A * a.DF[c * np + p] : (set ? a.DF[c * np + p] : 0.0);
        const double df = c < 3 ? ad + rinv * x[c] : (c < 6 ? ad + x[c] : ad + mu * x[c]);
        a.DF[c * np + p] = df;
        a.Fout[c * np + p] = F[c * np] + a.Bdt * df;
      }
    }
#pragma unroll
    for (int i = 0; i < 6; ++i)
#pragma unroll
      for (int c = 0; c < 6; ++c) qv[i][c] = qv[i + 1][c];
  }
}

template <bool CURV>
__global__ void __launch_bounds__(kF64Threads, 2) stencil_kernel_fp64(const __grid_constant__ F64Pair P) {
  const int b = (int)blockIdx.x >= P.n0 ? 1 : 0;
  fp64_tile<CURV>(P.a[b], P.p[b], (int)blockIdx.x - (b ? P.n0 : 0));
}

size_t smem_of(const StencilPlan64& p) {
  return sizeof(double) * (54 + 6 * (size_t)p.th * 12 +
                           2 * 3 * ((size_t)p.th * (p.tw + 6) + (size_t)(p.th + 6) * p.tw));
}

}  // namespace

// The split of a block: tiles of kq x kr over (q, r) and chunks of planes,
// chosen for the fewest warp-steps on the fullest SM: the total over all CTAs
// plus half a CTA's own (the tail), a chunk's six window planes counted as
// 0.3 of a step.  Axes have at least 12 points, so closure rows from both ends
// do not meet.
StencilPlan64 make_plan64(int nq, int nr, int ns, int sms) {
  StencilPlan64 best{};
  double best_cost = 1e300;
  for (int kq = 1; kq <= std::max(1, nq / 6); ++kq) {
    const int tw = (nq + kq - 1) / kq;
    if (tw > 128 || (tw < 12 && kq > 1)) continue;
    for (int kr = 1; kr <= std::max(1, nr / 6); ++kr) {
      const int th = (nr + kr - 1) / kr, warps = (tw * th + 31) / 32;
      if (tw * th > kF64Threads || (th < 6 && kr > 1)) continue;
      // halo fluxes: 9 of about 210 instructions each
      const double step = warps + 0.043 * (6.0 * (tw + th)) / 32.0;
      for (int c = 4; c <= 32; ++c) {
        const int nc = (ns + c - 1) / c;
        const double cta = step * (c + 0.3), total = step * (double)kq * kr * (ns + 0.3 * nc);
        const double cost = total / (2 * sms) + 0.5 * cta;
        if (cost < best_cost) {
          best_cost = cost;
          best = StencilPlan64{kq, kr, tw, th, c, 1};
        }
      }
    }
  }
  if (best.ok && smem_of(best) > kF64Smem) best.ok = 0;
  return best;
}

void launch_stencil_fp64(const VolumeArgs<double>& a0, const VolumeArgs<double>* a1, bool curv, void* stream) {
  F64Pair P;
  const VolumeArgs<double>* a[2] = {&a0, a1 ? a1 : &a0};
  int n[2], nt = 0;
  size_t smem = 0;
  for (int b = 0; b < 2; ++b) {
    P.a[b] = *a[b];
    P.p[b] = *static_cast<const StencilPlan64*>(a[b]->plan64);
    if (a[b]->schunk > 0) P.p[b].chunk = a[b]->schunk;
    n[b] = P.p[b].kq * P.p[b].kr * ((a[b]->ns + P.p[b].chunk - 1) / P.p[b].chunk);
    nt = std::max(nt, (P.p[b].tw * P.p[b].th + 31) / 32 * 32);
    smem = std::max(smem, smem_of(P.p[b]));
  }
  P.n0 = n[0];
  if (!a1) n[1] = 0;
  auto kern = curv ? stencil_kernel_fp64<true> : stencil_kernel_fp64<false>;
  // the same limit for every launch: threads stepping other scenarios set it too
  cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kF64Smem);
  kern<<<n[0] + n[1], nt, smem, (cudaStream_t)stream>>>(P);
}

}  // namespace wql
