// Building blocks of the plain FP64 TR-BDF2 form, shared by the time-advance kernel
// (kernels_fp64.cu) and the discrete-adjoint kernel (kernels_adjoint.cu): the per-warp shared
// memory view, FP64 right-hand side, Newton matrix, dense LU with partial pivoting and its
// solves, Newton iteration and the TR-BDF2 step loop.
#pragma once

#include "advance.hpp"
#include "engine.cuh"

namespace tchem_gb {
namespace fp64 {


struct WarpMem {
  double* x;     // [m] current iterate, for gathers
  double* keff;  // [R]
  double* q;     // [R] rates of progress
  double* d;     // [NF] Jacobian factor-slot derivatives
  double* w;     // [m] scratch of the factorisation and the solves
  int32_t* piv;  // [m]
  double* A;     // [m][lda] Newton matrix / LU factors
};

template <int NPL>
struct Ctx {
  const MechLayout& L;
  const SmemTables& T;
  const WarpMem& W;
  int lane;
  int lda;
  const int32_t* pos;  // [m] row and column of each species in the Newton matrix
  tchem_gb_sample_stats st;
};

// Size of the Newton system of a context (the aerosol context of kernels_aero.cu has its own).
template <int NPL>
__device__ __forceinline__ int sys_dim(const Ctx<NPL>& c) {
  return c.L.m;
}

// Row and column of unknown i in a context's Newton matrix. The species of Ctx stand in the sparse LU's order
// (at most 128 species), in which the steps of a
// 51-species factorisation hold 560 multipliers instead of 925.
template <class C>
__device__ __forceinline__ int place(const C&, int i) {
  return i;
}
template <int NPL>
__device__ __forceinline__ int place(const Ctx<NPL>& c, int i) {
  return __ldg(c.pos + i);
}

template <int NPL>
__device__ __forceinline__ void publish(Ctx<NPL>& c, const double (&y)[NPL]) {
#pragma unroll
  for (int k = 0; k < NPL; ++k) {
    const int i = c.lane + 32 * k;
    if (i < c.L.m) c.W.x[i] = y[k];
  }
  __syncwarp();
}

// f = omega(y): src/core/impl/TChem_Impl_ReactionRatesAerosol.hpp:80-138.
template <int NPL>
__device__ __forceinline__ void rhs(Ctx<NPL>& c, const double (&y)[NPL], double (&f)[NPL]) {
  publish(c, y);
  const SmemTables& T = c.T;
  for (int r = c.lane; r < c.L.R; r += 32) {
    double q = c.W.keff[r];
    for (int g = T.rf_ptr[r]; g < T.rf_ptr[r + 1]; ++g) q *= c.W.x[T.rf_sp[g]];
    c.W.q[r] = q;
  }
  __syncwarp();
#pragma unroll
  for (int k = 0; k < NPL; ++k) {
    const int i = c.lane + 32 * k;
    double acc = 0.0;
    if (i < c.L.m) {
      acc = T.emis[i];
      for (int e = T.pr_ptr[i]; e < T.pr_ptr[i + 1]; ++e) acc += T.pr_nu[e] * c.W.q[T.pr_r[e]];
    }
    f[k] = acc;
  }
  __syncwarp();
  ++c.st.n_rhs;
}

// A = I - coef * J(y), analytic Jacobian.
template <int NPL>
__device__ __forceinline__ void newton_matrix(Ctx<NPL>& c, const double (&y)[NPL], double coef) {
  publish(c, y);
  const SmemTables& T = c.T;
  const int m = c.L.m, lda = c.lda;
  for (int r = c.lane; r < c.L.R; r += 32) {
    const int f0 = T.rf_ptr[r], f1 = T.rf_ptr[r + 1];
    for (int f = f0; f < f1; ++f) {
      double dv = c.W.keff[r];
      for (int g = f0; g < f1; ++g)
        if (g != f) dv *= c.W.x[T.rf_sp[g]];
      c.W.d[f] = dv;
    }
  }
  double* A = c.W.A;
  for (int i = 0; i < m; ++i)
    for (int j = c.lane; j < m; j += 32) A[i * lda + j] = (i == j) ? 1.0 : 0.0;
  __syncwarp();
  for (int z = c.lane; z < c.L.NZ; z += 32) {
    const int rc = T.jz_rc[z];
    const int i = rc >> 16, j = rc & 0xffff;
    double J = 0.0;
    for (int e = T.jz_ptr[z]; e < T.jz_ptr[z + 1]; ++e) J += T.jc_nu[e] * c.W.d[T.jc_f[e]];
    A[place(c, i) * lda + place(c, j)] = (i == j ? 1.0 : 0.0) - coef * J;
  }
  __syncwarp();
  ++c.st.n_jac;
}

// In-place LU with partial pivoting (first maximum in current row order), row swaps; the diagonal of
// the factors holds the pivots' reciprocals.
// C: a per-sample context (Ctx, or the aerosol context) with W.A, W.piv, W.w, lane, lda and st.
//
// An FP64 instruction holds one warp's share of the FP64 units for 64 cycles, however many lanes take part, so
// their number is what counts. The pivot search compares the bit patterns of the magnitudes (three integer
// reductions instead of five rounds of FP64 compares), and a step updates only rows with a multiplier and
// columns with an entry of the pivot row: both are listed by ballots, and groups of lanes take a row each
// where few columns are left. What is left out are additions of zero. A 51-species factorisation
// takes 158 k cycles in one warp: 303 k with the unknowns in their own order, 272 k of them with a row's loads no
// longer behind the previous row's store; 61 k now are the pivots' reciprocals and the multipliers.
template <class C>
__device__ __forceinline__ bool lu_factor(C& c) {
  double* A = c.W.A;
  const int m = sys_dim(c), lda = c.lda, lane = c.lane;
  uint16_t* cols = reinterpret_cast<uint16_t*>(c.W.w);  // [m] columns of the step, then [m] its rows
  uint16_t* rows = cols + m;
  const uint32_t below = (1u << lane) - 1u;
  for (int k = 0; k < m; ++k) {
    unsigned long long best = 0;
    int bi = m;
    for (int i = k + lane; i < m; i += 32) {
      const unsigned long long v = __double_as_longlong(A[i * lda + k]) & 0x7fffffffffffffffull;
      if (v > best && v <= 0x7ff0000000000000ull) { best = v; bi = i; }  // a NaN is passed over
    }
    const uint32_t hi = static_cast<uint32_t>(best >> 32), lo = static_cast<uint32_t>(best);
    const uint32_t top = __reduce_max_sync(kFullMask, hi);
    const uint32_t low = __reduce_max_sync(kFullMask, hi == top ? lo : 0u);
    bi = __reduce_min_sync(kFullMask, hi == top && lo == low ? bi : m);
    if ((top | low) == 0u || top >= 0x7ff00000u) return false;
    const double inv = 1.0 / A[bi * lda + k];
    if (lane == 0) c.W.piv[k] = bi;
    __syncwarp();
    if (bi != k) {
      for (int j = lane; j < m; j += 32) {
        const double a = A[k * lda + j];
        A[k * lda + j] = A[bi * lda + j];
        A[bi * lda + j] = a;
      }
      __syncwarp();
    }
    // rows with an entry in the pivot's column, columns with one in its row, and whether any product with a
    // zero counts too: an infinity, a NaN or a pivot without a reciprocal
    int nc = 0, nr = 0;
    bool wild = top < 0x00300000u;
    for (int i0 = k + 1; i0 < m; i0 += 32) {
      const int i = i0 + lane;
      bool in_row = false, in_col = false;
      if (i < m) {
        const long long u = __double_as_longlong(A[k * lda + i]), l = __double_as_longlong(A[i * lda + k]);
        in_row = (u << 1) != 0;
        in_col = (l << 1) != 0;
        wild |= ((u >> 52) & 0x7ff) == 0x7ff || ((l >> 52) & 0x7ff) == 0x7ff;
      }
      const uint32_t rb = __ballot_sync(kFullMask, in_row), cb = __ballot_sync(kFullMask, in_col);
      if (in_row) cols[nc + __popc(rb & below)] = static_cast<uint16_t>(i);
      if (in_col) rows[nr + __popc(cb & below)] = static_cast<uint16_t>(i);
      nc += __popc(rb);
      nr += __popc(cb);
    }
    if (__any_sync(kFullMask, wild)) {
      __syncwarp();
      for (int i = k + 1 + lane; i < m; i += 32) cols[i - k - 1] = rows[i - k - 1] = static_cast<uint16_t>(i);
      nc = nr = m - k - 1;
    }
    __syncwarp();
    for (int r = lane; r < nr; r += 32) A[rows[r] * lda + k] *= inv;
    if (lane == 0) A[k * lda + k] = inv;
    __syncwarp();
    if (nc > 0) {
      const int width = nc > 16 ? 32 : nc > 8 ? 16 : nc > 4 ? 8 : 4;  // lanes to a row
      const int first = lane / width, step = 32 / width;
      for (int e = lane & (width - 1); e < nc; e += width) {
        const int j = cols[e];
        const double u = A[k * lda + j];
        for (int r0 = first; r0 < nr; r0 += 4 * step) {  // four rows' loads, then their updates, then their stores
          double* at[4];
          double v[4], l[4];
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const int r = r0 + q * step;
            const int i = rows[min(r, nr - 1)];
            at[q] = A + i * lda + j;
            v[q] = *at[q];
            l[q] = A[i * lda + k];
          }
#pragma unroll
          for (int q = 0; q < 4; ++q)
            if (r0 + q * step < nr) *at[q] = v[q] - l[q] * u;
        }
      }
    }
    __syncwarp();
  }
  ++c.st.n_lu;
  return true;
}

// The row swaps of lu_factor applied to w, in their order or backward; by the whole warp.
template <class C>
__device__ __forceinline__ void lu_swaps(C& c, double* w, bool backward) {
  const int m = sys_dim(c);
  const int chunks = (m + 31) / 32;
  for (int t = 0; t < chunks; ++t) {
    const int i0 = 32 * (backward ? chunks - 1 - t : t), i = i0 + c.lane;
    uint32_t moved = __ballot_sync(kFullMask, i < m && c.W.piv[i] != i);
    if (c.lane == 0) {
      while (moved) {
        const int b = backward ? 31 - __clz(moved) : __ffs(moved) - 1, k = i0 + b, p = c.W.piv[k];
        moved &= ~(1u << b);
        const double v = w[k];
        w[k] = w[p];
        w[p] = v;
      }
    }
  }
  __syncwarp();
}

// x = A^{-1} b with the factors of lu_factor. The vector stays in registers, an element per lane and
// 32 rows, and each step hands its element round by a shuffle: no store, barrier and load in the chain.
template <int NPL, class C>
__device__ __forceinline__ void lu_solve(C& c, const double (&b)[NPL], double (&x)[NPL]) {
  const double* A = c.W.A;
  double* w = c.W.w;
  const int m = sys_dim(c), lda = c.lda, lane = c.lane;
#pragma unroll
  for (int k = 0; k < NPL; ++k) {
    const int i = lane + 32 * k;
    if (i < m) w[place(c, i)] = b[k];
  }
  __syncwarp();
  lu_swaps(c, w, false);
#pragma unroll
  for (int k = 0; k < NPL; ++k) {
    const int i = lane + 32 * k;
    x[k] = (i < m) ? w[i] : 0.0;
  }
#pragma unroll
  for (int t = 0; t < NPL; ++t) {
#pragma unroll 4
    for (int k = 32 * t; k < min(m, 32 * t + 32); ++k) {
      const double xk = __shfl_sync(kFullMask, x[t], k - 32 * t);
#pragma unroll
      for (int a = t; a < NPL; ++a) {
        const int i = lane + 32 * a;
        if (i > k && i < m) x[a] -= A[i * lda + k] * xk;
      }
    }
  }
#pragma unroll
  for (int t = NPL - 1; t >= 0; --t) {
#pragma unroll 4
    for (int k = min(m, 32 * t + 32) - 1; k >= 32 * t; --k) {
      const double xk = __shfl_sync(kFullMask, x[t], k - 32 * t) * A[k * lda + k];
      if (lane == k - 32 * t) x[t] = xk;
#pragma unroll
      for (int a = 0; a <= t; ++a) {
        const int i = lane + 32 * a;
        if (i < k) x[a] -= A[i * lda + k] * xk;
      }
    }
  }
#pragma unroll
  for (int k = 0; k < NPL; ++k) {
    const int i = lane + 32 * k;
    if (i < m) w[i] = x[k];
  }
  __syncwarp();
#pragma unroll
  for (int k = 0; k < NPL; ++k) {
    const int i = lane + 32 * k;
    x[k] = (i < m) ? w[place(c, i)] : 0.0;
  }
  __syncwarp();
  ++c.st.n_solve;
}

struct NewtonSettings {
  int max_newton, jac_interval;
  double atol, rtol;
};

// Solves y - coef f(y) = rhs from the guess in y. rhs and newton_matrix resolve on the context type.
template <int NPL, class C>
__device__ __forceinline__ bool newton(C& c, double (&y)[NPL], const double (&rhs_v)[NPL], double coef, const NewtonSettings& s) {
  for (int it = 0; it < s.max_newton; ++it) {
    double f[NPL], g[NPL], dx[NPL];
    rhs(c, y, f);
#pragma unroll
    for (int k = 0; k < NPL; ++k) g[k] = -((y[k] - coef * f[k]) - rhs_v[k]);
    if (it % s.jac_interval == 0) {
      newton_matrix(c, y, coef);
      if (!lu_factor(c)) return false;
    }
    lu_solve(c, g, dx);
    ++c.st.n_newton_iter;
    double sdx = 0.0, sy = 0.0;
#pragma unroll
    for (int k = 0; k < NPL; ++k) {
      if (c.lane + 32 * k < sys_dim(c)) {
        y[k] += dx[k];
        sdx += dx[k] * dx[k];
        sy += y[k] * y[k];
      }
    }
    const double ndx = sqrt(warp_sum(sdx)), ny = sqrt(warp_sum(sy));
    if (!isfinite(ndx) || !isfinite(ny)) return false;
    if (ndx <= s.atol + s.rtol * ny) return true;
  }
  return false;
}

// One sample's trajectory record (dt == nullptr: not recorded): accepted step sizes and the
// state at the start of steps 0, kTapeSegment, 2 kTapeSegment, ...
struct Tape {
  double* dt;    // [cap]
  double* ckpt;  // [cap / kTapeSegment + 1][m]
  int cap;
};

// TR-BDF2 integration of one sample (same algorithm as the oracle's Sample::integrate).
template <int NPL, class C>
__device__ int integrate(C& c, double (&y)[NPL], const double (&atol)[NPL], const double (&rtol)[NPL],
                         double t_beg, double t_end, double dt_in, double dt_min, double dt_max, int max_iters,
                         const NewtonSettings& s, double& t_out, double& dt_out, const Tape& tape = Tape{}) {
  if (dt_in < 0.0) return TCHEM_GB_SAMPLE_NEGATIVE_DT;
  const double gamma = 2.0 - sqrt(2.0);
  const double d = 0.5 * gamma;
  const double cg = 1.0 / (gamma * (2.0 - gamma));
  const double cn = (1.0 - gamma) * (1.0 - gamma) / (gamma * (2.0 - gamma));
  const double kappa = (-3.0 * gamma * gamma + 4.0 * gamma - 2.0) / (12.0 * (2.0 - gamma));
  const double e0 = 1.0 / gamma, e1 = -1.0 / (gamma * (1.0 - gamma)), e2 = 1.0 / (1.0 - gamma);
  const int m = sys_dim(c);

  double fn[NPL], fg[NPL], f1[NPL], yg[NPL], y1[NPL], rv[NPL];
  double t = t_beg, dt = dt_in;
  int status = TCHEM_GB_SAMPLE_OK;
  rhs(c, y, fn);
  for (int iter = 0; iter < max_iters && t < t_end; ++iter) {
    bool converged = false, last = false;
    for (int ntry = 0; ntry < 4; ++ntry) {
      dt = fmin(fmax(dt, dt_min), dt_max);
      last = dt >= t_end - t;
      if (last) dt = t_end - t;
      if (!(dt > 0.0)) { status = TCHEM_GB_SAMPLE_DT_UNDERFLOW; break; }
      const double coef = d * dt;
#pragma unroll
      for (int k = 0; k < NPL; ++k) { rv[k] = y[k] + coef * fn[k]; yg[k] = y[k]; }
      bool ok = newton(c, yg, rv, coef, s);
      if (ok) {
        rhs(c, yg, fg);
#pragma unroll
        for (int k = 0; k < NPL; ++k) { rv[k] = cg * yg[k] - cn * y[k]; y1[k] = yg[k]; }
        ok = newton(c, y1, rv, coef, s);
      }
      if (ok) { converged = true; break; }
      ++c.st.n_newton_fail;
      dt *= 0.5;
    }
    if (status != TCHEM_GB_SAMPLE_OK) break;
    if (!converged) { status = TCHEM_GB_SAMPLE_NEWTON_FAIL; break; }
    rhs(c, y1, f1);
    double est[NPL], estf[NPL];
#pragma unroll
    for (int k = 0; k < NPL; ++k) est[k] = 2.0 * kappa * dt * (e0 * fn[k] + e1 * fg[k] + e2 * f1[k]);
    lu_solve(c, est, estf);
    double err = 0.0;
#pragma unroll
    for (int k = 0; k < NPL; ++k) {
      if (c.lane + 32 * k < m) {
        const double wgt = atol[k] + rtol[k] * fmax(fabs(y[k]), fabs(y1[k]));
        err = fmax(err, fabs(estf[k]) / wgt);
      }
    }
    err = warp_max(err);
    if (!isfinite(err)) { status = TCHEM_GB_SAMPLE_NONFINITE; break; }
    if (err <= 1.0 || dt <= dt_min) {
      if (tape.dt) {
        const int n = c.st.n_steps;
        if (n >= tape.cap) { status = TCHEM_GB_SAMPLE_TAPE_FULL; break; }
        if (c.lane == 0) tape.dt[n] = dt;
        if (n % kTapeSegment == 0) {
#pragma unroll
          for (int k = 0; k < NPL; ++k) {
            const int i = c.lane + 32 * k;
            if (i < m) tape.ckpt[static_cast<size_t>(n / kTapeSegment) * m + i] = y[k];
          }
        }
      }
      t = last ? t_end : t + dt;
#pragma unroll
      for (int k = 0; k < NPL; ++k) { y[k] = y1[k]; fn[k] = f1[k]; }
      ++c.st.n_steps;
      double fac = err > 0.0 ? 0.9 * cbrt(1.0 / err) : 2.0;
      fac = fmax(0.2, fmin(2.0, fac));
      dt = fmin(dt * fac, dt_max);
      if (t + dt > t_end) dt = t_end - t;
    } else {
      ++c.st.n_rejected;
      dt *= fmax(0.2, 0.9 * cbrt(1.0 / err));
    }
  }
  t_out = t;
  dt_out = dt;
  if (status != TCHEM_GB_SAMPLE_OK) {
#pragma unroll
    for (int k = 0; k < NPL; ++k) y[k] = 0.0;
    t_out = t_end;
    dt_out = -1.0;
  }
  return status;
}


}  // namespace fp64
}  // namespace tchem_gb
