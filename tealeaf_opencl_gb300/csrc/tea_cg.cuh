// CG tile bodies shared by the single-chunk kernels (tea_kernels.cu) and
// the batched kernels (tea_batch.cu): one lane's column x of one tile,
// rows y0 .. y0+TH-1, with the arithmetic of the reference kernels.
#pragma once

#include "tea_device.cuh"

namespace tea {

// Every tile body below works in groups of 4 rows and, within a group,
// issues all of its loads before its first store.  The fields are reached
// through the members of Dev, which the compiler must assume may alias, so
// a load written after a store cannot move above it; loading the group
// first keeps 4 rows of loads in flight instead of one.  The arithmetic and
// the order of the per-lane sums are those of the row-by-row form.

// w = A p and the lane's share of p.w (tea_leaf_cg_cl.cl:45-69), with the fields
// reached through restrict-qualified pointers: p and the coefficients are only
// read and w only written, so the compiler may issue a group's loads before
// the previous group's stores and keep more loads in flight.  Same
// arithmetic and per-lane summation order; with 4 blocks per SM (64
// registers) 192.2 -> 174.4 us at 4096^2 on non-zero fields.
template <int TH, int F, bool EMU = true>
__device__ __forceinline__ void cg_w_tile_r(const Dev& d, int x, int y0, bool xin,
                                            double* acc) {
  const double* __restrict__ p = d.p;
  const double* __restrict__ kx = d.Kx;
  const double* __restrict__ ky = d.Ky;
  const double* __restrict__ dg = d.diag;
  double* __restrict__ w = d.w;
  const long long S = d.S;
#pragma unroll 1
  for (int g = y0; g < y0 + TH; g += 4) {
    const long long c0 = cidx(d, x, g);
    double pv[4], wv[4];
#pragma unroll
    for (int j = 0; j < 4; j++) {
      pv[j] = 0.0;
      wv[j] = 0.0;
      if (xin && g + j < d.y_max) {
        const long long c = c0 + j * S;
        pv[j] = p[c];
        wv[j] = smvp_v<F, EMU>(__ldg(dg + c), __ldg(ky + c + S), __ldg(ky + c), __ldg(kx + c + 1),
                          __ldg(kx + c), pv[j], p[c + S], p[c - S], p[c + 1], p[c - 1]);
      }
    }
#pragma unroll
    for (int j = 0; j < 4; j++)
      if (xin && g + j < d.y_max) w[c0 + j * S] = wv[j];
#pragma unroll
    for (int j = 0; j < 4; j++) acc[0] = accum<F>(acc[0], pv[j], wv[j]);
  }
}

// u += alpha p; r -= alpha w (tea_leaf_cg_cl.cl:88-89) on loaded values
template <int F>
__device__ __forceinline__ void ur_values(double alpha, double& u, double p,
                                          double& r, double w) {
  if (F) {
    u = __fma_rn(alpha, p, u);
    r = __fma_rn(-alpha, w, r);
  } else {
    u = u + alpha * p;
    r = r - alpha * w;
  }
}

// u += alpha p, r -= alpha w, z = M^-1 r and the lane's share of r.z (no sum
// when NV == 0), tea_leaf_cg_cl.cl:73-137.  With SD it also starts PPCG's inner
// steps, sd = M^-1 r / theta (tea_leaf_ppcg_cl.cl:4-60), from the z it has just
// formed: the same values tea_leaf_ppcg_solve_init_sd computes from the stored
// r.  The fields are reached through restrict-qualified pointers and
// the strip coefficients loaded with u, p, r and w, before the stores of u
// and r, so that more loads are in flight.  The strip solve reads exactly
// the rows strip_solve reads (a strip may end in the halo row).  Same
// arithmetic and per-lane summation order; with 4 blocks per SM (64
// registers), on non-zero fields at 4096^2 (block Jacobi): calc_ur 246.4 ->
// 210.9 us, calc_ur + init_sd 223.7 -> 215.0 us.
template <int TH, int F, int NV, bool SD = false>
__device__ __forceinline__ void cg_ur_tile_r(const Dev& d, int x, int y0, bool xin,
                                             double* acc, double alpha,
                                             const DivConst& theta = DivConst{}) {
  double* __restrict__ u = d.u;
  const double* __restrict__ p = d.p;
  double* __restrict__ r = d.r;
  const double* __restrict__ w = d.w;
  double* __restrict__ z = d.z;
  double* __restrict__ sd = d.sd;
  const long long S = d.S;
  // the lane's sums and the z / sd stores of one group of 4 rows
  auto finish = [&](long long c0, const bool in[4], const double rv[4], const double zv[4],
                    bool prec) {
#pragma unroll
    for (int j = 0; j < 4; j++) {
      double av = 0.0, bv = 0.0;
      if (in[j]) {
        if (prec) z[c0 + j * S] = zv[j];
        if (SD) sd[c0 + j * S] = emu_ddiv(prec ? zv[j] : rv[j], theta);
        av = rv[j];
        bv = prec ? zv[j] : rv[j];
      }
      if (NV > 0) acc[0] = accum<F>(acc[0], av, bv);
    }
  };
  if (d.prec == PREC_JAC_BLOCK) {
    const double* __restrict__ bfp = d.bfp;
    const double* __restrict__ ky = d.Ky;
    const double* __restrict__ cp = d.cp;
#pragma unroll 1
    for (int g = y0; g < y0 + TH; g += 4) {
      const long long c0 = cidx(d, x, g);
      const int upper = xin && g < d.y_max ? strip_rows(d, g) : 0;
      bool in[4];
      double uv[4], rv[4], bl[4], kl[4], cl[4];
#pragma unroll
      for (int j = 0; j < 4; j++) {
        in[j] = xin && g + j < d.y_max;
        uv[j] = rv[j] = bl[j] = kl[j] = cl[j] = 0.0;
        const long long c = c0 + j * S;
        if (in[j]) {
          uv[j] = u[c];
          rv[j] = r[c];
          ur_values<F>(alpha, uv[j], p[c], rv[j], w[c]);
        }
        if (j < upper) {
          if (F || j > 0) bl[j] = __ldg(bfp + c);
          if (j > 0) kl[j] = __ldg(ky + c);
          if (j + 1 < upper) cl[j] = __ldg(cp + c);
        }
      }
      const double d0 = !F && upper > 0 ? __ldg(d.diag + c0) : 0.0;
#pragma unroll
      for (int j = 0; j < 4; j++)
        if (in[j]) {
          u[c0 + j * S] = uv[j];
          r[c0 + j * S] = rv[j];
        }
      double zv[4] = {0.0, 0.0, 0.0, 0.0};
      if (upper == 4)
        strip_solve_v<F, false, true>(4, rv, bl, kl, cl, d0, zv);
      else if (upper > 0)
        strip_solve_v<F, false>(upper, rv, bl, kl, cl, d0, zv);
      finish(c0, in, rv, zv, true);
    }
  } else {
    const bool dia = d.prec == PREC_JAC_DIAG;
    const double* __restrict__ mi = d.Mi;
#pragma unroll 1
    for (int g = y0; g < y0 + TH; g += 4) {
      const long long c0 = cidx(d, x, g);
      bool in[4];
      double uv[4], rv[4], zv[4];
#pragma unroll
      for (int j = 0; j < 4; j++) {
        in[j] = xin && g + j < d.y_max;
        uv[j] = rv[j] = zv[j] = 0.0;
        const long long c = c0 + j * S;
        if (in[j]) {
          uv[j] = u[c];
          rv[j] = r[c];
          ur_values<F>(alpha, uv[j], p[c], rv[j], w[c]);
          if (dia) zv[j] = rv[j] * mi[c];
        }
      }
#pragma unroll
      for (int j = 0; j < 4; j++)
        if (in[j]) {
          u[c0 + j * S] = uv[j];
          r[c0 + j * S] = rv[j];
        }
      finish(c0, in, rv, zv, dia);
    }
  }
}

// p = z + beta p, or r + beta p without a preconditioner
// (tea_leaf_cg_cl.cl:141-160)
template <int TH, int F>
__device__ __forceinline__ void cg_p_tile(const Dev& d, int x, int y0, bool xin,
                                          double beta) {
  if (!xin) return;
  const double* src = d.prec != PREC_NONE ? d.z : d.r;
#pragma unroll 1
  for (int g = y0; g < y0 + TH; g += 4) {
    const long long c0 = cidx(d, x, g);
    double sv[4], pv[4];
#pragma unroll
    for (int j = 0; j < 4; j++) {
      sv[j] = pv[j] = 0.0;
      if (g + j < d.y_max) {
        sv[j] = src[c0 + j * d.S];
        pv[j] = d.p[c0 + j * d.S];
      }
    }
#pragma unroll
    for (int j = 0; j < 4; j++)
      if (g + j < d.y_max)
        d.p[c0 + j * d.S] = F ? __fma_rn(beta, pv[j], sv[j]) : sv[j] + beta * pv[j];
  }
}

// ---- the two-pass CG iteration (tea_cg_loop.cu, tea_batch.cu) ----

// The exact form's product is one FP64 instruction more, and pass w forms p' of
// the cells around a tile a second time: on the integer pipes (bit-identical)
// it leaves the two passes ahead of three kernels, see k_cg_pass_r.
template <int F, bool EMU = false>
__device__ __forceinline__ double p_next(double beta, double p, double z) {
  return F ? __fma_rn(beta, p, z) : z + mul_e<EMU>(beta, p);
}

// Pass A on one tile: lane column x, rows y0 .. y0+TH-1.  p' of the rows
// above and below and of the columns either side is formed here too (the
// two columns by lanes 0-7, one multiply-add for four rows), so no pass and
// no grid barrier separates p' from w.  Halo cells keep the p they were given
// (they are read from d.p whichever buffer is current).  On the first
// iteration of a launch p is current already (it stays in pin, or with COPY
// goes to pout as it is) and u has nothing pending.
// p and z are written by other SMs during the launch: they are read through
// L2.  All loads of four rows are issued before anything waits for one; rows
// past the interior are clamped to the halo row above it and lanes past the
// last column read the row's padding, and neither is used.
// PE: the exact form's alpha p and beta p on the integer pipes.
template <int TH, int F, bool COPY = false, bool EMU = true, bool PE = EMU>
__device__ __forceinline__ double loop_w_tile(const Dev& d, const double* __restrict__ pin,
                                              double* __restrict__ pout,
                                              const double* __restrict__ zsrc, int x, int y0,
                                              double alpha, double beta, bool first) {
  const int lane = threadIdx.x & 31;
  const double* __restrict__ hal = d.p;
  const double* __restrict__ kx = d.Kx;
  const double* __restrict__ ky = d.Ky;
  const double* __restrict__ dg = d.diag;
  double* __restrict__ u = d.u;
  double* __restrict__ w = d.w;
  const long long S = d.S;
  const long long c0 = cidx(d, x, y0);
  const bool xin = x < d.x_max;
  const int rows = min(TH, d.y_max - y0);
  const bool top = y0 + rows == d.y_max;  // row `rows` is halo
  const double* __restrict__ pcol = xin ? pin : hal;
  // p' from the old p and z; halo cells keep p
  auto fresh = [&](double po, double zv, bool in) {
    return first || !in ? po : p_next<F, PE>(beta, po, zv);
  };
  double acc = 0.0;
  double pm = 0.0, pc = 0.0, pco = 0.0;  // p' of rows g-1 and g, old p of row g
#pragma unroll 1
  for (int g = 0; g < rows; g += 4) {
    const bool bottom = TH == 4 || g == 0;
    double po[6], zv[6], uv[4], kyv[5], kxc[4], kxe[4], dv[4];
    const int er = min(g + (lane >> 1), rows - 1);
    const int xe = (lane & 1) ? x - lane + 32 : x - lane - 1;
    const bool ein = xe >= 0 && xe < d.x_max;
    double ep = 0.0, ez = 0.0;
#pragma unroll
    for (int j = 0; j < 6; j++) {
      po[j] = zv[j] = 0.0;
      if (j < 2 && !bottom) continue;  // carried from the group below
      const int row = min(g + j - 1, rows);
      const bool rin = (row >= 0 || y0 > 0) && !(row == rows && top);
      const long long c = c0 + row * S;
      po[j] = __ldcg((rin ? pcol : hal) + c);
      zv[j] = __ldcg(zsrc + c);
    }
    if (lane < 8) {
      const long long c = cidx(d, xe, y0 + er);
      ep = __ldcg((ein ? pin : hal) + c);
      ez = __ldcg(zsrc + c);
    }
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const long long c = c0 + min(g + j, rows - 1) * S;
      uv[j] = u[c];
      kyv[j] = __ldg(ky + c);
      kxc[j] = __ldg(kx + c);
      kxe[j] = __ldg(kx + c + 1);
      dv[j] = __ldg(dg + c);
    }
    kyv[4] = __ldg(ky + c0 + min(g + 4, rows) * S);
    double pv[6];
    pv[0] = pm;
    pv[1] = pc;
    if (!bottom) po[1] = pco;
#pragma unroll
    for (int j = 0; j < 6; j++) {
      if (j < 2 && !bottom) continue;
      const int row = min(g + j - 1, rows);
      const bool rin = (row >= 0 || y0 > 0) && !(row == rows && top);
      pv[j] = fresh(po[j], zv[j], rin && xin);
    }
    const double ev = fresh(ep, ez, ein);
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const long long c = c0 + (g + j) * S;
      const bool own = xin && g + j < rows;
      if (own && !first)
        u[c] = F ? __fma_rn(alpha, po[j + 1], uv[j]) : uv[j] + mul_e<PE>(alpha, po[j + 1]);
      double pe = __shfl_down_sync(0xffffffffu, pv[j + 1], 1);
      double pw = __shfl_up_sync(0xffffffffu, pv[j + 1], 1);
      const double e = __shfl_sync(0xffffffffu, ev, 2 * j + 1);
      const double wst = __shfl_sync(0xffffffffu, ev, 2 * j);
      if (lane == 31) pe = e;
      if (lane == 0) pw = wst;
      const double kyn = j < 3 && g + j + 1 < rows ? kyv[j + 1] : kyv[4];
      const double wv = smvp_v<F, EMU>(dv[j], kyn, kyv[j], kxe[j], kxc[j], pv[j + 1], pv[j + 2], pv[j],
                                  pe, pw);
      if (own) {
        w[c] = wv;
        if (COPY || !first) pout[c] = pv[j + 1];
      }
      acc = accum<F>(acc, own ? pv[j + 1] : 0.0, own ? wv : 0.0);
    }
    pm = pv[4];
    pc = pv[5];
    pco = po[5];
  }
  return acc;
}

// Pass B on one tile: r -= alpha w, z = M^-1 r and the lane's share of r.z
// (cg_ur_tile_r without u, which pass A updates).  A lane reads back only
// the r and w that it wrote itself.  RE: the exact form's alpha w on the integer
// pipes.
template <int TH, int F, int NV = 1, bool EMU = true, bool RE = false>
__device__ __forceinline__ void loop_r_tile(const Dev& d, int x, int y0, double alpha,
                                            double* acc) {
  double* __restrict__ r = d.r;
  const double* __restrict__ w = d.w;
  double* __restrict__ z = d.z;
  const long long S = d.S;
  if (x >= d.x_max) return;
  const int rows = min(TH, d.y_max - y0);
  auto r_next = [&](double rr, double ww) {
    return F ? __fma_rn(-alpha, ww, rr) : rr - mul_e<RE>(alpha, ww);
  };
#pragma unroll 1
  for (int g = 0; g < rows; g += 4) {
    const long long c0 = cidx(d, x, y0 + g);
    double rv[4], wv[4], mv[4], zv[4];
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const long long c = c0 + min(j, rows - 1 - g) * S;
      wv[j] = w[c];
      rv[j] = r[c];
      mv[j] = d.prec == PREC_JAC_DIAG ? __ldg(d.Mi + c) : 0.0;
    }
    if (d.prec == PREC_JAC_BLOCK) {
      const int upper = strip_rows(d, y0 + g);
      double bl[4], kl[4], cl[4];
#pragma unroll
      for (int j = 0; j < 4; j++) {
        const long long c = c0 + min(j, upper - 1) * S;
        bl[j] = __ldg(d.bfp + c);
        kl[j] = __ldg(d.Ky + c);
        cl[j] = __ldg(d.cp + c);
      }
      const double d0 = F ? 0.0 : __ldg(d.diag + c0);
#pragma unroll
      for (int j = 0; j < 4; j++)
        rv[j] = g + j >= rows ? 0.0 : r_next(rv[j], wv[j]);
      if (upper == 4)
        strip_solve_v<F, false, true>(4, rv, bl, kl, cl, d0, zv);
      else
        strip_solve_v<F, false>(upper, rv, bl, kl, cl, d0, zv);
    } else {
#pragma unroll
      for (int j = 0; j < 4; j++) {
        rv[j] = r_next(rv[j], wv[j]);
        zv[j] = d.prec == PREC_JAC_DIAG ? mul_e<EMU>(rv[j], mv[j]) : rv[j];
      }
    }
#pragma unroll
    for (int j = 0; j < 4; j++) {
      if (g + j < rows) {
        r[c0 + j * S] = rv[j];
        if (d.prec != PREC_NONE) z[c0 + j * S] = zv[j];
        acc[0] = accum<F>(acc[0], rv[j], zv[j]);
        if (NV > 1 && d.prec != PREC_NONE) acc[NV - 1] = accum<F>(acc[NV - 1], rv[j], rv[j]);
      }
    }
  }
  if (NV > 1 && d.prec == PREC_NONE) acc[NV - 1] = acc[0];  // z is r
}

// tea_leaf_jacobi_copy_u and tea_leaf_jacobi_solve in one pass
// (tea_leaf_jacobi_cl.cl:3-42; un is vector_Mi, as in the reference,
// ocl_kernels.cpp:576-585): un = u over the interior, one sweep from un, the sum
// of |u - un|.  The sweep reads the old u where un would hold its copy, and
// un's own halo; the new u goes to unew with u's halo ring, and un gets the old
// u, so the fields end as the two kernels leave them.  48 bytes per cell in
// place of 56 and one launch in place of two.  The sums of each cell stay in
// the reference's association (its denominator differs from the stored
// diagonal); two of the four products run on the integer pipes beside the
// division (bit-identical).  One lane's column of one tile: the lane's share of
// the sum.  un, where the old u goes, may be null (the resident loop copies it
// once at its end).  CG: u through L2, where other SMs write it during the
// launch.
template <int TH, bool CG, bool EMU = true>
__device__ __forceinline__ double jacobi_tile(const Dev& d, const double* __restrict__ u,
                                              double* __restrict__ unew, double* __restrict__ un,
                                              int x, int y0) {
  const double* hal = d.un;  // read only outside the interior
  const long long S = d.S;
  const double* west = x > 0 ? u : hal;
  const double* east = x + 1 < d.x_max ? u : hal;
  const int rows = min(TH, d.y_max - y0);
  double acc = 0.0;
#pragma unroll 1
  for (int g = 0; g < rows; g += 4) {
    const long long c0 = cidx(d, x, y0 + g);
    const int last = rows - 1 - g;  // last interior row of the group, or more
    double uc[6], kyv[5], nw[4], v[4];
#pragma unroll
    for (int i = 0; i < 6; i++) {
      const int j = min(i - 1, last + 1), y = y0 + g + j;
      uc[i] = ldv<CG>((y < 0 || y >= d.y_max ? hal : u) + c0 + j * S);
    }
#pragma unroll
    for (int i = 0; i < 5; i++) kyv[i] = __ldg(d.Ky + c0 + min(i, last + 1) * S);
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const long long c = c0 + min(j, last) * S;
      const double kxc = __ldg(d.Kx + c), kxe = __ldg(d.Kx + c + 1);
      const double s = __ldg(d.u0 + c) + mul_e<EMU>(kxe, ldv<CG>(east + c + 1)) +
                       kxc * ldv<CG>(west + c - 1) + mul_e<EMU>(kyv[j + 1], uc[j + 2]) +
                       kyv[j] * uc[j];
      const double den = 1.0 + (kxc + kxe) + (kyv[j] + kyv[j + 1]);
      nw[j] = EMU ? emu_ddiv_var(s, den) : s / den;
      v[j] = j <= last ? fabs(nw[j] - uc[j + 1]) : 0.0;
    }
#pragma unroll
    for (int j = 0; j < 4; j++)
      if (j <= last) {
        unew[c0 + j * S] = nw[j];
        if (un) un[c0 + j * S] = uc[j + 1];
      }
#pragma unroll
    for (int j = 0; j < 4; j++) acc = acc + v[j];
  }
  return acc;
}

// The host steps of one CG iteration (tea_solve.f90:282-330) after calc_ur,
// on the device: beta = rrn/rro, rro = rrn, error = sqrt(rrn), and the exit
// test (on sqrt(r.z), or on ||r||_2 when NV == 2).  result[] holds the
// reduced sums; run by one thread.
template <int NV>
__device__ __forceinline__ void cg_scalar_step(ResState* st, double alpha,
                                               const double* result) {
  const double rrn = result[0];
  const int n = st->n;
  if (st->check) {
    // breakdown (the caller asked for the check; the reference runs on)
    const double pw = st->pw;
    const int b = !(pw > 0.0) || isinf(pw) ? 1 : (isfinite(rrn) ? 0 : 2);
    if (b) {
      st->breakdown = b;
      st->breakdown_n = n;
      st->stop = 1;
      st->p_pending = 0;
      return;
    }
  }
  const double beta = rrn / st->rro;
  if (st->alphas) {
    st->alphas[n] = alpha;
    st->betas[n] = beta;
  }
  st->alpha = alpha;
  st->beta = beta;
  st->rrn = rrn;
  st->rro = rrn;
  const double err = sqrt(rrn);
  st->error = err;
  st->p_pending = 1;
  const bool done = NV > 1 ? sqrt(result[NV - 1]) < st->eps_target
                           : fabs(err) < st->eps_target;
  if (NV > 1) st->rr_true = result[NV - 1];
  if (done) {
    st->converged = 1;
    st->stop = 1;
  } else if (n >= st->loop_max ||
             (st->switch_n > 0 && n + 1 >= st->switch_n && fabs(err) <= st->switch_eps)) {
    st->stop = 1;
  } else {
    st->n = n + 1;
  }
}

}  // namespace tea
