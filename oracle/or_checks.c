/*
 * or_checks.c -- ORACLE (test infrastructure only).  Array wrappers around
 * the shared scalar functions of cg_math.h / cg_cell.h so that tests can
 * check them against libm, numpy and HEALPix identities on the CPU.
 */
#include <stdint.h>
#include <stdlib.h>
#include <string.h>

#include "../colore_gb300/csrc/cg_exact.h"

void or_vec_expf(const float *x, float *y, long n) { for (long i = 0; i < n; i++) y[i] = cg_expf(x[i]); }
void or_vec_logf(const float *x, float *y, long n) { for (long i = 0; i < n; i++) y[i] = cg_logf(x[i]); }
void or_vec_log1pf(const float *x, float *y, long n) { for (long i = 0; i < n; i++) y[i] = cg_log1pf(x[i]); }
void or_vec_acosf(const float *x, float *y, long n) { for (long i = 0; i < n; i++) y[i] = cg_acosf(x[i]); }
void or_vec_atan2f(const float *y, const float *x, float *o, long n)
{
  for (long i = 0; i < n; i++) o[i] = cg_atan2f(y[i], x[i]);
}
void or_vec_sincosf(const float *x, float *s, float *c, long n)
{
  for (long i = 0; i < n; i++) cg_sincosf(x[i], &s[i], &c[i]);
}
/* Largest |cg_atan01_q(t) - atan(t) / (pi/2)| over every float t in [0, 1]
 * (libm's double atan as the reference). */
double or_atan_q_maxerr(void)
{
  const uint32_t top = 0x3f800000u; /* 1.0f */
  double mx = 0;
#pragma omp parallel for reduction(max : mx) schedule(static, 65536)
  for (long long b = 0; b <= (long long)top; b++) {
    const float t = cg_u2f((uint32_t)b);
    const double e = fabs((double)cg_atan01_q(t) - atan((double)t) * 0.63661977236758134308);
    if (e > mx) mx = e;
  }
  return mx;
}

void or_philox(const uint32_t *ctr, const uint32_t *key, uint32_t *out)
{
  cg_u32x4 r = cg_philox4x32_10(ctr[0], ctr[1], ctr[2], ctr[3], key[0], key[1]);
  for (int i = 0; i < 4; i++) out[i] = r.v[i];
}
void or_poisson(const float *lam, int *k, long n, uint32_t k0, uint32_t k1)
{
  for (long i = 0; i < n; i++) k[i] = cg_poisson(lam[i], k0, k1, (uint32_t)i, (uint32_t)(i >> 32));
}
void or_ang2pix(long nside, const float *cth, const float *phi, long long *pix, long n)
{
  for (long i = 0; i < n; i++) pix[i] = cg_ang2pix_ring(nside, cth[i], phi[i]);
}
void or_nest2ring(long nside, const long long *in, long long *out, long n)
{
  for (long i = 0; i < n; i++) out[i] = cg_nest2ring(nside, in[i]);
}
void or_ring2nest(long nside, const long long *in, long long *out, long n)
{
  for (long i = 0; i < n; i++) out[i] = cg_ring2nest(nside, in[i]);
}
void or_pix2vec_nest(long nside, const long long *in, float *v, long n)
{
  for (long i = 0; i < n; i++) cg_pix2vec_nest(nside, in[i], v + 3 * i);
}
void or_shell_index(const float *r0, const float *rf, int nr, const float *r, int *walk, int *bisect, long n)
{
  float rfm[4096];
  for (int i = 0; i < nr && i < 4096; i++) rfm[i] = i == 0 ? rf[0] : (rf[i] > rfm[i - 1] ? rf[i] : rfm[i - 1]);
  for (long i = 0; i < n; i++) {
    walk[i] = cg_shell_index(r0, rf, nr, r[i], 0);
    bisect[i] = cg_shell_index0(r0, rfm, nr, r[i]);
  }
}

/* RING pixels of float directions by the margin-checked single-precision
 * path (cg_pix_checked; -1 where it defers to double), with coordinate
 * error ein relative to r. */
void or_pix_checked(long nside, const float *xyz, long n, float ein, long long *pix)
{
  for (long i = 0; i < n; i++) {
    const cg_dir d = cg_dir_of(xyz[3 * i], xyz[3 * i + 1], xyz[3 * i + 2], ein);
    pix[i] = cg_pix_checked(&d, (int)nside, ein);
  }
}

/* The float-float operations of cg_ff.h on n operand pairs: op 0 sum,
 * 1 product, 2 quotient, 3 square root of x, 4 product by the float y.h;
 * x and y as (h, l) pairs in xh/xl, yh/yl, the result in oh/ol. */
void or_ff_ops(int op, const float *xh, const float *xl, const float *yh, const float *yl, long n, float *oh,
               float *ol)
{
  for (long i = 0; i < n; i++) {
    const cg_ff x = cg_ff_make(xh[i], xl[i]), y = cg_ff_make(yh[i], yl[i]);
    cg_ff r;
    if (op == 0) r = cg_ff_add(x, y);
    else if (op == 1) r = cg_ff_mul(x, y);
    else if (op == 2) r = cg_ff_div(x, y);
    else if (op == 3) r = cg_ff_sqrt(x);
    else r = cg_ff_mulf(x, y.h);
    oh[i] = r.h;
    ol[i] = r.l;
  }
}

/* RING pixels of float-float positions (6 floats each: x, its rest, y, ...)
 * by the float-float tier (cg_pix_ff; -1 where it defers to double), each
 * within eP[i] of the double position. */
void or_pix_ff(long nside, const float *p, const float *eP, long n, long long *pix)
{
  float att[2 * (CG_ATT_N + 1)];
  cg_att_table(att);
  for (long i = 0; i < n; i++) {
    const float *q = p + 6 * i;
    pix[i] = cg_pix_ff(cg_ff_make(q[0], q[1]), cg_ff_make(q[2], q[3]), cg_ff_make(q[4], q[5]), eP[i], (int)nside,
                       att);
  }
}

/* The same decision by the double restatement shared with the kernels
 * (cgx_cart2sph + cgx_ang2pix). */
void or_pix_cgx(long nside, const double *xyz, long n, long long *pix)
{
  for (long i = 0; i < n; i++) {
    double r, cth, ph;
    cgx_cart2sph(xyz[3 * i], xyz[3 * i + 1], xyz[3 * i + 2], &r, &cth, &ph);
    pix[i] = cgx_ang2pix(nside, cth, ph);
  }
}

/* cg_src_offset_checked on n (corner, uniform) pairs with one dx: out[i] the
 * float coordinate (0 when not certain), ok[i] 1 when certain; ref[i] the
 * double expression rounded to float (cgx_src_offset). */
void or_src_offset_checked(long n, const double *x0, double dx, const uint32_t *bits, float *out, int *ok, float *ref)
{
  const float dh = (float)dx, dl = (float)(dx - (double)(float)dx);
  for (long i = 0; i < n; i++) {
    const float c = (float)x0[i], l = (float)(x0[i] - (double)(float)x0[i]);
    float f = 0.0f;
    ok[i] = cg_src_offset_checked(c, l, dh, dl, bits[i], &f);
    out[i] = f;
    ref[i] = cgx_src_offset(x0[i], dx, bits[i]);
  }
}

/* cg_poisson_ptrs_checked against cgx_poisson_ptrs on n means: got[i] the
 * single-precision count (-1: left to double), ref[i] the double one, for
 * float means lam[i] known within elam[i] of the double mean lam64[i]. */
void or_ptrs_checked(long n, const float *lam, const float *elam, const double *lam64, const long long *cid, uint32_t k0,
                     uint32_t k1, int *got, int *ref)
{
  for (long i = 0; i < n; i++) {
    got[i] = cg_poisson_ptrs_checked(lam[i], elam[i], cid[i], k0, k1);
    ref[i] = cgx_poisson_ptrs(lam64[i], cid[i], k0, k1);
  }
}

/* The counts' first tier (cg_lambda_seg, cg_tier_*) on n cells of a table
 * of NA nodes at r_i = i / idr: lam[i] within elam[i] of lam64[i]
 * (cgx_lambda), got[i] the tier's count, -1 when it leaves the cell open or -2
 * when it leaves it to PTRS, ref[i] the double count for lambda < 10 with the
 * uniform bits[i] 2^-24. */
void or_count_seg(const double *r, const double *nz, const double *bz, const double *norm, double idr, double dx,
                  const double *pos, double cell_vol, double rlim, int model, long n, const int *cell, const float *d,
                  const uint32_t *bits, float *lam, float *elam, double *lam64, int *got, int *ref)
{
  cg_pois_args a;
  memset(&a, 0, sizeof(a));
  a.x.r = r;
  a.x.nz = nz;
  a.x.bz = bz;
  a.x.norm = norm;
  a.x.idr = idr;
  a.x.r_last = r[CG_NA - 1];
  a.x.bz0 = bz[0];
  a.x.dx = dx;
  a.x.cell_vol = cell_vol;
  a.x.rlim = rlim;
  for (int k = 0; k < 3; k++) a.x.p[k] = pos[k];
  a.x.bias_model = model;
  a.idr = (float)idr;
  a.r_last = (float)a.x.r_last;
  a.rlim = (float)rlim;
  a.bias_model = model;
  float lo, hi;
  cg_tier_limits(&a, &lo, &hi);
  cg_pois_seg *seg = malloc((CG_NA - 1) * sizeof(cg_pois_seg));
  for (int i = 0; i < CG_NA - 1; i++) seg[i] = cg_pois_seg_make(&a.x, CG_NA, i);
  for (long i = 0; i < n; i++) {
    const int *c = cell + 3 * i;
    const float x = (float)cgx_coord(c[0], dx, pos[0]), y = (float)cgx_coord(c[1], dx, pos[1]);
    const float z = (float)cgx_coord(c[2], dx, pos[2]);
    const float r2 = CG_FMA(x, x, CG_FMA(z, z, CG_MUL(y, y)));
    const float u = CG_MUL((float)bits[i], CG_E24);
    float rr;
    const float s = cg_seg_pos(r2, a.idr, &rr);
    int j = (int)s, pos1;
    j = r2 > 0.0f && j < CG_NA - 1 ? j : 0;
    lam[i] = cg_lambda_seg(&seg[j], CG_SUB(s, (float)j), d[i], model, &elam[i], &pos1);
    lam64[i] = cgx_lambda(&a.x, c[0], c[1], c[2], d[i]);
    got[i] = rr > hi ? 0 : -1;
    if (!(rr > hi) && cg_tier_inside(r2, rr, lo)) {
      int t = cg_tier_lambda(lam[i], elam[i], pos1);
      if (cg_tier_uniform(lam[i], elam[i], u)) t &= ~CG_TIER_MAY;
      if (t & CG_TIER_PTRS) got[i] = -2;
      else if (!(t & CG_TIER_MAY)) got[i] = 0;
      else if (t & CG_TIER_INV) got[i] = cg_poisson_inv_checked(lam[i], elam[i], u);
    }
    ref[i] = lam64[i] < 10 ? cgx_poisson(lam64[i], (double)u, i, 1u, 2u) : -1;
  }
  free(seg);
}

/* A source's direction from one octant angle (cg_dir_phi): ph its phi and
 * ref that of cg_cart2sph; pix the RING pixel at nside (-1 where its margin
 * fails).  Positions are the float xyz. */
void or_dir_phi(long nside, const float *xyz, long n, float *ph, float *ref, long long *pix)
{
  for (long i = 0; i < n; i++) {
    float r, cth;
    const cg_dir d = cg_dir_phi(xyz[3 * i], xyz[3 * i + 1], xyz[3 * i + 2], &ph[i]);
    cg_cart2sph(xyz[3 * i], xyz[3 * i + 1], xyz[3 * i + 2], &r, &cth, &ref[i]);
    pix[i] = cg_pix_checked(&d, (int)nside, 0.0f);
  }
}

/* cg_next_float of f[i] upwards (up[i] != 0) or downwards. */
void or_next_float(long n, const float *f, const int *up, float *out)
{
  for (long i = 0; i < n; i++) out[i] = cg_next_float(f[i], up[i]);
}

/* Samples of whole cells by the per-cell constants (cg_imap_fast_cell) against
 * the double arithmetic: cell (3 ints) of a box of N cells of side dx with the
 * observer at pos, nsub sub-cells per axis.  edge[i] > 0: the cell crosses the
 * shell edge edge[i] with radial shift drr[i] known within edrr of drr64[i]
 * (shells 0 below, 1 above); else one shell.  stat[0..4]: fast cells,
 * equatorial ones, their samples, samples decided, and decided wrongly. */
void or_imap_fast(long nside, int N, double dx, const double *pos, long n, const int *cell, const int *nsub,
                  const float *edge, const float *drr, const double *drr64, float edrr, long long *stat)
{
  float b[1];
  int shell_of[2] = {0, 1};
  cg_imap_args a;
  memset(&a, 0, sizeof(a));
  a.dx = (float)dx;
  a.nside = (int)nside;
  a.sh.b = b;
  a.sh.shell_of = shell_of;
  a.sh.nb = 1;
  a.sh.nr = 2;
  a.sh.contig = 1;
  for (int k = 0; k < 5; k++) stat[k] = 0;
  for (long i = 0; i < n; i++) {
    const int *ci = cell + 3 * i, ns = nsub[i];
    const float dxs = (float)(dx / ns);
    cg_imap_cell c;
    memset(&c, 0, sizeof(c));
    b[0] = edge[i];
    c.j = 0;
    c.drr = drr[i];
    c.edrr = edrr;
    c.mode = edge[i] > 0 ? CG_SH_EDGE : CG_SH_SINGLE;
    c.delta = edge[i] > 0 ? -1 : 0; /* intervals -1 and 0 */
    float h[3], l[3];
    for (int k = 0; k < 3; k++) {
      const double x = cgx_coord(ci[k], dx, pos[k]);
      h[k] = (float)x;
      l[k] = (float)(x - (double)h[k]);
    }
    cg_imap_fast F;
    const int cls = cg_cell_class(&a, &c, h[0], h[1], h[2]);
    if (cls == CG_CELL_GENERAL) continue;
    cg_imap_fast_cell(&a, &c, cls, h[0], h[1], h[2], &F);
    stat[0]++;
    stat[1] += cls == CG_CELL_EQ;
    for (int q = 0; q < ns * ns * ns; q++) {
      const int sx = q % ns, sy = q / ns % ns, sz = q / (ns * ns);
      const float x = cg_imap_coord(&h[0], &l[0], 0, sx, dxs), y = cg_imap_coord(&h[1], &l[1], 0, sy, dxs);
      const float z = cg_imap_coord(&h[2], &l[2], 0, sz, dxs);
      const float u = F.ymaj ? y : x, v = F.ymaj ? x : y;
      int up, pix, ok;
      if (cls == CG_CELL_EQ) {
        ok = cg_fast_eq(&F, (int)nside, cg_fast_eq_thr((int)nside), u, v, z, CG_FMA(z, z, CG_MUL(v, v)), &up, &pix);
      } else {
        const cg_fast_line line = cg_fast_polar_line(&F, (int)nside, u, v);
        ok = cg_fast_polar(&F, &line, cg_fast_polar_k0((int)nside), z, &up, &pix);
      }
      const int s = up ? F.s1 : F.s0;
      stat[2]++;
      if (!ok) continue;
      stat[3]++;
      const double step = X_DIV(dx, (double)ns);
      const double X = X_ADD(cgx_coord(ci[0], dx, pos[0]), X_MUL(X_ADD((double)sx, 0.5), step));
      const double Y = X_ADD(cgx_coord(ci[1], dx, pos[1]), X_MUL(X_ADD((double)sy, 0.5), step));
      const double Z = X_ADD(cgx_coord(ci[2], dx, pos[2]), X_MUL(X_ADD((double)sz, 0.5), step));
      double r, cth, ph;
      cgx_cart2sph(X, Y, Z, &r, &cth, &ph);
      const int want = edge[i] > 0 ? (X_ADD(r, drr64[i]) >= (double)edge[i]) : 0;
      stat[4] += pix != cgx_ang2pix(nside, cth, ph) || s != want;
    }
  }
  (void)N;
}
