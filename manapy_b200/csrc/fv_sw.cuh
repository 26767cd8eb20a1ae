// Arithmetic of the shallow-water step on triangles, shared by the face and cell kernels of the
// two-launch step (fv_sw.cu) and the one-launch step on tiles (fv_sw_tile.cu).
//
// Every operation is written with its rounding (multiply-adds where they are meant), so the
// compiler contracts nothing by itself and both steps give the same bits: a sharded run, which
// takes the two-launch step in parts, equals the single-domain run that takes the tiles.
#pragma once

#include "fv_tile.cuh"

namespace mb {

__device__ __forceinline__ double swm(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double swa(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double sws(double a, double b) { return __dsub_rn(a, b); }
__device__ __forceinline__ double swf(double a, double b, double c) { return __fma_rn(a, b, c); }   // a b + c
__device__ __forceinline__ double swd(double a, double b, double c, double d) {                     // a b + c d
  return swf(a, b, swm(c, d));
}
__device__ __forceinline__ double swx(double a, double b, double c, double d) {                     // a b - c d
  return swf(a, b, -swm(c, d));
}

// SRNH flux specialised to manapy's constant As = 0 (d = 0, beta = 0; flux[4] is identically
// zero), with the eigenvalues of manapy's cubic lambda (lambda^2 - 2 u lambda + u^2 - c^2) in
// closed form, a = u + c, b = u - c and 0.  Put into manapy's rows
//   r_k = sum_k sign(lambda_k) {gamma, alpha sums, c^2} / sigma_k
// they cancel: with l' the other two eigenvalues sigma_k = +-(lambda_k - l')(lambda_k - l''),
// gamma_k = c^2 - u^2 + l' l'' and c^2 - u^2 = -a b, so for lambda = a, b the three quotients
// are -b / 2c, -1 / 2c, c / 2a and a / 2c, 1 / 2c, -c / 2b; lambda = 0 has sign 0.  Rows 2
// and 3 (tangential velocity, tracer) are v and c_h times row 0 plus the wave of speed u.
// Results differ from manapy's by rounding only.
//
// The FP64 pipe bounds the face kernels (about 500 FP64 instructions per face when written
// row by row, with 9 divisions), so quotients that share a denominator, or whose
// denominators may be multiplied, take one division: 1 / (sl sr (sl + sr) mesure) for the Roe
// means (hu_l / h_l sl = hu_l / sl) and the unit normal, 1 / (2 c a b) for 1 / 2c, 1 / a and 1 / b,
// 1 / w_h.
__device__ __forceinline__ void srnh0(double hu_l, double hu_r, double hv_l, double hv_r, double h_l, double h_r,
                                      double hc_l, double hc_r, double Z_l, double Z_r, double n0, double n1,
                                      double mesure, double grav, double flux[4]) {
  const double sl = __dsqrt_rn(h_l), sr = __dsqrt_rn(h_r);
  const double ss = swm(swm(sl, sr), swa(sl, sr));
  const double R = __ddiv_rn(1., swm(ss, mesure));
  const double K = swm(R, mesure), im = swm(R, ss);
  const double u_h = swm(swd(hu_l, sr, hu_r, sl), K);
  const double v_h = swm(swd(hv_l, sr, hv_r, sl), K);
  const double c_h = swm(swd(hc_l, sr, hc_r, sl), K);
  const double m0 = swm(n0, im), m1 = swm(n1, im);   // unit normal; the tangent is (-m1, m0)
  const double u = swd(u_h, m0, v_h, m1);
  const double v = swx(v_h, m0, u_h, m1);
  const double uleft = swd(hu_l, m0, hv_l, m1), vleft = swx(hv_l, m0, hu_l, m1);
  const double uright = swd(hu_r, m0, hv_r, m1), vright = swx(hv_r, m0, hu_r, m1);
  const double hroe = swm(0.5, swa(h_l, h_r));
  const double wd0 = sws(h_r, h_l), wd1 = sws(uright, uleft), wd2 = sws(vright, vleft), wd3 = sws(hc_r, hc_l),
               wd4 = sws(Z_r, Z_l);
  const double c = __dsqrt_rn(swm(grav, hroe));
  const double a = swa(u, c), b = sws(u, c);
  const double eps = 1e-10;
  const bool za = fabs(a) < eps, zb = fabs(b) < eps;
  const double sa = za ? 0. : copysign(1.0, a);
  const double sb = zb ? 0. : copysign(1.0, b);
  const double s0 = fabs(u) < eps ? 0. : copysign(1.0, u);
  const double da = za ? 1. : a, db = zb ? 1. : b, c2 = swm(2., c);
  const double dab = swm(da, db);
  const double D = __ddiv_rn(1., swm(c2, dab));
  const double i2c = swm(D, dab), hc2 = swm(0.5, c);
  // sign(a) / a - sign(b) / b
  const double e = swm(swx(sa, db, sb, da), swm(D, c2));
  const double ds = sws(sa, sb), hw = swm(hc2, wd4);
  const double hnew = swf(e, hw, swm(swd(swx(sb, a, sa, b), wd0, ds, wd1), i2c));
  const double unew0 = swf(ds, hw, swm(swx(swx(a, sa, b, sb), wd1, swm(swm(a, b), ds), wd0), i2c));
  const double vnew0 = swf(v, hnew, swm(s0, swf(-v, wd0, wd2)));
  const double cnew = swf(c_h, hnew, swm(s0, swf(-c_h, wd0, wd3)));
  const double w_lrh = swf(-0.5, hnew, hroe);
  const double w_lrhu = swm(0.5, sws(swa(uleft, uright), unew0));
  const double w_lrhv = swm(0.5, sws(swa(vleft, vright), vnew0));
  const double w_lrhc = swm(0.5, sws(swa(hc_l, hc_r), cnew));
  const double unew = swx(w_lrhu, m0, w_lrhv, m1);
  const double vnew = swd(w_lrhu, m1, w_lrhv, m0);
  const double q_s = swd(n0, unew, n1, vnew);
  const double gh = swm(swm(0.5, grav), swm(w_lrh, w_lrh));
  const double qw = __ddiv_rn(q_s, w_lrh);
  flux[0] = q_s;
  flux[1] = swd(qw, unew, gh, n0);
  flux[2] = swd(qw, vnew, gh, n1);
  flux[3] = swm(qw, w_lrhc);
}

// h and hc of cell c at a face centre (second order; gr: gradients of h and hc, psi: hc's limiter)
__device__ __forceinline__ void sw_reconstruct(const double *const gr[4], const double *psi, const double *cc, int c,
                                               double fx, double fy, double &h, double &hc) {
  const double r0 = sws(fx, ld(cc + 3 * (long long)c)), r1 = sws(fy, ld(cc + 3 * (long long)c + 1));
  const double p = ld_after(psi + c);
  h = swf(p, swd(ld_after(gr[0] + c), r0, ld_after(gr[1] + c), r1), h);
  hc = swf(p, swd(ld_after(gr[2] + c), r0, ld_after(gr[3] + c), r1), hc);
}

// Momentum of a reflective-wall ghost: the interior momentum with its normal component
// reversed, q - 2 (q.n) n / |n|^2 (no counterpart in manapy).
__device__ __forceinline__ void wall_mirror(double hu, double hv, double n0, double n1, double &gu, double &gv) {
  const double k = __ddiv_rn(swm(2., swd(hu, n0, hv, n1)), swd(n0, n0, n1, n1));
  gu = swf(-k, n0, hu);
  gv = swf(-k, n1, hv);
}

// faces.mesure of a face of normal (n0, n1), as the host forms it
__device__ __forceinline__ double sw_measure(double n0, double n1) { return __dsqrt_rn(swa(swm(n0, n0), swm(n1, n1))); }

// CFL dt candidate of a cell (manapy/solvers/shallowater/fvm_utils.py:16-42, without diffusion) from
// its state and its three face normals; manapy's (|u.n| / mesure + velson) * mesure without the
// division.
__device__ __forceinline__ double sw_dt_candidate(double h, double hu, double hv, const double n0[3],
                                                  const double n1[3], const double mes[3], double vol, double cfl,
                                                  double grav) {
  const double velson = __dsqrt_rn(swm(grav, h));
  const double ih = __ddiv_rn(1.0, h);
  const double u = swm(hu, ih), v = swm(hv, ih);
  double lam = 0.;
#pragma unroll
  for (int j = 0; j < 3; ++j) lam = swa(lam, swf(velson, mes[j], fabs(swd(u, n0[j], v, n1[j]))));
  return __ddiv_rn(swm(cfl, vol), lam);
}

// What the update of a triangle reads: its state, volume, faces and the values across them.
struct SwCell {
  double h, hu, hv, hc, Z, vol;
  double ns0x, ns0y;           // (G - V_1) turned by a right angle: the source's inner normal
  double s0[3], s1[3];         // outward normals of the local faces (cells.nf)
  double hp[3], zp[3];         // h and Z the source reads across them
  bool own[3], inner[3];       // left cell of the face; not a boundary face
  uint8_t code;                // order in which manapy adds the faces
};

// Residuals in manapy's order (inner faces by ascending face id, then boundary faces), bathymetry
// source (manapy/solvers/shallowater/fvm_utils.py:72-148) and forward-Euler update (:3-14, no
// Coriolis, wind or diffusion).
__device__ __forceinline__ void sw_update_cell(const SwCell &c, const double F[3][4], double dt, double grav,
                                               double &h_n, double &hu_n, double &hv_n, double &hc_n) {
  double rez[4] = {0., 0., 0., 0.};
#pragma unroll
  for (int pass = 0; pass < 2; ++pass) {
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const int sl = (c.code >> (2 * k)) & 3;
      if (pick3(c.inner[0], c.inner[1], c.inner[2], sl) == (pass == 1)) continue;
      const bool own = pick3(c.own[0], c.own[1], c.own[2], sl);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const double v = pick3(F[0][e], F[1][e], F[2][e], sl);
        rez[e] = own ? sws(rez[e], v) : swa(rez[e], v);
      }
    }
  }
  double c_1 = 0., c_2 = 0., ma[3], mb[3];
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    ma[j] = swm(c.hp[j], c.s0[j]);
    mb[j] = swm(c.hp[j], c.s1[j]);
    const double hm = swm(0.5, swa(c.h, c.hp[j])), hm2 = swm(hm, hm);
    c_1 = swf(hm2, c.s0[j], c_1);
    c_2 = swf(hm2, c.s1[j], c_2);
  }
  const double c_3 = swm(3.0, c.h);
  const double d12 = swx(ma[1], mb[2], ma[2], mb[1]), d02 = swx(ma[0], mb[2], mb[0], ma[2]),
               d01 = swx(ma[0], mb[1], mb[0], ma[1]);
  const double e0 = swx(c_1, mb[0], c_2, ma[0]), e1 = swx(c_1, mb[1], c_2, ma[1]), e2 = swx(c_1, mb[2], c_2, ma[2]);
  const double rdelta = __ddiv_rn(1., swa(sws(d12, d02), d01));
  const double h_1 = swm(swa(swf(c_3, d12, -e2), e1), rdelta);
  const double h_2 = swm(sws(swf(-c_3, d02, e2), e0), rdelta);
  const double h_3 = swm(swa(sws(e0, e1), swm(c_3, d01)), rdelta);
  const double z = swa(c.Z, c.h);
  const double z_1 = sws(z, h_1), z_2 = sws(z, h_2), z_3 = sws(z, h_3);
  const double ns1x = sws(c.ns0x, c.s0[1]), ns1y = sws(c.ns0y, c.s1[1]);
  const double ns2x = swa(c.ns0x, c.s0[0]), ns2y = swa(c.ns0y, c.s1[0]);
  const double s1x = swm(h_1, swf(-z_3, ns2x, swd(c.zp[0], c.s0[0], z_2, c.ns0x)));
  const double s1y = swm(h_1, swf(-z_3, ns2y, swd(c.zp[0], c.s1[0], z_2, c.ns0y)));
  const double s2x = swm(h_2, swf(z_3, ns1x, swx(c.zp[1], c.s0[1], z_1, c.ns0x)));
  const double s2y = swm(h_2, swf(z_3, ns1y, swx(c.zp[1], c.s1[1], z_1, c.ns0y)));
  const double s3x = swm(h_3, swf(-z_2, ns1x, swd(c.zp[2], c.s0[2], z_1, ns2x)));
  const double s3y = swm(h_3, swf(-z_2, ns1y, swd(c.zp[2], c.s1[2], z_1, ns2y)));
  const double hg = swm(-0.5, grav);
  const double dtv = __ddiv_rn(dt, c.vol);
  h_n = swf(dtv, rez[0], c.h);
  hu_n = swf(dtv, swf(hg, swa(swa(s1x, s2x), s3x), rez[1]), c.hu);
  hv_n = swf(dtv, swf(hg, swa(swa(s1y, s2y), s3y), rez[2]), c.hv);
  hc_n = swf(dtv, rez[3], c.hc);
}

}  // namespace mb
