// Arithmetic of the Euler kernels (fv_euler.cu, fv_euler_tile.cu), manapy's expressions
// (manapy/solvers/euler/fvm_utils2d.py).  Both files are compiled without multiply-add contraction,
// so every operation rounds as manapy's code does.
#pragma once

#include "fv_compact.cuh"

namespace mb {

constexpr double kNoDt = 1e300;

struct EulerQ {
  const double *rho, *P, *rhou, *rhov, *rhoE;
};

struct EulerW {
  double *rho, *P, *rhou, *rhov, *rhoE;
};

__device__ __forceinline__ double dmax3(double a, double b, double c) {
  // Python's max(a, b, c): the first of the largest
  double m = a;
  if (b > m) m = b;
  if (c > m) m = c;
  return m;
}

__device__ __forceinline__ void rusanov(double rhol, double Pl, double rhoul, double rhovl, double rhoEl, double rhor,
                                        double Pr, double rhour, double rhovr, double rhoEr, double n0, double n1,
                                        double mesure, double gamma, double F[4]) {
  const double ql = (rhoul * n0 + rhovl * n1);
  const double qr = (rhour * n0 + rhovl * n1);
  const double cl = sqrt(gamma * Pl / rhol);
  const double cr = sqrt(gamma * Pr / rhor);
  const double fl_rho = (rhoul * n0 + rhovl * n1);
  const double fl_rhou = ((rhoul * rhoul / rhol + Pl) * n0 + (rhoul * rhovl / rhol) * n1);
  const double fl_rhov = ((rhovl * rhoul / rhol) * n0 + (rhovl * rhovl / rhol + Pl) * n1);
  const double fl_rhoE = (rhoul / rhol * (rhoEl + Pl) * n0 + rhovl / rhol * (rhoEl + Pl) * n1);
  const double fr_rho = (rhour * n0 + rhovr * n1);
  const double fr_rhou = ((rhour * rhour / rhor + Pr) * n0 + (rhour * rhovr / rhor) * n1);
  const double fr_rhov = ((rhovr * rhour / rhor) * n0 + (rhovr * rhovr / rhor + Pr) * n1);
  const double fr_rhoE = (rhour / rhor * (rhoEr + Pr) * n0 + rhovr / rhor * (rhoEr + Pr) * n1);
  const double Ll = dmax3(fabs(ql / rhol - cl), fabs(ql / rhol), fabs(ql / rhol + cl));
  const double Lr = dmax3(fabs(qr / rhor - cr), fabs(qr / rhor), fabs(qr / rhor + cr));
  const double S = Ll > Lr ? Ll : Lr;
  F[0] = (0.5 * (fl_rho + fr_rho) - 0.5 * S * (rhor - rhol)) * mesure;
  F[1] = (0.5 * (fl_rhou + fr_rhou) - 0.5 * S * (rhour - rhoul)) * mesure;
  F[2] = (0.5 * (fl_rhov + fr_rhov) - 0.5 * S * (rhovr - rhovl)) * mesure;
  F[3] = (0.5 * (fl_rhoE + fr_rhoE) - 0.5 * S * (rhoEr - rhoEl)) * mesure;
}

// time_step_euler_2d's per-cell dt, faces in the cell's own order
__device__ __forceinline__ double euler_cell_dt(double rho, double P, double rhou, double rhov, const double n0[3],
                                                const double n1[3], const double mes[3], double vol, double cfl,
                                                double gamma) {
  const double velson = sqrt(gamma * fabs(P / rho));   // mes: sqrt(n0 n0 + n1 n1), as the host forms it
  double lam = 0.;
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    const double u_n = fabs((rhou * n0[j] + rhov * n1[j]) / rho) / sqrt(n0[j] * n0[j] + n1[j] * n1[j]);
    lam += (u_n + velson) * mes[j];
  }
  return cfl * vol / lam;
}

// What Rusanov's flux takes of a cell that does not depend on the face: with these formed once per cell
// instead of on both sides of every face, a face has 4 divisions left of 18.
struct EulerCell {
  double rho, rhou, rhov, rhoE;
  double c;                  // sound speed
  double uuP, uv, vvP;       // rhou^2 / rho + P, rhou rhov / rho, rhov^2 / rho + P
  double uE, vE;             // rhou / rho (rhoE + P), rhov / rho (rhoE + P)
};
__device__ __forceinline__ EulerCell euler_cell(double rho, double P, double rhou, double rhov, double rhoE,
                                                double gamma) {
  EulerCell e;
  e.rho = rho; e.rhou = rhou; e.rhov = rhov; e.rhoE = rhoE;
  e.c = sqrt(gamma * P / rho);
  e.uuP = rhou * rhou / rho + P;
  e.uv = rhou * rhov / rho;
  e.vvP = rhov * rhov / rho + P;
  e.uE = rhou / rho * (rhoE + P);
  e.vE = rhov / rho * (rhoE + P);
  return e;
}
// rusanov() of two such cells, the same operations
__device__ __forceinline__ void rusanov_cells(const EulerCell &l, const EulerCell &r, double n0, double n1,
                                              double mesure, double F[4]) {
  const double ql = (l.rhou * n0 + l.rhov * n1);
  const double qr = (r.rhou * n0 + l.rhov * n1);
  const double ul = ql / l.rho, ur = qr / r.rho;
  const double Ll = dmax3(fabs(ul - l.c), fabs(ul), fabs(ul + l.c));
  const double Lr = dmax3(fabs(ur - r.c), fabs(ur), fabs(ur + r.c));
  const double S = Ll > Lr ? Ll : Lr;
  F[0] = (0.5 * (ql + (r.rhou * n0 + r.rhov * n1)) - 0.5 * S * (r.rho - l.rho)) * mesure;
  F[1] = (0.5 * ((l.uuP * n0 + l.uv * n1) + (r.uuP * n0 + r.uv * n1)) - 0.5 * S * (r.rhou - l.rhou)) * mesure;
  F[2] = (0.5 * ((l.uv * n0 + l.vvP * n1) + (r.uv * n0 + r.vvP * n1)) - 0.5 * S * (r.rhov - l.rhov)) * mesure;
  F[3] = (0.5 * ((l.uE * n0 + l.vE * n1) + (r.uE * n0 + r.vE * n1)) - 0.5 * S * (r.rhoE - l.rhoE)) * mesure;
}

}  // namespace mb
