// The 2D Euler step (first-order Rusanov) in one launch: each block carries one tile of cells with its
// faces (fv_tile.cuh, mb_face_tiles) through the step in shared memory.  Compiled without multiply-add
// contraction: bit-identical to k_euler_face + k_euler_cell, and to manapy's kernels.
//
// The two-launch step writes a 32-byte flux per face and reads it, and a 32-byte face record, back from
// both cells, and gathers five fields of two cells per face: about 340 B of traffic per cell-update.
// Here the state of a tile and of the cells across its outer faces is read once, and what a flux takes
// of a cell alone (its sound speed, momentum and energy fluxes) is formed once per cell: 4 divisions
// per face and 6 per cell instead of 18 per face.
//
// Measured (B200, per step in CUDA graphs of 24, two launches -> this, one session): 2M triangles
// 161 -> 141 us, 720,000 63.6 -> 60.6, 45,000 9.3 -> 5.8, 1,800 8.0 -> 4.6.  The latency of the FP64
// chains between barriers bounds it (issue slots 46 % busy, FP64 pipe 35 %, 30 % of the warps:
// registers and shared memory allow 5 blocks).  Other shapes at 720,000 cells, beside 56.6 us for
// this one in the same session: 192 threads x 4 blocks 57-60 us, 256 x 3 60, 96 x 7 59-61; without the
// per-cell pass 56 (256 cells).
#include "fv_euler.cuh"
#include "fv_tile.cuh"

namespace mb {

#ifndef MB_EULER_TILE_THREADS
#define MB_EULER_TILE_THREADS 128
#endif
#ifndef MB_EULER_TILE_MIN_BLOCKS
#define MB_EULER_TILE_MIN_BLOCKS 5
#endif
constexpr int kEulerThreads = MB_EULER_TILE_THREADS;

// shared memory of a tile, in doubles; every array starts on 16 bytes
struct EulerTileLayout {
  int q, qstride, fl, n0, n1, mes, face, rec, red, total;
  __host__ __device__ explicit EulerTileLayout(const mb_face_tiles &t) {
    int at = 2;                    // the mbarrier
    qstride = t.cells + ((t.out_cap + 1) & ~1);
    q = at; at += 10 * qstride;    // rho, P (then c), rhou, rhov, rhoE; uuP, uv, vvP, uE, vE
    fl = at; at += 4 * t.face_cap;
    n0 = at; at += t.face_cap;
    n1 = at; at += t.face_cap;
    mes = at; at += t.face_cap;
    face = at; at += t.face_cap / 2;
    rec = at; at += 2 * t.cells;
    red = at; at += kEulerThreads / 32;
    total = at;
  }
};

struct EulerTileArgs {
  const double *q[5];   // rho, P, rhou, rhov, rhoE
  double *out[5];
  double *dt, *dt_next, *dt_after, *time;
  double cfl, gamma;
};

__global__ void __launch_bounds__(kEulerThreads, MB_EULER_TILE_MIN_BLOCKS)
    k_euler_tile(mb_mesh m, mb_face_tiles t, EulerTileArgs a) {
  extern __shared__ __align__(16) double sm[];
  const EulerTileLayout L(t);
  uint64_t *bar = reinterpret_cast<uint64_t *>(sm);
  double *q = sm + L.q, *sn0 = sm + L.n0, *sn1 = sm + L.n1, *smes = sm + L.mes, *red = sm + L.red;
  double2 *fl = reinterpret_cast<double2 *>(sm + L.fl);
  const uint32_t *sface = reinterpret_cast<const uint32_t *>(sm + L.face);
  const uint4 *srec = reinterpret_cast<const uint4 *>(sm + L.rec);
  const int T = t.cells, b = blockIdx.x, c0 = b * T, tid = threadIdx.x, Q = L.qstride;
  const int nc = min(T, m.nbcells - c0);
  const int4 head = __ldg(reinterpret_cast<const int4 *>(t.head) + b);
  const int n1 = head.x, nf = head.y;
  const int32_t *out = t.out + (long long)b * t.out_cap;

  tile_let_next_start();
  if (tid == 0) {
    tile_bar_init(bar);
    const long long fb = (long long)b * t.face_cap;
    const unsigned f2 = 8u * ((nf + 1) & ~1), f4 = 4u * ((nf + 3) & ~3), own = 8u * (nc & ~1);
    tile_bar_expect(bar, 3 * f2 + f4 + 16u * nc + 5 * own);
    tile_bulk(sn0, t.face_n0 + fb, f2, bar);
    tile_bulk(sn1, t.face_n1 + fb, f2, bar);
    tile_bulk(smes, t.face_mes + fb, f2, bar);
    tile_bulk(sm + L.face, t.face + 2 * fb, f4, bar);
    tile_bulk(sm + L.rec, t.cell + 8 * (long long)b * T, 16u * nc, bar);
    tile_prefetch(m.cell_volume + c0, 8u * nc);
  }
  int first = 0;
  if (tid < n1) first = ld(out + tid);
  tile_after_previous();
  const double dt = ld_after(a.dt);
  if (tid == 0) {
#pragma unroll
    for (int k = 0; k < 5; ++k) {
      tile_bulk(q + k * Q, a.q[k] + c0, 8u * (nc & ~1), bar);
      if (nc & 1) q[k * Q + nc - 1] = ld_after(a.q[k] + c0 + nc - 1);
    }
    if (b == 0) {
      *a.dt_after = kNoDt;
      if (a.time) *a.time += dt;
    }
  }
  for (int e = tid; e < n1; e += kEulerThreads) {
    const int c = e == tid ? first : ld(out + e);
#pragma unroll
    for (int k = 0; k < 5; ++k) tile_copy8(q + k * Q + T + e, a.q[k] + c);
  }
  tile_copies_done();
  __syncthreads();
  if (!tile_arrived(bar, t.late)) return;   // never seen

  for (int k = tid; k < nc + n1; k += kEulerThreads) {
    double *s = q + (k < nc ? k : T + k - nc);
    const EulerCell e = euler_cell(s[0], s[Q], s[2 * Q], s[3 * Q], s[4 * Q], a.gamma);
    s[Q] = e.c;
    s[5 * Q] = e.uuP; s[6 * Q] = e.uv; s[7 * Q] = e.vvP; s[8 * Q] = e.uE; s[9 * Q] = e.vE;
  }
  __syncthreads();
  auto cell = [&](int k) {
    const double *s = q + k;
    return EulerCell{s[0], s[2 * Q], s[3 * Q], s[4 * Q], s[Q], s[5 * Q], s[6 * Q], s[7 * Q], s[8 * Q], s[9 * Q]};
  };

  for (int f = tid; f < nf; f += kEulerThreads) {
    const uint32_t lr = sface[f];
    const int l = lr & 0xffffu, r = (lr >> 16) == kNoCell ? l : (int)(lr >> 16);   // Neumann: the cell's own state
    const double mes = smes[f], nx = sn0[f] / mes, ny = sn1[f] / mes;
    double F[4];
    rusanov_cells(cell(l), cell(r), nx, ny, mes, F);
    fl[f] = make_double2(F[0], F[1]);
    fl[t.face_cap + f] = make_double2(F[2], F[3]);
  }
  __syncthreads();

  double best = kNoDt;
  for (int k = tid; k < nc; k += kEulerThreads) {
    const int i = c0 + k;
    const TileCell c = tile_cell(srec[k]);   // v: local faces
    const int code = (c.fl >> 3) & 63;
    double n0[3], n1c[3], mes[3], rez[4] = {0., 0., 0., 0.};
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      n0[j] = sn0[c.v[j]];
      n1c[j] = sn1[c.v[j]];
      mes[j] = smes[c.v[j]];
    }
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      const int s = (code >> (2 * j)) & 3, f = pick3(c.v[0], c.v[1], c.v[2], s);
      const bool left = (c.fl >> s) & 1u;
      const double2 x = fl[f], y = fl[t.face_cap + f];
      const double F[4] = {x.x, x.y, y.x, y.y};
#pragma unroll
      for (int e = 0; e < 4; ++e) rez[e] = left ? rez[e] - F[e] : rez[e] + F[e];
    }
    const double v = ld(m.cell_volume + i);
    const double r1 = q[k] + dt * (rez[0] / v);
    const double u1 = q[2 * Q + k] + dt * (rez[1] / v);
    const double w1 = q[3 * Q + k] + dt * (rez[2] / v);
    const double E1 = q[4 * Q + k] + dt * (rez[3] / v);
    const double P1 = (a.gamma - 1) * (E1 - 0.5 * (u1 * u1 + w1 * w1) / r1);
    a.out[0][i] = r1; a.out[1][i] = P1; a.out[2][i] = u1; a.out[3][i] = w1; a.out[4][i] = E1;
        // euler_cell_dt with faces.mesure, the same number, for its square root
    const double velson = sqrt(a.gamma * fabs(P1 / r1));
    double lam = 0.;
#pragma unroll
    for (int j = 0; j < 3; ++j) lam += (fabs((u1 * n0[j] + w1 * n1c[j]) / r1) / mes[j] + velson) * mes[j];
    best = pmin(best, a.cfl * v / lam);
  }
  for (int o = 16; o > 0; o >>= 1) best = pmin(best, __shfl_xor_sync(0xffffffffu, best, o));
  if ((tid & 31) == 0) red[tid >> 5] = best;
  __syncthreads();
  if (tid == 0) {
#pragma unroll
    for (int w = 1; w < kEulerThreads / 32; ++w) best = pmin(best, red[w]);
    if (best < kNoDt) atomic_min_pos(a.dt_next, best);
  }
}

}  // namespace mb

using namespace mb;

extern "C" int mb_euler_step_tile(const mb_mesh *m, const mb_face_tiles *t, const double *const q_in[5],
                                  double *const q_out[5], double cfl, double gamma, double *ring, int step,
                                  double *time, void *stream) {
  MB_NVTX();
  if (!m || m->dim != 2 || m->nbcells <= 0 || !m->cell_volume || !face_tiles_ok(m, t) || !q_in || !q_out || !ring ||
      step < 0)
    return MB_EINVAL;
  EulerTileArgs a{};
  for (int k = 0; k < 5; ++k) {
    if (!q_in[k] || ((uintptr_t)q_in[k] & 15) || !q_out[k] || q_out[k] == q_in[k]) return MB_EINVAL;
    a.q[k] = q_in[k];
    a.out[k] = q_out[k];
  }
  a.dt = ring + step % 3; a.dt_next = ring + (step + 1) % 3; a.dt_after = ring + (step + 2) % 3;
  a.time = time;
  a.cfl = cfl; a.gamma = gamma;
  return tile_launch<k_euler_tile>(t->count, kEulerThreads, 8 * EulerTileLayout(*t).total,
                     reinterpret_cast<cudaStream_t>(stream), *m, *t, a) == cudaSuccess
             ? MB_OK
             : MB_ECUDA;
}
