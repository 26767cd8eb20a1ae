// The FP64 second-order advection-diffusion step on tetrahedra in two launches.
//
// 1. k_tet_grad, one block per tile of cells (mb_tet_tiles): the sums of the tile's vertices and edges
//    over their cells, from the state of the tile and the cells around it in shared memory; per cell
//    the least-squares right-hand side by inclusion-exclusion (4 vertices - 6 edges + 4 face
//    neighbours), the Barth limiter and the reconstructed value at each of its four faces; the
//    centre -> vertex values.
// 2. k_tet_flux, one thread per cell: upwind fluxes of the face values, diffusion as a linear form with
//    static coefficients (k_tet_coef), forward Euler.
//
// The three-launch step (k_f3_sums, k_f3_grad, k_f3_phase2) gathers 18 rows of 32 bytes per cell for the
// gradient from L2 and recomputes the geometry of every face in its last pass (normals, diamond
// vectors, centres: 12 vertex rows, 4 centres and about 300 operations per cell).
//
// Sums are kept relative to the middle of the tile and of its values: G = sum x_j w'_j and S = sum w'_j
// with x_j the offset of a centre and w'_j = w_j - w_ref, so a vertex or edge is 4 doubles and a list
// entry 4 multiply-adds, and a uniform state has exact zeros.  w_ref is the middle of the tile's
// values if they are of one sign and within a factor of 5, else the least in magnitude, or 0 where
// they change sign: |w'_j| <= 2 |w_j| for its cells, so the cancellation in G - x_i S is never much
// above that of the earlier sums, which took the values themselves, wherever a tile holds a steep
// front, an outlier or a NaN.
//
// Large meshes keep the sums in memory (k_tet_sums, k_tet_cell below) and take the same fluxes.
//
// Measured (B200, per step in CUDA graphs of the tuned length, three launches -> this, one session):
// 2,058 tetrahedra 38.9 -> 17.7 us, 16,464 43.2 -> 18.3, 48,000 45.5 -> 21.6, 93,750 47.4 -> 37.6; with
// the sums in memory 384,000 125 -> 86, 1,572,864 389 -> 265.  k_tet_flux reads 208 B of DRAM per cell and takes 18 us at 384,000 cells
// where k_f3_phase2 took 45.  The gradient pass is bound by its chain of passes and by reading the
// cells around a tile (512 threads x 2 blocks; 384 x 2 100-118 us at 384,000 cells, 256 x 3 124).
#include "fv_tile.cuh"

namespace mb {

#ifndef MB_TET_THREADS
#define MB_TET_THREADS 512
#endif
#ifndef MB_TET_MIN_BLOCKS
#define MB_TET_MIN_BLOCKS 2
#endif
constexpr int kTetThreads = MB_TET_THREADS;

// shared memory of a tile, in doubles; every array starts on 16 bytes
struct TetLayout {
  int xy, z, w, nG, nS, eG, eS, rec, ninc, einc, ngrp, egrp, total;
  __host__ __device__ explicit TetLayout(const mb_tet_tiles &t) {
    const int ncell = t.cells + t.ext_cap + 2;    // and the zero past the lists' ends
    int at = 2;                                   // the mbarrier
    xy = at; at += 2 * ncell;
    z = at; at += ncell;
    w = at; at += ncell;
    nG = at; at += 2 * t.node_cap;                // {G_x, G_y}, {G_z, S}
    nS = at; at += 2 * t.node_cap;
    eG = at; at += 2 * t.edge_cap;
    eS = at; at += 2 * t.edge_cap;
    rec = at; at += 4 * t.cells;
    ninc = at; at += t.ninc_cap / 4;
    einc = at; at += t.einc_cap / 4;
    ngrp = at; at += t.ngrp_cap / 2;
    egrp = at; at += t.egrp_cap / 2;
    total = at;
  }
};

template <bool DF>
__global__ void __launch_bounds__(kTetThreads, MB_TET_MIN_BLOCKS)
    k_tet_grad(mb_mesh m, mb_tet_tiles t, mb_bc bc, const double *__restrict__ w, double *__restrict__ face_values,
               double *__restrict__ wn) {
  extern __shared__ __align__(16) double sm[];
  const TetLayout L(t);
  uint64_t *bar = reinterpret_cast<uint64_t *>(sm);
  double2 *xy = reinterpret_cast<double2 *>(sm + L.xy);
  double *z = sm + L.z, *cw = sm + L.w;
  double2 *nG = reinterpret_cast<double2 *>(sm + L.nG), *nS = reinterpret_cast<double2 *>(sm + L.nS);
  double2 *eG = reinterpret_cast<double2 *>(sm + L.eG), *eS = reinterpret_cast<double2 *>(sm + L.eS);
  const uint4 *rec = reinterpret_cast<const uint4 *>(sm + L.rec);
  const uint16_t *ninc = reinterpret_cast<const uint16_t *>(sm + L.ninc);
  const uint16_t *einc = reinterpret_cast<const uint16_t *>(sm + L.einc);
  const int *ngrp = reinterpret_cast<const int *>(sm + L.ngrp), *egrp = reinterpret_cast<const int *>(sm + L.egrp);
  const int T = t.cells, b = blockIdx.x, c0 = b * T, tid = threadIdx.x;
  const int nc = min(T, m.nbcells - c0);
  const int4 h0 = __ldg(reinterpret_cast<const int4 *>(t.head) + 2 * b);
  const int neinc = ld(t.head + 8 * (long long)b + 4);
  const int nout = h0.x, nn = h0.y, ne = h0.z, nninc = h0.w;
  const int32_t *ext = t.ext + (long long)b * t.ext_cap;

  if (tid == 0) {
    tile_bar_init(bar);
    const long long eb = (long long)b * t.ext_cap;
    const unsigned z0 = 8u * (nc & ~1), z1 = 8u * ((nout + 1) & ~1);
    const unsigned g0 = 4u * ((((nn + 31) >> 5) + 4) & ~3), g1 = 4u * ((((ne + 31) >> 5) + 4) & ~3);
    tile_bar_expect(bar, 16u * nc + z0 + 16u * nout + z1 + 32u * nc + 2u * nninc + 2u * neinc + g0 + g1);
    tile_bulk(xy, t.own_xy + 2 * (long long)c0, 16u * nc, bar);
    tile_bulk(z, t.own_z + c0, z0, bar);
    tile_bulk(xy + T, t.ext_xy + 2 * eb, 16u * nout, bar);
    tile_bulk(z + T, t.ext_z + eb, z1, bar);
    tile_bulk(sm + L.ninc, t.ninc + (long long)b * t.ninc_cap, 2u * nninc, bar);
    tile_bulk(sm + L.einc, t.einc + (long long)b * t.einc_cap, 2u * neinc, bar);
    tile_bulk(sm + L.ngrp, t.ngrp + (long long)b * t.ngrp_cap, g0, bar);
    tile_bulk(sm + L.egrp, t.egrp + (long long)b * t.egrp_cap, g1, bar);
    tile_bulk(sm + L.rec, t.cell + 16 * (long long)c0, 32u * nc, bar);
    for (int q = 0; q < 12; ++q) tile_prefetch(t.cell_q + q * (long long)m.nbcells + c0, 8u * nc);
    if (nc & 1) z[nc - 1] = ld(t.own_z + c0 + nc - 1);
    const int pad = T + t.ext_cap;
    xy[pad] = make_double2(0., 0.);
    z[pad] = cw[pad] = 0.;
  }
  int first = 0;
  if (tid < nout) first = ld(ext + tid);
  tile_after_previous();
  tile_let_next_start();
  const GhostAfter ghost{make_rule(m, bc, w)};
  for (int k = tid; k < nc; k += kTetThreads) cw[k] = ld_after(w + c0 + k);
#pragma unroll 4
  for (int k = tid; k < nout; k += kTetThreads) cw[T + k] = ld_after(w + (k == tid ? first : ld(ext + k)));
  __syncthreads();
  if (!tile_arrived(bar, t.late)) return;   // never seen

  // every warp finds w_ref for itself (no further barrier; NaN compares neither less nor greater)
  double least = INFINITY, most = -INFINITY;
  for (int k = tid & 31; k < nc; k += 32) {
    const double v = cw[k];
    if (v < least) least = v;
    if (v > most) most = v;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const double a = __shfl_xor_sync(0xffffffffu, least, o), c = __shfl_xor_sync(0xffffffffu, most, o);
    if (a < least) least = a;
    if (c > most) most = c;
  }
  double wref = 0.;
  if (least > 0.) wref = most <= 5. * least ? 0.5 * least + 0.5 * most : least;
  if (most < 0.) wref = least >= 5. * most ? 0.5 * least + 0.5 * most : most;
  if (!isfinite(wref)) wref = 0.;
  cw[T + t.ext_cap] = wref;         // the lists' padding adds zeros; every warp writes the same
  __syncwarp();

  // four lanes per vertex (its list is about four times an edge's), each a quarter of the list
  for (int k4 = tid; k4 < ((4 * nn + 31) & ~31); k4 += kTetThreads) {
    const int k = k4 >> 2, sub = k4 & 3;
    double gx = 0., gy = 0., gz = 0., s = 0.;
    if (k < nn) {
      const uint16_t *row = ninc + ngrp[k >> 5] + (k & 31);
      const int len = ngrp[(k >> 5) + 1] - ngrp[k >> 5];
#pragma unroll 4
      for (int q = 32 * sub; q < len; q += 128) {
        const int l = row[q];
        const double2 p = xy[l];
        const double v = cw[l] - wref;
        gx += p.x * v; gy += p.y * v; gz += z[l] * v;
        s += v;
      }
    }
#pragma unroll
    for (int o = 1; o < 4; o <<= 1) {
      gx += __shfl_xor_sync(0xffffffffu, gx, o);
      gy += __shfl_xor_sync(0xffffffffu, gy, o);
      gz += __shfl_xor_sync(0xffffffffu, gz, o);
      s += __shfl_xor_sync(0xffffffffu, s, o);
    }
    if (sub != 0 || k >= nn) continue;
    nG[k] = make_double2(gx, gy);
    nS[k] = make_double2(gz, s);
    if (DF) {
      const int id = ld(t.node + (long long)b * t.node_cap + k);
      if (id & kTetOwned) {
        const int v = id & (kTetGhosts - 1);
        double mx, my, mz, a;
        ld4d(t.node_mu + 4 * (long long)v, mx, my, mz, a);
        double val = a * s + (mx * gx + my * gy + mz * gz);
        if (id & kTetGhosts) {
          val += ld(t.node_kappa + v) * wref;
          const int e = ld(m.n2g_ptr + v + 1);
          for (int q = ld(m.n2g_ptr + v); q < e; q += 4) {
            int f[4];
            double g[4];
            ghost4(ghost.g, m.n2g_idx, q, e, f, g);
#pragma unroll
            for (int u = 0; u < 4; ++u)
              if (f[u] >= 0) val += ld(m.n2g_alpha + q + u) * g[u];
          }
        } else {
          val += wref;
        }
        st1_keep(wn + v, val, l2_keep());
      }
    }
  }
  for (int k = tid; k < ne; k += kTetThreads) {
    const uint16_t *row = einc + egrp[k >> 5] + (k & 31);
    const int len = egrp[(k >> 5) + 1] - egrp[k >> 5];
    double gx = 0., gy = 0., gz = 0., s = 0.;
#pragma unroll 4
    for (int q = 0; q < len; q += 32) {
      const int l = row[q];
      const double2 p = xy[l];
      const double v = cw[l] - wref;
      gx += p.x * v; gy += p.y * v; gz += z[l] * v;
      s += v;
    }
    eG[k] = make_double2(gx, gy);
    eS[k] = make_double2(gz, s);
  }
  __syncthreads();

  for (int k = tid; k < nc; k += kTetThreads) {
    const int i = c0 + k;
    const uint4 ra = rec[2 * k], rb = rec[2 * k + 1];
    const uint32_t words[8] = {ra.x, ra.y, ra.z, ra.w, rb.x, rb.y, rb.z, rb.w};
    auto entry = [&](int j) { return (int)((words[j >> 1] >> (16 * (j & 1))) & 0xffffu); };
    const double *Q = t.cell_q + i;
    const long long n = m.nbcells;
    const double w0 = cw[k], wi = w0 - wref;
    const double2 p = xy[k];
    const double pz = z[k];
    double gx = 0., gy = 0., gz = 0., s = 0.;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const double2 a = nG[entry(j)], c = nS[entry(j)];
      gx += a.x; gy += a.y; gz += c.x; s += c.y;
    }
#pragma unroll
    for (int j = 0; j < 6; ++j) {
      const double2 a = eG[entry(4 + j)], c = eS[entry(4 + j)];
      gx -= a.x; gy -= a.y; gz -= c.x; s -= c.y;
    }
    double hi = w0, lo = w0;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int o = entry(10 + j);
      double v;
      if (o != kNoCell) {
        v = cw[o];
        const double vr = v - wref;
        const double2 q = xy[o];
        gx += q.x * vr; gy += q.y * vr; gz += z[o] * vr;
        s += vr;
      } else {
        v = ghost(-1 - ld(m.cell_nbr + 4 * (long long)i + j));
      }
      hi = pmax(hi, v);
      lo = pmin(lo, v);
    }
    // the stencil's own part, sum (x_j - x_i) w'_j, takes - w'_i D (cell_q's last planes); ghosts are
    // differences as they stand
    double jx = (gx - p.x * s) - wi * ld(Q + 9 * n), jy = (gy - p.y * s) - wi * ld(Q + 10 * n),
           jz = (gz - pz * s) - wi * ld(Q + 11 * n);
    if (entry(14)) {
      const D3 c = ld3(m.cell_xy + 4 * (long long)i);
      const int e = ld(m.ghostnid_ptr + i + 1);
      for (int q = ld(m.ghostnid_ptr + i); q < e; q += 4) {
        int f[4];
        double g[4];
        ghost4(ghost.g, m.ghostnid_idx, q, e, f, g);
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          if (f[u] < 0) continue;
          const double *x = m.face_ghostcenter + 3 * (long long)f[u];
          const double d = g[u] - w0;
          jx += (ld(x) - c.x) * d; jy += (ld(x + 1) - c.y) * d; jz += (ld(x + 2) - c.z) * d;
        }
      }
    }
    double de[4];
#pragma unroll
    for (int q = 0; q < 3; ++q)
      de[q] = ld(Q + (3 * q) * n) * jx + ld(Q + (3 * q + 1) * n) * jy + ld(Q + (3 * q + 2) * n) * jz;
    de[3] = -((de[0] + de[1]) + de[2]);   // the face centres' mean is the centre
    const double ps = tile_barth(de, hi - w0, w0 - lo, 1e-10);
    st4_keep(face_values + 4 * (long long)i, w0 + ps * de[0], w0 + ps * de[1], w0 + ps * de[2], w0 + ps * de[3],
             l2_keep());
  }
}

#ifndef MB_TET_FLUX_BLOCK
#define MB_TET_FLUX_BLOCK 128
#endif
#ifndef MB_TET_FLUX_MIN_BLOCKS
#define MB_TET_FLUX_MIN_BLOCKS 7
#endif

template <bool DF, bool ROWS>
__global__ void __launch_bounds__(MB_TET_FLUX_BLOCK, MB_TET_FLUX_MIN_BLOCKS)
    k_tet_flux(mb_mesh m, const uint16_t *__restrict__ links, mb_bc bc, const double *__restrict__ w,
               double *__restrict__ w_out,
               const double *__restrict__ sign, const double *__restrict__ coef, const double *__restrict__ src,
               const double *__restrict__ dt_dev, const double *__restrict__ face_values,
               const double *__restrict__ wn, double *__restrict__ rows_out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const bool on = i < m.nbcells;
  const long long n = m.nbcells;
  int4 nb = make_int4(0, 0, 0, 0), vt = nb;
  unsigned link = 0;
  double s[4] = {0., 0., 0., 0.}, c1 = 0., c2 = 0., c3 = 0., B[4] = {0., 0., 0., 0.}, rv = 0.;
  if (on) {
    // written before the gradient pass passed its own wait, which lets this launch start
    const uint64_t once = l2_stream();
    nb = ld4(m.cell_nbr + 4 * (long long)i);
    if (DF) vt = ld4(m.cell_vtx + 4 * (long long)i);
    link = ld(links + i);
    ld4d_stream(sign + 4 * (long long)i, s[0], s[1], s[2], s[3], once);
    if (DF) {
      c1 = ldd_stream(coef + i, once); c2 = ldd_stream(coef + n + i, once); c3 = ldd_stream(coef + 2 * n + i, once);
#pragma unroll
      for (int j = 0; j < 4; ++j) B[j] = ldd_stream(coef + (3 + j) * n + i, once);
      rv = ldd_stream(coef + 7 * n + i, once);
    } else {
      rv = 1 / ld(m.cell_volume + i);
    }
  }
  tile_after_previous();
  tile_let_next_start();
  if (!on) return;
  const GhostAfter ghost{make_rule(m, bc, w)};
  const double wi = ld_after(w + i);
  double mine[4];
  ld4_after(face_values + 4 * (long long)i, mine[0], mine[1], mine[2], mine[3]);
  double wo[4], far[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int o = comp(nb, j);
    const bool take_me = (s[j] >= 0) == (bool)((link >> j) & 1u);
    if (o >= 0) {
      wo[j] = DF ? ld_after(w + o) : 0.;
      far[j] = take_me ? 0. : ld_after(face_values + 4 * (long long)o + ((link >> (4 + 2 * j)) & 3u));
    } else {
      wo[j] = far[j] = ghost(-1 - o);
    }
  }
  double acc = 0.;
  if (DF) {
    const double v0 = ld_after(wn + vt.x);
    acc = c1 * (ld_after(wn + vt.y) - v0) + c2 * (ld_after(wn + vt.z) - v0) + c3 * (ld_after(wn + vt.w) - v0);
  }
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const bool own = (link >> j) & 1u;
    const double F = s[j] * ((s[j] >= 0) == own ? mine[j] : far[j]);
    acc += own ? -F : F;
    if (DF) acc += B[j] * (wo[j] - wi);
  }
  const double wnew = wi + ld_after(dt_dev) * (acc * rv + (src ? ld_after(src + i) : 0.0));
  w_out[i] = wnew;
  if (ROWS) {
    const D3 c = ld3(m.cell_xy + 4 * (long long)i);
    st4_keep(rows_out + 4 * (long long)i, c.x, c.y, c.z, wnew, l2_keep());
  }
}

// ---------------------------------------------------------------- large meshes: sums in memory
//
// Where a tile's outside cells (four to five times its own at 256 cells) cost more than they save, the
// sums of vertices and edges are formed as k_f3_sums forms them, from rows {centre, value}
// gathered through L2, and the cells read them back; face values and fluxes as above.

// vertex blocks [0, nnb): the vertex's sums {P, Q} relative to itself and (DF) its value from them (no
// weight per incidence is read); edge blocks: the edge's sums relative to its first vertex
template <bool DF>
__global__ void __launch_bounds__(kBlock) k_tet_sums(mb_mesh m, mb_bc bc, const double *__restrict__ w,
                                                     const double *__restrict__ rows,
                                                     const double *__restrict__ node_mu, double *__restrict__ nrec,
                                                     double *__restrict__ erec, double *__restrict__ wn, int nnb) {
  const int lane = threadIdx.x & 31;
  const uint64_t pst = l2_stream();
  double px = 0., py = 0., pz = 0., q = 0.;
  const bool vertex = (int)blockIdx.x < nnb;
  const int k = (vertex ? blockIdx.x : blockIdx.x - nnb) * blockDim.x + threadIdx.x;
  if (k >= (vertex ? m.nbnodes : m.nbedges)) return;
  const D3 X = ld3(m.node_coord + 4 * (long long)(vertex ? k : ld(m.edge_origin + k)));
  const int32_t *ptr = vertex ? m.n2c_sum_ptr : m.edge_sell_ptr, *idx = vertex ? m.n2c_sum_idx : m.edge_sell_idx;
  const int sb = ld(ptr + (k >> 5)), se = ld(ptr + (k >> 5) + 1);
  for (int p = sb + lane; p < se; p += 32) {
    const int c = ld1_stream(idx + p, pst);
    if (c < 0) continue;       // empty slot
    double x, y, z, v;
    ld4d(rows + 4 * (long long)c, x, y, z, v);
    px += (x - X.x) * v; py += (y - X.y) * v; pz += (z - X.z) * v;
    q += v;
  }
  st4_keep((vertex ? nrec : erec) + 4 * (long long)k, px, py, pz, q, l2_keep());
  if (DF && vertex) {
    double mx, my, mz, rd;
    ld4d_stream(node_mu + 4 * (long long)k, mx, my, mz, rd, pst);
    double a = rd * q + (mx * px + my * py + mz * pz);
    const int gb = ld(m.n2g_ptr + k), ge = ld(m.n2g_ptr + k + 1);
    if (gb < ge) {
      const GhostRule ghost = make_rule(m, bc, w);
      for (int g = gb; g < ge; g += 4) {
        int f[4];
        double v[4];
        ghost4(ghost, m.n2g_idx, g, ge, f, v);
#pragma unroll
        for (int u = 0; u < 4; ++u)
          if (f[u] >= 0) a += ld(m.n2g_alpha + g + u) * v[u];
      }
    }
    wn[k] = a;
  }
}

#ifndef MB_TET_CELL_MIN_BLOCKS
#define MB_TET_CELL_MIN_BLOCKS 8
#endif

// the face values of every cell from the vertex, edge and face-neighbour sums
__global__ void __launch_bounds__(128, MB_TET_CELL_MIN_BLOCKS)
    k_tet_cell(mb_mesh m, mb_bc bc, const double *__restrict__ w, const double *__restrict__ cell_q,
               const double *__restrict__ rows, const double *__restrict__ nrec, const double *__restrict__ erec,
               double *__restrict__ face_values) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= m.nbcells) return;
  const GhostRule ghost = make_rule(m, bc, w);
  D3 c;
  double wi;
  ld4d(rows + 4 * (long long)i, c.x, c.y, c.z, wi);
  const int4 vt = ld4(m.cell_vtx + 4 * (long long)i), nb = ld4(m.cell_nbr + 4 * (long long)i);
  const int4 ea = ld4(m.cell_edges + 8 * (long long)i), eb = ld4(m.cell_edges + 8 * (long long)i + 4);
  // offsets of the vertices, origins of their sums and of their edges'
  D3 P[4];
#pragma unroll
  for (int v = 0; v < 4; ++v) P[v] = ld3(m.node_coord + 4 * (long long)comp(vt, v)) - c;
  double sx = 0., sy = 0., sz = 0.;
#pragma unroll
  for (int v = 0; v < 4; ++v) {
    double px, py, pz, q;
    ld4d(nrec + 4 * (long long)comp(vt, v), px, py, pz, q);
    sx += px + P[v].x * q; sy += py + P[v].y * q; sz += pz + P[v].z * q;
  }
#pragma unroll
  for (int k = 0; k < 6; ++k) {
    // local vertex pairs (0,1), (0,2), (0,3), (1,2), (1,3), (2,3); origin: the vertex of smaller index
    const int a = k < 3 ? 0 : (k < 5 ? 1 : 2), b = k < 3 ? k + 1 : (k < 5 ? k - 1 : 3);
    const int e = k == 0 ? ea.x : (k == 1 ? ea.y : (k == 2 ? ea.z : (k == 3 ? ea.w : (k == 4 ? eb.x : eb.y))));
    double px, py, pz, q;
    ld4d(erec + 4 * (long long)e, px, py, pz, q);
    const D3 d = comp(vt, a) < comp(vt, b) ? P[a] : P[b];
    sx -= px + d.x * q; sy -= py + d.y * q; sz -= pz + d.z * q;
  }
  double hi = wi, lo = wi;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int o = comp(nb, j);
    double v;
    if (o >= 0) {
      double x, y, z;
      ld4d(rows + 4 * (long long)o, x, y, z, v);
      sx += (x - c.x) * v; sy += (y - c.y) * v; sz += (z - c.z) * v;
    } else {
      v = ghost(-1 - o);
    }
    hi = pmax(hi, v);
    lo = pmin(lo, v);
  }
  const double *Q = cell_q + i;
  const long long n = m.nbcells;
  const uint64_t once = l2_stream();
  sx -= wi * ldd_stream(Q + 9 * n, once); sy -= wi * ldd_stream(Q + 10 * n, once); sz -= wi * ldd_stream(Q + 11 * n, once);
  const int ge = ld(m.ghostnid_ptr + i + 1);
  for (int g = ld(m.ghostnid_ptr + i); g < ge; g += 4) {
    int f[4];
    double v[4];
    ghost4(ghost, m.ghostnid_idx, g, ge, f, v);
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      if (f[u] < 0) continue;
      const double *gc = m.face_ghostcenter + 3 * (long long)f[u];
      const double d = v[u] - wi;
      sx += (ld(gc) - c.x) * d; sy += (ld(gc + 1) - c.y) * d; sz += (ld(gc + 2) - c.z) * d;
    }
  }
  double de[4];
#pragma unroll
  for (int q = 0; q < 3; ++q)
    de[q] = ldd_stream(Q + (3 * q) * n, once) * sx + ldd_stream(Q + (3 * q + 1) * n, once) * sy +
            ldd_stream(Q + (3 * q + 2) * n, once) * sz;
  de[3] = -((de[0] + de[1]) + de[2]);   // the face centres' mean is the centre
  const double ps = tile_barth(de, hi - wi, wi - lo, 1e-10);
  st4_keep(face_values + 4 * (long long)i, wi + ps * de[0], wi + ps * de[1], wi + ps * de[2], wi + ps * de[3],
           l2_keep());
}

}  // namespace mb

using namespace mb;

extern "C" {

int mb_tet_tile_bytes(const mb_tet_tiles *t) { return t ? 8 * TetLayout(*t).total : MB_EINVAL; }

int mb_advdiff_step_tet(const mb_mesh *m, const mb_tet_tiles *t, const mb_bc *bc, const mb_advdiff_params *p,
                        const double *w_in, double *w_out, const double *sign_cf, const double *coef,
                        const double *src, const double *dt_dev, double *face_values, double *node_scratch,
                        void *stream) {
  MB_NVTX();
  if (!m || m->dim != 3 || m->nbcells <= 0 || !t || !bc || !p || p->order != 2 || !w_in || !w_out || w_in == w_out ||
      !sign_cf || !dt_dev || !face_values || !bc->kind || !bc->value)
    return MB_EINVAL;
  const bool df = p->diffusion != 0;
  if (!m->cell_nbr || !m->cell_vtx || !m->cell_xy || !m->cell_volume || !m->face_cellid || !m->n2g_ptr ||
      !m->n2g_idx || !m->n2g_alpha || !m->ghostnid_ptr || !m->ghostnid_idx || !m->face_ghostcenter ||
      !tet_tiles_ok(m, t))
    return MB_EINVAL;
  if (((uintptr_t)face_values & 31) || ((uintptr_t)sign_cf & 31) || ((uintptr_t)m->cell_xy & 31) ||
      (df && (!coef || !node_scratch)))
    return MB_EINVAL;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  const int bytes = 8 * TetLayout(*t).total, fb = ceil_div(m->nbcells, MB_TET_FLUX_BLOCK);
  cudaError_t e;
  if (df) {
    e = tile_launch<k_tet_grad<true>>(t->count, kTetThreads, bytes, st, *m, *t, *bc, w_in, face_values, node_scratch);
    if (e == cudaSuccess)
      e = tile_launch<k_tet_flux<true, false>>(fb, MB_TET_FLUX_BLOCK, 0, st, *m, t->link, *bc, w_in, w_out, sign_cf, coef,
                      src, dt_dev, face_values, node_scratch, nullptr);
  } else {
    e = tile_launch<k_tet_grad<false>>(t->count, kTetThreads, bytes, st, *m, *t, *bc, w_in, face_values, node_scratch);
    if (e == cudaSuccess)
      e = tile_launch<k_tet_flux<false, false>>(fb, MB_TET_FLUX_BLOCK, 0, st, *m, t->link, *bc, w_in, w_out, sign_cf, coef,
                      src, dt_dev, face_values, node_scratch, nullptr);
  }
  return e == cudaSuccess ? MB_OK : MB_ECUDA;
}

int mb_advdiff_step_tet_sums(const mb_mesh *m, const mb_tet_tables *t, const mb_bc *bc, const mb_advdiff_params *p,
                             const double *w_in, double *w_out, const double *rows_in, double *rows_out,
                             const double *sign_cf, const double *coef, const double *src, const double *dt_dev,
                             double *scratch, double *node_scratch, void *stream) {
  MB_NVTX();
  if (!m || m->dim != 3 || m->nbcells <= 0 || !t || !bc || !p || p->order != 2 || !w_in || !w_out || w_in == w_out ||
      !rows_in || !rows_out || rows_in == rows_out || !sign_cf || !dt_dev || !scratch || !bc->kind || !bc->value)
    return MB_EINVAL;
  const bool df = p->diffusion != 0;
  if (!m->cell_nbr || !m->cell_vtx || !m->cell_xy || !m->node_coord || !m->cell_volume || !m->face_cellid ||
      !m->n2g_ptr || !m->n2g_idx || !m->n2g_alpha || !m->ghostnid_ptr || !m->ghostnid_idx || !m->face_ghostcenter ||
      !m->cell_edges || !m->edge_origin || !m->edge_sell_ptr || !m->edge_sell_idx || m->nbedges <= 0 ||
      !m->n2c_sum_ptr || !m->n2c_sum_idx || !t->cell_q || !t->link || !t->node_mu)
    return MB_EINVAL;
  auto a32 = [](const void *q) { return ((uintptr_t)q & 31) == 0; };
  if (!a32(scratch) || !a32(sign_cf) || !a32(m->cell_xy) || !a32(m->node_coord) || !a32(rows_in) || !a32(rows_out) ||
      !a32(t->node_mu) || (df && (!coef || !node_scratch)))
    return MB_EINVAL;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  double *fv = scratch, *nrec = scratch + 4 * (long long)m->nbcells, *erec = nrec + 4 * (long long)m->nbnodes;
  const int nnb = ceil_div(m->nbnodes, kBlock), neb = ceil_div(m->nbedges, kBlock);
  const int fb = ceil_div(m->nbcells, MB_TET_FLUX_BLOCK);
  if (df)
    k_tet_sums<true><<<nnb + neb, kBlock, 0, st>>>(*m, *bc, w_in, rows_in, t->node_mu, nrec, erec, node_scratch, nnb);
  else
    k_tet_sums<false><<<nnb + neb, kBlock, 0, st>>>(*m, *bc, w_in, rows_in, t->node_mu, nrec, erec, node_scratch, nnb);
  k_tet_cell<<<ceil_div(m->nbcells, 128), 128, 0, st>>>(*m, *bc, w_in, t->cell_q, rows_in, nrec, erec, fv);
  if (df)
    k_tet_flux<true, true><<<fb, MB_TET_FLUX_BLOCK, 0, st>>>(*m, t->link, *bc, w_in, w_out, sign_cf, coef, src, dt_dev,
                                                            fv, node_scratch, rows_out);
  else
    k_tet_flux<false, true><<<fb, MB_TET_FLUX_BLOCK, 0, st>>>(*m, t->link, *bc, w_in, w_out, sign_cf, coef, src, dt_dev,
                                                             fv, node_scratch, rows_out);
  return cudaGetLastError() == cudaSuccess ? MB_OK : MB_ECUDA;
}

}  // extern "C"
