// The FP64 advection-diffusion step on triangles in one launch: each block carries one tile
// of cells (fv_tile.cuh) through the whole step in shared memory.
//
// The two-launch step (k_f2_phase1, k_f2_phase2) writes a record per cell and a value per
// vertex to memory and gathers, per cell, about 12 least-squares neighbours (centre and
// value), 3 neighbour records and centres, 3 vertices and 3 vertex values through L1: 328 B
// of DRAM traffic per cell-update, and bound by the latency of those gathers.  Here a block
// reads the state of its tile and of the cells around it once, and
//   1. per vertex: sums over its cells in shared memory;
//   2. per cell of the tile and its face layer: the least-squares right-hand side from its three
//      vertices' sums minus its face neighbours (below), the Barth limiter, and the
//      reconstructed value at each of its faces;
//   3. per cell of the tile: upwind fluxes of those face values, diffusion as a linear form
//      with static coefficients (k_tile_coef), forward Euler.
// The face layer's cells are computed by each tile that needs them (a quarter more at 384 cells).
//
// Measured (B200, per step in CUDA graphs of the tuned length, two-launch step with tuned launch shapes
// -> this, one session): 2M triangles 188 -> 112 us, 500,000 48.7 -> 34.2, 180,000 21.6 -> 15.1,
// 62,658 15.7 -> 8.0, 1,152 13.9 -> 6.8; first order with diffusion 20,000 10.2 -> 4.7; no diffusion
// 245,000 27.3 -> 16.0.
// It moves 225 B of DRAM per cell-update (500,000 cells).  What bounds it is the chain of passes in
// a block (barriers 30 % of the stalls, bulk copies and smem latency most of the rest; the
// load/store pipe is 45 % busy, two fifths of that bank conflicts), so three blocks per SM overlap
// each other's passes.  What was tried on the way, 2M triangles: everything loaded through
// registers, 224 us; cp.async of 8 and 16 bytes, 142 us (its scattered writes alone took 5 of 15
// load/store wavefronts per cell); bulk copies of tables laid out per tile, 109 us; launches that
// may overlap their predecessor's end, 107 us (and 7.2 -> 6.2 us at 1,152 cells).
//
// Least squares: the stencil of triangle i (cells sharing a vertex, i excluded) is the union of
// its three vertices' lists; a face neighbour is in two of them, i in all three.  With, per
// vertex v, n its cells, c the mean of their centres, W the mean of their values and
// P = sum (c_j - c)(w_j - W),
//   sum_{j of v} (c_j - c_i)(w_j - w_i) = P + n (c - c_i)(W - w_i),
// so the right-hand side is sum_3 vertices [P + n (c - c_i)(W - w_i)] - sum_3 neighbours
// (c_o - c_i)(w_o - w_i) + the stencil ghosts.  Every term is a product of differences: a
// uniform state gives exact zeros, as the direct sum does.
#include "fv_tile.cuh"

namespace mb {

// 384 threads x 3 blocks (56 registers): 2M triangles 107 us; 512 x 2 with 768-cell tiles 108, 256 x 4
// with 256-cell tiles 111 us
#ifndef MB_TILE_MIN_BLOCKS
#define MB_TILE_MIN_BLOCKS 3
#endif

// shared memory of a tile, in doubles; every array starts on 16 bytes.  The sums of a node
// take the place of its weights and the face values of a cell that of its matrix: each is
// read and then written by one thread.
struct TileLayout {
  int w, xy, C, M, W, nv, q0, q1, rec, inc, cnt, grp, total;
  __host__ __device__ TileLayout(const mb_tiles &t, bool o2, bool df) {
    const int ncell = t.cells + ((t.ext_cap + 1) & ~1), nloc = t.cells + t.face_cap;
    int at = 2;                     // the mbarrier
    w = at; at += ncell;
    xy = at; at += 2 * ncell;
    C = at; at += 2 * t.node_cap;
    M = at; at += 2 * t.node_cap;   // mu, then the sums P
    W = at; at += o2 ? 2 * t.node_cap : 0;
    nv = at; at += df ? t.node_cap : 0;
    q0 = at; at += o2 ? 2 * nloc : 0;   // matrix rows, then face values 0, 1
    q1 = at; at += o2 ? 2 * nloc : 0;   // then face value 2
    rec = at; at += 2 * nloc;
    inc = at; at += t.inc_cap / 4;
    cnt = at; at += t.node_cap / 4;
    grp = at; at += t.grp_cap / 2;
    total = at;
  }
};

template <bool O2, bool DF>
__global__ void __launch_bounds__(kTileThreads, MB_TILE_MIN_BLOCKS)
    k_f2_tile(mb_mesh m, mb_tiles t, mb_bc bc, const double *__restrict__ w, double *__restrict__ w_out,
              const double *__restrict__ sign, const double *__restrict__ coef, const double *__restrict__ src,
              const double *__restrict__ dt_dev) {
  extern __shared__ __align__(16) double sm[];
  const TileLayout L(t, O2, DF);
  uint64_t *bar = reinterpret_cast<uint64_t *>(sm);
  double *cw = sm + L.w;
  double2 *cxy = reinterpret_cast<double2 *>(sm + L.xy);
  double2 *nC = reinterpret_cast<double2 *>(sm + L.C), *nM = reinterpret_cast<double2 *>(sm + L.M);
  double2 *nW = reinterpret_cast<double2 *>(sm + L.W);
  double *nv = sm + L.nv;
  double2 *q0 = reinterpret_cast<double2 *>(sm + L.q0), *q1 = reinterpret_cast<double2 *>(sm + L.q1);
  uint4 *srec = reinterpret_cast<uint4 *>(sm + L.rec);
  uint16_t *sinc = reinterpret_cast<uint16_t *>(sm + L.inc), *scnt = reinterpret_cast<uint16_t *>(sm + L.cnt);
  int *sgrp = reinterpret_cast<int *>(sm + L.grp);
  const int T = t.cells, b = blockIdx.x, c0 = b * T, tid = threadIdx.x;
  const int nc = min(T, m.nbcells - c0);
  const int4 head = __ldg(reinterpret_cast<const int4 *>(t.head) + b);
  const int n1 = head.x, next = head.y, nn = head.z;
  const GhostAfter ghost{make_rule(m, bc, w)};
  const int32_t *ext = t.ext + (long long)b * t.ext_cap;
  const int32_t *node = t.node + (long long)b * t.node_cap;

  // everything the node and cell passes read, copied at once; what the last pass reads, asked
  // for in L2
  tile_let_next_start();
  if (tid == 0) {
    tile_bar_init(bar);
    const long long lb = (long long)b * (T + t.face_cap), nb = (long long)b * t.node_cap;
    const unsigned nloc = n1 ? T + n1 : nc, n8 = (nn + 7) & ~7, wb = 8u * (nc & ~1);
    const unsigned gb = 4u * ((((nn + 31) >> 5) + 4) & ~3);
    const unsigned bytes = wb + 16u * nc + 16u * next + (O2 ? 48u : 16u) * nloc + 32u * nn + 2u * n8 + gb + 2u * head.w;
    tile_bar_expect(bar, bytes);
    tile_bulk(cxy, m.cell_xy + 2 * (long long)c0, 16u * nc, bar);
    tile_bulk(cxy + T, t.ext_xy + 2 * (long long)b * t.ext_cap, 16u * next, bar);
    tile_bulk(nC, t.node_c + 2 * nb, 16u * nn, bar);
    tile_bulk(nM, t.node_mu + 2 * nb, 16u * nn, bar);
    tile_bulk(sinc, t.inc + (long long)b * t.inc_cap, 2u * head.w, bar);
    tile_bulk(scnt, t.count16 + nb, 2u * n8, bar);
    tile_bulk(sgrp, t.grp + (long long)b * t.grp_cap, gb, bar);
    tile_bulk(srec, t.cell + 8 * lb, 16u * nloc, bar);
    if (O2) {
      tile_bulk(q0, t.cell_q0 + 2 * lb, 16u * nloc, bar);
      tile_bulk(q1, t.cell_q1 + 2 * lb, 16u * nloc, bar);
    }
    tile_prefetch(sign + 4 * (long long)c0, 32u * nc);
    if (DF)
      for (int q = 0; q < 6; ++q) tile_prefetch(coef + q * (long long)m.nbcells + c0, 8u * nc);
  }
  int first = 0;
  if (tid < next) first = ld(ext + tid);
  tile_after_previous();
  if (tid == 0) {
    tile_bulk(cw, w + c0, 8u * (nc & ~1), bar);
    if (nc & 1) cw[nc - 1] = ld_after(w + c0 + nc - 1);
  }
  for (int k = tid; k < next; k += kTileThreads) tile_copy8(cw + T + k, w + (k == tid ? first : ld(ext + k)));
  tile_copies_done();
  __syncthreads();
  if (!tile_arrived(bar, t.late)) return;   // never seen

  for (int k = tid; k < nn; k += kTileThreads) {
    const int gb = sgrp[k >> 5], ge = sgrp[(k >> 5) + 1];
    const uint16_t *row = sinc + gb + (k & 31);
    const double2 C = nC[k], mu = nM[k];
    const unsigned cnt = scnt[k];
    // sums relative to the mean centre and the first cell's value: past the end of a list its
    // first cell is repeated, which adds exact zeros
    const double w0 = cw[row[0]];
    double sw = 0., px = 0., py = 0.;
#pragma unroll 2
    for (int q = 32; q < ge - gb; q += 32) {
      const int l = row[q];
      const double2 p = cxy[l];
      const double dw = cw[l] - w0;
      sw += dw;
      px += (p.x - C.x) * dw;
      py += (p.y - C.y) * dw;
    }
    const double n = (double)(int)(cnt & ~kNodeGhosts);
    const double W = w0 + sw / n;
    if (O2) {
      nM[k] = make_double2(px, py);
      nW[k] = make_double2(W, n);
    }
    if (DF) {
      double a = W + (mu.x * px + mu.y * py);
      if (cnt & kNodeGhosts) {
        const int v = ld(node + k);
        a += (ld(t.node_kappa + v) - 1.) * W;
        const int e = ld(m.n2g_ptr + v + 1);
        for (int q = ld(m.n2g_ptr + v); q < e; q += 4) {
          int f[4];
          double g[4];
          ghost4(ghost.g, m.n2g_idx, q, e, f, g);
#pragma unroll
          for (int u = 0; u < 4; ++u)
            if (f[u] >= 0) a += ld(m.n2g_alpha + q + u) * g[u];
        }
      }
      nv[k] = a;
    }
  }
  __syncthreads();

  if (O2) {
    for (int k = tid; k < nc + n1; k += kTileThreads) {
      const int li = k < nc ? k : T + k - nc;
      const TileCell c = tile_cell(srec[li]);
      const double2 ci = cxy[li];
      const double wi = cw[li];
      double jx = 0., jy = 0.;
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        const double2 P = nM[c.v[j]], C = nC[c.v[j]], W = nW[c.v[j]];
        const double d = W.y * (W.x - wi);
        jx += P.x + (C.x - ci.x) * d;
        jy += P.y + (C.y - ci.y) * d;
      }
      double hi = wi, lo = wi;
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        double wo;
        if (c.n[j] != kNoCell) {
          wo = cw[c.n[j]];
          const double2 co = cxy[c.n[j]];
          const double d = wo - wi;
          jx -= (co.x - ci.x) * d;
          jy -= (co.y - ci.y) * d;
        } else {
          const int i = k < nc ? c0 + k : ld(ext + k - nc);
          wo = ghost(-1 - ld(m.cell_nbr + 4 * (long long)i + j));
        }
        hi = pmax(hi, wo);
        lo = pmin(lo, wo);
      }
      if (c.fl & kTileGhosts) {
        const int i = k < nc ? c0 + k : ld(ext + k - nc);
        const int e = ld(m.ghostnid_ptr + i + 1);
        for (int q = ld(m.ghostnid_ptr + i); q < e; q += 4) {
          int f[4];
          double g[4];
          ghost4(ghost.g, m.ghostnid_idx, q, e, f, g);
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            if (f[u] < 0) continue;
            const double d = g[u] - wi;
            jx += (ld(m.face_ghostcenter + 3 * (long long)f[u]) - ci.x) * d;
            jy += (ld(m.face_ghostcenter + 3 * (long long)f[u] + 1) - ci.y) * d;
          }
        }
      }
      // reconstruction offsets g . (face centre - centre) at the three faces; they sum to zero
      const double2 Q0 = q0[li], Q1 = q1[li];
      double de[3];
      de[0] = Q0.x * jx + Q0.y * jy;
      de[1] = Q1.x * jx + Q1.y * jy;
      de[2] = -(de[0] + de[1]);
      const double ps = tile_barth(de, hi - wi, wi - lo, 1e-8);
      q0[li] = make_double2(wi + ps * de[0], wi + ps * de[1]);
      q1[li].x = wi + ps * de[2];
    }
    __syncthreads();
  }

  const double dt = ld_after(dt_dev);
#pragma unroll 2
  for (int k = tid; k < nc; k += kTileThreads) {
    const int i = c0 + k;
    double s[3], pad;
    ld4d_stream(sign + 4 * (long long)i, s[0], s[1], s[2], pad, l2_stream());
    double k1, k2, B[3], rv;
    if (DF) {
      const double *q = coef + i;
      const long long n = m.nbcells;
      const uint64_t once = l2_stream();
      k1 = ldd_stream(q, once); k2 = ldd_stream(q + n, once);
      B[0] = ldd_stream(q + 2 * n, once); B[1] = ldd_stream(q + 3 * n, once); B[2] = ldd_stream(q + 4 * n, once);
      rv = ldd_stream(q + 5 * n, once);
    } else {
      rv = 1 / ld(m.cell_volume + i);
    }
    const TileCell c = tile_cell(srec[k]);
    const double wi = cw[k];
    double acc = 0., mine[3] = {wi, wi, wi};
    if (O2) {
      const double2 u = q0[k];
      mine[0] = u.x; mine[1] = u.y; mine[2] = q1[k].x;
    }
    if (DF) {
      const double v0 = nv[c.v[0]];
      acc = k1 * (nv[c.v[1]] - v0) + k2 * (nv[c.v[2]] - v0);
    }
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      const bool own = tile_own(c.fl, j), take_me = (s[j] >= 0) == own;
      double wo, far;
      if (c.n[j] != kNoCell) {
        wo = cw[c.n[j]];
        far = wo;
        if (O2 && !take_me) {
          const int p = tile_peer(c.fl, j);
          far = sm[(p == 2 ? L.q1 : L.q0 + p) + 2 * c.n[j]];
        }
      } else {
        wo = far = ghost(-1 - ld(m.cell_nbr + 4 * (long long)i + j));
      }
      const double sol = take_me ? mine[j] : far;
      const double F = s[j] * sol;
      acc += own ? -F : F;
      if (DF) acc += B[j] * (wo - wi);
    }
    w_out[i] = wi + dt * (acc * rv + (src ? ld_after(src + i) : 0.0));
  }
}

template <bool O2, bool DF>
static int run_tile(const mb_mesh &m, const mb_tiles &t, const mb_bc &bc, const double *w, double *w_out,
                    const double *sign, const double *coef, const double *src, const double *dt, cudaStream_t st) {
  const int bytes = 8 * TileLayout(t, O2, DF).total;
  return tile_launch<k_f2_tile<O2, DF>>(t.count, kTileThreads, bytes, st, m, t, bc, w, w_out, sign, coef, src, dt) ==
                 cudaSuccess
             ? MB_OK
             : MB_ECUDA;
}

}  // namespace mb

using namespace mb;

extern "C" {

int mb_tile_bytes(const mb_tiles *t) { return t ? 8 * TileLayout(*t, true, true).total : MB_EINVAL; }

int mb_advdiff_step_tile(const mb_mesh *m, const mb_tiles *t, const mb_bc *bc, const mb_advdiff_params *p,
                         const double *w_in, double *w_out, const double *sign_cf, const double *coef,
                         const double *src, const double *dt_dev, void *stream) {
  MB_NVTX();
  if (!m || m->dim != 2 || m->nbcells <= 0 || !t || !bc || !p || !w_in || !w_out || w_in == w_out || !sign_cf ||
      !dt_dev || !bc->kind || !bc->value)
    return MB_EINVAL;
  if (p->order != 1 && p->order != 2) return MB_EINVAL;
  const bool o2 = p->order == 2, df = p->diffusion != 0;
  if (!m->cell_nbr || !m->cell_xy || !m->cell_volume || !m->face_cellid || !m->n2g_ptr || !m->n2g_idx ||
      !m->n2g_alpha || !m->ghostnid_ptr || !m->ghostnid_idx || !m->face_ghostcenter || !tiles_ok(m, t))
    return MB_EINVAL;
  if (!o2 && !df) return MB_EINVAL;   // nothing to share: mb_advdiff_step is one launch already
  if (((uintptr_t)m->cell_xy & 15) || ((uintptr_t)w_in & 15)) return MB_EINVAL;
  if (((uintptr_t)sign_cf & 31) || (df && !coef)) return MB_EINVAL;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  if (!o2) return run_tile<false, true>(*m, *t, *bc, w_in, w_out, sign_cf, coef, src, dt_dev, st);
  return df ? run_tile<true, true>(*m, *t, *bc, w_in, w_out, sign_cf, coef, src, dt_dev, st)
            : run_tile<true, false>(*m, *t, *bc, w_in, w_out, sign_cf, coef, src, dt_dev, st);
}

}  // extern "C"
