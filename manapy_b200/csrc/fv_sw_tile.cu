// The FP64 shallow-water step on triangles in one launch: each block carries one tile of cells with
// its faces (fv_tile.cuh, mb_face_tiles) through the step in shared memory.
//
// The two-launch step (k_sw2_flux, k_sw2_cell) writes a 32-byte flux per face and reads it back from
// both cells, gathers five fields of two cells per face and again three neighbours per cell, and
// recomputes face normals from the vertices: about 400 B of traffic per cell-update, bound by the
// gathers' latency.  Here a block reads the state of its cells and of the cells across its outer
// faces once; a flux crosses shared memory only.  Faces between two tiles are evaluated by both
// (a tenth more at 256 cells).  Same arithmetic, same bits (fv_sw.cuh).
//
// Measured (B200, per step in a CUDA graph of 48, two launches -> this, one session): 1.28M triangles
// 133 -> 80 us, 245,000 27.9 -> 19.4, 80,000 12.9 -> 7.4, 45,000 10.1 -> 5.8, 5,000 8.0 -> 4.6; second
// order (three launches -> two) 1.28M 277 -> 233, 245,000 63.9 -> 48.1, 45,000 20.8 -> 14.3, 5,000
// 17.5 -> 12.0.  The passes are long serial chains of FP64 operations (square roots and divisions
// among them) between barriers, so many small blocks per SM do best: 1.28M triangles, 128 threads x
// 5 blocks (96 registers) 80 us with 256-cell tiles; 128 x 6 93; 256 x 3 96; 160 x 4 87; 384 x 2 101.
#include "fv_sw.cuh"
#include "fv_tile.cuh"

namespace mb {

#ifndef MB_SW_TILE_THREADS
#define MB_SW_TILE_THREADS 128
#endif
#ifndef MB_SW_TILE_MIN_BLOCKS
#define MB_SW_TILE_MIN_BLOCKS 5
#endif
constexpr int kSwTileThreads = MB_SW_TILE_THREADS;

// shared memory of a tile, in doubles; every array starts on 16 bytes
struct SwTileLayout {
  int q, qstride, fl, n0, n1, mes, face, rec, red, total;
  __host__ __device__ explicit SwTileLayout(const mb_face_tiles &t) {
    int at = 2;                    // the mbarrier
    qstride = t.cells + ((t.out_cap + 1) & ~1);
    q = at; at += 5 * qstride;
    fl = at; at += 4 * t.face_cap;
    n0 = at; at += t.face_cap;
    n1 = at; at += t.face_cap;
    mes = at; at += t.face_cap;
    face = at; at += t.face_cap / 2;
    rec = at; at += 2 * t.cells;
    red = at; at += kSwTileThreads / 32;
    total = at;
  }
};

struct SwTileArgs {
  const double *q[5];
  double *out[4];
  const double *gr[4], *psi;   // order 2: gradients of h and hc, hc's limiter
  const double *dt_cur;
  double *dt_next, *dt_after;
  double cfl, grav;
  int walls;
};

template <bool ORDER2>
__global__ void __launch_bounds__(kSwTileThreads, MB_SW_TILE_MIN_BLOCKS)
    k_sw2_tile(mb_mesh m, mb_face_tiles t, SwTileArgs a) {
  extern __shared__ __align__(16) double sm[];
  const SwTileLayout L(t);
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
    tile_prefetch(t.cell_ns + 2 * (long long)c0, 16u * nc);
  }
  int first = 0;
  if (tid < n1) first = ld(out + tid);
  tile_after_previous();
  if (tid == 0) {
#pragma unroll
    for (int k = 0; k < 5; ++k) {
      tile_bulk(q + k * Q, a.q[k] + c0, 8u * (nc & ~1), bar);
      if (nc & 1) q[k * Q + nc - 1] = ld_after(a.q[k] + c0 + nc - 1);
    }
    if (b == 0) *a.dt_after = 1e6;
  }
  for (int e = tid; e < n1; e += kSwTileThreads) {
    const int c = e == tid ? first : ld(out + e);
#pragma unroll
    for (int k = 0; k < 5; ++k) tile_copy8(q + k * Q + T + e, a.q[k] + c);
  }
  tile_copies_done();
  __syncthreads();
  if (!tile_arrived(bar, t.late)) return;   // never seen

  for (int f = tid; f < nf; f += kSwTileThreads) {
    const uint32_t lr = sface[f];
    const int l = lr & 0xffffu, r = lr >> 16;
    const bool rim = r == kNoCell;
    const int rr = rim ? l : r;     // Neumann ghost: the interior cell's state
    const double n0 = sn0[f], n1f = sn1[f];
    double h_l = q[l], hc_l = q[3 * Q + l], h_r = q[rr], hc_r = q[3 * Q + rr];
    const double hu_l = q[Q + l], hv_l = q[2 * Q + l];
    double hu_r = q[Q + rr], hv_r = q[2 * Q + rr];
    if (ORDER2) {
      // reconstruction as sw2_flux_face, from the cells' gradients; the face centre through the
      // left or right cell's own face list
      const int gl = l < T ? c0 + l : ld(out + l - T), gr = rim ? gl : (r < T ? c0 + r : ld(out + r - T));
      const TileCell c = tile_cell(srec[l < T ? l : r]);
      const int j = c.v[0] == f ? 0 : (c.v[1] == f ? 1 : 2);
      const int g = ld(m.cell_faces + 4 * (long long)(l < T ? gl : gr) + j);
      const double fx = ld(m.face_center + 3 * (long long)g), fy = ld(m.face_center + 3 * (long long)g + 1);
      sw_reconstruct(a.gr, a.psi, m.cell_center, gl, fx, fy, h_l, hc_l);
      if (!rim)                     // a ghost is the interior cell's own value
        sw_reconstruct(a.gr, a.psi, m.cell_center, gr, fx, fy, h_r, hc_r);
    }
    if (rim && a.walls == MB_WALLS_REFLECT) wall_mirror(hu_l, hv_l, n0, n1f, hu_r, hv_r);
    double F[4];
    srnh0(hu_l, hu_r, hv_l, hv_r, h_l, h_r, hc_l, hc_r, q[4 * Q + l], q[4 * Q + rr], n0, n1f, smes[f], a.grav, F);
    fl[f] = make_double2(F[0], F[1]);
    fl[t.face_cap + f] = make_double2(F[2], F[3]);
  }
  __syncthreads();

  const double dt = ld_after(a.dt_cur);
  double best = 1e300;
  for (int k = tid; k < nc; k += kSwTileThreads) {
    const int i = c0 + k;
    const TileCell c = tile_cell(srec[k]);   // v: local faces, n: local neighbours
    SwCell s;
    s.h = q[k]; s.hu = q[Q + k]; s.hv = q[2 * Q + k]; s.hc = q[3 * Q + k]; s.Z = q[4 * Q + k];
    s.vol = ld(m.cell_volume + i);
    const double2 ns = ldd2(t.cell_ns + 2 * (long long)i);
    s.ns0x = ns.x; s.ns0y = ns.y;
    s.code = (uint8_t)((c.fl >> 3) & 63u);
    double F[3][4], n0[3], n1c[3], mes[3];
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      const int f = c.v[j];
      const double2 x = fl[f], y = fl[t.face_cap + f];
      F[j][0] = x.x; F[j][1] = x.y; F[j][2] = y.x; F[j][3] = y.y;
      n0[j] = sn0[f]; n1c[j] = sn1[f]; mes[j] = smes[f];
      s.own[j] = (c.fl >> j) & 1u;
      s.inner[j] = c.n[j] != kNoCell;
      const bool neg = (c.fl >> (9 + j)) & 1u;
      s.s0[j] = neg ? -1.0 * n0[j] : n0[j];
      s.s1[j] = neg ? -1.0 * n1c[j] : n1c[j];
      const int o = s.inner[j] ? c.n[j] : k;
      s.hp[j] = q[o];
      s.zp[j] = q[4 * Q + o];
      // where the cell has a boundary face, cells.cellfid slot j is not the cell across face j
      if ((c.fl & kTileRim) && s.inner[j]) {
        const int g = ld(m.cell_cellfid + 4 * (long long)i + j);
        s.hp[j] = ld_after(a.q[0] + g);
        s.zp[j] = ld_after(a.q[4] + g);
      }
    }
    double h, hu, hv, hc;
    sw_update_cell(s, F, dt, a.grav, h, hu, hv, hc);
    a.out[0][i] = h; a.out[1][i] = hu; a.out[2][i] = hv; a.out[3][i] = hc;
    best = pmin(best, sw_dt_candidate(h, hu, hv, n0, n1c, mes, s.vol, a.cfl, a.grav));
  }
  for (int o = 16; o > 0; o >>= 1) best = pmin(best, __shfl_xor_sync(0xffffffffu, best, o));
  if ((tid & 31) == 0) red[tid >> 5] = best;
  __syncthreads();
  if (tid == 0) {
#pragma unroll
    for (int w = 1; w < kSwTileThreads / 32; ++w) best = pmin(best, red[w]);
    if (best < 1e300) atomic_min_pos(a.dt_next, best);
  }
}

// declared in fv_advdiff.cu
int sw_gradients(const mb_mesh &m, const double *h, const double *hc, double *hx, double *hy, double *cx,
                 double *cy, double *psi, cudaStream_t st);

}  // namespace mb

using namespace mb;

extern "C" int mb_sw_step_tile(const mb_mesh *m, const mb_face_tiles *t, const double *const q_in[5],
                               double *const q_out[4], double cfl, double grav, int32_t order, int32_t walls,
                               double *scratch, const double *dt_cur, double *dt_next, double *dt_after,
                               void *stream) {
  MB_NVTX();
  if (!m || m->dim != 2 || m->nbcells <= 0 || !q_in || !q_out || (order != 1 && order != 2) || !dt_cur || !dt_next ||
      !dt_after || dt_cur == dt_next || dt_cur == dt_after || dt_next == dt_after)
    return MB_EINVAL;
  if (walls != MB_WALLS_NEUMANN && walls != MB_WALLS_REFLECT) return MB_EINVAL;
  if (!face_tiles_ok(m, t) || !m->cell_volume || !m->cell_cellfid || !m->cell_faces || !m->face_center ||
      !m->cell_center || (order == 2 && !scratch))
    return MB_EINVAL;
  SwTileArgs a{};
  for (int k = 0; k < 5; ++k) {
    if (!q_in[k] || ((uintptr_t)q_in[k] & 15) || (k < 4 && (!q_out[k] || q_out[k] == q_in[k]))) return MB_EINVAL;
    a.q[k] = q_in[k];
    if (k < 4) a.out[k] = q_out[k];
  }
  a.dt_cur = dt_cur; a.dt_next = dt_next; a.dt_after = dt_after;
  a.cfl = cfl; a.grav = grav; a.walls = walls;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  const int bytes = 8 * SwTileLayout(*t).total;
  cudaError_t e;
  if (order == 2) {
    const long long n = m->nbcells;
    const int rc = sw_gradients(*m, q_in[0], q_in[3], scratch, scratch + n, scratch + 2 * n, scratch + 3 * n,
                                scratch + 4 * n, st);
    if (rc != MB_OK) return rc;
    for (int k = 0; k < 4; ++k) a.gr[k] = scratch + k * n;
    a.psi = scratch + 4 * n;
    e = tile_launch<k_sw2_tile<true>>(t->count, kSwTileThreads, bytes, st, *m, *t, a);
  } else {
    e = tile_launch<k_sw2_tile<false>>(t->count, kSwTileThreads, bytes, st, *m, *t, a);
  }
  return e == cudaSuccess ? MB_OK : MB_ECUDA;
}
