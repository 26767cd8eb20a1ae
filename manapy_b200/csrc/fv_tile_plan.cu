// Builds the tiles of a triangle mesh (fv_tile.cuh) on the device: one block per tile, two
// passes (sizes, then the tables at strides the caller chose from the sizes).  Set-up work,
// once per mesh.
#include "fv_tile_plan.cuh"

namespace mb {

constexpr int kHashCells = 4096, kHashNodes = 2048, kMaxOut = 2048, kMaxNodes = 1536;

struct TileShared {
  int ckey[kHashCells];
  uint16_t cval[kHashCells];
  int nkey[kHashNodes];
  uint16_t nval[kHashNodes];
  int out[kMaxOut];       // outside cells: the face layer, then the rest
  int rest[kMaxOut];
  int node[2048];
  int grp[kMaxNodes / 32 + 2];
  int n1, n2, nn, bad;
};

template <bool WRITE>
__global__ void __launch_bounds__(kTileThreads) k_tile_plan(mb_mesh m, mb_tiles t, int32_t *head, int32_t *status,
                                                            const double *minv, const double *node_w) {
  extern __shared__ unsigned char raw[];
  TileShared &s = *reinterpret_cast<TileShared *>(raw);
  const int T = t.cells, c0 = blockIdx.x * T, tid = threadIdx.x, nt = blockDim.x;
  const int nc = min(T, m.nbcells - c0);
  for (int i = tid; i < kHashCells; i += nt) s.ckey[i] = -1;
  for (int i = tid; i < kHashNodes; i += nt) s.nkey[i] = -1;
  if (tid == 0) { s.n1 = s.n2 = s.nn = s.bad = 0; }
  __syncthreads();
  // the face layer
  for (int k = tid; k < 3 * nc; k += nt) {
    const int i = c0 + k / 3, j = k % 3;
    const int o = ld(m.cell_nbr + 4 * (long long)i + j);
    if (o >= 0) {
      // the sums by inclusion-exclusion take the three neighbours of a cell as distinct
      for (int q = 0; q < j; ++q)
        if (ld(m.cell_nbr + 4 * (long long)i + q) == o) s.bad = 1;
      if (o < c0 || o >= c0 + nc) {
        bool was_new;
        const int h = hash_put(s.ckey, kHashCells, o, was_new);
        if (h < 0) s.bad = 1;
        if (was_new) {
          const int at = atomicAdd(&s.n1, 1);
          if (at < kMaxOut) s.out[at] = o; else s.bad = 1;
        }
      }
    }
  }
  __syncthreads();
  const int n1 = min(s.n1, kMaxOut);
  block_sort(s.out, n1);
  // the vertices of the tile and its face layer
  for (int k = tid; k < 3 * (nc + n1); k += nt) {
    const int l = k / 3;
    const int i = l < nc ? c0 + l : s.out[l - nc];
    const int v = ld(m.cell_vtx + 4 * (long long)i + k % 3);
    bool was_new;
    const int h = hash_put(s.nkey, kHashNodes, v, was_new);
    if (h < 0) s.bad = 1;
    if (was_new) {
      const int at = atomicAdd(&s.nn, 1);
      if (at < kMaxNodes) s.node[at] = v; else s.bad = 1;
    }
  }
  __syncthreads();
  const int nn = min(s.nn, kMaxNodes);
  block_sort(s.node, nn);
  // every other cell of these vertices
  for (int k = tid; k < nn; k += nt) {
    const int v = s.node[k];
    for (int q = ld(m.n2c_ptr + v); q < ld(m.n2c_ptr + v + 1); ++q) {
      const int c = ld(m.n2c_idx + q);
      if (c >= c0 && c < c0 + nc) continue;
      bool was_new;
      const int h = hash_put(s.ckey, kHashCells, c, was_new);
      if (h < 0) s.bad = 1;
      if (was_new) {
        const int at = atomicAdd(&s.n2, 1);
        if (at < kMaxOut) s.rest[at] = c; else s.bad = 1;
      }
    }
  }
  __syncthreads();
  const int n2 = min(s.n2, kMaxOut);
  block_sort(s.rest, n2);
  // rows of the node -> cells lists: per 32 nodes the longest list
  const int ng = (nn + 31) >> 5;
  for (int g = tid; g < ng; g += nt) {
    int longest = 0;
    for (int k = 32 * g; k < min(32 * g + 32, nn); ++k)
      longest = max(longest, ld(m.n2c_ptr + s.node[k] + 1) - ld(m.n2c_ptr + s.node[k]));
    if (longest >= (int)kNodeGhosts) s.bad = 1;
    s.grp[g + 1] = 32 * longest;
  }
  __syncthreads();
  if (tid == 0) {
    s.grp[0] = 0;
    for (int g = 0; g < ng; ++g) s.grp[g + 1] += s.grp[g];
    if (T + n1 + n2 >= kNoCell || s.grp[ng] > 65535) s.bad = 1;
    if (!WRITE) {
      head[4 * blockIdx.x] = n1;
      head[4 * blockIdx.x + 1] = n1 + n2;
      head[4 * blockIdx.x + 2] = nn;
      head[4 * blockIdx.x + 3] = s.grp[ng];
      if (s.bad) atomicMax(status, 1);
    }
  }
  if (!WRITE) return;
  __syncthreads();
  // this pass found the same sets; a tile that does not fit its strides writes nothing
  if (s.bad || n1 > t.face_cap || n1 + n2 > t.ext_cap || nn > t.node_cap || s.grp[ng] > t.inc_cap) return;
  for (int k = tid; k < n1 + n2; k += nt) {
    const int c = k < n1 ? s.out[k] : s.rest[k - n1];
    bool was_new;
    s.cval[hash_put(s.ckey, kHashCells, c, was_new)] = (uint16_t)(T + k);
    t.ext[(long long)blockIdx.x * t.ext_cap + k] = c;
  }
  for (int k = tid; k < nn; k += nt) {
    const int v = s.node[k];
    bool was_new;
    s.nval[hash_put(s.nkey, kHashNodes, v, was_new)] = (uint16_t)k;
    const bool ghosts = ld(m.n2g_ptr + v + 1) > ld(m.n2g_ptr + v);
    const long long at = (long long)blockIdx.x * t.node_cap + k;
    t.node[at] = v;
    t.count16[at] = (uint16_t)((ld(m.n2c_ptr + v + 1) - ld(m.n2c_ptr + v)) | (ghosts ? kNodeGhosts : 0u));
    const double *row = node_w + 4 * (long long)v;
    reinterpret_cast<double2 *>(t.node_c)[at] = make_double2(row[0], row[1]);
    reinterpret_cast<double2 *>(t.node_mu)[at] = make_double2(row[2], row[3]);
  }
  for (int k = tid; k < n1 + n2; k += nt)
    reinterpret_cast<double2 *>(t.ext_xy)[(long long)blockIdx.x * t.ext_cap + k] =
        ldd2(m.cell_xy + 2 * (long long)(k < n1 ? s.out[k] : s.rest[k - n1]));
  __syncthreads();
  auto local = [&](int c) -> int {
    return c >= c0 && c < c0 + nc ? c - c0 : (int)hash_get(s.ckey, s.cval, kHashCells, c);
  };
  for (int k = tid; k < nc + n1; k += nt) {
    const int i = k < nc ? c0 + k : s.out[k - nc];
    const int li = k < nc ? k : T + k - nc;
    const int4 nb = ld4(m.cell_nbr + 4 * (long long)i), vt = ld4(m.cell_vtx + 4 * (long long)i);
    const unsigned own = ld(m.cell_flags + i) & 7u;
    unsigned fl = own;
    int n[3];
    for (int j = 0; j < 3; ++j) {
      const int o = comp(nb, j);
      n[j] = o < 0 ? kNoCell : local(o);
      if (o >= 0) {
        const int4 back = ld4(m.cell_nbr + 4 * (long long)o);
        const int peer = back.x == i ? 0 : (back.y == i ? 1 : 2);
        fl |= (unsigned)peer << (3 + 2 * j);
      }
    }
    if (ld(m.ghostnid_ptr + i + 1) > ld(m.ghostnid_ptr + i)) fl |= kTileGhosts;
    uint4 u;
    u.x = hash_get(s.nkey, s.nval, kHashNodes, vt.x) | ((unsigned)hash_get(s.nkey, s.nval, kHashNodes, vt.y) << 16);
    u.y = hash_get(s.nkey, s.nval, kHashNodes, vt.z) | ((unsigned)n[0] << 16);
    u.z = (unsigned)n[1] | ((unsigned)n[2] << 16);
    u.w = fl;
    const long long at = (long long)blockIdx.x * (T + t.face_cap) + li;
    reinterpret_cast<uint4 *>(t.cell)[at] = u;
    // (de_0, de_1) = Q J: reconstruction offsets at the first two faces from the right-hand side
    // (a face's centre minus the cell's: a sixth of the differences to the opposite vertex, which round to
    // the size of the cell, not to that of its coordinates)
    const double2 X0 = ldd2(m.node_coord + 2 * (long long)vt.x), X1 = ldd2(m.node_coord + 2 * (long long)vt.y),
                  X2 = ldd2(m.node_coord + 2 * (long long)vt.z);
    const double ia = minv[4 * (long long)i], ib = minv[4 * (long long)i + 1], ic = minv[4 * (long long)i + 2];
    const double ax = ((X0.x - X2.x) + (X1.x - X2.x)) * (1. / 6), ay = ((X0.y - X2.y) + (X1.y - X2.y)) * (1. / 6);
    const double bx = ((X1.x - X0.x) + (X2.x - X0.x)) * (1. / 6), by = ((X1.y - X0.y) + (X2.y - X0.y)) * (1. / 6);
    reinterpret_cast<double2 *>(t.cell_q0)[at] = make_double2(ax * ia + ay * ib, ax * ib + ay * ic);
    reinterpret_cast<double2 *>(t.cell_q1)[at] = make_double2(bx * ia + by * ib, bx * ib + by * ic);
  }
  for (int g = tid; g <= ng; g += nt) t.grp[(long long)blockIdx.x * t.grp_cap + g] = s.grp[g];
  uint16_t *inc = t.inc + (long long)blockIdx.x * t.inc_cap;
  for (int k = tid; k < 32 * ng; k += nt) {
    const int g = k >> 5, len = (s.grp[g + 1] - s.grp[g]) >> 5;
    const int v = k < nn ? s.node[k] : -1;
    const int b = v < 0 ? 0 : ld(m.n2c_ptr + v), e = v < 0 ? 0 : ld(m.n2c_ptr + v + 1);
    for (int q = 0; q < len; ++q)
      inc[s.grp[g] + 32 * q + (k & 31)] = b < e ? (uint16_t)local(ld(m.n2c_idx + (b + q < e ? b + q : b))) : 0;
  }
}

// A step launched next may read its tables before it waits for its predecessor in the stream: that
// predecessor is this launch, which waits for the tables.
__global__ void k_tile_filled() {}
void tile_filled(cudaStream_t st) { k_tile_filled<<<1, 32, 0, st>>>(); }

// inverse of the least-squares moment matrix of every cell (manapy/ast/functions2d.py:5-104),
// summed over the lsq_sell slots and the stencil ghosts: {i_yy, -i_xy, i_xx} / det, 0
__global__ void __launch_bounds__(kBlock) k_tile_minv(mb_mesh m, double *__restrict__ out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= m.nbcells) return;
  const double2 c = ldd2(m.cell_xy + 2 * (long long)i);
  double ixx = 0., iyy = 0., ixy = 0.;
  const int sb = ld(m.lsq_sell_ptr + (i >> 5)), se = ld(m.lsq_sell_ptr + (i >> 5) + 1);
  for (int k = sb + (threadIdx.x & 31); k < se; k += 32) {
    const int o = ld(m.lsq_sell_idx + k);
    if (o < 0) continue;
    const double2 p = ldd2(m.cell_xy + 2 * (long long)o);
    const double dx = p.x - c.x, dy = p.y - c.y;
    ixx += dx * dx; iyy += dy * dy; ixy += dx * dy;
  }
  for (int k = ld(m.ghostnid_ptr + i); k < ld(m.ghostnid_ptr + i + 1); ++k) {
    const double *g = m.face_ghostcenter + 3 * (long long)ld(m.ghostnid_idx + k);
    const double dx = ld(g) - c.x, dy = ld(g + 1) - c.y;
    ixx += dx * dx; iyy += dy * dy; ixy += dx * dy;
  }
  const double det = ixx * iyy - ixy * ixy;
  st4d_plain(out + 4 * (long long)i, iyy / det, -ixy / det, ixx / det, 0.0);
}

// of every node, {c_x, c_y, mu_x, mu_y}: the mean c of the centres c_j of its n cells, and its
// centre -> vertex weights in terms of the node sums: with the vertex X,
// alpha_j = (1 + lambda . (c_j - X)) / den (manapy/ast/functions2d.py:199-276, weights
// manapy/ddm/ddm_utils2d.py:608-705),
//   sum alpha_j w_j = kappa mean(w) + mu . sum (c_j - c) (w_j - mean(w)),
// kappa = sum alpha_j (1 up to rounding where the node has no ghosts), mu = lambda / den
__global__ void __launch_bounds__(kBlock) k_tile_node(mb_mesh m, double *__restrict__ out,
                                                      double *__restrict__ kappa_out) {
  const int v = blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= m.nbnodes) return;
  const double2 X = ldd2(m.node_coord + 2 * (long long)v);
  double ixx = 0., iyy = 0., ixy = 0., rx = 0., ry = 0., kappa = 0.;
  const int cb = ld(m.n2c_ptr + v), ce = ld(m.n2c_ptr + v + 1);
  const int gb = ld(m.n2g_ptr + v), ge = ld(m.n2g_ptr + v + 1);
  for (int k = cb; k < ce; ++k) {
    const double2 p = ldd2(m.cell_xy + 2 * (long long)ld(m.n2c_idx + k));
    const double dx = p.x - X.x, dy = p.y - X.y;
    ixx += dx * dx; iyy += dy * dy; ixy += dx * dy;
    rx += dx; ry += dy;
    kappa += ld(m.n2c_alpha + k);
  }
  const double n = (double)max(1, ce - cb);
  const double cx = X.x + rx / n, cy = X.y + ry / n;
  for (int k = gb; k < ge; ++k) {
    const double *g = m.face_ghostcenter + 3 * (long long)ld(m.n2g_idx + k);
    const double dx = ld(g) - X.x, dy = ld(g + 1) - X.y;
    ixx += dx * dx; iyy += dy * dy; ixy += dx * dy;
    rx += dx; ry += dy;
  }
  const double D = ixx * iyy - ixy * ixy;
  const double lx = (ixy * ry - iyy * rx) / D, ly = (ixy * rx - ixx * ry) / D;
  const double den = (double)(ce - cb + ge - gb) + lx * rx + ly * ry;
  st4d_plain(out + 4 * (long long)v, cx, cy, lx / den, ly / den);
  kappa_out[v] = kappa;
}

// the diamond diffusion of a cell as a linear form, planes c1, c2, B_0, B_1, B_2, 1 / V, with
//   sum_j D grad(w) . N_j = c1 (V_1 - V_0) + c2 (V_2 - V_0) + sum_j B_j (w_j - w_i),
// V the values at the cell's vertices, w_j the value across face j.  manapy's face flux
// (manapy/ast/functions2d.py:108-196, manapy/solvers/advecdiff/fvm_utils.py:5-26) grouped by
// value is A (V_a - V_b) + B (w_L - w_R) (see f2_phase2); B_j = 0 on faces without a gradient
__global__ void __launch_bounds__(kBlock) k_tile_coef(mb_mesh m, mb_bc bc, mb_advdiff_params p,
                                                      double *__restrict__ out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= m.nbcells) return;
  const int4 vt = ld4(m.cell_vtx + 4 * (long long)i), nb = ld4(m.cell_nbr + 4 * (long long)i);
  const uint32_t fl = ld(m.cell_flags + i);
  const double2 P[3] = {ldd2(m.node_coord + 2 * (long long)vt.x), ldd2(m.node_coord + 2 * (long long)vt.y),
                        ldd2(m.node_coord + 2 * (long long)vt.z)};
  const double2 ci = ldd2(m.cell_xy + 2 * (long long)i);
  double a[3], B[3];
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    const int o = comp(nb, j), f = -1 - o;
    a[j] = B[j] = 0.;
    if (o < 0 && !ld(bc.face_grad_on + f)) continue;
    const bool own = f2_own(fl, j), rev = f2_rev(fl, j);
    const double2 Pj = P[j], Pk = P[(j + 1) % 3];
    const double2 Xa = rev ? Pk : Pj, Xb = rev ? Pj : Pk;
    const double2 co = o < 0 ? make_double2(ld(m.face_ghostcenter + 3 * (long long)f),
                                            ld(m.face_ghostcenter + 3 * (long long)f + 1))
                             : ldd2(m.cell_xy + 2 * (long long)o);
    const double2 v1 = own ? ci : co, v2 = own ? co : ci;
    const double air = 0.5 * ((Xb.x - Xa.x) * (v2.y - v1.y) + (v1.x - v2.x) * (Xb.y - Xa.y));
    const double rda = 1 / (2 * air);
    double n0 = Xa.y - Xb.y, n1 = Xb.x - Xa.x;
    if (f2_flip(fl, j)) { n0 = -n0; n1 = -n1; }
    const double gx = rda * p.Dxx * n0, gy = rda * p.Dyy * n1;
    const double A = gx * (v1.y - v2.y) - gy * (v1.x - v2.x);
    B[j] = gy * (Xb.x - Xa.x) - gx * (Xb.y - Xa.y);
    a[j] = own != rev ? A : -A;
  }
  const long long n = m.nbcells;
  out[i] = a[1] - a[0];
  out[n + i] = a[2] - a[1];
  out[2 * n + i] = B[0];
  out[3 * n + i] = B[1];
  out[4 * n + i] = B[2];
  out[5 * n + i] = 1 / ld(m.cell_volume + i);
}

// the wait of a step for copies that were never issued
__global__ void k_tile_wait_check(int32_t *late, int limit) {
  __shared__ __align__(16) uint64_t bar;
  if (threadIdx.x == 0) {
    tile_bar_init(&bar);
    tile_bar_expect(&bar, 16);
  }
  __syncthreads();
  tile_arrived(&bar, late, limit);
}

// ---------------------------------------------------------------- tiles with their faces
//
// For the steps that exchange fluxes (shallow water, Euler): a tile's local cells are its own and,
// at cells + e, the cells across its outer faces; its local faces those of its cells, in the
// order of their first cell in the tile.

struct FaceTileShared {
  int ckey[kHashNodes];
  uint16_t cval[kHashNodes];
  int out[kMaxOut];
  int base[MB_TILE_MAX_CELLS];   // faces of the tile's cells before each cell
  int n1, bad;
};

template <bool WRITE>
__global__ void __launch_bounds__(kTileThreads) k_face_plan(mb_mesh m, mb_face_tiles t, int32_t *head,
                                                            int32_t *status) {
  extern __shared__ unsigned char raw[];
  FaceTileShared &s = *reinterpret_cast<FaceTileShared *>(raw);
  const int T = t.cells, c0 = blockIdx.x * T, tid = threadIdx.x, nt = blockDim.x;
  const int nc = min(T, m.nbcells - c0);
  for (int i = tid; i < kHashNodes; i += nt) s.ckey[i] = -1;
  if (tid == 0) s.n1 = s.bad = 0;
  __syncthreads();
  auto inside = [&](int c) { return c >= c0 && c < c0 + nc; };
  // a face is listed by its first cell in the tile; two cells sharing two faces are refused (the
  // search for a face in its neighbour would find the other one)
  for (int k = tid; k < nc; k += nt) {
    const int i = c0 + k;
    const int4 nb = ld4(m.cell_nbr + 4 * (long long)i);
    int mine = 0;
    for (int j = 0; j < 3; ++j) {
      const int o = comp(nb, j);
      for (int q = 0; q < j; ++q)
        if (o >= 0 && comp(nb, q) == o) s.bad = 1;
      if (o < 0 || !inside(o) || o > i) ++mine;
      if (o >= 0 && !inside(o)) {
        bool was_new;
        if (hash_put(s.ckey, kHashNodes, o, was_new) < 0) s.bad = 1;
        if (was_new) {
          const int at = atomicAdd(&s.n1, 1);
          if (at < kMaxOut) s.out[at] = o; else s.bad = 1;
        }
      }
    }
    s.base[k] = mine;
  }
  __syncthreads();
  const int n1 = min(s.n1, kMaxOut);
  block_sort(s.out, n1);
  __shared__ int nfaces;
  if (tid == 0) {
    int sum = 0;
    for (int k = 0; k < nc; ++k) { const int x = s.base[k]; s.base[k] = sum; sum += x; }
    nfaces = sum;
    if (T + n1 >= kNoCell) s.bad = 1;
    if (!WRITE) {
      head[4 * blockIdx.x] = n1;
      head[4 * blockIdx.x + 1] = sum;
      head[4 * blockIdx.x + 2] = head[4 * blockIdx.x + 3] = 0;
      if (s.bad) atomicMax(status, 1);
    }
  }
  if (!WRITE) return;
  __syncthreads();
  if (s.bad || n1 > t.out_cap || nfaces > t.face_cap) return;
  for (int k = tid; k < n1; k += nt) {
    bool was_new;
    s.cval[hash_put(s.ckey, kHashNodes, s.out[k], was_new)] = (uint16_t)(T + k);
    t.out[(long long)blockIdx.x * t.out_cap + k] = s.out[k];
  }
  __syncthreads();
  // local index of local face j of tile cell i
  auto face_of = [&](int i, int j) {
    const int4 nb = ld4(m.cell_nbr + 4 * (long long)i);
    int at = s.base[i - c0];
    for (int q = 0; q < j; ++q) {
      const int o = comp(nb, q);
      if (o < 0 || !inside(o) || o > i) ++at;
    }
    return at;
  };
  for (int k = tid; k < nc; k += nt) {
    const int i = c0 + k;
    const int4 nb = ld4(m.cell_nbr + 4 * (long long)i);
    const uint32_t f = ld(m.cell_flags + i);
    unsigned fl = (f & 7u) | ((unsigned)ld(m.cell_order + i) << 3) | (((f >> 9) & 7u) << 9);
    int face[3], n[3];
    for (int j = 0; j < 3; ++j) {
      const int o = comp(nb, j);
      n[j] = o < 0 ? kNoCell : (inside(o) ? o - c0 : (int)hash_get(s.ckey, s.cval, kHashNodes, o));
      if (o < 0) fl |= kTileRim;
      if (o >= 0 && inside(o) && o < i) {
        const int4 back = ld4(m.cell_nbr + 4 * (long long)o);
        face[j] = face_of(o, back.x == i ? 0 : (back.y == i ? 1 : 2));
      } else {
        face[j] = face_of(i, j);
        // this cell lists the face: its cells (left first) and geometry
        const bool left = (f >> j) & 1u;
        const int g = ld(m.cell_faces + 4 * (long long)i + j);
        const long long at = (long long)blockIdx.x * t.face_cap + face[j];
        reinterpret_cast<uint32_t *>(t.face)[at] =
            (unsigned)(left ? k : n[j]) | ((unsigned)(left ? n[j] : k) << 16);
        t.face_n0[at] = ld(m.face_normal + 3 * (long long)g);
        t.face_n1[at] = ld(m.face_normal + 3 * (long long)g + 1);
        t.face_mes[at] = ld(m.face_mesure + g);
      }
    }
    uint4 u;
    u.x = (unsigned)face[0] | ((unsigned)face[1] << 16);
    u.y = (unsigned)face[2] | ((unsigned)n[0] << 16);
    u.z = (unsigned)n[1] | ((unsigned)n[2] << 16);
    u.w = fl;
    reinterpret_cast<uint4 *>(t.cell)[(long long)blockIdx.x * T + k] = u;
    const int4 vt = ld4(m.cell_vtx + 4 * (long long)i);
    const double2 P1 = ldd2(m.node_coord + 2 * (long long)vt.y), G = ldd2(m.cell_xy + 2 * (long long)i);
    reinterpret_cast<double2 *>(t.cell_ns)[i] = make_double2(__dsub_rn(G.y, P1.y), -__dsub_rn(G.x, P1.x));
  }
}

}  // namespace mb

using namespace mb;

#define ST(s) reinterpret_cast<cudaStream_t>(s)

static int tile_mesh_bad(const mb_mesh *m) {
  return !m || m->dim != 2 || m->nlf != 3 || m->nbcells <= 0 || m->nbnodes <= 0 || !m->cell_vtx || !m->cell_nbr ||
         !m->cell_flags || !m->node_coord || !m->cell_xy || !m->cell_volume || !m->n2c_ptr || !m->n2c_idx ||
         !m->n2c_alpha || !m->n2g_ptr || !m->n2g_idx || !m->ghostnid_ptr || !m->ghostnid_idx || !m->face_ghostcenter;
}

template <bool WRITE>
static int run_plan(const mb_mesh *m, const mb_tiles *t, int32_t *head, int32_t *status, const double *minv,
                    const double *node_w, cudaStream_t st) {
  if (cudaFuncSetAttribute(k_tile_plan<WRITE>, cudaFuncAttributeMaxDynamicSharedMemorySize, sizeof(TileShared)) !=
      cudaSuccess)
    return MB_ECUDA;
  k_tile_plan<WRITE><<<t->count, kTileThreads, sizeof(TileShared), st>>>(*m, *t, head, status, minv, node_w);
  return cudaGetLastError() == cudaSuccess ? MB_OK : MB_ECUDA;
}

extern "C" {

int mb_tile_sizes(const mb_mesh *m, int32_t cells, int32_t *head, int32_t *status, void *stream) {
  MB_NVTX();
  if (tile_mesh_bad(m) || cells < 32 || cells > MB_TILE_MAX_CELLS || !head || !status) return MB_EINVAL;
  mb_tiles t{};
  t.cells = cells;
  t.count = ceil_div(m->nbcells, cells);
  return run_plan<false>(m, &t, head, status, nullptr, nullptr, ST(stream));
}

int mb_tile_fill(const mb_mesh *m, const mb_tiles *t, double *scratch, void *stream) {
  MB_NVTX();
  if (tile_mesh_bad(m) || !m->lsq_sell_ptr || !m->lsq_sell_idx || !scratch || ((uintptr_t)scratch & 31) ||
      !mb::tiles_ok(m, t))
    return MB_EINVAL;
  cudaStream_t st = ST(stream);
  double *minv = scratch, *node_w = scratch + 4 * (long long)m->nbcells;
  k_tile_minv<<<ceil_div(m->nbcells, kBlock), kBlock, 0, st>>>(*m, minv);
  k_tile_node<<<ceil_div(m->nbnodes, kBlock), kBlock, 0, st>>>(*m, node_w, t->node_kappa);
  const int rc = run_plan<true>(m, t, nullptr, nullptr, minv, node_w, st);
  if (rc != MB_OK) return rc;
  tile_filled(st);
  return cudaGetLastError() == cudaSuccess ? MB_OK : MB_ECUDA;
}

int mb_tile_coef(const mb_mesh *m, const mb_bc *bc, const mb_advdiff_params *p, double *coef, void *stream) {
  MB_NVTX();
  if (tile_mesh_bad(m) || !bc || !bc->face_grad_on || !p || !coef ) return MB_EINVAL;
  k_tile_coef<<<ceil_div(m->nbcells, kBlock), kBlock, 0, ST(stream)>>>(*m, *bc, *p, coef);
  return cudaGetLastError() == cudaSuccess ? MB_OK : MB_ECUDA;
}

}  // extern "C"

template <bool WRITE>
static int run_face_plan(const mb_mesh *m, const mb_face_tiles *t, int32_t *head, int32_t *status, cudaStream_t st) {
  k_face_plan<WRITE><<<t->count, kTileThreads, sizeof(FaceTileShared), st>>>(*m, *t, head, status);
  return cudaGetLastError() == cudaSuccess ? MB_OK : MB_ECUDA;
}

static bool face_mesh_bad(const mb_mesh *m) {
  return !m || m->dim != 2 || m->nlf != 3 || m->nbcells <= 0 || !m->cell_vtx || !m->cell_nbr || !m->cell_flags ||
         !m->cell_order || !m->cell_faces || !m->node_coord || !m->cell_xy || !m->face_normal || !m->face_mesure;
}

extern "C" {

int mb_face_tile_sizes(const mb_mesh *m, int32_t cells, int32_t *head, int32_t *status, void *stream) {
  MB_NVTX();
  if (face_mesh_bad(m) || cells < 32 || (cells & 1) || cells > MB_TILE_MAX_CELLS || !head || !status) return MB_EINVAL;
  mb_face_tiles t{};
  t.cells = cells;
  t.count = ceil_div(m->nbcells, cells);
  return run_face_plan<false>(m, &t, head, status, ST(stream));
}

int mb_face_tile_fill(const mb_mesh *m, const mb_face_tiles *t, void *stream) {
  MB_NVTX();
  if (face_mesh_bad(m) || !face_tiles_ok(m, t)) return MB_EINVAL;
  const int rc = run_face_plan<true>(m, t, nullptr, nullptr, ST(stream));
  if (rc != MB_OK) return rc;
  tile_filled(ST(stream));
  return cudaGetLastError() == cudaSuccess ? MB_OK : MB_ECUDA;
}

int mb_tile_wait_check(int32_t limit, int32_t *late, void *stream) {
  MB_NVTX();
  if (limit < 1 || limit > 4096 || !late) return MB_EINVAL;
  k_tile_wait_check<<<1, 32, 0, ST(stream)>>>(late, limit);
  return cudaGetLastError() == cudaSuccess ? MB_OK : MB_ECUDA;
}

}  // extern "C"
