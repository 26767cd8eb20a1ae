// Builds the tiles of a tetrahedral mesh (mb_tet_tiles, fv_tet_tile.cu) on the device: one block per
// tile, two passes (sizes, then the tables at strides the caller chose from the sizes).  Set-up
// work, once per mesh.
#include "fv_tile_plan.cuh"

namespace mb {

constexpr int kTetThreadsPlan = 256;
constexpr int kTetHashCells = 8192, kTetHashEdges = 4096, kTetHashNodes = 1024;
constexpr int kTetMaxOut = 4096, kTetMaxEdges = 2048, kTetMaxNodes = 512;

struct TetShared {
  int ckey[kTetHashCells];
  int ekey[kTetHashEdges];
  int nkey[kTetHashNodes];
  uint16_t cval[kTetHashCells], eval[kTetHashEdges], nval[kTetHashNodes];
  int out[kTetMaxOut], edge[kTetMaxEdges], node[kTetMaxNodes];
  int ngrp[kTetMaxNodes / 32 + 2], egrp[kTetMaxEdges / 32 + 2];
  int nout, ne, nn, bad;
};

// Centre -> vertex weights of a vertex X: alpha_j = (1 + lambda . (c_j - X)) / den over its cells and
// ghosts (manapy/ast/functions3d.py:251-362, weights manapy/ddm/ddm_utils3d.py:813-981), so
// sum alpha_j w_j = rden sum w_j + mu . sum (c_j - X) w_j with mu = lambda / den; kappa: the sum of
// alpha_j over its cells.
struct TetNode {
  D3 mu;
  double rden, kappa;
};
__device__ TetNode tet_node(const mb_mesh &m, int v) {
  const D3 X = ld3(m.node_coord + 4 * (long long)v);
  double ixx = 0., iyy = 0., izz = 0., ixy = 0., ixz = 0., iyz = 0., rx = 0., ry = 0., rz = 0., kappa = 0.;
  auto add = [&](double dx, double dy, double dz) {
    ixx += dx * dx; iyy += dy * dy; izz += dz * dz;
    ixy += dx * dy; ixz += dx * dz; iyz += dy * dz;
    rx += dx; ry += dy; rz += dz;
  };
  const int cb = ld(m.n2c_ptr + v), ce = ld(m.n2c_ptr + v + 1);
  const int gb = ld(m.n2g_ptr + v), ge = ld(m.n2g_ptr + v + 1);
  for (int q = cb; q < ce; ++q) {
    const D3 d = ld3(m.cell_xy + 4 * (long long)ld(m.n2c_idx + q)) - X;
    add(d.x, d.y, d.z);
    kappa += ld(m.n2c_alpha + q);
  }
  for (int q = gb; q < ge; ++q) {
    const double *g = m.face_ghostcenter + 3 * (long long)ld(m.n2g_idx + q);
    add(ld(g) - X.x, ld(g + 1) - X.y, ld(g + 2) - X.z);
  }
  const double D = ixx * iyy * izz + 2 * ixy * ixz * iyz - ixx * iyz * iyz - iyy * ixz * ixz - izz * ixy * ixy;
  const double lx = ((iyz * iyz - iyy * izz) * rx + (ixy * izz - ixz * iyz) * ry + (ixz * iyy - ixy * iyz) * rz) / D;
  const double ly = ((ixy * izz - ixz * iyz) * rx + (ixz * ixz - ixx * izz) * ry + (iyz * ixx - ixz * ixy) * rz) / D;
  const double lz = ((ixz * iyy - ixy * iyz) * rx + (iyz * ixx - ixz * ixy) * ry + (ixy * ixy - ixx * iyy) * rz) / D;
  const double den = (double)(ce - cb + ge - gb) + lx * rx + ly * ry + lz * rz;
  return TetNode{d3(lx / den, ly / den, lz / den), 1.0 / den, kappa};
}

// own bits and the face in the neighbour, of every cell (mb_tet_tiles.link)
__device__ unsigned tet_link(const mb_mesh &m, int i) {
  const int4 nb = ld4(m.cell_nbr + 4 * (long long)i);
  const uint32_t f = ld(m.cell_flags + i);
  unsigned link = 0;
  for (int j = 0; j < 4; ++j) {
    const int o = comp(nb, j);
    link |= ((f >> (6 * j)) & 1u) << j;
    if (o >= 0) {
      const int4 back = ld4(m.cell_nbr + 4 * (long long)o);
      link |= (unsigned)(back.x == i ? 0 : (back.y == i ? 1 : (back.z == i ? 2 : 3))) << (4 + 2 * j);
    }
  }
  return link;
}

template <bool WRITE>
__global__ void __launch_bounds__(kTetThreadsPlan) k_tet_plan(mb_mesh m, mb_tet_tiles t, int32_t *head,
                                                              int32_t *status) {
  extern __shared__ unsigned char raw[];
  TetShared &s = *reinterpret_cast<TetShared *>(raw);
  const int T = t.cells, b = blockIdx.x, c0 = b * T, tid = threadIdx.x, nt = blockDim.x;
  const int nc = min(T, m.nbcells - c0);
  for (int i = tid; i < kTetHashCells; i += nt) s.ckey[i] = -1;
  for (int i = tid; i < kTetHashEdges; i += nt) s.ekey[i] = -1;
  for (int i = tid; i < kTetHashNodes; i += nt) s.nkey[i] = -1;
  if (tid == 0) s.nout = s.ne = s.nn = s.bad = 0;
  __syncthreads();
  // inclusion-exclusion and the search for a face in its neighbour take the neighbours as distinct
  for (int k = tid; k < nc; k += nt) {
    const int4 nb = ld4(m.cell_nbr + 4 * (long long)(c0 + k));
    for (int j = 1; j < 4; ++j)
      for (int q = 0; q < j; ++q)
        if (comp(nb, j) >= 0 && comp(nb, j) == comp(nb, q)) s.bad = 1;
  }
  // the tile's vertices and edges
  for (int k = tid; k < 10 * nc; k += nt) {
    const int i = c0 + k / 10, q = k % 10;
    bool was_new;
    if (q < 4) {
      const int v = ld(m.cell_vtx + 4 * (long long)i + q);
      if (hash_put(s.nkey, kTetHashNodes, v, was_new) < 0) s.bad = 1;
      if (was_new) {
        const int at = atomicAdd(&s.nn, 1);
        if (at < kTetMaxNodes) s.node[at] = v; else s.bad = 1;
      }
    } else {
      const int e = ld(m.cell_edges + 8 * (long long)i + q - 4);
      if (hash_put(s.ekey, kTetHashEdges, e, was_new) < 0) s.bad = 1;
      if (was_new) {
        const int at = atomicAdd(&s.ne, 1);
        if (at < kTetMaxEdges) s.edge[at] = e; else s.bad = 1;
      }
    }
  }
  __syncthreads();
  const int nn = min(s.nn, kTetMaxNodes), ne = min(s.ne, kTetMaxEdges);
  block_sort(s.node, nn);
  block_sort(s.edge, ne);
  // the cells around the vertices (those around the edges are among them)
  for (int k = tid; k < nn; k += nt) {
    const int v = s.node[k];
    for (int q = ld(m.n2c_ptr + v); q < ld(m.n2c_ptr + v + 1); ++q) {
      const int c = ld(m.n2c_idx + q);
      if (c >= c0 && c < c0 + nc) continue;
      bool was_new;
      if (hash_put(s.ckey, kTetHashCells, c, was_new) < 0) s.bad = 1;
      if (was_new) {
        const int at = atomicAdd(&s.nout, 1);
        if (at < kTetMaxOut) s.out[at] = c; else s.bad = 1;
      }
    }
  }
  __syncthreads();
  const int nout = min(s.nout, kTetMaxOut);
  block_sort(s.out, nout);
  const int ng = (nn + 31) >> 5, eg = (ne + 31) >> 5;
  auto edge_cells = [&](int e) {   // cells listed for edge e
    const int sb = ld(m.edge_sell_ptr + (e >> 5)), se = ld(m.edge_sell_ptr + (e >> 5) + 1);
    int n = 0;
    for (int k = sb + (e & 31); k < se; k += 32) n += ld(m.edge_sell_idx + k) >= 0;
    return n;
  };
  for (int g = tid; g < ng + eg; g += nt) {
    const bool edges = g >= ng;
    const int h = edges ? g - ng : g, n = edges ? ne : nn;
    int longest = 0;
    for (int k = 32 * h; k < min(32 * h + 32, n); ++k)
      longest = max(longest, edges ? edge_cells(s.edge[k]) : ld(m.n2c_ptr + s.node[k] + 1) - ld(m.n2c_ptr + s.node[k]));
    (edges ? s.egrp : s.ngrp)[h + 1] = 32 * longest;
  }
  __syncthreads();
  if (tid == 0) {
    s.ngrp[0] = s.egrp[0] = 0;
    for (int g = 0; g < ng; ++g) s.ngrp[g + 1] += s.ngrp[g];
    for (int g = 0; g < eg; ++g) s.egrp[g + 1] += s.egrp[g];
    if (T + nout + 2 >= kNoCell || m.nbnodes >= (1 << 29)) s.bad = 1;
    if (!WRITE) {
      int32_t *h = head + 8 * (long long)b;
      h[0] = nout; h[1] = nn; h[2] = ne; h[3] = s.ngrp[ng]; h[4] = s.egrp[eg]; h[5] = h[6] = h[7] = 0;
      if (s.bad) atomicMax(status, 1);
    }
  }
  if (!WRITE) return;
  __syncthreads();
  if (s.bad || nout > t.ext_cap || nn > t.node_cap || ne > t.edge_cap || s.ngrp[ng] > t.ninc_cap ||
      s.egrp[eg] > t.einc_cap)
    return;
  // coordinates relative to the mean of the cells' centres (every warp forms the same)
  D3 org = {0., 0., 0.};
  for (int k = tid & 31; k < nc; k += 32) org = org + ld3(m.cell_xy + 4 * (long long)(c0 + k));
  for (int o = 16; o > 0; o >>= 1)
    org = org + D3{__shfl_xor_sync(0xffffffffu, org.x, o), __shfl_xor_sync(0xffffffffu, org.y, o),
                   __shfl_xor_sync(0xffffffffu, org.z, o)};
  org = (1. / nc) * org;
  auto put_xyz = [&](double *xy, double *z, long long at, int c) {
    const D3 p = ld3(m.cell_xy + 4 * (long long)c);
    reinterpret_cast<double2 *>(xy)[at] = make_double2(p.x - org.x, p.y - org.y);
    z[at] = p.z - org.z;
  };
  for (int k = tid; k < nc; k += nt) put_xyz(t.own_xy, t.own_z, c0 + k, c0 + k);
  for (int k = tid; k < nout; k += nt) {
    const int c = s.out[k];
    const long long at = (long long)b * t.ext_cap + k;
    bool was_new;
    s.cval[hash_put(s.ckey, kTetHashCells, c, was_new)] = (uint16_t)(T + k);
    t.ext[at] = c;
    put_xyz(t.ext_xy, t.ext_z, at, c);
  }
  for (int k = tid; k < ne; k += nt) {
    bool was_new;
    s.eval[hash_put(s.ekey, kTetHashEdges, s.edge[k], was_new)] = (uint16_t)k;
  }
  for (int k = tid; k < nn; k += nt) {
    const int v = s.node[k];
    bool was_new;
    s.nval[hash_put(s.nkey, kTetHashNodes, v, was_new)] = (uint16_t)k;
    const int first = ld(m.n2c_idx + ld(m.n2c_ptr + v));
    const bool own = first >= c0 && first < c0 + nc;   // one tile writes a vertex's value
    const bool ghosts = ld(m.n2g_ptr + v + 1) > ld(m.n2g_ptr + v);
    t.node[(long long)b * t.node_cap + k] = v | (own ? kTetOwned : 0) | (ghosts ? kTetGhosts : 0);
    if (own) {
      // a = 1 / den - mu . X: the sums are relative to the tile's origin
      const TetNode u = tet_node(m, v);
      const D3 X = ld3(m.node_coord + 4 * (long long)v) - org;
      st4d_plain(t.node_mu + 4 * (long long)v, u.mu.x, u.mu.y, u.mu.z, u.rden - dot(u.mu, X));
      t.node_kappa[v] = ghosts ? u.kappa : 1.0;
    }
  }
  __syncthreads();
  auto local = [&](int c) -> int {
    return c >= c0 && c < c0 + nc ? c - c0 : (int)hash_get(s.ckey, s.cval, kTetHashCells, c);
  };
  for (int g = tid; g <= ng; g += nt) t.ngrp[(long long)b * t.ngrp_cap + g] = s.ngrp[g];
  for (int g = tid; g <= eg; g += nt) t.egrp[(long long)b * t.egrp_cap + g] = s.egrp[g];
  uint16_t *ninc = t.ninc + (long long)b * t.ninc_cap, *einc = t.einc + (long long)b * t.einc_cap;
  // past the end of a list: the slot of a zero value at T + ext_cap
  for (int k = tid; k < 32 * ng; k += nt) {
    const int len = (s.ngrp[(k >> 5) + 1] - s.ngrp[k >> 5]) >> 5, v = k < nn ? s.node[k] : -1;
    const int q0 = v < 0 ? 0 : ld(m.n2c_ptr + v), q1 = v < 0 ? 0 : ld(m.n2c_ptr + v + 1);
    for (int q = 0; q < len; ++q)
      ninc[s.ngrp[k >> 5] + 32 * q + (k & 31)] = q0 + q < q1 ? (uint16_t)local(ld(m.n2c_idx + q0 + q)) : (uint16_t)(T + t.ext_cap);
  }
  for (int k = tid; k < 32 * eg; k += nt) {
    const int len = (s.egrp[(k >> 5) + 1] - s.egrp[k >> 5]) >> 5, e = k < ne ? s.edge[k] : -1;
    int q = 0;
    if (e >= 0) {
      const int sb = ld(m.edge_sell_ptr + (e >> 5)), se = ld(m.edge_sell_ptr + (e >> 5) + 1);
      for (int p = sb + (e & 31); p < se; p += 32) {
        const int c = ld(m.edge_sell_idx + p);
        if (c >= 0) einc[s.egrp[k >> 5] + 32 * q++ + (k & 31)] = (uint16_t)local(c);
      }
    }
    for (; q < len; ++q) einc[s.egrp[k >> 5] + 32 * q + (k & 31)] = (uint16_t)(T + t.ext_cap);
  }
  for (int k = tid; k < nc; k += nt) {
    const int i = c0 + k;
    const int4 vt = ld4(m.cell_vtx + 4 * (long long)i), nb = ld4(m.cell_nbr + 4 * (long long)i);
    uint16_t r[16];
    for (int j = 0; j < 4; ++j) {
      r[j] = (uint16_t)hash_get(s.nkey, s.nval, kTetHashNodes, comp(vt, j));
      const int o = comp(nb, j);
      r[10 + j] = o < 0 ? kNoCell : (uint16_t)local(o);
    }
    for (int j = 0; j < 6; ++j) r[4 + j] = (uint16_t)hash_get(s.ekey, s.eval, kTetHashEdges, ld(m.cell_edges + 8 * (long long)i + j));
    r[14] = ld(m.ghostnid_ptr + i + 1) > ld(m.ghostnid_ptr + i) ? 1 : 0;
    r[15] = 0;
    for (int j = 0; j < 16; ++j) t.cell[16 * (long long)i + j] = r[j];
    t.link[i] = (uint16_t)tet_link(m, i);
  }
}

// planes of a cell's reconstruction: (de_0, de_1, de_2) = Q J, rows Q_k = (face centre k - centre)^T
// times the inverse moment matrix (cell_lsq: cofactors, determinant, and D, the sum of the
// stencil's centre offsets): Q (9 planes), D (3)
__global__ void __launch_bounds__(kBlock) k_tet_q(mb_mesh m, double *__restrict__ out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= m.nbcells) return;
  const int4 vt = ld4(m.cell_vtx + 4 * (long long)i);
  const D3 P[4] = {ld3(m.node_coord + 4 * (long long)vt.x), ld3(m.node_coord + 4 * (long long)vt.y),
                   ld3(m.node_coord + 4 * (long long)vt.z), ld3(m.node_coord + 4 * (long long)vt.w)};
  double a0, a1, a2, a3, a4, a5, dia, pad, Dx, Dy, Dz;
  ld4d(m.cell_lsq + 12 * (long long)i, a0, a1, a2, a3);
  ld4d(m.cell_lsq + 12 * (long long)i + 4, a4, a5, dia, pad);
  ld4d(m.cell_lsq + 12 * (long long)i + 8, Dx, Dy, Dz, pad);
  const long long n = m.nbcells;
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    // face centre - centre: a twelfth of the differences to the opposite vertex o, which round to the
    // size of the cell, not to that of its coordinates as a difference of two centres does
    const int o = j == 0 ? 3 : (j == 1 ? 1 : 2);
    const D3 f = (1. / 12) * (((P[0] - P[o]) + (P[1] - P[o])) + ((P[2] - P[o]) + (P[3] - P[o])));
    const double qx = (f.x * a0 + f.y * a1 + f.z * a2) / dia, qy = (f.x * a1 + f.y * a3 + f.z * a4) / dia,
                 qz = (f.x * a2 + f.y * a4 + f.z * a5) / dia;
    out[(3 * j) * n + i] = qx;
    out[(3 * j + 1) * n + i] = qy;
    out[(3 * j + 2) * n + i] = qz;
  }
  out[9 * n + i] = Dx;
  out[10 * n + i] = Dy;
  out[11 * n + i] = Dz;
}

__global__ void __launch_bounds__(kBlock) k_tet_tables(mb_mesh m, mb_tet_tables t) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k < m.nbcells) {
    t.link[k] = (uint16_t)tet_link(m, k);
    // the link's search for a face in its neighbour takes the neighbours as distinct
    const int4 nb = ld4(m.cell_nbr + 4 * (long long)k);
    for (int j = 1; j < 4; ++j)
      for (int q = 0; q < j; ++q)
        if (comp(nb, j) >= 0 && comp(nb, j) == comp(nb, q)) atomicMax(t.status, 1);
  }
  if (k < m.nbnodes) {
    const TetNode u = tet_node(m, k);
    st4d_plain(t.node_mu + 4 * (long long)k, u.mu.x, u.mu.y, u.mu.z, u.rden);
  }
}

// the diamond diffusion of a tetrahedron as a linear form, planes c_1, c_2, c_3 (vertex differences
// V_k - V_0), B_0..B_3 (value differences across the faces), 1 / V: diamond3's
// [(V_A - V_C) (Q3 - Q2).t / 2 + (V_B - V_C) (Q1 - Q3).t / 2 + (V_R - V_L) N.DN] / (N . (v2 - v1))
__global__ void __launch_bounds__(kBlock) k_tet_coef(mb_mesh m, mb_bc bc, mb_advdiff_params p,
                                                     double *__restrict__ out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= m.nbcells) return;
  const int4 vt = ld4(m.cell_vtx + 4 * (long long)i), nb = ld4(m.cell_nbr + 4 * (long long)i);
  const uint32_t fl = ld(m.cell_flags + i);
  const D3 ci = ld3(m.cell_xy + 4 * (long long)i);
  double cv[4] = {0., 0., 0., 0.}, B[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int o = comp(nb, j), f = -1 - o;
    B[j] = 0.;
    if (o < 0 && !ld(bc.face_grad_on + f)) continue;
    const bool own = (fl >> (6 * j)) & 1u;
    int d0, d1, d2;
    face_desc(fl, j, d0, d1, d2);
    const D3 V0 = ld3(m.node_coord + 4 * (long long)comp(vt, d0)), V1 = ld3(m.node_coord + 4 * (long long)comp(vt, d1)),
             V2 = ld3(m.node_coord + 4 * (long long)comp(vt, d2));
    const double *gc = m.face_ghostcenter + 3 * (long long)(o < 0 ? f : 0);
    const D3 co = o < 0 ? d3(ld(gc), ld(gc + 1), ld(gc + 2)) : ld3(m.cell_xy + 4 * (long long)o);
    const D3 Nd = 0.5 * cross(V1 - V0, V2 - V0);
    const D3 N = ((fl >> (6 * j + 5)) & 1u) ? (-1.0) * Nd : Nd;
    const bool swp = (fl >> (6 * j + 4)) & 1u;
    const D3 Q2 = swp ? V2 : V1, Q3 = swp ? V1 : V2;
    const int l2 = swp ? d2 : d1, l3 = swp ? d1 : d2;
    const D3 v1 = own ? ci : co, v2 = own ? co : ci;
    const D3 DN = d3(p.Dxx * N.x, p.Dyy * N.y, p.Dzz * N.z);
    const D3 t = cross(v1 - v2, DN);
    const double r = 1 / dot(N, v2 - v1);
    double fa = 0.5 * dot(Q3 - Q2, t) * r, fb = 0.5 * dot(V0 - Q3, t) * r;
    B[j] = dot(N, DN) * r;      // times V_R - V_L, and the flux enters the cell with the same sign
    if (!own) { fa = -fa; fb = -fb; }
#pragma unroll
    for (int v = 0; v < 4; ++v) cv[v] += (v == d0 ? fa : 0.) + (v == l2 ? fb : 0.) - (v == l3 ? fa + fb : 0.);
  }
  const long long n = m.nbcells;
#pragma unroll
  for (int v = 0; v < 3; ++v) out[v * n + i] = cv[v + 1];
#pragma unroll
  for (int j = 0; j < 4; ++j) out[(3 + j) * n + i] = B[j];
  out[7 * n + i] = 1 / ld(m.cell_volume + i);
}

}  // namespace mb

using namespace mb;

#define ST(s) reinterpret_cast<cudaStream_t>(s)

static bool tet_mesh_bad(const mb_mesh *m) {
  return !m || m->dim != 3 || m->nlf != 4 || m->nbcells <= 0 || m->nbnodes <= 0 || !m->cell_vtx || !m->cell_nbr ||
         !m->cell_flags || !m->node_coord || !m->cell_xy || !m->cell_volume || !m->n2c_ptr || !m->n2c_idx ||
         !m->n2c_alpha || !m->n2g_ptr || !m->n2g_idx || !m->ghostnid_ptr || !m->ghostnid_idx ||
         !m->face_ghostcenter || !m->cell_edges || !m->edge_sell_ptr || !m->edge_sell_idx || !m->cell_lsq ||
         ((uintptr_t)m->cell_xy & 31) || ((uintptr_t)m->node_coord & 31) || ((uintptr_t)m->cell_lsq & 31);
}

template <bool WRITE>
static int run_tet_plan(const mb_mesh *m, const mb_tet_tiles *t, int32_t *head, int32_t *status, cudaStream_t st) {
  if (cudaFuncSetAttribute(k_tet_plan<WRITE>, cudaFuncAttributeMaxDynamicSharedMemorySize, sizeof(TetShared)) !=
      cudaSuccess)
    return MB_ECUDA;
  k_tet_plan<WRITE><<<t->count, kTetThreadsPlan, sizeof(TetShared), st>>>(*m, *t, head, status);
  return cudaGetLastError() == cudaSuccess ? MB_OK : MB_ECUDA;
}

extern "C" {

int mb_tet_tile_sizes(const mb_mesh *m, int32_t cells, int32_t *head, int32_t *status, void *stream) {
  MB_NVTX();
  if (tet_mesh_bad(m) || cells < 32 || (cells & 1) || cells > MB_TET_TILE_MAX_CELLS || !head || !status)
    return MB_EINVAL;
  mb_tet_tiles t{};
  t.cells = cells;
  t.count = ceil_div(m->nbcells, cells);
  return run_tet_plan<false>(m, &t, head, status, ST(stream));
}

int mb_tet_tile_fill(const mb_mesh *m, const mb_tet_tiles *t, void *stream) {
  MB_NVTX();
  if (tet_mesh_bad(m) || !tet_tiles_ok(m, t)) return MB_EINVAL;
  cudaStream_t st = ST(stream);
  k_tet_q<<<ceil_div(m->nbcells, kBlock), kBlock, 0, st>>>(*m, t->cell_q);
  const int rc = run_tet_plan<true>(m, t, nullptr, nullptr, st);
  if (rc != MB_OK) return rc;
  tile_filled(st);
  return cudaGetLastError() == cudaSuccess ? MB_OK : MB_ECUDA;
}

int mb_tet_tables_fill(const mb_mesh *m, const mb_tet_tables *t, void *stream) {
  MB_NVTX();
  if (tet_mesh_bad(m) || !t || !t->cell_q || !t->link || !t->node_mu || !t->status || ((uintptr_t)t->node_mu & 31))
    return MB_EINVAL;
  cudaStream_t st = ST(stream);
  k_tet_q<<<ceil_div(m->nbcells, kBlock), kBlock, 0, st>>>(*m, t->cell_q);
  const int n = m->nbcells > m->nbnodes ? m->nbcells : m->nbnodes;
  k_tet_tables<<<ceil_div(n, kBlock), kBlock, 0, st>>>(*m, *t);
  tile_filled(st);
  return cudaGetLastError() == cudaSuccess ? MB_OK : MB_ECUDA;
}

int mb_tet_coef(const mb_mesh *m, const mb_bc *bc, const mb_advdiff_params *p, double *coef, void *stream) {
  MB_NVTX();
  if (tet_mesh_bad(m) || !bc || !bc->face_grad_on || !p || !coef) return MB_EINVAL;
  k_tet_coef<<<ceil_div(m->nbcells, kBlock), kBlock, 0, ST(stream)>>>(*m, *bc, *p, coef);
  return cudaGetLastError() == cudaSuccess ? MB_OK : MB_ECUDA;
}

}  // extern "C"
