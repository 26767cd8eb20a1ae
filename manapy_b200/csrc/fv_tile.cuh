// Tiles of a triangle mesh: contiguous ranges of cells (device numbering, a Morton curve)
// that one thread block carries through a whole step in shared memory, with the cells
// around them.
//
// Tile k holds the cells [k T, (k + 1) T).  Its local cells are those (local index = offset
// in the range), then at T + e the outside cells ext[e]: first the n1 cells across a face of
// the tile, then every other cell that shares a vertex with one of these T + n1 cells.  Its
// local nodes are the vertices of the T + n1 cells.  All local indices fit 16 bits.
#pragma once

#include <atomic>

#include "fv_compact.cuh"

namespace mb {

#ifndef MB_TILE_THREADS
#define MB_TILE_THREADS 384
#endif
constexpr int kTileThreads = MB_TILE_THREADS;
constexpr uint16_t kNoCell = 0xffffu;
constexpr unsigned kNodeGhosts = 0x8000u;   // in a node's cell count: the node has boundary faces

// flags word of a local cell record {v0, v1, v2, n0, n1, n2, flags, 0}
__device__ __forceinline__ bool tile_own(unsigned fl, int j) { return (fl >> j) & 1u; }
__device__ __forceinline__ int tile_peer(unsigned fl, int j) { return (fl >> (3 + 2 * j)) & 3u; }  // the face in the neighbour
constexpr unsigned kTileGhosts = 1u << 9;   // boundary faces at a vertex of the cell

// asynchronous copies global -> shared: no register holds the data, so a thread keeps as many in
// flight as it issues before tile_copies_done()
__device__ __forceinline__ void tile_copy8(void *dst, const void *src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}
// bulk copies global -> shared (addresses and sizes multiples of 16), counted by an mbarrier: one
// thread issues them and they pass the load/store pipe by
__device__ __forceinline__ void tile_bar_init(uint64_t *bar) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"((unsigned)__cvta_generic_to_shared(bar)) : "memory");
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void tile_bar_expect(uint64_t *bar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(
                   (unsigned)__cvta_generic_to_shared(bar)),
               "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void tile_bulk(void *dst, const void *src, unsigned bytes, uint64_t *bar) {
  if (bytes)
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     (unsigned)__cvta_generic_to_shared(dst)),
                 "l"(src), "r"(bytes), "r"((unsigned)__cvta_generic_to_shared(bar))
                 : "memory");
}
// waits for phase 0 of the barrier; false when the copies have not arrived after `limit` tries
constexpr int kTileWait = 1 << 22;
__device__ __forceinline__ bool tile_bar_wait(uint64_t *bar, int limit) {
  const unsigned a = (unsigned)__cvta_generic_to_shared(bar);
  for (int k = 0; k < limit; ++k) {
    unsigned ok;
    asm volatile("{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], 0;\nselp.u32 %0, 1, 0, p;\n}"
                 : "=r"(ok)
                 : "r"(a)
                 : "memory");
    if (ok) return true;
  }
  return false;
}
// The wait of a step for the copies of its tile.  When it runs out the block reports in *late, waits once
// more for what is still in flight towards its shared memory, and has to return with its cells
// unwritten: the state is then not a step's, which the host sees in *late.
__device__ __forceinline__ bool tile_arrived(uint64_t *bar, int32_t *late, int limit = kTileWait) {
  if (tile_bar_wait(bar, limit)) return true;
  // no fence: the host reads the word after the launch has ended (a fence here, though never run, cost
  // the shallow-water step 1.9 %: 80.6 -> 82.1 us at 1.28M triangles)
  if (late) asm volatile("st.relaxed.sys.global.s32 [%0], 1;" ::"l"(late) : "memory");
  tile_bar_wait(bar, limit);
  return false;
}
__device__ __forceinline__ void tile_copies_done() { asm volatile("cp.async.wait_all;" ::: "memory"); }
// asks for [p, p + bytes) in L2, but for a ragged end of less than 16 bytes on either side
__device__ __forceinline__ void tile_prefetch(const void *p, unsigned bytes) {
  const uint64_t a = ((uint64_t)p + 15) & ~15ull, e = ((uint64_t)p + bytes) & ~15ull;
  if (e > a) asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(a), "r"((unsigned)(e - a)) : "memory");
}

// the tables of t are there, aligned and with strides a step can use
inline bool tiles_ok(const mb_mesh *m, const mb_tiles *t) {
  if (!t || t->cells < 32 || (t->cells & 1) || t->cells > MB_TILE_MAX_CELLS ||
      t->count != ceil_div(m->nbcells, t->cells) || t->face_cap < 0 || t->ext_cap < t->face_cap || t->node_cap < 1 ||
      (t->node_cap & 7) || (t->grp_cap & 3) || t->grp_cap < ceil_div(t->node_cap, 32) + 1 || t->inc_cap < 32 ||
      (t->inc_cap & 31))
    return false;
  const void *p[] = {t->head, t->ext, t->ext_xy, t->node, t->count16, t->node_c, t->node_mu, t->cell, t->cell_q0,
                     t->cell_q1, t->grp, t->inc, t->node_kappa};
  for (const void *q : p)
    if (!q || ((uintptr_t)q & 15)) return false;
  return true;
}

inline bool face_tiles_ok(const mb_mesh *m, const mb_face_tiles *t) {
  if (!t || t->cells < 32 || (t->cells & 1) || t->cells > MB_TILE_MAX_CELLS ||
      t->count != ceil_div(m->nbcells, t->cells) || t->out_cap < 0 || t->face_cap < 4 || (t->face_cap & 3))
    return false;
  const void *p[] = {t->head, t->out, t->face, t->face_n0, t->face_n1, t->face_mes, t->cell, t->cell_ns};
  for (const void *q : p)
    if (!q || ((uintptr_t)q & 15)) return false;
  return true;
}

inline bool tet_tiles_ok(const mb_mesh *m, const mb_tet_tiles *t) {
  if (!t || t->cells < 32 || (t->cells & 1) || t->cells > MB_TET_TILE_MAX_CELLS ||
      t->count != ceil_div(m->nbcells, t->cells) || t->ext_cap < 0 || (t->ext_cap & 1) || t->node_cap < 1 ||
      t->edge_cap < 1 || (t->ngrp_cap & 3) || (t->egrp_cap & 3) || t->ngrp_cap < ceil_div(t->node_cap, 32) + 1 ||
      t->egrp_cap < ceil_div(t->edge_cap, 32) + 1 || t->ninc_cap < 32 || (t->ninc_cap & 31) || t->einc_cap < 32 ||
      (t->einc_cap & 31))
    return false;
  const void *p[] = {t->head, t->ext, t->ext_xy, t->ext_z, t->own_xy, t->own_z, t->node, t->node_mu, t->node_kappa,
                     t->ngrp, t->ninc, t->egrp, t->einc, t->cell, t->cell_q, t->link};
  for (const void *q : p)
    if (!q || ((uintptr_t)q & 31)) return false;
  return true;
}
// a tetrahedral tile's node entry: the vertex, and
constexpr int kTetOwned = 1 << 30;    // this tile writes its value
constexpr int kTetGhosts = 1 << 29;   // it has boundary faces

// programmatic dependent launch: a step's blocks may start while the previous step's last ones
// run; before tile_after_previous() they touch only tables that no step writes
__device__ __forceinline__ void tile_let_next_start() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void tile_after_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// Loads of what an earlier launch wrote.  The read-only path (ld, const __restrict__) may be moved
// above tile_after_previous() by the compiler, since it promises that nothing writes the data
// while the kernel runs; these are not.
__device__ __forceinline__ double ld_after(const double *p) {
  double v;
  asm volatile("ld.global.f64 %0, [%1];" : "=d"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void ld4_after(const double *p, double &a, double &b, double &c, double &d) {
  asm volatile("ld.global.v4.f64 {%0, %1, %2, %3}, [%4];" : "=d"(a), "=d"(b), "=d"(c), "=d"(d) : "l"(p) : "memory");
}
// GhostRule with the state loaded so
struct GhostAfter {
  GhostRule g;
  __device__ __forceinline__ double operator()(int f) const {
    const int k = g.kind[f];
    if (k == MB_G_DIRICHLET) return ld(g.value + f);
    const double wc = ld_after(g.w + ld(g.face_cellid + 2 * (long long)f));
    if (k == MB_G_NEUMANN) return wc;
    if (k == MB_G_NONSLIP) return -1 * wc;
    if (k == MB_G_NEUMANN_NH) return wc + ld(g.value + f) * ld(g.dist + f);
    if (k == MB_G_CELL_AT_FACE) return ld_after(g.w + (long long)ld(g.value + f));
    return 0.0;
  }
};

// Ghost values of the boundary faces idx[q .. min(q + 4, e)): the four chains index -> rule, cell -> value
// run side by side (one after the other, the lists of boundary vertices and cells were the longest
// chain of a small mesh's step).  f < 0 and v = 0 past the end.
__device__ __forceinline__ void ghost4(const GhostRule &g, const int32_t *idx, int q, int e, int f[4], double v[4]) {
  int k[4], c[4];
#pragma unroll
  for (int u = 0; u < 4; ++u) f[u] = q + u < e ? ld(idx + q + u) : -1;
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    const long long at = f[u] < 0 ? 0 : f[u];
    k[u] = f[u] < 0 ? MB_G_NONE : (int)g.kind[at];
    v[u] = ld(g.value + at);
    c[u] = ld(g.face_cellid + 2 * at);
  }
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    const int k_ = k[u];
    const double val = v[u];
    double wc = 0.;
    if (k_ != MB_G_NONE && k_ != MB_G_DIRICHLET) wc = ld_after(g.w + (k_ == MB_G_CELL_AT_FACE ? (long long)val : c[u]));
    v[u] = k_ == MB_G_DIRICHLET ? val : (k_ == MB_G_NONSLIP ? -1 * wc : wc);
    if (k_ == MB_G_NEUMANN_NH) v[u] = wc + val * ld(g.dist + f[u]);
  }
}

// Lets kernel K take all the shared memory that a block of the device may have.  The limit belongs to the
// kernel, which every solver in the process launches with the bytes of its own tiles, from any
// thread: it is set to that one value, before the first launch on a device, and never lowered.
template <auto K>
inline cudaError_t tile_shared_limit() {
  static std::atomic<uint64_t> done{0};          // devices, a bit each; beyond 64 it is set every time
  int dev = 0, most = 0;
  cudaError_t e = cudaGetDevice(&dev);
  const uint64_t bit = dev < 64 ? 1ull << dev : 0;
  if (e != cudaSuccess || (done.load(std::memory_order_acquire) & bit)) return e;
  cudaFuncAttributes fa;
  if ((e = cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev)) != cudaSuccess) return e;
  if ((e = cudaFuncGetAttributes(&fa, K)) != cudaSuccess) return e;
  e = cudaFuncSetAttribute(K, cudaFuncAttributeMaxDynamicSharedMemorySize, most - (int)fa.sharedSizeBytes);
  if (e == cudaSuccess) done.fetch_or(bit, std::memory_order_release);
  return e;
}

// Barth limiter of a cell (manapy/ast/functions2d.py:280-325, functions3d.py:364-408): the smallest of 1 and of
// room / |de_j| over the faces whose offset de_j is `least` or more, room = up where the offset is
// positive, else dn.  Found by multiplying across, so that one division is left.  Those products could
// overflow where an offset is above 2^510 (3e153): there every quotient is formed.  The offsets sum
// to zero, so the others bound the last one.  (2M triangles 109.9 us a step without the branch, 109.7
// with it; 110.5-110.7 with the branch around both ways of finding it.)
template <int N>
__device__ __forceinline__ double tile_barth(const double (&de)[N], double up, double dn, double least) {
  double num = 1., den = 1.;
#pragma unroll
  for (int j = 0; j < N; ++j) {
    const double ad = fabs(de[j]), room = de[j] > 0. ? up : dn;
    if (ad >= least && room * den < num * ad) { num = room; den = ad; }
  }
  double most = fabs(de[0]);
#pragma unroll
  for (int j = 1; j + 1 < N; ++j) most += fabs(de[j]);
  double ps = num / den;
  if (__double2hiint(most) >= 0x5fd00000) {
    ps = 1.;
#pragma unroll
    for (int j = 0; j < N; ++j) {
      const double ad = fabs(de[j]), r = (de[j] > 0. ? up : dn) / ad;
      if (ad >= least && r < ps) ps = r;
    }
  }
  return ps;
}

template <class... P, class... A>
inline cudaError_t tile_launch_ex(const cudaLaunchConfig_t &cfg, void (*k)(P...), A... args) {
  return cudaLaunchKernelEx(&cfg, k, P(args)...);
}
// a refusal is reported by the call that met it, not again by the next one that asks for the last error
inline cudaError_t tile_done(cudaError_t e) {
  if (e != cudaSuccess) cudaGetLastError();
  return e;
}
template <auto K, class... A>
inline cudaError_t tile_launch(int blocks, int threads, int bytes, cudaStream_t st, A... args) {
  if (bytes > 48 * 1024) {                       // what every kernel may take
    const cudaError_t e = tile_done(tile_shared_limit<K>());
    if (e != cudaSuccess) return e;
  }
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(blocks);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = bytes;
  cfg.stream = st;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return tile_done(tile_launch_ex(cfg, K, args...));
}

// flags of a cell record of the tiles with faces: bit j left cell of face j, bits 3-8 manapy's order of
// the faces (cell_order), bit 9+j cells.nf is minus the face normal, and
constexpr unsigned kTileRim = 1u << 12;     // the cell has a boundary face

struct TileCell {
  int v[3], n[3];
  unsigned fl;
};
__device__ __forceinline__ TileCell tile_cell(const uint4 &u) {
  TileCell c;
  c.v[0] = u.x & 0xffffu; c.v[1] = u.x >> 16; c.v[2] = u.y & 0xffffu;
  c.n[0] = u.y >> 16; c.n[1] = u.z & 0xffffu; c.n[2] = u.z >> 16;
  c.fl = u.w & 0xffffu;
  return c;
}

}  // namespace mb
