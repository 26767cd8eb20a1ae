// Tiles of a triangle mesh: contiguous ranges of cells (device numbering, a Morton curve)
// that one thread block carries through a whole step in shared memory, with the cells
// around them.
//
// Tile k holds the cells [k T, (k + 1) T).  Its local cells are those (local index = offset
// in the range), then at T + e the outside cells ext[e]: first the n1 cells across a face of
// the tile, then every other cell that shares a vertex with one of these T + n1 cells.  Its
// local nodes are the vertices of the T + n1 cells.  All local indices fit 16 bits.
#pragma once

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
__device__ __forceinline__ bool tile_bar_wait(uint64_t *bar, int limit = 1 << 22) {
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

// programmatic dependent launch: a step's blocks may start while the previous step's last ones
// run; before tile_after_previous() they touch only tables that no step writes
__device__ __forceinline__ void tile_let_next_start() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void tile_after_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

template <class... P, class... A>
inline cudaError_t tile_launch(void (*k)(P...), int blocks, int threads, int bytes, cudaStream_t st, A... args) {
  if (bytes > 48 * 1024) {
    const cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
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
  return cudaLaunchKernelEx(&cfg, k, P(args)...);
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
