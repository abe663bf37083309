// ha_ptx.cuh -- the device core's loads, stores and atomics in explicit PTX.
//
// ha_core.cuh reaches the memory that warps share only through these functions
// and cuda::atomic_ref, so a host build of the core (tests/hostcore) replaces
// this file by one whose every access is a point where another warp may run.
#ifndef HA_PTX_CUH_
#define HA_PTX_CUH_

#include <stdint.h>

#include "ha_types.h"

namespace ha {

// ---------------------------------------------------------------------------
// PTX helpers: explicit scope and ordering
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint32_t lane_id() {
  uint32_t l;
  asm("mov.u32 %0, %%laneid;" : "=r"(l));
  return l;
}
__device__ __forceinline__ uint32_t lanemask_lt() {
  uint32_t m;
  asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
  return m;
}
// Whether this lane is the first of group `grp` it belongs to (three times
// quicker than comparing its id with the group's lowest set bit).
__device__ __forceinline__ bool first_of(uint32_t grp) { return (grp & lanemask_lt()) == 0; }
__device__ __forceinline__ uint32_t sm_id() {
  uint32_t v;
  asm("mov.u32 %0, %%smid;" : "=r"(v));
  return v;
}
__device__ __forceinline__ uint64_t globaltimer_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
__device__ __forceinline__ uint32_t ld_relaxed(const uint32_t *p) {
  uint32_t v;
  asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p));
  return v;
}
// may return a value that this SM read earlier in the same launch
__device__ __forceinline__ uint32_t ld_cached(const uint32_t *p) {
  uint32_t v;
  asm volatile("ld.global.ca.u32 %0, [%1];" : "=r"(v) : "l"(p));
  return v;
}
__device__ __forceinline__ void st_relaxed(uint32_t *p, uint32_t v) {
  asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ void st_release(uint32_t *p, uint32_t v) {
  asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ uint32_t atom_add(uint32_t *p, uint32_t v) {
  uint32_t o;
  asm volatile("atom.relaxed.gpu.global.add.u32 %0, [%1], %2;"
               : "=r"(o) : "l"(p), "r"(v));
  return o;
}
__device__ __forceinline__ uint32_t atom_or(uint32_t *p, uint32_t v) {
  uint32_t o;
  asm volatile("atom.relaxed.gpu.global.or.b32 %0, [%1], %2;"
               : "=r"(o) : "l"(p), "r"(v));
  return o;
}
__device__ __forceinline__ uint32_t atom_and(uint32_t *p, uint32_t v) {
  uint32_t o;
  asm volatile("atom.relaxed.gpu.global.and.b32 %0, [%1], %2;"
               : "=r"(o) : "l"(p), "r"(v));
  return o;
}
__device__ __forceinline__ void red_add(uint32_t *p, uint32_t v) {
  asm volatile("red.relaxed.gpu.global.add.u32 [%0], %1;" ::"l"(p), "r"(v));
}
__device__ __forceinline__ void red_add_release(uint32_t *p, uint32_t v) {
  asm volatile("red.release.gpu.global.add.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ void red_or(uint32_t *p, uint32_t v) {
  asm volatile("red.relaxed.gpu.global.or.b32 [%0], %1;" ::"l"(p), "r"(v));
}
__device__ __forceinline__ void red_and(uint32_t *p, uint32_t v) {
  asm volatile("red.relaxed.gpu.global.and.b32 [%0], %1;" ::"l"(p), "r"(v));
}
__device__ __forceinline__ uint32_t atom_cas(uint32_t *p, uint32_t expect, uint32_t v) {
  uint32_t o;
  asm volatile("atom.acq_rel.gpu.global.cas.b32 %0, [%1], %2, %3;"
               : "=r"(o) : "l"(p), "r"(expect), "r"(v) : "memory");
  return o;
}
__device__ __forceinline__ uint32_t atom_exch(uint32_t *p, uint32_t v) {
  uint32_t o;
  asm volatile("atom.acq_rel.gpu.global.exch.b32 %0, [%1], %2;"
               : "=r"(o) : "l"(p), "r"(v) : "memory");
  return o;
}
__device__ __forceinline__ uint32_t atom_exch_acquire(uint32_t *p, uint32_t v) {
  uint32_t o;
  asm volatile("atom.acquire.gpu.global.exch.b32 %0, [%1], %2;"
               : "=r"(o) : "l"(p), "r"(v) : "memory");
  return o;
}
__device__ __forceinline__ void fence_acq_rel() {
  asm volatile("fence.acq_rel.gpu;" ::: "memory");
}
__device__ __forceinline__ void fence_sc() { asm volatile("fence.sc.gpu;" ::: "memory"); }

// Slab metadata accesses (bit arrays, size nibbles, slab counters) carry an
// L2 evict-last cache policy, so that the metadata of the slabs in use stays
// in L2 while payload streams through it -- for every kernel that calls
// hamalloc / hafree, not only those launched on a stream with an access-
// policy window (ha_l2_persist_c).  Build with -DHA_L2_HINTS=0 for plain
// accesses.  (halloc's analogue: cudaFuncCachePreferL1 and ld.global.ca
// metadata loads, src/halloc.cu:279, src/utils.h:141-157.)
#ifndef HA_L2_HINTS
#define HA_L2_HINTS 1
#endif
#if HA_L2_HINTS
__device__ __forceinline__ uint64_t meta_policy() {
  uint64_t p;
  asm("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(p));
  return p;
}
__device__ __forceinline__ uint32_t ld_meta(const uint32_t *p) {
  uint32_t v;
  asm volatile("ld.relaxed.gpu.global.L2::cache_hint.u32 %0, [%1], %2;"
               : "=r"(v) : "l"(p), "l"(meta_policy()));
  return v;
}
__device__ __forceinline__ uint32_t atom_add_meta(uint32_t *p, uint32_t v) {
  uint32_t o;
  asm volatile("atom.relaxed.gpu.global.add.L2::cache_hint.u32 %0, [%1], %2, %3;"
               : "=r"(o) : "l"(p), "r"(v), "l"(meta_policy()));
  return o;
}
__device__ __forceinline__ uint32_t atom_or_meta(uint32_t *p, uint32_t v) {
  uint32_t o;
  asm volatile("atom.relaxed.gpu.global.or.L2::cache_hint.b32 %0, [%1], %2, %3;"
               : "=r"(o) : "l"(p), "r"(v), "l"(meta_policy()));
  return o;
}
__device__ __forceinline__ uint32_t atom_and_meta(uint32_t *p, uint32_t v) {
  uint32_t o;
  asm volatile("atom.relaxed.gpu.global.and.L2::cache_hint.b32 %0, [%1], %2, %3;"
               : "=r"(o) : "l"(p), "r"(v), "l"(meta_policy()));
  return o;
}
__device__ __forceinline__ void red_or_meta(uint32_t *p, uint32_t v) {
  asm volatile("red.relaxed.gpu.global.or.L2::cache_hint.b32 [%0], %1, %2;"
               ::"l"(p), "r"(v), "l"(meta_policy()));
}
__device__ __forceinline__ void red_and_meta(uint32_t *p, uint32_t v) {
  asm volatile("red.relaxed.gpu.global.and.L2::cache_hint.b32 [%0], %1, %2;"
               ::"l"(p), "r"(v), "l"(meta_policy()));
}
#else
__device__ __forceinline__ uint32_t ld_meta(const uint32_t *p) { return ld_relaxed(p); }
__device__ __forceinline__ uint32_t atom_add_meta(uint32_t *p, uint32_t v) { return atom_add(p, v); }
__device__ __forceinline__ uint32_t atom_or_meta(uint32_t *p, uint32_t v) { return atom_or(p, v); }
__device__ __forceinline__ uint32_t atom_and_meta(uint32_t *p, uint32_t v) { return atom_and(p, v); }
__device__ __forceinline__ void red_or_meta(uint32_t *p, uint32_t v) { red_or(p, v); }
__device__ __forceinline__ void red_and_meta(uint32_t *p, uint32_t v) { red_and(p, v); }
#endif

// a slab descriptor, word by word atomic
__device__ __forceinline__ Desc ld_desc(const Desc *p) {
  Desc d;
  asm volatile("ld.relaxed.gpu.global.v4.u32 {%0, %1, %2, %3}, [%4];"
               : "=r"(d.size_id), "=r"(d.chunk_id), "=r"(d.is_head), "=r"(d.chunk_enc)
               : "l"(p));
  return d;
}

}  // namespace ha

#endif  // HA_PTX_CUH_
