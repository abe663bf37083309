// host_ptx.h -- the device core as host C++: CUDA's keywords and warp
// intrinsics, and in place of csrc/ha_ptx.cuh the loads, stores and atomics
// with a point before each where the scheduler may switch to another lane
// (hostcore.cpp).  Force-included before the core's own headers.
#ifndef HA_HOST_PTX_H_
#define HA_HOST_PTX_H_
#define HA_PTX_CUH_  // keeps csrc/ha_ptx.cuh out

// every system header comes before the keywords are defined away
#include <setjmp.h>
#include <stdint.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>
#include <time.h>
#include <ucontext.h>

#include <memory>
#include <vector>

#define __device__
#define __constant__
#define __forceinline__ inline
#define __noinline__ __attribute__((noinline))

struct uint4 {
  uint32_t x, y, z, w;
};

// ---- the scheduler's side (hostcore.cpp) -----------------------------------
void hc_point();                 // another lane may run here
void hc_pause(uint32_t ns);      // this lane sleeps
uint64_t hc_time_ns();           // grows with every point
uint32_t hc_lane();
uint32_t hc_mask();              // the lanes of the calling lane's warp
uint32_t hc_sm();
void hc_wrote(const uint32_t *p, uint32_t from, uint32_t to);  // by a swap or an exchange
// the values that the lanes of `mask` bring, once all have come
const uint64_t *hc_meet(uint32_t mask, uint64_t value);

// ---- warp intrinsics ---------------------------------------------------------
static inline int __popc(uint32_t x) { return __builtin_popcount(x); }
static inline int __ffs(uint32_t x) { return __builtin_ffs((int)x); }
static inline int __clz(uint32_t x) { return x ? __builtin_clz(x) : 32; }
static inline uint64_t __umul64hi(uint64_t a, uint64_t b) {
  return (uint64_t)(((unsigned __int128)a * b) >> 64);
}
static inline uint32_t __activemask() { return hc_mask(); }
static inline uint32_t __ballot_sync(uint32_t mask, bool p) {
  const uint64_t *v = hc_meet(mask, p);
  uint32_t r = 0;
  for (uint32_t i = 0; i < 32; i++)
    if (((mask >> i) & 1u) && v[i]) r |= 1u << i;
  return r;
}
static inline bool __any_sync(uint32_t mask, bool p) { return __ballot_sync(mask, p) != 0; }
template <class T>
static inline T __shfl_sync(uint32_t mask, T value, uint32_t src) {
  const uint64_t *v = hc_meet(mask, (uint64_t)value);
  return (T)v[src & 31u];
}
static inline uint32_t __match_any_sync(uint32_t mask, uint32_t value) {
  const uint64_t *v = hc_meet(mask, value);
  uint32_t r = 0;
  for (uint32_t i = 0; i < 32; i++)
    if (((mask >> i) & 1u) && v[i] == value) r |= 1u << i;
  return r;
}
template <class T>
static inline T __ldg(const T *p) { return *p; }
static inline void __nanosleep(uint32_t ns) { hc_pause(ns); }
static inline uint32_t hc_clock() { return (uint32_t)hc_time_ns(); }
#define clock() hc_clock()
template <class T>
static inline T atomicExch(T *p, T v) {
  hc_point();
  T o = *p;
  *p = v;
  return o;
}

#include "ha_types.h"

namespace ha {
inline uint32_t lane_id() { return hc_lane(); }
inline uint32_t lanemask_lt() { return (1u << hc_lane()) - 1u; }
inline bool first_of(uint32_t grp) { return (grp & lanemask_lt()) == 0; }
inline uint32_t sm_id() { return hc_sm(); }
inline uint64_t globaltimer_ns() { return hc_time_ns(); }
template <class T>
inline T hc_load(const T *p) {
  hc_point();
  return *(const volatile T *)p;
}
template <class T>
inline void hc_store(T *p, T v) {
  hc_point();
  *(volatile T *)p = v;
}
inline uint32_t ld_relaxed(const uint32_t *p) { return hc_load(p); }
inline uint32_t ld_cached(const uint32_t *p) { return hc_load(p); }
inline uint32_t ld_meta(const uint32_t *p) { return hc_load(p); }
inline void st_relaxed(uint32_t *p, uint32_t v) { hc_store(p, v); }
inline void st_release(uint32_t *p, uint32_t v) { hc_store(p, v); }
#define HC_RMW(name, T, expr)           \
  inline T name(T *p, T v) {            \
    hc_point();                         \
    const T o = *p;                     \
    *p = (expr);                        \
    return o;                           \
  }
HC_RMW(atom_add, uint32_t, o + v)
HC_RMW(atom_or, uint32_t, o | v)
HC_RMW(atom_and, uint32_t, o & v)
HC_RMW(exchanged, uint32_t, v)
HC_RMW(atom_exch_acquire, uint32_t, v)
HC_RMW(atom_add_meta, uint32_t, o + v)
HC_RMW(atom_or_meta, uint32_t, o | v)
HC_RMW(atom_and_meta, uint32_t, o & v)
template <class T>
inline T hc_cas(T *p, T expect, T v) {
  hc_point();
  const T o = *p;
  if (o == expect) *p = v;
  return o;
}
inline uint32_t atom_cas(uint32_t *p, uint32_t expect, uint32_t v) {
  const uint32_t o = hc_cas(p, expect, v);
  if (o == expect) hc_wrote(p, o, v);
  return o;
}
inline uint32_t atom_exch(uint32_t *p, uint32_t v) {
  const uint32_t o = exchanged(p, v);
  hc_wrote(p, o, v);
  return o;
}
inline void red_add(uint32_t *p, uint32_t v) { atom_add(p, v); }
inline void red_add_release(uint32_t *p, uint32_t v) { atom_add(p, v); }
inline void red_or(uint32_t *p, uint32_t v) { atom_or(p, v); }
inline void red_and(uint32_t *p, uint32_t v) { atom_and(p, v); }
inline void red_or_meta(uint32_t *p, uint32_t v) { atom_or(p, v); }
inline void red_and_meta(uint32_t *p, uint32_t v) { atom_and(p, v); }
inline void fence_acq_rel() {}
inline void fence_sc() {}
inline Desc ld_desc(const Desc *p) {
  Desc d;
  d.size_id = hc_load(&p->size_id);
  d.chunk_id = hc_load(&p->chunk_id);
  d.is_head = hc_load(&p->is_head);
  d.chunk_enc = hc_load(&p->chunk_enc);
  return d;
}
}  // namespace ha

#endif  // HA_HOST_PTX_H_
