// ha_samples.cu -- the reference's sample programs as workloads of the C ABI
// (halloc_c.h): grid-points (samples/grid-points/grid-points.cu) and
// add-strings (samples/add-strings/add-strings.cu).  Each step is its own
// entry point so that a caller can time it; the check entry points read the
// results back on the device for the tests.
#include <cuda_runtime.h>
#include <limits.h>
#include <stdint.h>
#include <stdio.h>

#include "halloc.h"
#include "halloc_c.h"
#include "ha_types.h"

namespace ha {
extern __constant__ Config c_cfg;
}

namespace {

cudaStream_t as_stream(void *s) { return reinterpret_cast<cudaStream_t>(s); }

int launch_status() {
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) {
    fprintf(stderr, "halloc-b200: launch failed: %s\n", cudaGetErrorString(e));
    return HA_ECUDA;
  }
  return HA_OK;
}

uint32_t blocks_for(uint64_t n, uint32_t block) { return (uint32_t)((n + block - 1) / block); }

__device__ __forceinline__ uint32_t mix32(uint32_t x) {
  x ^= x >> 16;
  x *= 0x7feb352du;
  x ^= x >> 15;
  x *= 0x846ca68bu;
  x ^= x >> 16;
  return x;
}

// ---- grid-points -------------------------------------------------------------
//
// One thread per point: a 16-byte list node from hamalloc (or from a
// pre-allocated array, the sample's comparison mode) is pushed onto the list
// of the point's grid cell with an atomic exchange
// (grid-points.cu:82-137).  The lists are then walked and their nodes freed
// (grid-points.cu:101-153).

struct PointNode {
  int ip;
  PointNode *next;
};
static_assert(sizeof(PointNode) == 16, "one 16-byte block per node");

__device__ __forceinline__ uint32_t cell_of(const float *pts, uint32_t ip, uint32_t ncells) {
  const int nc = (int)ncells;
  int c[3];
  for (int d = 0; d < 3; d++) {
    const int v = (int)floorf(pts[3 * (size_t)ip + d] * (float)nc);
    c[d] = max(min(v, nc - 1), 0);
  }
  return (uint32_t)(c[0] + nc * (c[1] + nc * c[2]));
}

__global__ void ha_grid_insert_k(uint32_t n, uint32_t ncells, const float *__restrict__ pts,
                                 PointNode **grid, PointNode *pre, unsigned long long *nfail) {
  const uint32_t ip = blockIdx.x * blockDim.x + threadIdx.x;
  if (ip >= n) return;
  // the point is on its way while the node is allocated
  unsigned long long *cell = reinterpret_cast<unsigned long long *>(grid + cell_of(pts, ip, ncells));
  PointNode *node = pre ? pre + ip : static_cast<PointNode *>(hamalloc(sizeof(PointNode)));
  if (!node) {
    atomicAdd(nfail, 1ull);
    return;
  }
  // No fence before the exchange: the node's link is only known after it, so
  // a list can be walked from the end of this kernel on, never during it
  // (the fence was 17 % of the kernel's stalls).
  node->ip = (int)ip;
  const unsigned long long old = atomicExch(cell, (unsigned long long)(uintptr_t)node);
  node->next = reinterpret_cast<PointNode *>((uintptr_t)old);
}

// per cell: number of points and the sum of mix32(point index)
__global__ void ha_grid_check_k(uint32_t ncells3, PointNode *const *grid, uint32_t *count,
                                unsigned long long *hsum) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= ncells3) return;
  uint32_t c = 0;
  unsigned long long h = 0;
  for (const PointNode *p = grid[i]; p && c <= (1u << 30); p = p->next) {
    c++;
    h += mix32((uint32_t)p->ip);
  }
  count[i] = c;
  hsum[i] = h;
}

// Bound by dependent round trips: a list is a pointer chase (about 400 cycles
// a node) and a hafree takes about 2,500 cycles.  One thread per cell doing
// both in turn kept 1,024 warps busy for a 32^3 grid, a warp as long as its
// longest list.  Here the first warp of a block walks 32 lists, up to
// kGridDepth nodes of each, into shared memory, and the whole block frees what it
// found, so every hafree call has full warps and four times as many warps are
// in flight: 1 M nodes in 32^3 cells took 140-199 us before and
// 47 now (131 without the order by slab below).
//
// The nodes of a cell come from the heads of many SMs, so a warp's 32 nodes
// lay in seven slabs or more, each with a counter to lower and a descriptor
// to read: hot lines.  Freed in slab order a warp meets one or two.
constexpr uint32_t kGridBlock = 128;
constexpr uint32_t kGridDepth = 32;

__device__ __forceinline__ uint32_t slab_bucket(const PointNode *p) {
  return (uint32_t)((uint64_t)((const char *)p - ha::c_cfg.pool) >> ha::c_cfg.sb_sh) & 31u;
}

// kWide: every warp of the block walks 32 lists, a quarter as deep, for grids of
// many cells, which fill the GPU with walkers either way and for which one
// walker per block means four times the blocks.  The line lies by the cells:
// what counts is how many walkers there are, however long the lists.  The free
// alone, one walker and all warps walking, in us: 1 M points in 24^3 cells 78
// and 164, 32^3 53 and 87, 40^3 45 and 62, 48^3 41 and 50, 64^3 64-74 and 47,
// 100^3 96 and 61; 4 M points in 40^3 211 and 211, 48^3 208 and 160, 64^3 (16
// a cell) 201 and 152; 8 M points in 64^3 (32 a cell) 423 and 288.
constexpr uint32_t kGridWide = 1u << 16;  // cells from which on every warp walks

template <bool kWide>
__global__ void __launch_bounds__(kGridBlock) ha_grid_free_k(uint32_t ncells3, PointNode **grid,
                                                             int pre) {
  constexpr uint32_t kWalkers = kWide ? kGridBlock : 32;
  constexpr uint32_t kSteps = 32 * kGridDepth / kWalkers;
  __shared__ PointNode *s_node[32 * kGridDepth], *s_sorted[32 * kGridDepth];
  __shared__ uint32_t s_count, s_more, s_bucket[32];
  const uint32_t lane = threadIdx.x & 31;
  const bool first = threadIdx.x < 32, walker = kWide || first;
  PointNode *p = nullptr;
  if (walker) {
    const uint32_t i = blockIdx.x * kWalkers + threadIdx.x;
    if (i < ncells3) {
      p = grid[i];
      if (p) grid[i] = nullptr;
    }
  }
  if (pre) return;
  if (kWide && !__syncthreads_or(p != nullptr)) return;  // nothing but empty lists
  for (;;) {
    if (first) s_bucket[lane] = 0;
    if (kWide) {
      if (threadIdx.x == 0) s_count = s_more = 0;
      __syncthreads();
    }
    if (walker) {
      uint32_t n = 0, left = __ballot_sync(0xffffffffu, p != nullptr);
      for (uint32_t d = 0; d < kSteps && left; d++) {
        if (kWide) {  // the warps share one queue
          if (lane == 0) n = atomicAdd(&s_count, (uint32_t)__popc(left));
          n = __shfl_sync(0xffffffffu, n, 0);
        }
        if (p) {
          s_node[n + __popc(left & ((1u << lane) - 1))] = p;
          p = p->next;
        }
        n += __popc(left);
        left = __ballot_sync(0xffffffffu, p != nullptr);
      }
      if (lane == 0) {
        if (!kWide) {
          s_count = n;
          s_more = left;
        } else if (left) {
          atomicOr(&s_more, left);
        }
      }
    }
    __syncthreads();
    const uint32_t n = s_count, more = s_more;
    PointNode **list = s_node;
    if (n > kGridBlock) {
      // order the nodes by slab (modulo 32)
      uint32_t at[32 * kGridDepth / kGridBlock];
#pragma unroll
      for (uint32_t j = 0; j < 32 * kGridDepth / kGridBlock; j++) {
        const uint32_t k = j * kGridBlock + threadIdx.x;
        if (k < n) at[j] = atomicAdd(&s_bucket[slab_bucket(s_node[k])], 1u);
      }
      __syncthreads();
      if (first) {
        const uint32_t c = s_bucket[lane];
        uint32_t sum = c;
        for (int o = 1; o < 32; o *= 2) {
          const uint32_t v = __shfl_up_sync(0xffffffffu, sum, o);
          if (lane >= (uint32_t)o) sum += v;
        }
        s_bucket[lane] = sum - c;
      }
      __syncthreads();
#pragma unroll
      for (uint32_t j = 0; j < 32 * kGridDepth / kGridBlock; j++) {
        const uint32_t k = j * kGridBlock + threadIdx.x;
        if (k < n) s_sorted[s_bucket[slab_bucket(s_node[k])] + at[j]] = s_node[k];
      }
      __syncthreads();
      list = s_sorted;
    }
    for (uint32_t k = threadIdx.x; k < n; k += kGridBlock) hafree(list[k]);
    if (!more) return;
    __syncthreads();  // the lists are free again
  }
}

// ---- add-strings -------------------------------------------------------------
//
// Strings of spaces, zero-terminated, in blocks from hamalloc; every block is
// at least 8-byte aligned and a multiple of 8 bytes long, so strings are read
// and written as 64-bit words (add-strings.cu:71-205), two at a time.  1 M
// pairs of 0 to 31 characters, word by word -> by pairs: concatenation 83 ->
// 73 us, check (byte by byte) 47 -> 28 us, allocation 49 -> 43 us.
//
// Every pair is one 16-byte granule: a string that starts in the upper half of
// one (24-byte blocks do) is read a single word first.  So no load leaves the
// granules that hold a byte of the string, wherever the string lies; what a
// pair holds past its string is not used.

constexpr uint64_t kSpaces = 0x2020202020202020ull;

struct Pair {
  uint64_t x, y;
};
// words from p to the end of its 16-byte granule: 1 or 2
__device__ __forceinline__ uint32_t words_at(const uint64_t *p) {
  return 2 - (((uintptr_t)p >> 3) & 1u);
}
// the words_at(p) words from p on; the second of one word reads as all ones,
// which holds no zero byte
__device__ __forceinline__ Pair load_pair(const uint64_t *p) {
  Pair v;
  if (((uintptr_t)p & 15u) == 0) {
    const ulonglong2 q = *reinterpret_cast<const ulonglong2 *>(p);
    v.x = q.x;
    v.y = q.y;
  } else {
    v.x = p[0];
    v.y = ~0ull;
  }
  return v;
}
__device__ __forceinline__ void store_pair(uint64_t *p, uint64_t x, uint64_t y) {
  if (((uintptr_t)p & 15u) == 0) {
    *reinterpret_cast<ulonglong2 *>(p) = make_ulonglong2(x, y);
  } else {
    p[0] = x;
    p[1] = y;
  }
}

// first zero byte of v (8 when none)
__device__ __forceinline__ uint32_t zero_byte(uint64_t v) {
  const uint64_t t = (v - 0x0101010101010101ull) & ~v & 0x8080808080808080ull;
  return t ? (uint32_t)(__ffsll((long long)t) - 1) >> 3 : 8u;
}
// length of the string whose pair v starts at byte `at`; `len` unchanged when
// the pair holds no zero byte
__device__ __forceinline__ bool ends_in(const Pair &v, uint32_t at, uint32_t &len) {
  const uint32_t zx = zero_byte(v.x), zy = zero_byte(v.y);
  if (zx < 8) {
    len = at + zx;
    return true;
  }
  if (zy < 8) {
    len = at + 8 + zy;
    return true;
  }
  return false;
}

__global__ void ha_strings_alloc_k(uint32_t n, const int *__restrict__ lens, char **strs,
                                   unsigned long long *nfail) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const uint32_t l = (uint32_t)lens[i];
  // l + 1 bytes rounded up to whole words: the same size class for blocks up
  // to 3 KiB, and room for the last word in CUDA's heap above that
  const uint32_t words = l / 8 + 1;  // the word holding the zero byte is the last
  uint64_t *s = static_cast<uint64_t *>(hamalloc(8 * words));
  strs[i] = reinterpret_cast<char *>(s);
  if (!s) {
    atomicAdd(nfail, 1ull);
    return;
  }
  const uint32_t tail = l % 8;  // spaces in the last word
  const uint64_t last = tail ? kSpaces >> (8 * (8 - tail)) : 0ull;
  uint32_t k = 0;
  for (; k + 2 < words; k += 2) store_pair(s + k, kSpaces, kSpaces);
  if (k + 1 < words)
    store_pair(s + k, kSpaces, last);
  else
    s[k] = last;
}

// c = a followed by b: word k of c takes a's word k while a covers it, then
// a's tail and b's head, then b's words shifted by a's length modulo 8.
// Both lengths are found in one loop, a pair of each string per round trip (a
// 31-character pair takes two; word after word and string after string took
// eight), and c is written by pairs.
__global__ void ha_strings_concat_k(uint32_t n, char **c, char *const *a, char *const *b,
                                    unsigned long long *nfail) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const uint64_t *sa = reinterpret_cast<const uint64_t *>(a[i]);
  const uint64_t *sb = reinterpret_cast<const uint64_t *>(b[i]);
  if (!sa || !sb) {
    c[i] = nullptr;
    atomicAdd(nfail, 1ull);
    return;
  }
  uint32_t la = 0, lb = 0;
  bool enda = false, endb = false;
  for (uint32_t i = 0, j = 0; !enda || !endb;) {
    Pair va = {0, 0}, vb = {0, 0};
    if (!enda) va = load_pair(sa + i);
    if (!endb) vb = load_pair(sb + j);
    if (!enda) enda = ends_in(va, 8 * i, la);
    if (!endb) endb = ends_in(vb, 8 * j, lb);
    i += words_at(sa + i);
    j += words_at(sb + j);
  }
  const uint32_t lc = la + lb;
  const uint32_t cwords = lc / 8 + 1;
  uint64_t *sc = static_cast<uint64_t *>(hamalloc(8 * cwords));
  c[i] = reinterpret_cast<char *>(sc);
  if (!sc) {
    atomicAdd(nfail, 1ull);
    return;
  }
  const uint32_t bwords = lb / 8 + 1;  // words of b up to and including its zero byte
  const uint32_t sh = la % 8, ka = la / 8;
  uint64_t before = sh ? sa[ka] & ((1ull << (8 * sh)) - 1) : 0ull;  // what precedes b's next word
  // word k of c, k ascending
  auto word = [&](uint32_t k) -> uint64_t {
    uint64_t w;
    if (k < ka) {
      w = sa[k];
    } else {
      const uint32_t j = k - ka;  // b's word that starts in this one
      const uint64_t v = j < bwords ? sb[j] : 0ull;
      w = before | (v << (8 * sh));
      before = sh ? v >> (8 * (8 - sh)) : 0ull;
    }
    if (k == cwords - 1) {  // clear whatever follows the zero byte
      const uint32_t z = lc % 8;
      w &= z ? ((1ull << (8 * z)) - 1) : 0ull;
    }
    return w;
  };
  uint32_t k = 0;
  for (; k + 1 < cwords; k += 2) {
    const uint64_t x = word(k), y = word(k + 1);
    store_pair(sc + k, x, y);
  }
  if (k < cwords) sc[k] = word(k);
}

__global__ void ha_strings_free_k(uint32_t n, char **strs) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  hafree(strs[i]);
  strs[i] = nullptr;
}

// counts strings that are not la[i] + lb[i] spaces followed by a zero byte
// (by pairs of words; a pair is read only once all before it are spaces, so
// the string reaches at least to its start).  Strings may lie anywhere: one
// that does not start on a word is read byte by byte.
__global__ void ha_strings_check_k(uint32_t n, char *const *c, const int *la, const int *lb,
                                   unsigned long long *bad) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const uint64_t *s = reinterpret_cast<const uint64_t *>(c[i]);
  const uint32_t want = (uint32_t)(la[i] + lb[i]);
  bool ok = s != nullptr;
  if (((uintptr_t)s & 7u) != 0) {
    const char *t = c[i];
    for (uint32_t k = 0; ok && k < want; k++) ok = t[k] == ' ';
    if (ok) ok = t[want] == 0;
  } else if (ok) {
    const uint32_t full = want / 8, z = want % 8;  // the zero byte: byte z of word `full`
    const uint64_t mask = z == 7 ? ~0ull : (1ull << (8 * (z + 1))) - 1;
    const uint64_t tail = z ? kSpaces >> (8 * (8 - z)) : 0ull;
    uint32_t k = 0;
    if (full && words_at(s) == 1) ok = s[k++] == kSpaces;
    for (; ok && k + 1 < full; k += 2) {
      const Pair v = load_pair(s + k);
      ok = v.x == kSpaces && v.y == kSpaces;
    }
    if (ok && k < full) {  // one whole word left, then the last, in one granule
      const Pair v = load_pair(s + k);
      ok = v.x == kSpaces && (v.y & mask) == tail;
    } else if (ok) {
      ok = (s[k] & mask) == tail;
    }
  }
  if (!ok) atomicAdd(bad, 1ull);
}

}  // namespace

extern "C" int ha_grid_insert_c(uint32_t n, uint32_t ncells, const float *pts, void **grid,
                                void *pre_nodes, uint64_t *nfail, void *stream) {
  if (!pts || !grid || !nfail || ncells == 0 || ncells > 1024) return HA_EINVAL;
  if (n == 0) return HA_OK;
  ha_grid_insert_k<<<blocks_for(n, 128), 128, 0, as_stream(stream)>>>(
      n, ncells, pts, reinterpret_cast<PointNode **>(grid),
      static_cast<PointNode *>(pre_nodes), reinterpret_cast<unsigned long long *>(nfail));
  return launch_status();
}

extern "C" int ha_grid_check_c(uint32_t ncells, void *const *grid, uint32_t *count,
                               uint64_t *hsum, void *stream) {
  if (!grid || !count || !hsum || ncells == 0 || ncells > 1024) return HA_EINVAL;
  const uint32_t n3 = ncells * ncells * ncells;
  ha_grid_check_k<<<blocks_for(n3, 128), 128, 0, as_stream(stream)>>>(
      n3, reinterpret_cast<PointNode *const *>(grid), count,
      reinterpret_cast<unsigned long long *>(hsum));
  return launch_status();
}

extern "C" int ha_grid_free_c(uint32_t ncells, void **grid, int pre_nodes, void *stream) {
  if (!grid || ncells == 0 || ncells > 1024) return HA_EINVAL;
  const uint32_t n3 = ncells * ncells * ncells;
  if (n3 >= kGridWide)
    ha_grid_free_k<true><<<blocks_for(n3, kGridBlock), kGridBlock, 0, as_stream(stream)>>>(
        n3, reinterpret_cast<PointNode **>(grid), pre_nodes);
  else
    ha_grid_free_k<false><<<blocks_for(n3, 32), kGridBlock, 0, as_stream(stream)>>>(
        n3, reinterpret_cast<PointNode **>(grid), pre_nodes);
  return launch_status();
}

extern "C" int ha_strings_alloc_c(uint32_t n, const int *lens, char **strs, uint64_t *nfail,
                                  void *stream) {
  if (!lens || !strs || !nfail) return HA_EINVAL;
  if (n == 0) return HA_OK;
  ha_strings_alloc_k<<<blocks_for(n, 128), 128, 0, as_stream(stream)>>>(
      n, lens, strs, reinterpret_cast<unsigned long long *>(nfail));
  return launch_status();
}

extern "C" int ha_strings_concat_c(uint32_t n, char **c, char *const *a, char *const *b,
                                   uint64_t *nfail, void *stream) {
  if (!c || !a || !b || !nfail) return HA_EINVAL;
  if (n == 0) return HA_OK;
  ha_strings_concat_k<<<blocks_for(n, 128), 128, 0, as_stream(stream)>>>(
      n, c, a, b, reinterpret_cast<unsigned long long *>(nfail));
  return launch_status();
}

extern "C" int ha_strings_free_c(uint32_t n, char **strs, void *stream) {
  if (!strs) return HA_EINVAL;
  if (n == 0) return HA_OK;
  ha_strings_free_k<<<blocks_for(n, 128), 128, 0, as_stream(stream)>>>(n, strs);
  return launch_status();
}

extern "C" int ha_strings_check_c(uint32_t n, char *const *c, const int *la, const int *lb,
                                  uint64_t *bad, void *stream) {
  if (!c || !la || !lb || !bad) return HA_EINVAL;
  if (n == 0) return HA_OK;
  ha_strings_check_k<<<blocks_for(n, 128), 128, 0, as_stream(stream)>>>(
      n, c, la, lb, reinterpret_cast<unsigned long long *>(bad));
  return launch_status();
}
