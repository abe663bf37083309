// hostcore.cpp -- the device core (csrc/ha_core.cuh) compiled as host C++ and
// run by warps whose every access to shared memory is a point where a seeded
// scheduler may switch to another lane.  TEST INFRASTRUCTURE ONLY.
//
// Each lane is a fiber.  The lanes of a warp meet at its votes and shuffles
// and otherwise run independently; memory is sequentially consistent.  Now and
// then the scheduler holds a lane back for up to a few thousand points, so
// that others overtake it anywhere in a change of a head.  Time is virtual: it
// grows by 20 ns a point.
//
// The pool has tiny slabs (64 KiB at least): what matters is how often heads
// are used up and slabs filed, not how large they are.
#include "host_ptx.h"

#include "ha_core.cuh"

namespace ha {
Config c_cfg;
Class g_cls[kNSizes];
uint4 g_mod[kNSizes];
State g_st;
}  // namespace ha

namespace {

constexpr size_t kStack = 128 << 10;

struct Warp;
struct Lane {
  ucontext_t start;
  jmp_buf at;
  std::unique_ptr<char[]> stack;
  Warp *warp = nullptr;
  uint32_t id = 0;
  bool begun = false, done = false, met = true;
  uint64_t wake = 0;  // not run before this point (sleeping or held back)
  uint64_t vals[32];
};
struct Meeting {
  uint32_t mask, here;
  uint64_t vals[32];
};
struct Warp {
  uint32_t all = 0, mask = 0, sm = 0;  // mask: the lanes in the present call
  std::vector<Lane> lanes;
  std::vector<Meeting> open;
  const int64_t *ops = nullptr;
  int64_t *res = nullptr;
  int64_t nops = 0;
};

std::vector<Warp> g_warps;
std::vector<Lane *> g_lanes;
Lane *g_cur = nullptr;
jmp_buf g_main;
uint64_t g_points = 0, g_rng = 1;
uint32_t g_hold = 0;  // one point in g_hold holds its lane back (0: none)
uint32_t g_level_moves = 0;  // changes of the level in a set-0 head word
std::vector<uint32_t> g_meta;
bool g_stuck = false;

uint64_t rnd() {
  g_rng ^= g_rng << 13;
  g_rng ^= g_rng >> 7;
  g_rng ^= g_rng << 17;
  return g_rng;
}

void to_main() {
  if (!_setjmp(g_cur->at)) _longjmp(g_main, 1);
}

char *pool() { return ha::c_cfg.pool; }

// ops of a warp: nops x lanes values; v > 0: the lane allocates v bytes, v < 0:
// it frees its result of op -v - 1, v = 0: it does nothing (all lanes of the
// warp then take part in neither).  res holds offsets from the pool, -1 for
// NULL.
void lane_main() {
  Lane *l = g_cur;
  Warp *w = l->warp;
  const uint32_t nl = (uint32_t)w->lanes.size();
  for (int64_t i = 0; i < w->nops; i++) {
    const int64_t op = w->ops[i * nl + l->id];
    int64_t &r = w->res[i * nl + l->id];
    if (op > 0) {
      void *p = ha::malloc_small((uint32_t)op);
      r = p ? (char *)p - pool() : -1;
    } else if (op < 0) {
      int64_t &from = w->res[(-op - 1) * nl + l->id];
      // a warp's lanes free together: a lane with nothing frees nothing, so
      // such a free is left to the others through the warp's mask
      const bool have = from >= 0;
      const uint32_t m = __ballot_sync(w->all, have);
      if (have) {
        w->mask = m;
        ha::free_small((uint64_t)from);
      }
      __ballot_sync(w->all, true);
      w->mask = w->all;
      from = -2;
    }
  }
  l->done = true;
  to_main();
}

}  // namespace

void hc_point() {
  g_points++;
  if (g_hold && rnd() % g_hold == 0) g_cur->wake = g_points + rnd() % 4000;
  to_main();
}
void hc_pause(uint32_t ns) {
  g_cur->wake = g_points + ns / 20 + 1;
  to_main();
}
void hc_wrote(const uint32_t *p, uint32_t from, uint32_t to) {
  if (p >= ha::g_st.head && p < ha::g_st.head + ha::kNSizes)
    g_level_moves += ha::head_level(from) != ha::head_level(to);
}
uint64_t hc_time_ns() { return g_points * 20; }
uint32_t hc_lane() { return g_cur->id; }
uint32_t hc_mask() { return g_cur->warp->mask; }
uint32_t hc_sm() { return g_cur->warp->sm; }
const uint64_t *hc_meet(uint32_t mask, uint64_t value) {
  Lane *l = g_cur;
  if (mask == 1u << l->id) {
    l->vals[l->id] = value;
    return l->vals;
  }
  Warp *w = l->warp;
  Meeting *m = nullptr;
  for (Meeting &o : w->open)
    if (o.mask == mask) m = &o;
  if (!m) {
    w->open.push_back(Meeting{mask, 0, {}});
    m = &w->open.back();
  }
  m->here |= 1u << l->id;
  m->vals[l->id] = value;
  if (m->here == mask) {
    for (Lane &o : w->lanes)
      if ((mask >> o.id) & 1u) {
        memcpy(o.vals, m->vals, sizeof(o.vals));
        o.met = true;
      }
    w->open.erase(w->open.begin() + (m - w->open.data()));
  } else {
    l->met = false;
    to_main();
  }
  return l->vals;
}

extern "C" {

// cls: 16 x 8 words as in ha_types.h; every slab starts in the free set
void hc_init(uint32_t nsbs, uint32_t sb_sh, const uint32_t *cls, uint32_t nheads, uint32_t surge,
             uint32_t spec_mask) {
  using namespace ha;
  memset(&g_st, 0, sizeof(g_st));
  g_level_moves = 0;
  memset(&c_cfg, 0, sizeof(c_cfg));
  memcpy(g_cls, cls, sizeof(g_cls));
  for (uint32_t s = 0; s < kNSizes; s++) {
    const uint64_t mn = ~0ull / g_cls[s].nchunks + 1, mh = ~0ull / g_cls[s].hash_step + 1;
    g_mod[s] = {(uint32_t)mn, (uint32_t)(mn >> 32), (uint32_t)mh, (uint32_t)(mh >> 32)};
  }
  c_cfg.pool = (char *)((uintptr_t)1 << 40);  // never dereferenced
  c_cfg.pool_bytes = (uint64_t)nsbs << sb_sh;
  c_cfg.nsbs = nsbs;
  c_cfg.sb_sh = sb_sh;
  c_cfg.bit_words_sh = sb_sh - 9;
  c_cfg.nib_words_sh = sb_sh - 7;
  c_cfg.set_words = (nsbs + 31) / 32;
  c_cfg.sum_words = (c_cfg.set_words + 31) / 32;
  c_cfg.nheads = nheads;
  c_cfg.surge = surge;
  c_cfg.spec_mask = spec_mask;
  const size_t bits = (size_t)nsbs << c_cfg.bit_words_sh, nibs = (size_t)nsbs << c_cfg.nib_words_sh;
  g_meta.assign(bits + nibs, 0);
  c_cfg.bits = g_meta.data();
  c_cfg.nibs = g_meta.data() + bits;
  for (uint32_t s = 0; s < kMaxHeads * kNSizes; s++) {
    g_st.ticket[s * kTicketStride] = kFirstTicket;
    g_st.head[s] = kSlabField;
    g_st.cached[s] = kNone;
  }
  g_st.wait_limit_us = 1000000;
  g_st.committed = g_st.n_free = nsbs;
  for (uint32_t sb = 0; sb < nsbs; sb++) {
    g_st.ctr[ctr_index(sb)] = kCtrInit;
    g_st.desc[desc_index(sb)].size_id = kNone;
    g_st.desc[desc_index(sb)].chunk_id = kNone;
    g_st.sets[kSetFree][sb >> 5] |= 1u << (sb & 31);
    g_st.sums[kSetFree][sb >> 10] |= 1u << ((sb >> 5) & 31);
  }
}

// Runs the warps' programs to their ends in an order drawn from `seed`.
// Returns the number of points, or -1 when no lane can go on or after
// max_points.
int64_t hc_run(uint32_t nwarps, const uint32_t *nlanes, const uint32_t *sm, const int64_t *const *ops,
               const int64_t *nops, int64_t *const *res, uint64_t seed, uint32_t hold,
               int64_t max_points) {
  g_rng = seed * 0x9E3779B97F4A7C15ull + 0x1234567;
  for (int i = 0; i < 8; i++) rnd();
  g_points = 0;
  g_hold = hold;
  g_warps.clear();
  g_warps.resize(nwarps);
  g_lanes.clear();
  for (uint32_t i = 0; i < nwarps; i++) {
    Warp &w = g_warps[i];
    w.lanes.resize(nlanes[i]);
    w.all = w.mask = nlanes[i] == 32 ? ~0u : (1u << nlanes[i]) - 1;
    w.sm = sm[i];
    w.ops = ops[i];
    w.nops = nops[i];
    w.res = res[i];
    for (uint32_t k = 0; k < nlanes[i]; k++) {
      Lane &l = w.lanes[k];
      l.id = k;
      l.warp = &w;
      l.stack.reset(new char[kStack]);
      getcontext(&l.start);
      l.start.uc_stack.ss_sp = l.stack.get();
      l.start.uc_stack.ss_size = kStack;
      l.start.uc_link = nullptr;
      makecontext(&l.start, lane_main, 0);
      g_lanes.push_back(&l);
    }
  }
  std::vector<Lane *> run;
  for (;;) {
    run.clear();
    uint64_t next = ~0ull;
    bool left = false;
    for (Lane *l : g_lanes) {
      if (l->done) continue;
      left = true;
      if (!l->met) continue;
      if (l->wake <= g_points)
        run.push_back(l);
      else if (l->wake < next)
        next = l->wake;
    }
    if (!left) return (int64_t)g_points;
    if (run.empty()) {
      if (next == ~0ull) return -1;  // every lane waits at a meeting
      g_points = next;
      continue;
    }
    if ((int64_t)g_points > max_points) return -1;
    g_cur = run[rnd() % run.size()];
    if (!_setjmp(g_main)) {
      if (!g_cur->begun) {
        g_cur->begun = true;
        setcontext(&g_cur->start);
      }
      _longjmp(g_cur->at, 1);
    }
  }
}

uint32_t hc_status() { return ha::g_st.status; }
uint32_t hc_nulls() { return ha::g_st.n_null; }
uint32_t hc_head_changes() { return ha::g_st.n_head_changes; }
uint32_t hc_surge_changes() { return ha::g_st.n_surge_changes; }
uint32_t hc_level_moves() { return g_level_moves; }
// whether size sid may open surge level `level`
uint32_t hc_room(uint32_t sid, uint32_t level, uint32_t nfree, uint32_t committed) {
  return ha::room_for_level(sid, level, nfree, committed);
}
// whether a free looks at the sets of a slab whose descriptor showed size sid
uint32_t hc_crosses(uint32_t sid, uint32_t n0, uint32_t n) { return ha::crosses(sid, n0, n); }
// head slab, prefetched slab and level of head set k of size sid; the copy
// of the level beside it
void hc_head(uint32_t sid, uint32_t k, uint32_t out[4]) {
  using namespace ha;
  const uint32_t hs = k * kNSizes + sid;
  out[0] = head_slab(g_st.head[hs]);
  out[1] = g_st.cached[hs];
  out[2] = head_level(g_st.head[hs]);
  out[3] = g_st.level[sid];
}
// a slab: used chunks, head flag in its counter, chunk field, size id, chunk
// id, is_head, and the number of the sets it is in
void hc_slab(uint32_t sb, uint32_t out[7]) {
  using namespace ha;
  const uint32_t c = g_st.ctr[ctr_index(sb)];
  const Desc &d = g_st.desc[desc_index(sb)];
  out[0] = c >> kCntShift;
  out[1] = (c & kHeadFlag) != 0;
  out[2] = (c >> kChunkShift) & kChunkField;
  out[3] = d.size_id;
  out[4] = d.chunk_id;
  out[5] = d.is_head;
  out[6] = 0;
  for (uint32_t k = 0; k < kNSets; k++) out[6] += (g_st.sets[k][sb >> 5] >> (sb & 31)) & 1u;
}

}  // extern "C"
