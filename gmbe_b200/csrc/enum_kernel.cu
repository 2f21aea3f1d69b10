// The enumeration engine: one persistent kernel, one task per warp.
//
// Semantics follow the reference's GMBE path (the -s 2 kernel):
//   task set-up      IterFinderWithMultipleVertex   src/IterFinderGpu.cu:772-887
//   stack DFS        IterProcess                    src/IterFinderGpu.cu:12-69
//   push / pop       finder_push / finder_pop       src/IterFinderGpu.h:206-303 (PRUNE_EN)
//   task splitting   split test + LargeToTiny       src/IterFinderGpu.cu:835-858, 889-910
//   scheduling       IterFinderKernel_6             src/IterFinderGpu.cu:918-1053
// The data layout and the work per step are this engine's own:
//   * Task set-up counts the two-hop multiset once through a per-warp dense
//     map (no union merges, no binary searches) and lays the candidate set C
//     out as [Q part | P part] instead of sorting it.
//   * Tier 1 (|L| above the bitmap limit) keeps GMBE's per-candidate
//     neighbour counts and level bounds, but walks per-task local adjacency
//     (L position -> C index and C index -> L position) instead of binary
//     searching global rows on every push and pop.
//   * Tier 2 (|L| <= 32*K) re-expresses the same DFS over K-word bitmaps of
//     the current L: a push is an AND, the maximality test a compare, the
//     pro-active pruning test an AND with the removed vertices.  Candidates
//     of one neighbourhood are one class, and a sub-problem of at most 32
//     classes over 32 L vertices is walked in registers, a class per lane.
//   * Split tasks go to a bounded MPMC ring; every device wait is bounded and
//     reports a status instead of hanging.
#include <cuda_runtime.h>

#include <climits>
#include <cstdio>

#include "enum_common.cuh"
#include "enum_launch.h"

// Loops are kept rolled unless they say otherwise, and what several places call
// stays out of line.  The kernel is bound by instruction fetch: its warps are
// each in another part of the code, and half of their stalls are for want of an
// instruction, the instruction caches at three quarters of their peak (a
// 32-graph batch).  Rolled it is 336 KB, with loops unrolled as the compiler
// would 498 KB; whole calls, rolled / unrolled: 256-graph batch 163 / 262 ms,
// 300,000-edge graph 44 / 64 ms, medium graph 302 / 391 ms.
#define ROLLED _Pragma("unroll 1")

namespace gmbe {

namespace {

constexpr int32_t kFree = 0x7fffffff;     // live at every level (reference 0x7fff)
constexpr int32_t kTouched = 0x3fffffff;  // marked by the pop restore pass (reference 0x3fff)
constexpr unsigned kFull = 0xffffffffu;

__device__ __forceinline__ unsigned lanemask_lt() {
  unsigned r;
  asm volatile("mov.u32 %0, %%lanemask_lt;" : "=r"(r));
  return r;
}

__device__ __noinline__ void set_status(EnumCtl* ctl, int32_t code, unsigned long long info) {
  if (atomicCAS(&ctl->status, 0, code) == 0) ctl->err_info = info;
  atomicExch(&ctl->abort, 1);
}

// Sums over the warp, out of line: a score of call sites would each hold the
// reduction.
__device__ __noinline__ unsigned long long warp_sum64(unsigned long long v) { return warp_sum(v); }
// Exclusive prefix sum within the warp, and above it (32 bits up) the total.
__device__ __noinline__ unsigned long long scan32(int v) {
  int tot;
  const int ex = warp_excl_scan(v, &tot);
  return ((unsigned long long)(unsigned)tot << 32) | (unsigned)ex;
}
__device__ __forceinline__ int excl_scan(int v, int* tot) {
  const unsigned long long r = scan32(v);
  *tot = (int)(r >> 32);
  return (int)r;
}

// Visits every entry of a list of rows with all 32 lanes busy, in order.
// row_of(r, beg, len) describes row r; load(valid, pos) reads what the visit
// needs, pos indexing the global entry array, and visit(valid, r, k, v) gets it,
// k counting the entries; both are called by every lane (uniform control flow).
// Two loads per lane are issued before the first visit: a walk is bound by
// their latency (and, unrolled further, by its own code).  flat_rows2: more(v)
// reads what hangs on the first load, again two per lane before the first visit.
template <typename RowOf, typename Load, typename More, typename Visit>
__device__ __forceinline__ void flat_rows2(int nr, RowOf row_of, Load load, More more,
                                           Visit visit) {
  const int lane = (int)lane_id();
  int done = 0;
  ROLLED for (int r0 = 0; r0 < nr; r0 += 32) {
    int beg = 0, len = 0;
    if (r0 + lane < nr) row_of(r0 + lane, beg, len);
    int tot;
    const int ex = excl_scan(len, &tot);
    beg -= ex;
    ROLLED for (int e0 = 0; e0 < tot; e0 += 64) {
      int r[2];
      decltype(load(true, 0)) v[2];
      decltype(more(v[0])) w[2];
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        r[u] = 0;
        if (e0 + 32 * u < tot) {
          const int e = e0 + 32 * u + lane;
          int lo = 0;
#pragma unroll
          for (int step = 16; step > 0; step >>= 1) {
            const int cand = lo + step;
            if (__shfl_sync(kFull, ex, cand) <= e) lo = cand;
          }
          r[u] = r0 + lo;
          v[u] = load(e < tot, __shfl_sync(kFull, beg, lo) + e);
        }
      }
#pragma unroll
      for (int u = 0; u < 2; ++u)
        if (e0 + 32 * u < tot) w[u] = more(v[u]);
#pragma unroll
      for (int u = 0; u < 2; ++u)
        if (e0 + 32 * u < tot)
          visit(e0 + 32 * u + lane < tot, r[u], done + e0 + 32 * u + lane, v[u], w[u]);
    }
    done += tot;
  }
}
template <typename RowOf, typename Load, typename Visit>
__device__ __forceinline__ void flat_rows(int nr, RowOf row_of, Load load, Visit visit) {
  flat_rows2(nr, row_of, load, [](int v) { return v; },
             [&](bool valid, int r, int k, int v, int) { visit(valid, r, k, v); });
}

// What every warp of a block shares, and each warp's own state.  Both live in
// shared memory: functions that are not inlined reach them at a fixed address,
// and nothing of them takes up registers or local memory (whose traffic would
// evict the warps' working sets from L1).
struct Block {
  const EnumParams* p;   // the rest of the launch's parameters
  EnumCtl* ctl;
  Task* q_tasks;
  unsigned long long* q_seq;
  const DevGraph* graphs;  // every graph of the launch
  int32_t* slots;        // exported bitmap sub-problems (nslot x kSlotWords)
  uint32_t* slot_bits;   // slot occupancy
  int32_t* bigslots;     // large slots (nbig x kBigSlotWords)
  uint32_t* big_bits;
  int32_t* emit;
  uint64_t deadline;      // %globaltimer after which the launch gives up (0: never)
  long long import_words; // arena words every warp of the launch has
  int nslot, nbig;
  int import_cap;        // most candidates any warp of the launch can take in
  int import_l, import_s; // most L vertices / two-hop entries any warp can take in
  // Copies of parameters read often.
  int32_t prune, server, share_min_work, slot_records, eager_share, share_counts, touch_scan;
  int32_t smem_words;
  int32_t lookout;  // 1 while an idle warp of the block watches the queue
  unsigned long long last_ns, busy_ns;  // per-block timing, at the launch's end
};

struct Warp {
  int32_t* base;           // this warp's scratch
  const DevGraph* gp;      // graph of the task being run
  int32_t gid;
  int32_t tier;            // index of the warp's layout in s_sl
  // Accumulators, kept by lane 0 (acc).
  unsigned long long cnt, hash, nonmax, splits;
  unsigned long long ns_t2, n_t2;  // time inside the bitmap tier, sub-problems run
  unsigned long long pushes;       // pushes so far: counts tier | bitmap tier << 32
  unsigned long long shape;        // last task set up: |C| | (part << 32) | (parts << 48)
  unsigned long long ns_t1;        // time inside the counts tier (bitmap tier excluded)
  unsigned long long dead;         // counts tier: entries of aadj known to be retired (lane 0)
  bool seen;                       // first-touch bitmaps in shared memory (this_smem)
  long long dem_t;                 // clock64 of the last export-demand reading (lane 0)
  int dem;                         // that reading

  __device__ __forceinline__ const ScratchLayout& sl() const;
  __device__ __forceinline__ int32_t* A(int64_t off) const { return base + off; }
  __device__ __forceinline__ uint64_t* A64(int64_t off) const {
    return reinterpret_cast<uint64_t*>(base + off);
  }
  // This warp's first-touch bitmap in global memory.
  __device__ __forceinline__ uint32_t* gseen() const;
};

__shared__ Block s_blk;
__shared__ ScratchLayout s_sl[2];
__shared__ Warp s_warp[kEnumWarps];
static_assert(sizeof(Block) + 2 * sizeof(ScratchLayout) + kEnumWarps * sizeof(Warp) + 64 +
                      kEnumWarps * sizeof(uint32_t) *
                          (kSeenMaxWords > kSmemWords ? kSeenMaxWords : kSmemWords) <=
                  kBlockSmemBytes,
              "a block's shared memory (64 bytes: alignment)");
extern __shared__ uint4 enum_smem4[];

__device__ __forceinline__ Warp& this_warp() { return s_warp[threadIdx.x >> 5]; }
// This warp's part of the dynamic shared memory.
__device__ __forceinline__ uint32_t* this_smem() {
  return reinterpret_cast<uint32_t*>(enum_smem4) + (size_t)(threadIdx.x >> 5) * s_blk.smem_words;
}
__device__ __forceinline__ const ScratchLayout& Warp::sl() const { return s_sl[tier]; }
__device__ __forceinline__ uint32_t* Warp::gseen() const {
  return reinterpret_cast<uint32_t*>(base + sl().gseen);
}
// Adds to one of the warp's accumulators (v: the same in every lane).
__device__ __forceinline__ void acc(unsigned long long& a, unsigned long long v) {
  if (lane_id() == 0) a += v;
}

// Whether this warp should leave its task (lane-uniform): the launch is
// aborting, or its time limit has passed (which starts the abort).
__device__ __noinline__ bool must_stop() {
  int s = 0;
  if (lane_id() == 0) {
    s = *(volatile int32_t*)&s_blk.ctl->abort;
    if (!s && s_blk.deadline != 0) {
      const uint64_t now = globaltimer_ns();
      if (now > s_blk.deadline) {
        set_status(s_blk.ctl, kStDeadline, now - s_blk.deadline);
        s = 1;
      }
    }
  }
  return __shfl_sync(0xffffffffu, s, 0) != 0;
}

// Before a counting pass over `words` bitmap words: the bitmap tier, which uses
// the same shared memory, may have left anything there.
__device__ __forceinline__ void clear_seen(const Warp& W, int words) {
  if (!W.seen) return;
  uint32_t* seen = this_smem();
  ROLLED for (int i = (int)lane_id(); i < words; i += 32) seen[i] = 0u;
  __syncwarp();
}

// Adds 1 to counts[i] and tells whether this was i's first touch since the
// counts were last cleared.  With a shared-memory bitmap the first touch is a
// shared atomic and the count a fire-and-forget global one, so the warp does
// not wait for an L2 round trip per entry; without it, the returned old count
// tells.  seen: this_smem(), so that the compiler sees a shared address (through
// a pointer kept in memory the atomic took the generic path: 18.5 -> 18.0 ms on
// 8,000 roots of about 144,000 entries).
__device__ __forceinline__ bool count_first(bool shared, uint32_t* seen, int32_t* counts, int i) {
  if (shared) {
    const uint32_t bit = 1u << (i & 31);
    atomicAdd(&counts[i], 1);
    return (atomicOr(&seen[i >> 5], bit) & bit) == 0u;
  }
  return atomicAdd(&counts[i], 1) == 0;
}

// After a counting pass: makes every lane's count increments visible to the
// warp, and clears the bitmap bits of the `n` indices touched (listed in idx).
__device__ __forceinline__ void counts_done(const Warp& W, const int32_t* idx, int n) {
  __threadfence_block();
  __syncwarp();
  if (W.seen) {
    uint32_t* seen = this_smem();
    ROLLED for (int i = (int)lane_id(); i < n; i += 32) seen[idx[i] >> 5] = 0u;
    __syncwarp();
  }
}

// Whether a counting pass of `entries` entries over an index space of
// `words` bitmap words collects its first touches from the global bitmap:
// only without the shared-memory bitmap, and when the pass is large enough
// that a scan of the words costs less than an atomic round trip per 32
// entries.
__device__ __forceinline__ bool use_gseen(const Warp& W, long long entries, int words) {
  if (s_blk.touch_scan != 0) return s_blk.touch_scan > 0;
  return !W.seen && entries >= (long long)words;
}

// Lists the set bits of bits[0, words) in increasing index order into
// out[0, cap) (indices beyond cap are not written) and clears the words;
// returns the number of set bits.  Every lane takes one word per round, so
// the loads are independent and coalesced.  The bits were set by this warp's
// atomics: the fence before the call makes them visible here.
__device__ __noinline__ int collect_bits(uint32_t* bits, int words, int32_t* out, int cap) {
  const int lane = (int)lane_id();
  int n = 0;
  ROLLED for (int w0 = 0; w0 < words; w0 += 32) {
    const int w = w0 + lane;
    uint32_t m = w < words ? __ldcg(bits + w) : 0u;
    if (m) bits[w] = 0u;
    int tot;
    int o = n + excl_scan(__popc(m), &tot);
    while (m) {
      if (o < cap) out[o] = (w << 5) + __ffs(m) - 1;
      ++o;
      m &= m - 1;
    }
    n += tot;
  }
  __syncwarp();
  return n;
}

// Emission (opt-in): appends a maximal biclique's L to the launch's record
// buffer as [|L|, graph, internal U ids of L...]; R is N(L).  Two forms:
//  - a buffer (rd null): a record that does not fit entirely is dropped (the
//    reserved word count keeps growing past the buffer, which tells the
//    host); the host zeroes the buffer first and reads it after the launch;
//  - a ring in host-mapped memory (rd = the host's consumed word count):
//    positions grow without bound and index the ring modulo its size; a
//    producer whose record would overrun words the host has not consumed
//    waits for it (bounded by wait_ns: past it the launch fails with a
//    timeout status and the record is dropped).  The host drains the ring
//    while the launch runs and zeroes what it consumed.
// In both, the body and graph words are made visible system-wide before the
// length word, which commits the record (the host waits for a non-zero
// length at the next position).  Kept out of line and given plain
// arguments: inlined at its four call sites, the code grew the
// enumeration's hot loops enough to slow every launch by a quarter.
struct EmitDst {
  int32_t* buf;
  long long cap;                        // words
  const unsigned long long* rd;         // ring: words the host has consumed
  long long wait_ns;                    // ring: longest wait for room
};

__device__ __forceinline__ EmitDst emit_dst(const EnumParams& p) {
  return EmitDst{p.emit, p.emit_cap, p.emit_read, p.idle_ns_limit};
}

// Reserves a record of `count` ids (lane-uniform); -1 if it is dropped.
__device__ __noinline__ long long emit_reserve(EnumCtl* ctl, const EmitDst& d, int count) {
  const unsigned long long need = (unsigned long long)count + 2;
  long long pos = 0;
  if (lane_id() == 0) {
    const unsigned long long at = atomicAdd(&ctl->emit_pos, need);
    if (!d.rd) {
      pos = at + need > (unsigned long long)d.cap ? -1LL : (long long)at;
    } else if (need > (unsigned long long)d.cap) {
      pos = -1;
      set_status(ctl, kStCapacity, ((unsigned long long)6 << 32) | (unsigned)count);
    } else {
      pos = (long long)at;
      const uint64_t t0 = globaltimer_ns();
      while (at + need > *(volatile const unsigned long long*)d.rd + (unsigned long long)d.cap) {
        if (*(volatile int32_t*)&ctl->abort || globaltimer_ns() - t0 > (uint64_t)d.wait_ns) {
          set_status(ctl, kStTimeout, at);
          pos = -1;
          break;
        }
        __nanosleep(1000);
      }
    }
  }
  return __shfl_sync(kFull, pos, 0);
}

__device__ __forceinline__ int32_t& emit_at(const EmitDst& d, long long pos) {
  return d.buf[(unsigned long long)pos % (unsigned long long)d.cap];
}

__device__ __forceinline__ void emit_header(const EmitDst& d, long long pos, int count, int gid) {
  __threadfence_system();
  __syncwarp();
  if (lane_id() == 0) {
    emit_at(d, pos + 1) = gid;
    __threadfence_system();
    emit_at(d, pos) = count;
  }
  __syncwarp();
}

// L = ids[idx[i]] (or ids[i] when idx is null) for i < n.
__device__ __noinline__ void emit_list(EnumCtl* ctl, EmitDst d, int gid, int n,
                                       const int32_t* ids, const int32_t* idx) {
  const long long pos = emit_reserve(ctl, d, n);
  if (pos < 0) return;
  ROLLED for (int i = (int)lane_id(); i < n; i += 32) emit_at(d, pos + 2 + i) = idx ? ids[idx[i]] : ids[i];
  emit_header(d, pos, n, gid);
}

// L = ids[l] for the l < nscan with llevel[l] == level, count of them.
__device__ __noinline__ void emit_level(EnumCtl* ctl, EmitDst d, int gid, int count, int nscan,
                                        const int32_t* llevel, int level, const int32_t* ids) {
  const long long pos = emit_reserve(ctl, d, count);
  if (pos < 0) return;
  int out = 0;
  ROLLED for (int b0 = 0; b0 < nscan; b0 += 32) {
    const int l = b0 + (int)lane_id();
    const bool s = l < nscan && llevel[l] == level;
    const unsigned bal = __ballot_sync(kFull, s);
    if (s) emit_at(d, pos + 2 + out + __popc(bal & lanemask_lt())) = ids[l];
    out += __popc(bal);
  }
  emit_header(d, pos, count, gid);
}

// L = lid[b] for the set bits b of a K-word mask (lane w: word w), count of them.
__device__ __noinline__ void emit_words(EnumCtl* ctl, EmitDst d, int gid, int count, int K,
                                        uint32_t mw, const int32_t* lid) {
  const long long pos = emit_reserve(ctl, d, count);
  if (pos < 0) return;
  const int lane = (int)lane_id();
  int out = 0;
  ROLLED for (int w = 0; w < K; ++w) {
    const uint32_t m = __shfl_sync(kFull, mw, w);
    const bool s = (m >> lane) & 1u;
    if (s) emit_at(d, pos + 2 + out + __popc(m & lanemask_lt())) = lid[w * 32 + lane];
    out += __popc(m);
  }
  emit_header(d, pos, count, gid);
}

// Serving block of graph `gid` (a block index into the arena, which the
// launch receives in place of the descriptor array).
__device__ __forceinline__ ServeGraph* serve_graph(const Warp& W, int32_t gid) {
  char* arena = const_cast<char*>(reinterpret_cast<const char*>(s_blk.graphs));
  return reinterpret_cast<ServeGraph*>(arena + ((size_t)(uint32_t)gid << kServeBlockShift));
}

// Descriptor of graph `gid` of this launch.
__device__ __forceinline__ const DevGraph* graph_at(const Warp& W, int32_t gid) {
  return s_blk.server ? &serve_graph(W, gid)->g : s_blk.graphs + gid;
}

// Most parts a root is split into.
constexpr int kMaxParts = 1024;

// Bucket of candidate w among `parts` (Knuth's multiplicative hash, scaled):
// spreads consecutive ids, hence the work, evenly over the parts.
__device__ __forceinline__ int part_of(int w, int parts) {
  return (int)(((unsigned long long)((uint32_t)w * 2654435761u) * (unsigned)parts) >> 32);
}

// Children of the current graph about to be queued (serving: a graph
// completes when its roots and every queued child have finished).
__device__ __forceinline__ void graph_spawned(const Warp& W, unsigned long long n) {
  if (s_blk.server) atomicAdd(&serve_graph(W, W.gid)->pending, n);
}

// ---------------------------------------------------------------------------
// Bitmap sub-problems.
//
// A sub-problem is an L of kn vertices (K words of bits) and a list of
// candidate classes.  A class is one or more candidates with the same
// neighbourhood inside L: its K mask words, the sum of its P candidates' hash
// keys, and an info word with their number and two flags, kInfoQ (some
// candidate of it is in Q) and kInfoP (some candidate of it is in P, i.e. is
// still to be pushed).  Classes are in push order: those with a P candidate
// stand at the position of their first one.
//
// Merging candidates into classes leaves GMBE's search tree as it is.  When a
// candidate x is popped, finder_pop retires every candidate whose
// neighbourhood lies inside x's, so of several candidates with one
// neighbourhood only the first P candidate is ever pushed at that level; that
// push is non-maximal exactly if one of them is in Q (or another Q candidate
// covers it).  A biclique that is counted is covered by no Q candidate, and a
// retired candidate always has a popped one (in Q from then on) above it, so
// R consists of P candidates that are still live: summing a class's P keys
// gives the same R.  Without pruning the rule does not hold, and nothing is
// merged.
//
// What a push costs is the list it goes through.  On a 300,000-edge graph the
// average push met 848 candidates and meets 88 classes (319 and 62, 190 and 34
// on graphs of 20,000 to 40,000 edges), and 73 % of the pushes have at most 32,
// one per lane.  Kernel times with single candidates (unrolled code) / now: 28 x
// 40 vertices at density 0.8 8.2 / 1.65 ms, 300 x 200 with planted blocks 0.83 /
// 0.25 ms, 20,000 edges 1.09 / 0.79 ms.  Where next to no candidates are equal, a
// child of 33 to 128 classes costs more than it did, and a launch that waits for
// one warp's chain of them longer: 60 x 40 at density 0.6 5.1 / 6.8 ms in one
// vertex order, 5.5 / 5.4 in the other, 80 x 36 7.4 / 10.6 ms.
//
// Lists live in memory as planes (word w of class i at m[w * stride + i]), so
// a warp's sweep over 32 classes reads one line per mask word.
constexpr uint32_t kInfoQ = 1u << 31;
constexpr uint32_t kInfoP = 1u << 30;
constexpr uint32_t kInfoCnt = kInfoP - 1u;

struct ClsList {
  uint32_t* m;     // K planes of `stride` words
  uint64_t* key;   // [stride] sum of the P candidates' hash keys
  uint32_t* info;  // [stride] number of P candidates | flags
  int n, stride, K;
};

__device__ __forceinline__ ClsList cls_list_at(uint32_t* base, int n, int K) {
  ClsList l;
  l.n = n;
  l.K = K;
  l.stride = (n + 31) & ~31;
  l.m = base;
  l.key = reinterpret_cast<uint64_t*>(base + (size_t)l.stride * K);
  l.info = base + (size_t)l.stride * (K + 2);
  return l;
}

// One level of the walk while a deeper one runs, in the warp's arena: the list
// it works on, its live bits (a bit per class), and the class it pushed last;
// its L words follow.  The list's own Q and P bits serve every level on it:
// classes are pushed in order, so that at each level, of the live ones, those
// up to the last pushed one are Q and the rest are what they were when the list
// was made (q_bits, p_bits).  So a level costs one bit a class, and the scratch
// holds a level per L vertex of the widest child (cls_sub_words).  With Q and P
// bits at every level it held half of them, and wider children went down the
// counts tier instead: 900 candidates below a row of 140 vertices, 800 of them
// below one of 128, 17 ms on one B200 against 63 with the other warps' help and
// 156 without.
struct ClsFrame {
  ClsList l;
  const uint64_t* lk;  // hash key of each L bit
  const int32_t* lid;  // internal U id of each L bit (emission only)
  uint64_t sR;         // R of the push that opened the level
  ClsFrame* prev;
  uint32_t* A;         // live bits
  const uint32_t* QP;  // the list's Q bits, then its P bits
  uint32_t *top, *stop;  // first free word above the level: arena, shared memory
  uint32_t nR;
  int nend;            // classes [0, nend) may be pushed here
  int last;            // the last pushed class (-1: none; a level on its parent's
                       // list starts from the parent's)
};
static_assert(sizeof(ClsFrame) <= 4 * kFrameWords, "frame size");

__device__ __forceinline__ int words_k(int n) {
  int w = (n + 31) >> 5;
  return w <= 2 ? (w < 1 ? 1 : w) : (w <= 4 ? 4 : w);
}

// Slot layout (int32 words): header, L words, L keys, L ids, then the list.
constexpr int kSlotWords = 32768;
constexpr int kSlotHdr = 16;
constexpr int kSlotL = kSlotHdr;
constexpr int kSlotLk = kSlotL + kKMax;             // 32 kKMax uint64
constexpr int kSlotLid = kSlotLk + 2 * 32 * kKMax;  // 32 kKMax int32
constexpr int kSlotList = (kSlotLid + 32 * kKMax + 31) & ~31;
__host__ __device__ constexpr int slot_cap(int K) {
  return ((kSlotWords - kSlotList) / (K + 3)) & ~31;
}
__host__ __device__ constexpr int big_slot_cap(int K) {
  return ((kBigSlotWords - kSlotList) / (K + 3)) & ~31;
}
static_assert(slot_cap(1) <= kSlotMaxRecords && slot_cap(1) >= slot_cap(2) &&
                  slot_cap(2) >= slot_cap(4) && kSlotWords == kSlotWordsHost,
              "host view of the slot size");
// header words: 0 K, 1 n, 2 kn, 3 graph, 4..5 sR, 6 nR

// Claims a free slot of an occupancy bitmap of n slots (lane 0); -1 if none.
__device__ __noinline__ int bits_alloc(uint32_t* bits, int n) {
  const int nw = n >> 5;
  if (nw == 0) return -1;
  int start = (int)(((blockIdx.x * 32u + (threadIdx.x >> 5)) * 2654435761u) % (unsigned)nw);
  ROLLED for (int t = 0; t < nw; ++t) {
    int wi = (start + t) % nw;
    unsigned cur = *(volatile unsigned*)&bits[wi];
    while (cur != 0xffffffffu) {
      int b = __ffs(~cur) - 1;
      unsigned old = atomicOr(&bits[wi], 1u << b);
      if (!(old & (1u << b))) return wi * 32 + b;
      cur = old | (1u << b);
    }
  }
  return -1;
}

// A regular slot (lane 0); -1 if none.
__device__ int slot_alloc(Warp& W) { return bits_alloc(s_blk.slot_bits, s_blk.nslot); }

__device__ __forceinline__ bool regular_fits(const Warp& W, int n, int K) {
  return n <= slot_cap(K) && (s_blk.slot_records <= 0 || n <= s_blk.slot_records);
}

// A slot for a sub-problem of n classes with K-word masks (lane 0): a regular
// one when it fits, else a large one; -1 if none.
__device__ int slot_alloc_for(Warp& W, int n, int K) {
  if (regular_fits(W, n, K)) return slot_alloc(W);
  if (n > big_slot_cap(K)) return -1;
  const int b = bits_alloc(s_blk.big_bits, s_blk.nbig);
  return b < 0 ? -1 : s_blk.nslot + b;
}

// Whether a child of n classes and so many levels can be exported at all:
// some kind of slot holds it, and every warp of the launch can run it.
__device__ __forceinline__ bool slot_fits(const Warp& W, int n, int K, int levels) {
  if (s_blk.nslot == 0 || cls_need(n, K, levels) + cls_key_words(K) > s_blk.import_words)
    return false;
  return regular_fits(W, n, K) || (s_blk.nbig > 0 && n <= big_slot_cap(K));
}

__device__ __forceinline__ int32_t* slot_ptr(const Warp& W, int s) {
  return s < s_blk.nslot ? s_blk.slots + (size_t)s * kSlotWords
                     : s_blk.bigslots + (size_t)(s - s_blk.nslot) * kBigSlotWords;
}

__device__ void slot_free(Warp& W, int s) {
  if (s < s_blk.nslot) atomicAnd(&s_blk.slot_bits[s >> 5], ~(1u << (s & 31)));
  else {
    const int b = s - s_blk.nslot;
    atomicAnd(&s_blk.big_bits[b >> 5], ~(1u << (b & 31)));
  }
}

__device__ bool queue_push_one(Warp& W, const Task& t);

// Demand for exported work (lane-uniform): 0 none, 1 idle warps outnumber
// queued work, 2 more than an eighth of all warps are idle as well.
// The counters are global loads the warp would wait for on every sizable
// child, so a reading is reused for kDemandCycles SM clocks (about 2 us):
// demand moves with warps going idle, far more slowly than children come.
constexpr long long kDemandCycles = 4096;
__device__ __noinline__ int export_demand() {
  Warp& W = this_warp();
  int want = 0;
  if (lane_id() == 0) {
    const long long now = clock64();
    if (now - W.dem_t < kDemandCycles) {
      want = W.dem;
    } else {
      EnumCtl* c = s_blk.ctl;
      int idle = *(volatile int32_t*)&c->idle_warps;
      unsigned long long queued = *(volatile unsigned long long*)&c->q_tail -
                                  *(volatile unsigned long long*)&c->q_head;
      if (idle > 0 && (unsigned long long)idle > queued) {
        const int warps = (int)(gridDim.x * (blockDim.x >> 5));
        want = idle > (warps >> 3) ? 2 : 1;
      }
      W.dem = want;
      W.dem_t = now;
    }
  }
  return __shfl_sync(0xffffffffu, want, 0);
}

// GMBE's split test on a child: (|P| > h or |L| > h) and |P| * |L| > s.
__device__ __forceinline__ bool big_enough(const Warp& W, int nP, int nL) {
  return (nP > W.gp->bound_height || nL > W.gp->bound_height) &&
         (long long)nP * nL > (long long)W.gp->bound_size;
}

// Whether to hand a child (nP classes to push, |L| = nL) to another warp.  A
// child that passes GMBE's split test goes whenever warps wait for work.
// When many warps wait, smaller children go too: the size test misjudges
// dense graphs, where a few dozen candidates can hold millions of
// bicliques.  The floor (share_min_work) keeps the tiniest children, whose
// copy would cost the exporting warp more than running them, at home.
// `eager`: a child that passes the split test goes even when no warp waits
// (the counts tier's parents are the heaviest tasks of a launch and are
// claimed first; their children, queued ahead of new roots, keep every warp
// busy instead of lengthening the parent).
__device__ __forceinline__ bool should_export(Warp& W, int nP, int nL, bool eager = false) {
  if (nP < 2 || nL < 2) return false;
  const bool sizable = (long long)nP * nL >= s_blk.share_min_work;
  const bool big = big_enough(W, nP, nL);
  if (!big && !sizable) return false;  // goes at no demand: skip reading it
  if (eager && big) return true;
  const int d = export_demand();
  return (d == 2 && (big || sizable)) || (d == 1 && big);
}

// Enqueues a filled slot as a task; false if the ring is full.
// kind 0: a bitmap sub-problem; kind 1: a counts-tier child (vertex lists).
__device__ __noinline__ bool slot_publish(int slot, int kind) {
  Warp& W = this_warp();
  __syncwarp();
  __threadfence();
  Task t;
  t.v[0] = -2 - slot;
  t.v[1] = kind ? 1 : -1;
  t.v[2] = t.v[3] = -1;
  t.graph = t.part = t.parts = t.pad = 0;
  return queue_push_one(W, t);
}

__device__ void slot_header(int32_t* sp, int K, int n, int kn, uint64_t sR, uint64_t nR, int gid) {
  sp[0] = K;
  sp[1] = n;
  sp[2] = kn;
  sp[3] = gid;
  *reinterpret_cast<uint64_t*>(sp + 4) = sR;
  sp[6] = (int32_t)nR;
}

// Bit i of word w set below i classes: the first n bits of a bit string.
__device__ __forceinline__ uint32_t first_bits(int n, int w) {
  return ~__funnelshift_lc(0u, 0xffffffffu, (unsigned)max(n - 32 * w, 0));  // (clamped at 32)
}

// ---------------------------------------------------------------------------
// Shared memory of a warp, in words: the merge table, the level being walked,
// the indices of a child's classes, and an arena for the masks and the live, Q
// and P bits of the levels being walked.  A warp waits about 30 cycles for
// shared memory and ten times that for a line another lane's store has sent to
// L2, and a push is a chain of such accesses.
constexpr int kSlots = 256;  // entries of the merge table
constexpr int kSmTab = 0;    // five arrays: mask, leader, key sum (low, high), info
constexpr int kSmCur = kSmTab + 5 * kSlots;
constexpr int kSmIdx = kSmCur + 40;
constexpr int kSmArena = kSmIdx + kChildMax;
static_assert(kSmArena < kSmemWords && kSmArena % 8 == 0, "shared memory layout");
static_assert(kChildMax * 2 <= kSlots, "probing ends");

struct MergeTab {  // all-zero between merges
  uint32_t *mask, *lead, *lo, *hi, *info;
};
__device__ __forceinline__ MergeTab this_tab() {
  uint32_t* t = this_smem() + kSmTab;
  return MergeTab{t, t + kSlots, t + 2 * kSlots, t + 3 * kSlots, t + 4 * kSlots};
}
// Adds a class to the sums of its leader's entry.  Shared-memory atomics: a
// popular mask (one vertex of L, say) takes in hundreds of candidates, and
// that many global atomics on one address held up every warp's memory traffic
// (432,000 cycles for a merge).
__device__ __forceinline__ void merge_add(const MergeTab& t, uint32_t h, uint64_t key,
                                          uint32_t info) {
  if (info & kInfoP) {
    const uint32_t lo = (uint32_t)key;
    const uint32_t old = atomicAdd(&t.lo[h], lo);
    atomicAdd(&t.hi[h], (uint32_t)(key >> 32) + (old + lo < lo ? 1u : 0u));
    atomicAdd(&t.info[h], info & kInfoCnt);
  }
  atomicOr(&t.info[h], info & (kInfoQ | kInfoP));
}

__device__ __forceinline__ uint32_t hash_mix(uint32_t h) {
  h *= 0x9e3779b1u;
  h ^= h >> 15;
  return h * 0x85ebca6bu;
}

// Merges the classes of a list that have one mask, in place and in order
// (pruning on only); returns the new length, and in `nend` (a prefix length)
// the number of kept classes among the first nend.  The table holds, per hash
// of a mask, the class that stands first among those with a P candidate (or,
// without any, first of all); every other class of the slot with the leader's
// mask joins it, and one with another mask stays as it is (the merge may miss
// some: duplicates are retired later, as single candidates would be).  A list
// longer than the table holds is merged in parts, by hash.  The planes move to
// the new, smaller stride.  S: one word per 32 classes of scratch.
__device__ __noinline__ int cls_merge(uint32_t* m, uint64_t* key, uint32_t* info, int n, int K,
                                      int* stride_io, uint32_t* S, int* nend_io) {
  const int lane = (int)lane_id();
  const MergeTab t = this_tab();
  const size_t st = (size_t)*stride_io;
  constexpr int U = 2;
  // The hashes of U chunks of classes, their loads in flight together.
  const auto hashes = [&](int b, uint32_t* h) {
#pragma unroll
    for (int u = 0; u < U; ++u) h[u] = 0x51ed270bu;
    ROLLED for (int w = 0; w < K; ++w) {
      uint32_t x[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int i = b + 32 * u + lane;
        x[u] = i < n ? m[w * st + i] : 0u;
      }
#pragma unroll
      for (int u = 0; u < U; ++u) h[u] = (h[u] ^ x[u]) * 0x9e3779b1u;
    }
#pragma unroll
    for (int u = 0; u < U; ++u) h[u] = hash_mix(h[u]);
  };
  uint32_t parts = n <= 1024 ? 1u : (n <= 2048 ? 2u : (n <= 4096 ? 4u : (n <= 8192 ? 8u : 16u)));
  if (parts > 1u) {
    // One part is enough where the masks fill no more than half of the table: a
    // pass to see saves the others (8,000 roots, each with up to 7,800 prefixes
    // of a 48-vertex row below it, 46 masks: 20.1 ms a call in eight parts, 18.5
    // so).
    ROLLED for (int b = 0; b < n; b += 32 * U) {
      uint32_t h[U];
      hashes(b, h);
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (b + 32 * u + lane < n) t.lead[h[u] >> 24] = 1u;
    }
    __syncwarp();
    uint32_t used = 0u;
    ROLLED for (int h = lane; h < kSlots; h += 32) {
      used += t.lead[h];
      t.lead[h] = 0u;
    }
    if (__reduce_add_sync(kFull, used) <= kSlots / 2) parts = 1u;
  }
  ROLLED for (int w = lane; w < ((n + 31) >> 5); w += 32) S[w] = first_bits(n, w);
  ROLLED for (uint32_t part = 0; part < parts; ++part) {
    ROLLED for (int b = 0; b < n; b += 32 * U) {
      uint32_t h[U], v[U];
      hashes(b, h);
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int i = b + 32 * u + lane;
        v[u] = 0u;
        if (i < n) {
          v[u] = ((info[i] & kInfoP) ? 0x7fffffffu : 0x3fffffffu) - (uint32_t)i;
        }
      }
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (v[u] && (h[u] & (parts - 1u)) == part) atomicMax(&t.lead[h[u] >> 24], v[u]);
    }
    __syncwarp();
    ROLLED for (int b = 0; b < n; b += 32 * U) {
      int j[U];
      uint32_t h[U];
      hashes(b, h);
      bool gone[U], any = false;
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int i = b + 32 * u + lane;
        j[u] = i;
        if (i < n && (h[u] & (parts - 1u)) == part) {
          const uint32_t v = t.lead[h[u] >> 24];
          j[u] = (int)(v > 0x3fffffffu ? 0x7fffffffu - v : 0x3fffffffu - v);
        }
        gone[u] = j[u] != i;
        any |= gone[u];
      }
      if (!__any_sync(kFull, any)) continue;
      ROLLED for (int w = 0; w < K; ++w) {
        uint32_t x[U], y[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
          x[u] = gone[u] ? m[w * st + b + 32 * u + lane] : 0u;
          y[u] = gone[u] ? m[w * st + j[u]] : 0u;
        }
#pragma unroll
        for (int u = 0; u < U; ++u) gone[u] &= x[u] == y[u];
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int i = b + 32 * u + lane;
        if (gone[u]) {
          const uint32_t f = info[i];
          merge_add(t, h[u] >> 24, (f & kInfoP) ? key[i] : 0ULL, f);
        }
        const unsigned bal = __ballot_sync(kFull, gone[u]);
        if (lane == 0 && bal) S[(b >> 5) + u] &= ~bal;
      }
    }
    __syncwarp();
    // the leaders' sums; the table back to zero
    ROLLED for (int h = lane; h < kSlots; h += 32) {
      const uint32_t v = t.lead[h];
      if (v) {
        const uint32_t f = t.info[h];
        if (f) {
          const int j = (int)(v > 0x3fffffffu ? 0x7fffffffu - v : 0x3fffffffu - v);
          key[j] += (uint64_t)t.lo[h] | ((uint64_t)t.hi[h] << 32);
          info[j] = (info[j] + (f & kInfoCnt)) | (f & (kInfoQ | kInfoP));
          t.lo[h] = t.hi[h] = t.info[h] = 0u;
        }
        t.lead[h] = 0u;
      }
    }
    __syncwarp();
  }
  const int nend = *nend_io;
  int kept = 0, kend = 0;
  ROLLED for (int w = lane; w < ((n + 31) >> 5); w += 32) {
    const uint32_t k = S[w];
    kept += __popc(k);
    kend += __popc(k & first_bits(nend, w));
  }
  kept = (int)__reduce_add_sync(kFull, (unsigned)kept);
  *nend_io = (int)__reduce_add_sync(kFull, (unsigned)kend);
  if (kept == n) return n;
  const size_t ns = (size_t)((kept + 31) & ~31);
  // Every class moves down, plane after plane: what is written lies below
  // everything still to be read.
  ROLLED for (int w = 0; w < K; ++w) {
    int o = 0;
    ROLLED for (int b = 0; b < n; b += 32 * U) {
      uint32_t x[U], bal[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int i = b + 32 * u;
        bal[u] = i < n ? S[i >> 5] : 0u;
        x[u] = (bal[u] >> lane) & 1u ? m[w * st + i + lane] : 0u;
      }
      __syncwarp();
#pragma unroll
      for (int u = 0; u < U; ++u) {
        if ((bal[u] >> lane) & 1u) m[w * ns + o + __popc(bal[u] & lanemask_lt())] = x[u];
        o += __popc(bal[u]);
      }
      __syncwarp();
    }
  }
  int o = 0;
  ROLLED for (int b = 0; b < n; b += 32 * U) {
    uint64_t k[U];
    uint32_t f[U], bal[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int i = b + 32 * u;
      bal[u] = i < n ? S[i >> 5] : 0u;
      const bool mine = (bal[u] >> lane) & 1u;
      k[u] = mine ? key[i + lane] : 0ULL;
      f[u] = mine ? info[i + lane] : 0u;
    }
    __syncwarp();
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if ((bal[u] >> lane) & 1u) {
        const int d = o + __popc(bal[u] & lanemask_lt());
        key[d] = k[u];
        info[d] = f[u];
      }
      o += __popc(bal[u]);
    }
    __syncwarp();
  }
  *stride_io = (int)ns;
  return kept;
}

__device__ __noinline__ void emit_bits(int count, int K, uint32_t mw, const int32_t* lid) {
  emit_words(s_blk.ctl, emit_dst(*s_blk.p), this_warp().gid, count, K, mw, lid);
}

// ---------------------------------------------------------------------------
// Leaf sub-problems: at most 32 classes over at most 32 L vertices.  Lane i
// holds class i's mask, key sum and count, lane b the key of L bit b, and a
// level is four words (live, Q and P classes and L) that every lane knows;
// lane d keeps level d's while a deeper one runs.  A push is then a handful of
// ballots: the walk touches no memory at all.  Maximal bicliques are only
// noted (their L), one per lane, and hashed 32 at a time, every lane its own.
struct Leaf {
  uint32_t m;  // this lane's class: mask
  uint32_t cnt;
  uint64_t key;
  uint64_t lk;  // key of L bit `lane`
  uint32_t A, Q, P, L;
  uint32_t lim;  // classes the first level may push
  uint32_t nR;   // R of the sub-problem's root biclique
  uint64_t sR;
};

// Hashes the noted bicliques (one L per lane, `nb` of them): L's keys over its
// bits, R as the classes of P0 covering it.
__device__ __forceinline__ uint64_t leaf_flush(const Leaf& f, uint32_t P0, uint32_t L0,
                                               uint32_t buf, int nb, int swapped) {
  uint64_t sL = 0, sR = f.sR, nR = f.nR;
  ROLLED for (uint32_t b = L0; b; b &= b - 1) {
    const int i = __ffs(b) - 1;
    const uint64_t k = __shfl_sync(kFull, f.lk, i);
    if ((buf >> i) & 1u) sL += k;
  }
  ROLLED for (uint32_t b = P0; b; b &= b - 1) {
    const int i = __ffs(b) - 1;
    const uint32_t mi = __shfl_sync(kFull, f.m, i);
    const uint64_t k = __shfl_sync(kFull, f.key, i);
    const uint32_t c = __shfl_sync(kFull, f.cnt, i);
    if ((mi & buf) == buf) {
      sR += k;
      nR += c;
    }
  }
  return (int)lane_id() < nb ? biclique_hash_s(swapped, sL, (uint64_t)__popc(buf), sR, nR) : 0ULL;
}

// Hands the child (classes sel, of them p to push and q in Q, L = ln) of a
// leaf sub-problem to an idle warp; all: every class of R of its push.
__device__ __noinline__ bool leaf_export(uint32_t m, uint64_t key, uint32_t cnt,
                                         uint64_t lk, const int32_t* lid, uint64_t sR, uint32_t nR,
                                         uint32_t sel, uint32_t q, uint32_t p, uint32_t ln,
                                         uint32_t all) {
  Warp& W = this_warp();
  const int lane = (int)lane_id();
  const int n = __popc(sel), kn = __popc(ln);
  if (!slot_fits(W, n, 1, cls_levels(kn, __popc(p))) || !should_export(W, __popc(p), kn))
    return false;
  int slot = lane == 0 ? slot_alloc_for(W, n, 1) : 0;
  slot = __shfl_sync(kFull, slot, 0);
  if (slot < 0) return false;
  int32_t* sp = slot_ptr(W, slot);
  const ClsList d = cls_list_at(reinterpret_cast<uint32_t*>(sp + kSlotList), n, 1);
  if ((sel >> lane) & 1u) {
    const int o = __popc(sel & lanemask_lt());
    d.m[o] = m & ln;
    d.key[o] = key;
    d.info[o] = cnt | (((q >> lane) & 1u) ? kInfoQ : 0u) | (((p >> lane) & 1u) ? kInfoP : 0u);
  }
  reinterpret_cast<uint64_t*>(sp + kSlotLk)[lane] = lk;
  if (s_blk.emit) sp[kSlotLid + lane] = lid[lane];
  const bool r = (all >> lane) & 1u;
  const uint64_t sR1 = warp_sum64(r ? key : 0ULL) + sR;
  const uint32_t nR1 = __reduce_add_sync(kFull, r ? cnt : 0u) + nR;
  if (lane == 0) {
    sp[kSlotL] = (int32_t)ln;
    slot_header(sp, 1, n, kn, sR1, nR1, W.gid);
  }
  if (slot_publish(slot, 0)) return true;
  if (lane == 0) slot_free(W, slot);
  __syncwarp();
  return false;
}

// What a walk adds to its warp's totals, in registers.  The two counts go to
// the 64-bit totals at every look at the stop flag: a step adds one to one of
// them at most and some loop of the walk looks whenever `steps` passes a
// multiple of kLookSteps, so that they stay at or below it, however many
// bicliques the sub-problem has.
constexpr uint32_t kLookSteps = 4096;
struct Tally {
  unsigned long long hl;  // this lane's part of the hash sum
  uint32_t cnt, nonmax;   // bicliques found, pushes rejected, since the last look
  uint32_t steps;
  int swapped;
  int share_floor;        // |P|*|L| from which a child may be shared out
};
// Adds the counts to the totals; at a look, whether the walk should stop.
__device__ __noinline__ bool tally_add(uint32_t cnt, uint32_t nonmax, bool look) {
  Warp& W = this_warp();
  acc(W.cnt, cnt);
  acc(W.nonmax, nonmax);
  acc(W.pushes, (unsigned long long)(cnt + nonmax) << 32);
  return look && must_stop();
}
// Counts a step; whether the walk should stop.  `every`: steps between looks, a
// divisor of kLookSteps.
__device__ __forceinline__ bool tally_step(Tally& y, uint32_t every) {
  if ((++y.steps & (every - 1u)) != 0u) return false;
  const bool stop = tally_add(y.cnt, y.nonmax, true);
  y.cnt = y.nonmax = 0u;
  return stop;
}

// Walks a leaf sub-problem (lid: the internal U id of each L bit, for
// emission); false if the launch is stopping.
__device__ __forceinline__ bool leaf_run(Tally& y, const Leaf& f, const int32_t* const* lid) {
  const int lane = (int)lane_id();
  const bool prune = s_blk.prune != 0;
  const uint32_t m = f.m, P0 = f.P;
  uint32_t A = f.A, Q = f.Q, P = f.P, L = f.L, lim = f.lim;
  uint32_t sA = 0, sQ = 0, sP = 0, sL = 0, buf = 0;
  int depth = 0, nb = 0;
  while (true) {
    const uint32_t t = P & A & lim;
    const bool stop = t == 0u && depth == 0;
    if (nb == 32 || (stop && nb > 0)) {
      y.hl += leaf_flush(f, P0, f.L, buf, nb, y.swapped);
      nb = 0;
    }
    if (t == 0u) {
      if (stop) return true;
      --depth;
      A = __shfl_sync(kFull, sA, depth);
      Q = __shfl_sync(kFull, sQ, depth);
      P = __shfl_sync(kFull, sP, depth);
      L = __shfl_sync(kFull, sL, depth);
      if (depth == 0) lim = f.lim;
      continue;
    }
    if (tally_step(y, kLookSteps)) return false;
    // ---- push (finder_push) of class c, and what its pop leaves ----
    const int c = __ffs(t) - 1;
    const uint32_t cb = t & (0u - t);
    const uint32_t mc = __shfl_sync(kFull, m, c);
    const uint32_t ln = L & mc;
    const uint32_t x = m & ln;
    const uint32_t all = __ballot_sync(kFull, x == ln);
    const uint32_t meet = __ballot_sync(kFull, x != 0u);
    const uint32_t out = __ballot_sync(kFull, (m & L & ~mc) != 0u);
    const uint32_t cov = all & A;
    const uint32_t sel = A & meet & ~cov;
    const bool bad = (cov & Q) != 0u;
    if (prune) A &= out | cb;  // retired: nothing outside the popped one's neighbourhood
    P &= ~cb;
    Q |= cb;
    if (bad) {
      ++y.nonmax;
      continue;
    }
    ++y.cnt;
    if (lane == nb) buf = ln;
    ++nb;
    if (s_blk.emit) emit_bits(__popc(ln), 1, ln, *lid);
    const uint32_t p = sel & P;
    const int kn = __popc(ln);
    if (p != 0u && kn > 1) {
      // (a class of an upper level's R covers ln too: all & P0 is all of R)
      if (__popc(p) * kn >= y.share_floor &&
          leaf_export(m, f.key, f.cnt, f.lk, *lid, f.sR, f.nR, sel, sel & Q, p, ln, all & P0))
        continue;
      if (lane == depth) {
        sA = A;
        sQ = Q;
        sP = P;
        sL = L;
      }
      ++depth;
      A = sel;
      Q &= sel;
      P = p;
      L = ln;
      lim = kFull;
    }
  }
}

// ---------------------------------------------------------------------------
// The walk over larger sub-problems: the DFS of IterProcess / finder_push /
// finder_pop, a level at a time.  One sweep over a level's live classes does a
// push and its pop together: which classes cover the new L (absorbed, or a Q
// one that makes the push non-maximal), which go to the child, and which the
// pop retires.  A child that comes down to 32 classes over 32 L vertices is a
// leaf; a larger one gets a list of its own, its masks cut down to the L
// vertices left and merged again, or, when the arena has no room for it, works
// on its parent's list with live, Q and P bits of its own.
struct ClsCur {             // the level being walked, in shared memory
  ClsList l;
  const uint64_t* lk;
  const int32_t* lid;
  uint32_t* A;              // live bits
  const uint32_t* QP;       // the list's Q bits, then its P bits (nwp words each)
  uint32_t *S, *C;          // bits of the child being made, and of the covering classes
  ClsFrame* fr;
  uint32_t *top, *stop;     // first free word of the arena, and of the shared one
  const int32_t* leaf_lid;  // of the leaf being walked (emission)
  uint64_t sR;
  uint32_t nR;
  int nw, nwp;              // words of the bit strings (nwp: the even number from nw)
  int nend;
};
static_assert(sizeof(ClsCur) <= 40 * 4, "shared memory layout");
__device__ __forceinline__ ClsCur& this_cur() {
  return *reinterpret_cast<ClsCur*>(this_smem() + kSmCur);
}

// Word w of a level's Q and P bits, the live classes' at least, while class `at`
// is being pushed.
__device__ __forceinline__ uint32_t q_bits(const ClsCur& c, int at, int w) {
  return c.QP[w] | (c.QP[c.nwp + w] & first_bits(at, w));
}
__device__ __forceinline__ uint32_t p_bits(const ClsCur& c, int at, int w) {
  return c.QP[c.nwp + w] & ~first_bits(at + 1, w);
}

// Visits four words of classes at a time, those whose bit is set in `live`
// (word sb + j for bit j): word(w, x) is called for each of the K mask words
// with x[0..3], this lane's class of each of the four, then done(j) with the
// four's numbers (fewer left: the last one again).  Four loads per lane are in
// flight at once: little else hides a warp's latency.
template <typename Word, typename Done>
__device__ __forceinline__ void cls_words4(const uint32_t* m, int st, int K, int sb, unsigned live,
                                           Word word, Done done) {
  const int lane = (int)lane_id();
  while (live) {
    int j[4], i[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      j[u] = live ? __ffs(live) - 1 : j[u > 0 ? u - 1 : 0];
      live &= live - 1;
      i[u] = (sb + j[u]) * 32 + lane;
    }
    const uint32_t* p = m;
    ROLLED for (int w = 0; w < K; ++w, p += st) {
      uint32_t x[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) x[u] = p[i[u]];
      word(w, x);
    }
    done(j);
  }
}

struct SweepOut {
  bool nm;            // a Q class covers the new L
  int nsel, nselp;    // classes of the child, P classes among them
};

// One push's sweep over the level's live classes.  lnw and rmw (lane w: word
// w) are the new L and the L vertices it leaves; cpos is the pushed class,
// which stays live.  Bits C: the classes covering the new L; bits S: the
// child's.
__device__ __forceinline__ SweepOut cls_sweep(const ClsCur& c, uint32_t lnw, uint32_t rmw,
                                              int cpos) {
  const int lane = (int)lane_id();
  const int K = c.l.K, st = c.l.stride, nw = c.nw;
  const uint32_t* m = c.l.m;
  uint32_t* A = c.A;
  const bool prune = s_blk.prune != 0;
  uint32_t bad = 0u, nsel = 0u, nselp = 0u;
  ROLLED for (int sb = 0; sb < nw; sb += 32) {
    const int wl = sb + lane;
    const bool in = wl < nw;
    const uint32_t aw = in ? A[wl] : 0u;
    const uint32_t qw = in ? q_bits(c, cpos, wl) : 0u;
    const uint32_t pw = in ? p_bits(c, cpos, wl) : 0u;
    uint32_t sel = 0u, out = 0u, cv = 0u;
    uint32_t miss[4] = {0u, 0u, 0u, 0u}, meet[4] = {0u, 0u, 0u, 0u}, leave[4] = {0u, 0u, 0u, 0u};
    cls_words4(
        m, st, K, sb, __ballot_sync(kFull, aw != 0u),
        [&](int w, const uint32_t* x) {
          const uint32_t ln = __shfl_sync(kFull, lnw, w), rm = __shfl_sync(kFull, rmw, w);
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            miss[u] |= ln & ~x[u];
            meet[u] |= ln & x[u];
            leave[u] |= rm & x[u];
          }
        },
        [&](const int* j) {
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const uint32_t b0 = __ballot_sync(kFull, miss[u] == 0u);
            const uint32_t b1 = __ballot_sync(kFull, meet[u] != 0u);
            const uint32_t b2 = __ballot_sync(kFull, leave[u] != 0u);
            miss[u] = meet[u] = leave[u] = 0u;
            if (lane == j[u]) {
              cv = b0;
              sel = b1;
              out = b2;
            }
          }
        });
    cv &= aw;
    sel &= aw & ~cv;
    bad |= cv & qw;
    if (in) {
      if (prune) A[wl] = (aw & out) | (wl == (cpos >> 5) ? 1u << (cpos & 31) : 0u);
      c.S[wl] = sel;
      c.C[wl] = cv;
    }
    nsel += __popc(sel);
    nselp += __popc(sel & pw);
  }
  SweepOut o;
  o.nm = __any_sync(kFull, bad != 0u);
  o.nsel = (int)__reduce_add_sync(kFull, nsel);
  o.nselp = (int)__reduce_add_sync(kFull, nselp);
  return o;
}

// A mask's bits inside ln moved together: bit r of the result is the r-th set
// bit of ln (lane w of lnw: word w, of base: the number of set bits below it).
// Word 0 of the result; the others, up to four, in hi when asked for.
template <bool kHi>
__device__ __forceinline__ uint32_t cls_pack(const uint32_t* m, int stride, int K, uint32_t lnw,
                                             uint32_t base, int i, bool valid, uint32_t* hi) {
  uint32_t lo = 0u;
  if (kHi) hi[0] = hi[1] = hi[2] = 0u;
  ROLLED for (int w = 0; w < K; ++w) {
    const uint32_t lw = __shfl_sync(kFull, lnw, w);
    const uint32_t bw = __shfl_sync(kFull, base, w);
    if (lw == 0u) continue;
    uint32_t x = valid ? m[(size_t)w * stride + i] & lw : 0u;
    ROLLED for (; x; x &= x - 1) {
      const uint32_t r = bw + __popc(lw & ((x & (0u - x)) - 1u));
      const uint32_t bit = 1u << (r & 31);
      if (!kHi) {
        lo |= bit;
      } else {
        const uint32_t ww = r >> 5;
        lo |= ww == 0u ? bit : 0u;
        hi[0] |= ww == 1u ? bit : 0u;
        hi[1] |= ww == 2u ? bit : 0u;
        hi[2] |= ww == 3u ? bit : 0u;
      }
    }
  }
  return lo;
}

// Keys (and ids) of the L bits kept in ln, moved together.
__device__ __noinline__ void cls_pack_keys(const uint64_t* slk, const int32_t* slid, int K,
                                           uint32_t lnw, uint32_t base, uint64_t* lk,
                                           int32_t* lid) {
  const int lane = (int)lane_id();
  ROLLED for (int w = 0; w < K; ++w) {
    const uint32_t lw = __shfl_sync(kFull, lnw, w);
    const uint32_t bw = __shfl_sync(kFull, base, w);
    if ((lw >> lane) & 1u) {
      const uint32_t r = bw + __popc(lw & lanemask_lt());
      lk[r] = slk[w * 32 + lane];
      if (lid) lid[r] = slid[w * 32 + lane];
    }
  }
  __syncwarp();
}

// Writes the child's classes (selection bits S of the push of class cpos) to
// list d: masks cut down to ln, moved together to dK words when that is fewer
// (at most four then).
__device__ __noinline__ void cls_copy_child(uint32_t lnw, uint32_t base, uint32_t* dbase, int dn,
                                            int dK, int cpos) {
  const ClsCur& c = this_cur();
  const int lane = (int)lane_id();
  const ClsList d = cls_list_at(dbase, dn, dK);
  const ClsList l = c.l;
  const bool pack = dK < l.K;
  int o = 0;
  ROLLED for (int b0 = 0; b0 < c.nw; b0 += 32) {
    const uint32_t sl = b0 + lane < c.nw ? c.S[b0 + lane] : 0u;
    ROLLED for (unsigned todo = __ballot_sync(kFull, sl != 0u); todo; todo &= todo - 1) {
      const int j = __ffs(todo) - 1;
      const uint32_t sw = __shfl_sync(kFull, sl, j);
      const int b = b0 + j, i = b * 32 + lane;
      const bool mine = (sw >> lane) & 1u;
      const int t = o + __popc(sw & lanemask_lt());
      if (mine) {
        d.key[t] = l.key[i];
        d.info[t] = (l.info[i] & kInfoCnt) | (((q_bits(c, cpos, b) >> lane) & 1u) ? kInfoQ : 0u) |
                    (((p_bits(c, cpos, b) >> lane) & 1u) ? kInfoP : 0u);
      }
      if (pack) {
        uint32_t hi[3];
        const uint32_t lo = cls_pack<true>(l.m, l.stride, l.K, lnw, base, i, mine, hi);
        if (mine) {
          d.m[t] = lo;
#pragma unroll
          for (int w = 1; w < 4; ++w)
            if (w < dK) d.m[(size_t)w * d.stride + t] = hi[w - 1];
        }
      } else {
        ROLLED for (int w = 0; w < l.K; ++w) {
          const uint32_t lw = __shfl_sync(kFull, lnw, w);
          if (mine) d.m[(size_t)w * d.stride + t] = l.m[(size_t)w * l.stride + i] & lw;
        }
      }
      o += __popc(sw);
    }
  }
  __syncwarp();
}

// Hands the child just selected to an idle warp.
__device__ __noinline__ bool cls_export(uint32_t lnw, uint32_t base, int nsel, int nselp, int kn,
                                        uint64_t sR, uint32_t nR, int cpos) {
  Warp& W = this_warp();
  const ClsCur& c = this_cur();
  const int lane = (int)lane_id();
  const int kc = words_k(kn);
  const int cK = c.l.K, K = kc <= kKMax && kc < cK ? kc : cK;
  if (!slot_fits(W, nsel, K, cls_levels(kn, nselp)) || !should_export(W, nselp, kn)) return false;
  int slot = lane == 0 ? slot_alloc_for(W, nsel, K) : 0;
  slot = __shfl_sync(kFull, slot, 0);
  if (slot < 0) return false;
  int32_t* sp = slot_ptr(W, slot);
  cls_copy_child(lnw, base, reinterpret_cast<uint32_t*>(sp + kSlotList), nsel, K, cpos);
  uint64_t* lk = reinterpret_cast<uint64_t*>(sp + kSlotLk);
  int32_t* lid = s_blk.emit ? sp + kSlotLid : nullptr;
  if (K < cK) {
    cls_pack_keys(c.lk, c.lid, cK, lnw, base, lk, lid);
  } else {
    ROLLED for (int b = lane; b < 32 * K; b += 32) {
      lk[b] = c.lk[b];
      if (lid) lid[b] = c.lid[b];
    }
  }
  if (lane < K) sp[kSlotL + lane] = K < cK ? (int32_t)first_bits(kn, lane) : (int32_t)lnw;
  if (lane == 0) slot_header(sp, K, nsel, kn, sR, nR, W.gid);
  if (slot_publish(slot, 0)) return true;
  if (lane == 0) slot_free(W, slot);
  __syncwarp();
  return false;
}

// The classes of a list of at most 32 one-word classes, a class per lane.
__device__ __forceinline__ void leaf_of_list(const ClsList& l, Leaf& f) {
  const int lane = (int)lane_id();
  const bool in = lane < l.n;
  const uint32_t info = in ? l.info[lane] : 0u;
  f.m = in ? l.m[lane] : 0u;
  f.key = in ? l.key[lane] : 0ULL;
  f.cnt = info & kInfoCnt;
  f.A = first_bits(l.n, 0);
  f.Q = __ballot_sync(kFull, (info & kInfoQ) != 0u);
  f.P = __ballot_sync(kFull, (info & kInfoP) != 0u);
}
// Its L (keys lk), what its first level may push, and R of its root biclique.
__device__ __forceinline__ void leaf_at(Leaf& f, uint32_t L, const uint64_t* lk, uint32_t lim,
                                        uint64_t sR, uint32_t nR) {
  const int lane = (int)lane_id();
  f.L = L;
  f.lk = (L >> lane) & 1u ? lk[lane] : 0ULL;
  f.lim = lim;
  f.sR = sR;
  f.nR = nR;
}

// The indices of the selected classes, in order, into g.
__device__ __forceinline__ void cls_indices(const uint32_t* S, int nw, uint32_t* g) {
  int o = 0;
  if (nw <= 8) {  // a class per lane; more words: a word per lane.  (60 rows of
                  // half of 40 vertices: 7.8 ms a word per lane, 6.6 so.)
    const int lane = (int)lane_id();
    ROLLED for (int w = 0; w < nw; ++w) {
      const uint32_t s = S[w];
      if ((s >> lane) & 1u) g[o + __popc(s & lanemask_lt())] = (uint32_t)(w * 32 + lane);
      o += __popc(s);
    }
    __syncwarp();
    return;
  }
  ROLLED for (int b0 = 0; b0 < nw; b0 += 32) {
    const int w = b0 + (int)lane_id();
    uint32_t s = w < nw ? S[w] : 0u;
    int t;
    int at = o + excl_scan(__popc(s), &t);
    ROLLED for (; s; s &= s - 1) g[at++] = (uint32_t)(w * 32 + __ffs(s) - 1);
    o += t;
  }
  __syncwarp();
}

// A child of 33 to kChildMax selected classes over at most 32 L vertices, its
// classes merged on the way (pruning on): the table (one entry per mask, found
// by probing) keeps each mask's leader and the sums, and the leaders, in order,
// are the child's classes; their number is returned, they themselves go to lm
// (masks), key and info.
__device__ __noinline__ int cls_child(uint32_t lnw, uint32_t base, int nsel, uint32_t* lm,
                                      uint64_t* key, uint32_t* info, int cpos) {
  const ClsCur& c = this_cur();
  const int lane = (int)lane_id();
  const MergeTab t = this_tab();
  uint32_t* g = this_smem() + kSmIdx;
  const bool merge = s_blk.prune != 0;
  const ClsList l = c.l;
  cls_indices(c.S, c.nw, g);
  const uint32_t ln0 = __shfl_sync(kFull, lnw, 0);
  int n = 0;
  // Without merging every class is its own leader: one pass.
  ROLLED for (int pass = merge ? 0 : 1; pass < 2; ++pass) {
    ROLLED for (int b = 0; b < nsel; b += 32) {
      const int at = b + lane;
      const bool in = at < nsel;
      uint32_t x = 0u, f = 0u, h = 0u;
      uint64_t k = 0ULL;
      const int i = in ? (int)g[at] : 0;  // the class, or (second pass) its entry
      if (pass == 0 || !merge) {
        // (one-word masks keep their bits where they are)
        x = l.K == 1 ? (in ? l.m[i] & ln0 : 0u)
                     : cls_pack<false>(l.m, l.stride, l.K, lnw, base, i, in, nullptr);
        if (in) {
          f = (((q_bits(c, cpos, i >> 5) >> (i & 31)) & 1u) << 31) |
              (((p_bits(c, cpos, i >> 5) >> (i & 31)) & 1u) << 30);
          if (f & kInfoP) {
            f |= l.info[i] & kInfoCnt;
            k = l.key[i];
          }
        }
      }
      if (pass == 0) {
        if (x) {
          h = hash_mix(x) >> 24;
          while (true) {
            const uint32_t old = atomicCAS(&t.mask[h], 0u, x);
            if (old == 0u || old == x) break;
            h = (h + 1) & (kSlots - 1);
          }
          // the earlier the larger, P classes first
          const uint32_t rank = ((f & kInfoP) ? 0x8000u : 0x4000u) - (uint32_t)at;
          atomicMax(&t.lead[h], rank);
          merge_add(t, h, k, f);
          g[at] = h;
        }
      } else {
        bool is = x != 0u;
        if (merge && in) {
          h = (uint32_t)i;
          const uint32_t v = t.lead[h];
          is = (v > 0x4000u ? 0x8000u : 0x4000u) - v == (uint32_t)at;
          if (is) {
            x = t.mask[h];
            f = t.info[h];
            k = (uint64_t)t.lo[h] | ((uint64_t)t.hi[h] << 32);
          }
        }
        const unsigned bal = __ballot_sync(kFull, is);
        if (is) {
          const int r = n + __popc(bal & lanemask_lt());
          lm[r] = x;
          key[r] = k;
          info[r] = f;
        }
        n += __popc(bal);
      }
    }
    __syncwarp();
  }
  if (merge) {
    ROLLED for (int at = lane; at < nsel; at += 32) {
      const uint32_t h = g[at];
      t.mask[h] = t.lead[h] = t.lo[h] = t.hi[h] = t.info[h] = 0u;
    }
  }
  __syncwarp();
  return n;
}

// A level: live bits and a frame.  last < 0: for a fresh list (masks at l.m),
// whose Q and P bits are made here too; else on the parent's list, where class
// `last` was pushed, for the classes selected there.
__device__ __noinline__ void cls_enter(ClsList l, uint32_t L, int nend, const uint64_t* lk,
                                       const int32_t* lid, uint64_t sR, uint32_t nR,
                                       uint32_t* top, uint32_t* stop, int last) {
  ClsCur& c = this_cur();
  const int lane = (int)lane_id();
  const uint32_t* send = this_smem() + kSmemWords;
  ClsFrame* fr = reinterpret_cast<ClsFrame*>(top);
  const int nw = (l.n + 31) >> 5, nwp = (nw + 1) & ~1;
  const int bits = last < 0 ? 3 * nwp : nwp;
  uint32_t* Lw = top + kFrameWords;
  top = Lw + ((l.K + 1) & ~1);
  uint32_t* A;
  if (bits <= send - stop) {
    A = stop;
    stop += bits;
  } else {
    A = top;
    top += bits;
  }
  const uint32_t* QP = c.QP;
  if (last < 0) {  // everything is live, Q and P as the info words say
    uint32_t *Q = A + nwp, *P = Q + nwp;
    QP = Q;
    ROLLED for (int b = 0; b < nw; ++b) {
      const int i = b * 32 + lane;
      const uint32_t f = i < l.n ? l.info[i] : 0u;
      const uint32_t q = __ballot_sync(kFull, (f & kInfoQ) != 0u);
      const uint32_t p = __ballot_sync(kFull, (f & kInfoP) != 0u);
      if (lane == 0) {
        A[b] = first_bits(l.n, b);
        Q[b] = q;
        P[b] = p;
      }
    }
    // The masks too, when there is room.
    const int words = l.K * l.stride;
    if (words <= send - stop && (l.m < this_smem() || l.m >= send)) {
      ROLLED for (int i = lane; i < words; i += 32) stop[i] = l.m[i];
      l.m = stop;
      stop += words;
    }
  } else {
    const uint32_t* S = c.S;
    ROLLED for (int b = lane; b < nw; b += 32) A[b] = S[b];
  }
  if (lane < l.K) Lw[lane] = L;
  ClsFrame* prev = c.fr;
  __syncwarp();
  if (lane == 0) {
    fr->l = l;
    fr->lk = lk;
    fr->lid = lid;
    fr->sR = sR;
    fr->prev = prev;
    fr->A = A;
    fr->QP = QP;
    fr->top = top;
    fr->stop = stop;
    fr->nR = nR;
    fr->nend = nend;
    fr->last = last;
    c.l = l;
    c.lk = lk;
    c.lid = lid;
    c.A = A;
    c.QP = QP;
    c.fr = fr;
    c.top = top;
    c.stop = stop;
    c.nw = nw;
    c.nwp = nwp;
    c.sR = sR;
    c.nR = nR;
    c.nend = nend;
  }
  __syncwarp();
}

// Back to the level above (false: there is none); its L in L (lane w: word w),
// and the class it pushed last in `last`.
__device__ __forceinline__ bool cls_leave(ClsCur& c, uint32_t& L, int& last) {
  const int lane = (int)lane_id();
  const ClsFrame* fr = c.fr->prev;
  if (!fr) return false;
  __syncwarp();
  const int K = fr->l.K;
  L = lane < K ? (reinterpret_cast<const uint32_t*>(fr) + kFrameWords)[lane] : 0u;
  last = fr->last;
  if (lane == 0) {
    c.l = fr->l;
    c.lk = fr->lk;
    c.lid = fr->lid;
    c.nw = (fr->l.n + 31) >> 5;
    c.nwp = (c.nw + 1) & ~1;
    c.A = fr->A;
    c.QP = fr->QP;
    c.fr = const_cast<ClsFrame*>(fr);
    c.top = fr->top;
    c.stop = fr->stop;
    c.sR = fr->sR;
    c.nR = fr->nR;
    c.nend = fr->nend;
  }
  __syncwarp();
  return true;
}

// Starts a sub-problem: merges its list, sets up the first level.  True if the
// list came down to a leaf, left as l.
__device__ __noinline__ bool cls_begin(ClsList* lp, uint32_t L, int* nend, const uint64_t* lk,
                                       const int32_t* lid, uint64_t sR0, uint32_t nR0,
                                       uint32_t* top) {
  ClsCur& c = this_cur();
  uint32_t* sm = this_smem();
  ClsList l = *lp;
  uint32_t* S = top;
  uint32_t* C = top + cls_bit_words(l.n);
  top += 2 * cls_bit_words(l.n);
  if (s_blk.prune && l.n > 32) l.n = cls_merge(l.m, l.key, l.info, l.n, l.K, &l.stride, S, nend);
  *lp = l;
  if (l.n <= 32 && l.K == 1) return true;
  // The two bit strings a push makes go to the shared arena.
  uint32_t* stop = sm + kSmArena;
  const int nwp = (int)cls_bit_words(l.n);
  if (2 * nwp <= sm + kSmemWords - stop) {
    S = stop;
    C = stop + nwp;
    stop += 2 * nwp;
  }
  __syncwarp();
  if (lane_id() == 0) {
    c.fr = nullptr;
    c.S = S;
    c.C = C;
  }
  __syncwarp();
  cls_enter(l, L, *nend, lk, lid, sR0, nR0, top, stop, -1);
  return false;
}

// A maximal push's biclique: R (the covering classes, all of them live P ones)
// into sR and nR, its hash returned.
__device__ __forceinline__ uint64_t cls_biclique(const ClsCur& c, uint32_t lnw, int kn, int swapped,
                                                 uint64_t& sR, uint32_t& nR) {
  const int lane = (int)lane_id();
  sR = 0;
  nR = 0;
  uint64_t sL = 0;
  const uint32_t* C = c.C;
  ROLLED for (int w = lane; w < c.nw; w += 32)
    ROLLED for (uint32_t b = C[w]; b; b &= b - 1) {
      const int i = w * 32 + __ffs(b) - 1;
      sR += c.l.key[i];
      nR += c.l.info[i] & kInfoCnt;
    }
  const uint64_t* lk = c.lk;
  ROLLED for (int w = 0; w < c.l.K; ++w)
    if ((__shfl_sync(kFull, lnw, w) >> lane) & 1u) sL += lk[w * 32 + lane];
  sR = warp_sum64(sR) + c.sR;
  nR = __reduce_add_sync(kFull, nR) + c.nR;
  sL = warp_sum64(sL);
  return biclique_hash_s(swapped, sL, (uint64_t)kn, sR, (uint64_t)nR);
}

// Runs a sub-problem: the list l (in the warp's scratch; its classes may be
// merged), L words `L` (lane w: word w), the first level pushing classes
// [0, nend) only.  [top, end) is the arena.
__device__ __noinline__ void cls_run(ClsList l, uint32_t L, int nend, const uint64_t* lk,
                                     const int32_t* lid, uint64_t sR0, uint64_t nR0, uint32_t* top,
                                     uint32_t* end) {
  const int lane = (int)lane_id();
  const uint64_t t0 = globaltimer_ns();
  ClsCur& c = this_cur();
  Tally y;
  y.hl = 0;
  y.cnt = y.nonmax = y.steps = 0;
  {
    const DevGraph* g = this_warp().gp;
    y.swapped = g->swapped;
    y.share_floor =
        s_blk.nslot == 0 ? INT_MAX : min(s_blk.share_min_work, max(g->bound_size, 0));
  }
  unsigned long long hash = 0;
  Leaf f;
  int last = -1;
  bool leaf = cls_begin(&l, L, &nend, lk, lid, sR0, (uint32_t)nR0, top);
  const bool root_leaf = leaf;
  if (leaf) {
    leaf_of_list(l, f);
    leaf_at(f, __shfl_sync(kFull, L, 0), lk, first_bits(nend, 0), sR0, (uint32_t)nR0);
    if (lane == 0) c.leaf_lid = lid;
    __syncwarp();
  }
  while (true) {
    if (leaf) {
      leaf = false;
      if (!leaf_run(y, f, &c.leaf_lid) || root_leaf) break;
    }
    // ---- the next class to push: the first live P one ----
    int cpos = -1;
    {
      const uint32_t* A = c.A;
      const int nw = c.nw, e = c.nend;
      ROLLED for (int b0 = (last + 1) >> 5; b0 < nw; b0 += 32) {
        const int w = b0 + lane;
        const uint32_t t = w < nw ? A[w] & p_bits(c, last, w) & first_bits(e, w) : 0u;
        const unsigned bal = __ballot_sync(kFull, t != 0u);
        if (bal) {
          const int j = __ffs(bal) - 1;
          cpos = (b0 + j) * 32 + __ffs(__shfl_sync(kFull, t, j)) - 1;
          break;
        }
      }
    }
    if (cpos < 0) {
      if (!cls_leave(c, L, last)) break;
      continue;
    }
    if (tally_step(y, 1024u)) break;
    last = cpos;
    const int K = c.l.K;
    const uint32_t mc = lane < K ? c.l.m[(size_t)lane * c.l.stride + cpos] : 0u;
    const uint32_t lnw = L & mc, rmw = L & ~mc;
    const int kn = (int)__reduce_add_sync(kFull, (unsigned)__popc(lnw));
    const SweepOut o = cls_sweep(c, lnw, rmw, cpos);
    if (o.nm) {
      ++y.nonmax;
      continue;
    }
    ++y.cnt;
    uint64_t sR;
    uint32_t nR;
    hash += cls_biclique(c, lnw, kn, y.swapped, sR, nR);
    if (s_blk.emit) emit_bits(kn, K, lnw, c.lid);
    const int nsel = o.nsel, nselp = o.nselp;
    if (kn <= 1 || nselp == 0) continue;
    // Bits of the new L below each word (lane w: word w).
    uint32_t base = 0u;
    if (K > 1) {
      int tot;
      base = (uint32_t)excl_scan(__popc(lnw), &tot);
    }
    // A big enough child goes to an idle warp instead, at any depth, so that a
    // subtree that started here can still be shared once warps run out of work.
    if (nselp * (long long)kn >= y.share_floor &&
        cls_export(lnw, base, nsel, nselp, kn, sR, nR, cpos))
      continue;
    const int kc = words_k(kn);
    const int dK = kc <= kKMax && kc < K ? kc : K;
    const bool pack = dK < K;
    const long long keys = pack ? 64LL * dK + (s_blk.emit ? 32LL * dK : 0) : 0;
    const bool tiny = kn <= 32 && nsel <= 32;
    uint32_t* at = c.top;
    if (lane == 0) c.fr->last = cpos;
    if (!tiny && cls_need(nsel, dK, cls_levels(kn, nselp)) + keys > end - at) {
      // ---- no room: a level on the parent's list ----
      cls_enter(c.l, lnw, c.l.n, c.lk, c.lid, sR, nR, at, c.stop, cpos);
      L = lnw;
      continue;
    }
    const uint64_t* clk = c.lk;
    const int32_t* clid = c.lid;
    if (pack) {
      uint64_t* nlk = reinterpret_cast<uint64_t*>(at);
      int32_t* nlid = s_blk.emit ? reinterpret_cast<int32_t*>(at + 64 * dK) : nullptr;
      cls_pack_keys(clk, clid, K, lnw, base, nlk, nlid);
      clk = nlk;
      clid = nlid;
      at += keys;
    }
    const uint32_t nl = pack ? first_bits(kn, lane) : lnw;
    if (tiny) {
      // ---- straight into the lanes ----
      uint32_t* g = this_smem() + kSmIdx;
      cls_indices(c.S, c.nw, g);
      const bool in = lane < nsel;
      const int i = in ? (int)g[lane] : 0;
      f.A = first_bits(nsel, 0);
      f.Q = __ballot_sync(kFull, in && ((q_bits(c, cpos, i >> 5) >> (i & 31)) & 1u));
      f.P = __ballot_sync(kFull, in && ((p_bits(c, cpos, i >> 5) >> (i & 31)) & 1u));
      const bool p = (f.P >> lane) & 1u;
      f.key = p ? c.l.key[i] : 0ULL;
      f.cnt = p ? c.l.info[i] & kInfoCnt : 0u;
      if (K == 1) {
        const uint32_t l0 = __shfl_sync(kFull, lnw, 0);
        f.m = in ? c.l.m[i] & l0 : 0u;
      } else {
        f.m = cls_pack<false>(c.l.m, c.l.stride, K, lnw, base, i, in, nullptr);
      }
      leaf = true;
    } else {
      ClsList d = cls_list_at(at, nsel, dK);
      uint32_t* stop = c.stop;
      if (kn <= 32 && nsel <= kChildMax) {
        uint32_t* lm = d.m;
        if (d.stride <= this_smem() + kSmemWords - stop) lm = stop;
        d.n = cls_child(lnw, base, nsel, lm, d.key, d.info, cpos);
        d.stride = (d.n + 31) & ~31;
        d.m = lm;
        leaf = d.n <= 32;
        if (leaf) leaf_of_list(d, f);
        else if (lm == stop) stop += d.stride;
      } else {
        cls_copy_child(lnw, base, d.m, nsel, dK, cpos);
        int dend = nsel;
        if (s_blk.prune && nsel > 32)
          d.n = cls_merge(d.m, d.key, d.info, nsel, dK, &d.stride, c.S, &dend);
        if (d.n <= 32 && dK == 1) {
          leaf_of_list(d, f);
          leaf = true;
        }
      }
      if (!leaf) {
        cls_enter(d, nl, d.n, clk, clid, sR, nR, at + cls_list_words(nsel, dK), stop, -1);
        L = lane < dK ? nl : 0u;
        last = -1;
      }
    }
    if (leaf) {
      leaf_at(f, __shfl_sync(kFull, nl, 0), clk, kFull, sR, nR);
      __syncwarp();
      if (lane == 0) c.leaf_lid = clid;
      __syncwarp();
    }
  }
  hash += warp_sum64(y.hl);
  tally_add(y.cnt, y.nonmax, false);
  Warp& W = this_warp();
  acc(W.hash, hash);
  acc(W.ns_t2, globaltimer_ns() - t0);
  acc(W.n_t2, 1);
  __syncwarp();
}

// Sub-problem list in the warp's own scratch over n L vertices (all bits):
// [top, ...) is what follows the list.
__device__ __forceinline__ void tier2(Warp& W, const ClsList& l, int n, int nend, uint64_t sR0,
                                      uint64_t nR0) {
  cls_run(l, first_bits(n, (int)lane_id()), nend, W.A64(W.sl().lkey), W.A(W.sl().lid), sR0, nR0,
          l.m + cls_list_words(l.n, l.K), reinterpret_cast<uint32_t*>(W.A(W.sl().ar_end)));
}

// Runs an exported sub-problem and releases its slot.  The slot was written
// by another warp, possibly on another SM, and this SM may hold lines of it
// from an older owner in its (non-coherent) L1: the header is read with
// volatile loads and the body is copied through L2 (ld.global.cg) into this
// warp's own scratch, where the sub-problem then runs.  The slot is freed as
// soon as it is copied; nothing here writes it, so no store can land on the
// classes of its next owner.
__device__ __noinline__ void tier2_from_slot(int slot) {
  Warp& W = this_warp();
  const int lane = (int)lane_id();
  int32_t* sp = slot_ptr(W, slot);
  volatile const int32_t* vh = sp;
  const int K = vh[0];
  const int n = vh[1];
  const int32_t gid = vh[3];
  const uint64_t sR = (uint64_t)(uint32_t)vh[4] | ((uint64_t)(uint32_t)vh[5] << 32);
  const uint64_t nR = (uint32_t)vh[6];
  const uint32_t L = lane < K ? (uint32_t)vh[kSlotL + lane] : 0u;
  uint32_t* at = reinterpret_cast<uint32_t*>(W.A(W.sl().ar_root));
  uint64_t* lkey = reinterpret_cast<uint64_t*>(at);
  int32_t* lid = reinterpret_cast<int32_t*>(at + 64 * K);
  const ClsList l = cls_list_at(at + cls_key_words(K), n, K);
  const int nw = (int)cls_list_words(n, K);
  const uint4* src = reinterpret_cast<const uint4*>(sp + kSlotList);
#pragma unroll 4
  for (int i = lane; i < nw / 4; i += 32) reinterpret_cast<uint4*>(l.m)[i] = __ldcg(src + i);
  const unsigned long long* slk = reinterpret_cast<const unsigned long long*>(sp + kSlotLk);
  ROLLED for (int i = lane; i < 32 * K; i += 32) lkey[i] = __ldcg(slk + i);
  const unsigned* sli = reinterpret_cast<const unsigned*>(sp + kSlotLid);
  if (s_blk.emit)
    ROLLED for (int i = lane; i < 32 * K; i += 32) lid[i] = (int32_t)__ldcg(sli + i);
  __syncwarp();
  if (lane == 0) slot_free(W, slot);
  __syncwarp();
  W.gid = gid;
  W.gp = graph_at(W, gid);
  __syncwarp();
  cls_run(l, L, n, lkey, lid, sR, nR, l.m + nw, reinterpret_cast<uint32_t*>(W.A(W.sl().ar_end)));
}

// The edges between a sub-problem's candidates and its vertices: edge e joins
// candidate tab[ids[e]] - bias (below 0: none) and vertex rows[e]; without
// rows, ids holds both, id << 7 | vertex.  Without ids (n = 0), vertex r's are
// the ids col[off[L[r]] .. off[L[r] + 1]) (below 0: none).
struct ClsEdges {
  const int32_t *ids, *rows, *tab;
  int n, bias;
  const int32_t *L, *off, *col;
};

// The candidates of a list being built that get masks (bits and ranks, MB and
// MP), and their masks (K planes of st words).
struct ClsRaw {
  const uint32_t *MB, *MP;
  uint32_t* raw;
  int st, nq;
};

// An edge between candidate i and vertex r: a bit of the candidate's mask, or,
// where it gets none, into the vertex's sums.
__device__ __forceinline__ void cls_edge(const ClsRaw& b, const MergeTab& t, const uint64_t* keys,
                                         const int32_t* vidx, int i, int r) {
  const uint32_t w = b.MB[i >> 5], bit = 1u << (i & 31);
  if (w & bit) {
    const uint32_t d = b.MP[i >> 5] + __popc(w & (bit - 1u));
    atomicOr(&b.raw[(size_t)(r >> 5) * b.st + d], 1u << (r & 31));
  } else if (i < b.nq) {
    atomicOr(&t.info[r], kInfoQ);
  } else {
    atomicMax(&t.lead[r], 0x7fffffffu - (uint32_t)i);
    const int v = vidx[i];
    const uint64_t k = keys[v < 0 ? ~v : v];
    const uint32_t lo = (uint32_t)k;
    const uint32_t old = atomicAdd(&t.lo[r], lo);
    atomicAdd(&t.hi[r], (uint32_t)(k >> 32) + (old + lo < lo ? 1u : 0u));
    atomicAdd(&t.info[r], 1u);
  }
}

// All edges of rows that are not laid out.
__device__ __noinline__ void cls_edges_of_rows(ClsRaw b, const uint64_t* keys, const int32_t* vidx,
                                               ClsEdges ed, int nL) {
  const MergeTab t = this_tab();
  flat_rows2(
      nL,
      [&](int r, int& beg, int& len) {
        const int u = ed.L[r];
        beg = ed.off[u];
        len = ed.off[u + 1] - beg;
      },
      [&](bool valid, int pos) { return valid ? ed.col[pos] : -1; },
      [&](int w) { return w >= 0 ? ed.tab[w] - ed.bias : -1; },
      [&](bool, int r, int, int, int i) {
        if (i >= 0) cls_edge(b, t, keys, vidx, i, r);
      });
}

// Builds the class list of n candidates, [Q | P], the first nq of them Q, over
// nL vertices, at `at` ([at, end): at least cls_list_words + cls_build_words).
// Candidate i has cnt[i] of the vertices and hash key keys[vidx[i]]; without
// cnt, vidx[i] is complemented if it has one of them only.  *nend: candidates
// [0, nend) may be pushed at the first level; classes [0, nend) on return.
// mpos: room for n words, or null (it is taken from the end then).
//
// Most candidates of a root have one of its vertices only (on the 300,000-edge
// serving graph a root has 1,565 candidates and 1,867 edges to them).  Those
// need no record: the candidates of one vertex are one class from the start,
// summed up per vertex as the edges are walked, and only the others get masks.
__device__ __noinline__ ClsList cls_build(uint32_t* at, uint32_t* end, int n, int nq, int K, int nL,
                                          int* nend, const int32_t* cnt, const uint64_t* keys,
                                          const int32_t* vidx, ClsEdges ed, uint32_t* mpos) {
  const int lane = (int)lane_id();
  const bool merge = s_blk.prune != 0;
  const int nw = (n + 31) >> 5;
  // Bits and ranks of the candidates with masks (M) and of all classes (F).
  uint32_t* sm = this_smem() + kSmArena;
  uint32_t* send = this_smem() + kSmemWords;
  uint32_t* MB;
  if (4 * nw <= send - sm) {
    MB = sm;
    sm += 4 * nw;
  } else {
    end -= 4 * ((nw + 1) & ~1);
    MB = end;
  }
  uint32_t *MP = MB + nw, *FB = MP + nw, *FP = FB + nw;
  int nm = 0;
#pragma unroll 2
  for (int b = 0; b < nw; ++b) {
    const int i = b * 32 + lane;
    const unsigned bal =
        __ballot_sync(kFull, i < n && (!merge || (cnt ? cnt[i] >= 2 : vidx[i] >= 0)));
    if (lane == 0) {
      MB[b] = FB[b] = bal;
      MP[b] = (uint32_t)nm;
    }
    nm += __popc(bal);
  }
  const int st = (nm + 31) & ~31;
  if (!mpos) {
    end -= st;
    mpos = end;  // candidate of each mask
  }
  const auto key_of = [&](int i) {
    const int v = vidx[i];
    return keys[v < 0 ? ~v : v];
  };
  uint32_t* raw;
  if (K * st <= send - sm) {
    raw = sm;
  } else {
    end -= (size_t)K * st;
    raw = end;
  }
  ROLLED for (int i = lane; i < K * st; i += 32) raw[i] = 0u;
  // Sums per vertex: the table's entries.
  static_assert(32 * kKMax <= kSlots, "an entry per vertex");
  const MergeTab t = this_tab();
  uint32_t* first = t.lead;  // 0x7fffffff - the first P candidate, or 0
  uint32_t* info = t.info;
  __syncwarp();
  ROLLED for (int w = lane; w < nw; w += 32) {
    const uint32_t o = MP[w];
    int k = 0;
    ROLLED for (uint32_t b = MB[w]; b; b &= b - 1) mpos[o + k++] = (uint32_t)(w * 32 + __ffs(b) - 1);
  }
  __syncwarp();
  const ClsRaw b{MB, MP, raw, st, nq};
  if (!ed.ids) cls_edges_of_rows(b, keys, vidx, ed, nL);
  ROLLED for (int e0 = 0; e0 < ed.n; e0 += 64) {
    int id[2], ci[2];
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int e = e0 + 32 * u + lane;
      id[u] = e < ed.n ? ed.ids[e] : -1;
    }
#pragma unroll
    for (int u = 0; u < 2; ++u)
      ci[u] = id[u] >= 0 ? ed.tab[ed.rows ? id[u] : id[u] >> 7] - ed.bias : -1;
#pragma unroll
    for (int u = 0; u < 2; ++u)
      if (ci[u] >= 0)
        cls_edge(b, t, keys, vidx, ci[u], ed.rows ? ed.rows[e0 + 32 * u + lane] : id[u] & 127);
  }
  __threadfence_block();
  __syncwarp();
  int nqs = 0;  // vertices whose only candidates are Q
  ROLLED for (int r0 = 0; r0 < nL; r0 += 32) {
    const int r = r0 + lane;
    const uint32_t v = r < nL ? first[r] : 0u;
    if (v) {
      const uint32_t i = 0x7fffffffu - v;
      atomicOr(&FB[i >> 5], 1u << (i & 31));
    }
    nqs += __popc(__ballot_sync(kFull, r < nL && !v && (info[r] & kInfoQ)));
  }
  __syncwarp();
  int nf = 0;
  ROLLED for (int w0 = 0; w0 < nw; w0 += 32) {
    const int w = w0 + lane;
    int tot;
    const int ex = excl_scan(w < nw ? __popc(FB[w]) : 0, &tot);
    if (w < nw) FP[w] = (uint32_t)(nf + ex);
    nf += tot;
  }
  __syncwarp();
  // Classes before candidate i, the Q-only vertices' (they stand after the
  // other Q classes) left out.
  const auto rank = [&](int i) {
    return i >= n ? nf : (int)FP[i >> 5] + __popc(FB[i >> 5] & ((1u << (i & 31)) - 1u));
  };
  const int nqm = rank(nq);
  *nend = rank(*nend) + nqs;
  const ClsList l = cls_list_at(at, nf + nqs, K);
  ROLLED for (int d = lane; d < nm; d += 32) {
    const int i = (int)mpos[d];
    const int f = rank(i) + (i >= nq ? nqs : 0);
    ROLLED for (int w = 0; w < K; ++w) l.m[(size_t)w * l.stride + f] = raw[(size_t)w * st + d];
    l.info[f] = i < nq ? kInfoQ : kInfoP | 1u;
    // Only P candidates' keys can enter an R that is counted.
    l.key[f] = i < nq ? 0ULL : key_of(i);
  }
  int oq = nqm;
  ROLLED for (int r0 = 0; r0 < nL; r0 += 32) {
    const int r = r0 + lane;
    const uint32_t v = r < nL ? first[r] : 0u;
    const uint32_t fl = r < nL ? info[r] : 0u;
    const unsigned bal = __ballot_sync(kFull, !v && fl != 0u);
    if (v || fl) {
      const int f = v ? rank((int)(0x7fffffffu - v)) + nqs : oq + __popc(bal & lanemask_lt());
      ROLLED for (int w = 0; w < K; ++w)
        l.m[(size_t)w * l.stride + f] = w == (r >> 5) ? 1u << (r & 31) : 0u;
      l.info[f] = fl | (v ? kInfoP : 0u);
      l.key[f] = (uint64_t)t.lo[r] | ((uint64_t)t.hi[r] << 32);
      first[r] = info[r] = t.lo[r] = t.hi[r] = 0u;
    }
    oq += __popc(bal);
  }
  __syncwarp();
  return l;
}

// ---------------------------------------------------------------------------
// Tier 1: GMBE counts + level bounds over the task's C, local adjacency.
struct T1 {
  const int32_t* L;   // L vertices (internal U ids)
  int nL, nC, nq;
  int nend;  // the first level pushes positions [nq, nend) only
  uint64_t sRtask, nRtask;
};

// What a walk over rows does at each entry's candidate p.
enum T1Op {
  kOpAdd,      // count it
  kOpSub,      // take its count back
  kOpRestore,  // count it, and mark it touched if its bound is at least `level`
  kOpRetire,   // retire it below `level` unless touched (or x itself)
  kOpFree,     // touched: free again
  kOpSetBit,   // its bit in bits
  kOpClearBit, // its word in bits to zero
};

// Walks rows of aadj: with x >= 0 the rows of candidate x's L positions (cadj)
// whose llevel is lvl (those a push of x keeps, found without a pass over all
// of L), else every L position with llevel == lvl.  One function for all walks
// of a push and a pop: inlined at each of them, the walk was a third of the
// counts tier's code.
__device__ __noinline__ void t1_walk(int nL, int x, int lvl, int op, int level, uint32_t* bits) {
  Warp& W = this_warp();
  const int32_t* llevel = W.A(W.sl().llevel);
  const int32_t* aoff = W.A(W.sl().aoff);
  const int32_t* aadj = W.A(W.sl().aadj);
  const int32_t* cadj = W.A(W.sl().cadj);
  int32_t* ncnt = W.A(W.sl().ncnt);
  int32_t* bound = W.A(W.sl().bound);
  const int lane = (int)lane_id();
  int rb = 0, re = nL;
  if (x >= 0) {
    const int32_t* coff = W.A(W.sl().coff);
    rb = coff[x];
    re = coff[x + 1];
  }
  const int xx = x;
  // Only these read bounds; the others do not wait for an entry before they ask
  // for the next (pruning off, 900 candidates below a row of 140 vertices:
  // 552 -> 485 ms).
  const bool bounds = op >= kOpRestore && op <= kOpFree;
  ROLLED for (int c0 = rb; c0 < re; c0 += 32) {
    const int j = c0 + lane;
    const int l = j < re ? (x >= 0 ? cadj[j] : j) : 0;
    const unsigned bal = __ballot_sync(kFull, j < re && llevel[l] == lvl);
    const int nsel = __popc(bal);
    if (nsel == 0) continue;
    // Lane k takes the k-th selected row of the chunk.
    unsigned m = bal;
    ROLLED for (int k = 0; k < lane && m; ++k) m &= m - 1;
    const int row = __shfl_sync(kFull, l, m ? __ffs(m) - 1 : 0);
    flat_rows2(
        nsel,
        [&](int, int& beg, int& len) {
          beg = aoff[row];
          len = aoff[row + 1] - beg;
        },
        [&](bool valid, int pos) { return valid ? aadj[pos] : -1; },
        [&](int p) { return bounds && p >= 0 ? bound[p] : 0; },
        [&](bool, int, int, int p, int b) {
          if (p < 0) return;
          switch (op) {
            case kOpAdd: atomicAdd(&ncnt[p], 1); break;
            case kOpSub: atomicSub(&ncnt[p], 1); break;
            case kOpRestore:
              atomicAdd(&ncnt[p], 1);
              if (b >= level) bound[p] = kTouched;
              break;
            case kOpRetire:
              if (p != xx && b >= level && b != kTouched) bound[p] = level - 1;
              break;
            case kOpFree:
              if (b == kTouched) bound[p] = kFree;
              break;
            case kOpSetBit: atomicOr(&bits[p >> 5], 1u << (p & 31)); break;
            default: bits[p >> 5] = 0u; break;
          }
        });
  }
  __threadfence_block();
  __syncwarp();
}

// finder_pop (src/IterFinderGpu.h:266-303) of candidate x at `level`, walking
// only the rows of the level above it: the removed rows (llevel == level-1)
// restore their counts and mark the candidates they meet, and the kept rows
// (llevel == level, the rows of x) decide the pruning.  A pass over every
// candidate is not needed: a candidate adjacent to neither kept nor removed
// rows has count 0 at this level and every level below it, so no push, scan,
// maximality test or later pop at or below this level reads its bound, and
// the pop one level up treats every bound >= level-1 alike.
__device__ __noinline__ void t1_pop(int nL, int x, int level) {
  Warp& W = this_warp();
  int32_t* llevel = W.A(W.sl().llevel);
  int32_t* bound = W.A(W.sl().bound);
  const int32_t* coff = W.A(W.sl().coff);
  const int32_t* cadj = W.A(W.sl().cadj);
  const int lane = (int)lane_id();
  // restore counts over L_parent \ L_child and mark touched candidates
  t1_walk(nL, -1, level - 1, kOpRestore, level, nullptr);
  if (s_blk.prune) {
    // Candidates of the kept rows that no removed row met are retired at this
    // level (a candidate in several kept rows is visited several times: the
    // write is the same each time, and touched ones are left for the pass
    // below).
    t1_walk(nL, x, level, kOpRetire, level, nullptr);
    // touched candidates -> free
    t1_walk(nL, -1, level - 1, kOpFree, level, nullptr);
  }
  if (lane == 0) bound[x] = kFree;
  __syncwarp();
  // the kept rows go back to the level above (deeper levels are popped already)
  ROLLED for (int j = coff[x] + lane; j < coff[x + 1]; j += 32) {
    const int l = cadj[j];
    if (llevel[l] == level) llevel[l] = level - 1;
  }
  __syncwarp();
}

// Hands the child sub-problem of a maximal push (x at `level`, |L_new| = kept)
// to tier 2.  Candidates: C entries live below this level with
// 0 < count < kept; Q = those before x.  Pruning is off here: with it, the
// sparse push takes every child that the bitmap tier may run (its indices, -1
// between pushes, would not survive this one).
__device__ __noinline__ void t1_handoff(const T1 t, int x, int level, int kept, uint64_t sR,
                                        uint64_t nR) {
  Warp& W = this_warp();
  const int lane = (int)lane_id();
  const int32_t* llevel = W.A(W.sl().llevel);
  const int32_t* ncnt = W.A(W.sl().ncnt);
  const int32_t* bound = W.A(W.sl().bound);
  const uint64_t* ckey = W.A64(W.sl().ckey);
  int32_t* sidx = W.A(W.sl().sidx);
  int32_t* lp = W.A(W.sl().lp);
  uint64_t* lkey = W.A64(W.sl().lkey);
  const int32_t* aoff = W.A(W.sl().aoff);
  const int32_t* aadj = W.A(W.sl().aadj);
  // L_sub positions
  int n = 0;
  ROLLED for (int c0 = 0; c0 < t.nL; c0 += 32) {
    int l = c0 + lane;
    bool sel = l < t.nL && llevel[l] == level;
    unsigned bal = __ballot_sync(kFull, sel);
    if (sel) {
      int j = n + __popc(bal & lanemask_lt());
      lp[j] = l;
      lkey[j] = W.gp->ukey[t.L[l]];
      if (s_blk.emit) W.A(W.sl().lid)[j] = t.L[l];
    }
    n += __popc(bal);
  }
  // candidates, their C indices at the arena's end
  uint32_t* end = reinterpret_cast<uint32_t*>(W.A(W.sl().ar_end)) - cls_stride(t.nC);
  int32_t* cpos = reinterpret_cast<int32_t*>(end);
  int nsub = 0, nq = 0;
  ROLLED for (int c0 = 0; c0 < t.nC; c0 += 64) {
    int b[2], c[2];
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int i = c0 + 32 * u + lane;
      b[u] = i < t.nC ? bound[i] : -1;
      c[u] = i < t.nC ? ncnt[i] : 0;
    }
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int i = c0 + 32 * u + lane;
      const bool sel = b[u] > level && c[u] > 0 && c[u] < kept;
      const unsigned bal = __ballot_sync(kFull, sel);
      const int s = nsub + __popc(bal & lanemask_lt());
      if (sel) cpos[s] = i;
      if (i < t.nC) sidx[i] = sel ? s : -1;
      nsub += __popc(bal);
      nq += __popc(__ballot_sync(kFull, sel && i < x));  // candidates before x are Q
    }
  }
  __syncwarp();
  if (nsub > 0) {
    int nend = nsub;
    const ClsList l = cls_build(
        reinterpret_cast<uint32_t*>(W.A(W.sl().ar_sub)), end, nsub, nq, words_k(kept), n, &nend,
        nullptr, ckey, cpos, ClsEdges{nullptr, nullptr, sidx, 0, 0, lp, aoff, aadj},
        reinterpret_cast<uint32_t*>(W.A(W.sl().tcls)));
    tier2(W, l, n, nend, sR, nR);
  }
  __syncwarp();
}

// A push at `level` whose child L (the `kept` rows, marked llevel == level)
// fits the bitmap tier, done without touching the level's counts: the child's
// neighbour counts are built from the kept rows alone, the child sub-problem
// goes to tier 2, and the state after finder_pop is written directly.  With
// pruning on, finder_pop leaves a candidate c of bound >= level at FREE if c
// is adjacent to a removed vertex (its count inside the kept rows is below
// its count at this level) or is x itself, and at level-1 otherwise; every
// candidate of bound >= level is FREE before the push, and candidates not
// adjacent to the kept rows are either touched (stay FREE) or irrelevant
// below this level (count 0), so only candidates adjacent to the kept rows
// change.
__device__ __noinline__ void t1_sparse_push(const T1 t, int x, int level, int kept, uint64_t sL) {
  Warp& W = this_warp();
  const int lane = (int)lane_id();
  int32_t* llevel = W.A(W.sl().llevel);
  const int32_t* ncnt = W.A(W.sl().ncnt);
  int32_t* bound = W.A(W.sl().bound);
  const int32_t* coff = W.A(W.sl().coff);
  const int32_t* cadj = W.A(W.sl().cadj);
  const int32_t* aoff = W.A(W.sl().aoff);
  const int32_t* aadj = W.A(W.sl().aadj);
  int32_t* cc = W.A(W.sl().fill);   // child counts, all-zero between pushes
  int32_t* sidx = W.A(W.sl().sidx); // -1 between pushes
  int32_t* tl = W.A(W.sl().tlist);
  int32_t* lp = W.A(W.sl().lp);
  uint64_t* lkey = W.A64(W.sl().lkey);
  // kept rows -> lp[0..kept), with their hash keys
  int n = 0;
  {
    int rb = coff[x], re = coff[x + 1];
    ROLLED for (int b0 = rb; b0 < re; b0 += 32) {
      int j = b0 + lane;
      int l = j < re ? cadj[j] : 0;
      bool sel = j < re && llevel[l] == level;
      unsigned bal = __ballot_sync(kFull, sel);
      if (sel) {
        int q = n + __popc(bal & lanemask_lt());
        lp[q] = l;
        if (q < 32 * kKMax) {
          lkey[q] = W.gp->ukey[t.L[l]];
          if (s_blk.emit) W.A(W.sl().lid)[q] = t.L[l];
        }
      }
      n += __popc(bal);
    }
  }
  __syncwarp();
  // Child counts over the kept rows.  tl = candidates met (each once);
  // ent = every (candidate, row) entry met, packed p << 7 | r (r < 128), so
  // that the child's masks come from one linear pass instead of a second walk.
  int32_t* ent = W.A(W.sl().ent);
  int32_t* tcls = W.A(W.sl().tcls);
  const uint64_t* ckey = W.A64(W.sl().ckey);
  int nt = 0, ne = 0;
  // Whether the met candidates come out in the order of their first touch or of
  // their ids decides the order of the child's P: by the rows' whole lengths, so
  // that dropping dead entries (t1_compact) changes no search tree.
  int kent = 0;
  if (!W.seen) {
    const int32_t* rev_off = W.gp->rev_off;
    ROLLED for (int q = lane; q < n; q += 32) {
      const int u = t.L[lp[q]];
      kent += rev_off[u + 1] - rev_off[u];
    }
    kent = warp_sum64(kent);
  }
  const int cwords = (t.nC + 31) >> 5;
  // (with `scan`: fire-and-forget counts and touch bits, and the touched list
  // from the bitmap)
  const bool scan = use_gseen(W, kent, cwords);
  if (!scan) clear_seen(W, cwords);
  const bool shared = W.seen;
  uint32_t* seen = this_smem();
  flat_rows(
      n,
      [&](int r, int& beg, int& len) {
        int l = lp[r];
        beg = aoff[l];
        len = aoff[l + 1] - beg;
      },
      [&](bool valid, int pos) { return valid ? aadj[pos] : -1; },
      [&](bool, int r, int, int p) {
        const unsigned lt = lanemask_lt();
        bool first = false;
        if (p >= 0) {
          if (scan) {
            atomicAdd(&cc[p], 1);
            atomicOr(&W.gseen()[p >> 5], 1u << (p & 31));
          } else {
            first = count_first(shared, seen, cc, p);
          }
        }
        const unsigned bal = __ballot_sync(kFull, first);
        if (first) tl[nt + __popc(bal & lt)] = p;
        nt += __popc(bal);
        const unsigned be = __ballot_sync(kFull, p >= 0);
        if (p >= 0) ent[ne + __popc(be & lt)] = (p << 7) | r;
        ne += __popc(be);
      });
  if (scan) {
    __threadfence_block();
    __syncwarp();
    nt = collect_bits(W.gseen(), cwords, tl, t.nC);
  } else {
    counts_done(W, tl, nt);
  }
  // R of the child, maximality, and each touched candidate's class (0 none,
  // 1 Q, 2 P).  Lane-local counters keep the iterations independent, so
  // their loads overlap.
  bool ism = true;
  uint64_t sR = 0;
  unsigned long long nR = 0;
  int ncand = 0, nqc = 0;
#pragma unroll 4
  for (int q = lane; q < nt; q += 32) {
    const int p = tl[q];
    const int c = cc[p];
    const int b = bound[p];
    int cls = 0;
    if (c == kept) {
      sR += ckey[p];
      ++nR;
      if (p < x && b >= level) ism = false;
    } else if (b >= level) {
      cls = p < x ? 1 : 2;
      ++ncand;
      nqc += cls == 1;
    }
    tcls[q] = cls;
  }
  ism = __all_sync(kFull, ism);
  ncand = (int)__reduce_add_sync(kFull, (unsigned)ncand);
  nqc = (int)__reduce_add_sync(kFull, (unsigned)nqc);
  const int K = words_k(n);
  const int levels = cls_levels(kept, ncand - nqc);
  sR = warp_sum64(sR) + t.sRtask;
  nR = warp_sum64(nR) + t.nRtask;
  if (ism) {
    acc(W.cnt, 1);
    acc(W.hash, biclique_hash(*W.gp, sL, (uint64_t)kept, sR, nR));
    if (s_blk.emit) emit_list(s_blk.ctl, emit_dst(*s_blk.p), W.gid, n, t.L, lp);
  } else {
    acc(W.nonmax, 1);
  }
  __syncwarp();
  if (ism && kept > 1 && ncand > 0) {
    // child indices: Q from the front, P from the back
    uint32_t* at = reinterpret_cast<uint32_t*>(W.A(W.sl().ar_sub));
    uint32_t* end = reinterpret_cast<uint32_t*>(W.A(W.sl().ar_end)) - cls_stride(ncand);
    // C index of each child candidate, complemented if it meets one kept row
    int32_t* cpos = reinterpret_cast<int32_t*>(end);
    int nq = 0, np = 0;
    ROLLED for (int b0 = 0; b0 < nt; b0 += 32) {
      int q = b0 + lane;
      const int cls = q < nt ? tcls[q] : 0;
      const int p = q < nt ? tl[q] : 0;
      unsigned bq = __ballot_sync(kFull, cls == 1);
      unsigned bp = __ballot_sync(kFull, cls == 2);
      int s = -1;
      if (cls == 1) s = nq + __popc(bq & lanemask_lt());
      if (cls == 2) s = ncand - 1 - (np + __popc(bp & lanemask_lt()));
      if (s >= 0) {
        sidx[p] = s;
        cpos[s] = cc[p] >= 2 ? p : ~p;
      }
      nq += __popc(bq);
      np += __popc(bp);
    }
    __syncwarp();
    int nend = ncand;
    const ClsList l =
        cls_build(at, end, ncand, nqc, K, n, &nend, nullptr, ckey, cpos,
                  ClsEdges{ent, nullptr, sidx, ne, 0, nullptr, nullptr, nullptr},
                  reinterpret_cast<uint32_t*>(tcls));
    // To an idle warp when some want work and the child is big enough by
    // GMBE's split test, else it runs here.
    int slot = -1;
    if (slot_fits(W, l.n, K, levels) && should_export(W, ncand - nqc, n, s_blk.eager_share != 0)) {
      slot = lane == 0 ? slot_alloc_for(W, l.n, K) : 0;
      slot = __shfl_sync(kFull, slot, 0);
    }
    if (slot >= 0) {
      int32_t* sp = slot_ptr(W, slot);
      uint32_t* dst = reinterpret_cast<uint32_t*>(sp + kSlotList);
      const int words = (int)cls_list_words(l.n, K);
      ROLLED for (int i = lane; i < words; i += 32) dst[i] = l.m[i];
      uint64_t* lk = reinterpret_cast<uint64_t*>(sp + kSlotLk);
      ROLLED for (int b = lane; b < n; b += 32) lk[b] = lkey[b];
      if (s_blk.emit) {
        int32_t* li = sp + kSlotLid;
        const int32_t* lid = W.A(W.sl().lid);
        ROLLED for (int b = lane; b < n; b += 32) li[b] = lid[b];
      }
      if (lane < K) sp[kSlotL + lane] = (int32_t)first_bits(n, lane);
      if (lane == 0) slot_header(sp, K, l.n, n, sR, nR, W.gid);
      if (!slot_publish(slot, 0)) {  // ring full
        if (lane == 0) slot_free(W, slot);
        __syncwarp();
        slot = -1;
      }
    }
    if (slot < 0) tier2(W, l, n, nend, sR, nR);
  }
  __syncwarp();
  // state after finder_pop(x, level), then clear the child scratch
  unsigned gone = 0;  // entries of the candidates retired
#pragma unroll 4
  for (int q = lane; q < nt; q += 32) {
    const int p = tl[q];
    const int c = cc[p];
    if (bound[p] >= level && p != x && c == ncnt[p]) {
      bound[p] = level - 1;
      gone += c;
    }
    cc[p] = 0;
    sidx[p] = -1;
  }
  if (level == 1) acc(W.dead, __reduce_add_sync(kFull, gone));
  ROLLED for (int q = lane; q < n; q += 32) llevel[lp[q]] = level - 1;
  __syncwarp();
}

// A push at `level` that keeps one or two rows (la; lb, or -1), whole: what
// t1_sparse_push would do, without counts, an entry list or a sub-problem.
// With pruning on, the child of two rows has candidates on one row each; its
// pushes keep that row alone, one push per row that has a P candidate (the
// others of the row are retired with it), non-maximal exactly if the row has a
// Q candidate.  So the rows are walked and summed up: row a's candidates are
// marked in cc, row b's walk tells the common ones (R of the push) from its
// own, row a's second walk sees the rest.  Each walk keeps kNarrow rounds of
// loads in flight, for a push is a chain of them and one warp's pushes are a
// root's critical path.
//
// On the 300,000-edge graph three fifths of a heavy root's first-level pushes
// keep one or two rows (3,042 of 5,028).  Whole calls, before -> after: that
// graph 50.2 -> 48.5 ms, one shard of the large graph (rows of 10^5 entries)
// 915 -> 839 ms.
constexpr int kNarrow = 4;
__device__ __noinline__ void t1_narrow_push(const T1 t, int x, int level, int la, int lb,
                                            uint64_t sL) {
  Warp& W = this_warp();
  const int lane = (int)lane_id();
  int32_t* llevel = W.A(W.sl().llevel);
  const int32_t* ncnt = W.A(W.sl().ncnt);
  int32_t* bound = W.A(W.sl().bound);
  const int32_t* aoff = W.A(W.sl().aoff);
  const int32_t* aadj = W.A(W.sl().aadj);
  const uint64_t* ckey = W.A64(W.sl().ckey);
  int32_t* cc = W.A(W.sl().fill);  // all-zero between pushes
  const bool two = lb >= 0;
  if (two) {
    const int end = aoff[la + 1];
#pragma unroll 4
    for (int j = aoff[la] + lane; j < end; j += 32) {
      const int p = aadj[j];
      if (p >= 0) cc[p] = 1;
    }
    __syncwarp();
  }
  bool ism = true;
  uint64_t sR = 0;       // R of the push
  unsigned nR = 0, gone = 0;  // gone: entries of the candidates retired
  uint64_t key[2];       // R of the child's push that keeps row b (0), row a (1)
  unsigned np[2], nq[2];
#pragma unroll
  for (int s = 0; s < 2; ++s) {
    key[s] = 0;
    np[s] = nq[s] = 0;
    if (s == 0 && !two) continue;
    const int row = s == 0 ? lb : la;
    const int end = aoff[row + 1];
    ROLLED for (int j0 = aoff[row] + lane; j0 < end; j0 += 32 * kNarrow) {
      int p[kNarrow], b[kNarrow], nc[kNarrow], m[kNarrow];
      uint64_t k[kNarrow];
#pragma unroll
      for (int u = 0; u < kNarrow; ++u) p[u] = j0 + 32 * u < end ? aadj[j0 + 32 * u] : -1;
#pragma unroll
      for (int u = 0; u < kNarrow; ++u) {
        if (p[u] < 0) continue;
        b[u] = bound[p[u]];
        nc[u] = ncnt[p[u]];
        k[u] = ckey[p[u]];
        m[u] = two ? cc[p[u]] : 1;  // row b: 1 in row a too; row a: 2 in row b too
      }
#pragma unroll
      for (int u = 0; u < kNarrow; ++u) {
        if (p[u] < 0) continue;
        const bool live = b[u] >= level;
        if (two) {
          if (s == 0 && m[u]) cc[p[u]] = 2;
          if (s == 1) cc[p[u]] = 0;
          if (s == 1 && m[u] == 2) continue;  // common: done with row b
        }
        const bool covers = !two || (s == 0 && m[u]);
        if (covers) {
          sR += k[u];
          ++nR;
          ism = ism && !(live && p[u] < x);
        } else if (live) {
          if (p[u] < x) {
            ++nq[s];
          } else {
            key[s] += k[u];
            ++np[s];
          }
        }
        // finder_pop: retired if it meets no removed row
        const int c = covers && two ? 2 : 1;
        if (live && p[u] != x && nc[u] == c) {
          bound[p[u]] = level - 1;
          gone += c;
        }
      }
    }
    __syncwarp();
  }
  if (level == 1) acc(W.dead, __reduce_add_sync(kFull, gone));
  ism = __all_sync(kFull, ism);
  if (ism) {
    sR = warp_sum64(sR) + t.sRtask;
    const uint64_t nRs = __reduce_add_sync(kFull, nR) + t.nRtask;
    acc(W.cnt, 1);
    acc(W.hash, biclique_hash(*W.gp, sL, two ? 2 : 1, sR, nRs));
    int32_t* lp = W.A(W.sl().lp);
    if (s_blk.emit) {
      if (lane <= (int)two) lp[lane] = lane < (int)two ? lb : la;
      __syncwarp();
      emit_list(s_blk.ctl, emit_dst(*s_blk.p), W.gid, two ? 2 : 1, t.L, lp);
    }
    if (two) {
      const uint64_t ka = W.gp->ukey[t.L[la]];
#pragma unroll
      for (int s = 0; s < 2; ++s) {
        const unsigned n = __reduce_add_sync(kFull, np[s]);
        if (n == 0) continue;
        acc(W.pushes, 1ULL << 32);
        if (__any_sync(kFull, nq[s] != 0)) {
          acc(W.nonmax, 1);
          continue;
        }
        const uint64_t ks = warp_sum64(key[s]);
        acc(W.cnt, 1);
        acc(W.hash, biclique_hash(*W.gp, s == 0 ? sL - ka : ka, 1, sR + ks, nRs + n));
        if (s_blk.emit) emit_list(s_blk.ctl, emit_dst(*s_blk.p), W.gid, 1, t.L, lp + s);
      }
    }
  } else {
    acc(W.nonmax, 1);
  }
  if (lane == 0) {
    llevel[la] = level - 1;
    if (two) llevel[lb] = level - 1;
  }
  __syncwarp();
}

// Levels 2 .. kLevelBits + 1 of the counts tier keep a bitmap of the
// candidates the level's L meets (count != 0 there): the scan for the next
// live candidate and a recount walk its words instead of every candidate.
__device__ __forceinline__ uint32_t* level_bits(const Warp& W, int level) {
  if (level < 2 || level > kLevelBits + 1) return nullptr;
  return reinterpret_cast<uint32_t*>(W.A(W.sl().lbits)) +
         (size_t)(level - 2) * (size_t)((W.sl().capC + 31) >> 5);
}

__device__ __forceinline__ unsigned long long warp_min_u64(unsigned long long v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = min(v, __shfl_xor_sync(kFull, v, o));
  return v;
}

// First candidate i in [start, end) with bound[i] > level-1 and ncnt[i] != 0
// (src/IterFinderGpu.cu:26-34), or -1.  bits, when given, holds the
// candidates with ncnt != 0.
__device__ __forceinline__ int t1_next_live(const int32_t* bound, const int32_t* ncnt,
                                            const uint32_t* bits, int start, int end, int level) {
  const int lane = (int)lane_id();
  if (!bits) {
    ROLLED for (int b0 = start; b0 < end; b0 += 32) {
      const int i = b0 + lane;
      const bool ok = i < end && bound[i] > level - 1 && ncnt[i] != 0;
      const unsigned bal = __ballot_sync(kFull, ok);
      if (bal) return b0 + __ffs(bal) - 1;
    }
    return -1;
  }
  if (start >= end) return -1;
  const int w0 = start >> 5, wend = (end + 31) >> 5;
  ROLLED for (int wb = w0; wb < wend; wb += 32) {
    const int w = wb + lane;
    uint32_t m = w < wend ? bits[w] : 0u;
    if (w == w0) m &= ~0u << (start & 31);
    if (w == wend - 1 && (end & 31)) m &= (1u << (end & 31)) - 1u;
    int first = -1;
    while (m) {
      const int i = (w << 5) + __ffs(m) - 1;
      if (bound[i] > level - 1) {
        first = i;
        break;
      }
      m &= m - 1;
    }
    const unsigned bal = __ballot_sync(kFull, first >= 0);
    if (bal) return __shfl_sync(kFull, first, __ffs(bal) - 1);
  }
  return -1;
}

// Counts-tier child export.  A push at `level` of candidate x whose new L
// (the `kept` rows, llevel == level) is too large for the bitmap tier
// descends in place; when warps wait for work the child goes to one of them
// instead, as vertex lists in a slot: L' = the kept rows' vertices, C' = the
// candidates live below this level (bound > level) with 0 < count < kept,
// in index order (those before x are its Q), and the R sum and size of the
// push.  Every bound of C' is free at the child's first level (a bound above
// `level` is FREE or TOUCHED there), so the importer starts from a clean
// frame, and the child's levels leave this level's state as they found it:
// the exporter pops x at once.  nbits holds the candidates the kept rows
// meet (the bitmap of level + 1).  Slot: header of 16 words {|L'|, |C'|,
// |Q'|, graph, sR (2 words), |R|}, then L' ids, then C' ids.
constexpr int kFrameHdr = 16;

// Whether a counts-tier child of `kept` rows (`kent` entries left in them) may
// be shared out now: slots exist, every warp has room for that much, warps wait
// for work.
__device__ __forceinline__ bool t1_export_wanted(Warp& W, int kept, long long kent) {
  if (!s_blk.share_counts || (s_blk.nslot == 0 && s_blk.nbig == 0)) return false;
  if (kept > s_blk.import_l || kent > (long long)s_blk.import_s) return false;
  return export_demand() != 0;
}

__device__ __noinline__ bool t1_try_export(const T1 t, int x, int level, int kept, uint64_t sR,
                                           uint64_t nR, const uint32_t* nbits) {
  Warp& W = this_warp();
  const int lane = (int)lane_id();
  const int32_t* bound = W.A(W.sl().bound);
  const int32_t* ncnt = W.A(W.sl().ncnt);
  const int32_t* cv = W.A(W.sl().cv);
  const int32_t* coff = W.A(W.sl().coff);
  const int32_t* cadj = W.A(W.sl().cadj);
  const int32_t* llevel = W.A(W.sl().llevel);
  const int cwords = (t.nC + 31) >> 5;
  int m = 0, mq = 0;
  ROLLED for (int w0 = 0; w0 < cwords; w0 += 32) {
    const int w = w0 + lane;
    uint32_t b = w < cwords ? nbits[w] : 0u;
    while (b) {
      const int p = (w << 5) + __ffs(b) - 1;
      if (bound[p] > level && ncnt[p] < kept) {
        ++m;
        mq += p < x;
      }
      b &= b - 1;
    }
  }
  m = (int)__reduce_add_sync(kFull, (unsigned)m);
  mq = (int)__reduce_add_sync(kFull, (unsigned)mq);
  if (m == 0 || m > s_blk.import_cap || !should_export(W, m - mq, kept)) return false;
  if (s_blk.import_s < W.sl().capS) {
    // The importer lays the graph's whole rows out; those here may have lost
    // entries since (t1_compact).
    const int32_t* rev_off = W.gp->rev_off;
    long long whole = 0;
    ROLLED for (int j = coff[x] + lane; j < coff[x + 1]; j += 32) {
      const int l = cadj[j];
      if (llevel[l] == level) whole += rev_off[t.L[l] + 1] - rev_off[t.L[l]];
    }
    if (warp_sum64(whole) > (unsigned long long)s_blk.import_s) return false;
  }
  const long long words = kFrameHdr + (long long)kept + m;
  int slot = -1;
  if (lane == 0) {
    if (words <= kSlotWords) slot = slot_alloc(W);
    if (slot < 0 && words <= kBigSlotWords) {
      const int b = bits_alloc(s_blk.big_bits, s_blk.nbig);
      if (b >= 0) slot = s_blk.nslot + b;
    }
  }
  slot = __shfl_sync(kFull, slot, 0);
  if (slot < 0) return false;
  int32_t* sp = slot_ptr(W, slot);
  // L' ids: the kept rows, from x's row of cadj
  int nl = 0;
  ROLLED for (int j0 = coff[x]; j0 < coff[x + 1]; j0 += 32) {
    const int j = j0 + lane;
    const int l = j < coff[x + 1] ? cadj[j] : 0;
    const bool sel = j < coff[x + 1] && llevel[l] == level;
    const unsigned bal = __ballot_sync(kFull, sel);
    if (sel) sp[kFrameHdr + nl + __popc(bal & lanemask_lt())] = t.L[l];
    nl += __popc(bal);
  }
  // C' ids in index order: lane k takes word k of each round
  int32_t* cdst = sp + kFrameHdr + kept;
  int o = 0;
  ROLLED for (int w0 = 0; w0 < cwords; w0 += 32) {
    const int w = w0 + lane;
    uint32_t b = w < cwords ? nbits[w] : 0u;
    uint32_t keep = 0u;
    ROLLED for (uint32_t bb = b; bb; bb &= bb - 1) {
      const int bit = __ffs(bb) - 1;
      const int p = (w << 5) + bit;
      if (bound[p] > level && ncnt[p] < kept) keep |= 1u << bit;
    }
    int tot;
    int at = o + excl_scan(__popc(keep), &tot);
    ROLLED for (; keep; keep &= keep - 1) cdst[at++] = cv[(w << 5) + __ffs(keep) - 1];
    o += tot;
  }
  if (lane == 0) {
    sp[0] = kept;
    sp[1] = m;
    sp[2] = mq;
    sp[3] = W.gid;
    *reinterpret_cast<uint64_t*>(sp + 4) = sR;
    sp[6] = (int32_t)nR;
  }
  if (slot_publish(slot, 1)) {
    acc(W.splits, 1);
    return true;
  }
  if (lane == 0) slot_free(W, slot);
  __syncwarp();
  return false;
}

// Drops the entries of retired candidates (bound 0) from the rows, between two
// pushes of the first level.  Such a candidate lies inside one already popped,
// and the chain of these ends at one that is live and in Q from then on.  So
// nothing below reads it: it is not pushed or handed to a child, and a push it
// covers is covered by that Q candidate too, which makes the push non-maximal
// and its R unread.  (A push of this level that it covered would lie inside the
// popped one as well, and be retired itself.)
//
// A vertex of the hub kind has tens of thousands of candidates that meet no
// other row; the first push that keeps its row retires them all, and every
// later one walked past them: of a root with 33 rows, 35,857 candidates and
// 37,503 entries, 161 pushes took 400 ms.  The pass is made when a quarter of
// the entries are known to be dead, so that all passes of a task together cost
// a few walks of its rows.  Whole calls, before -> after: one shard of the large
// graph 839 -> 642 ms, medium graph 355 -> 292-322 ms, a shard of eight of it
// 183 -> 151 ms, the 300,000-edge graph 48.5 -> 41-43 ms.
__device__ __noinline__ void t1_compact(int nL) {
  const Warp& W = this_warp();
  const int lane = (int)lane_id();
  int32_t* aoff = W.A(W.sl().aoff);
  int32_t* aadj = W.A(W.sl().aadj);
  const int32_t* bound = W.A(W.sl().bound);
  // Per 32 entries: their live bits, and the live ones before them.
  uint32_t* rank = reinterpret_cast<uint32_t*>(W.A(W.sl().ent));
  const int total = aoff[nL];
  int n = 0;
  ROLLED for (int e0 = 0; e0 < total; e0 += 256) {
    int p[8];
    bool on[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int e = e0 + 32 * u + lane;
      p[u] = e < total ? aadj[e] : -1;
    }
#pragma unroll
    for (int u = 0; u < 8; ++u) on[u] = p[u] >= 0 && bound[p[u]] >= 1;
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const unsigned bal = __ballot_sync(kFull, on[u]);
      const int c = (e0 >> 5) + u;
      if (lane == 0 && 32 * c < total) {
        rank[2 * c] = bal;
        rank[2 * c + 1] = (uint32_t)n;
      }
      if (on[u]) aadj[n + __popc(bal & lanemask_lt())] = p[u];
      n += __popc(bal);
    }
  }
  __syncwarp();
  ROLLED for (int r = lane; r <= nL; r += 32) {
    const int old = aoff[r];
    const int c = old >> 5;
    aoff[r] = old >= total ? n
                           : (int)rank[2 * c + 1] +
                                 __popc(rank[2 * c] & ((1u << (old & 31)) - 1u));
  }
  __syncwarp();
}
// Entries from which it pays, and fit its scratch (two words per 32 of them).
constexpr int kCompactMin = 256;

__device__ __noinline__ void tier1_run(const T1 t) {
  Warp& W = this_warp();
  const int lane = (int)lane_id();
  int32_t* llevel = W.A(W.sl().llevel);
  int32_t* ncnt = W.A(W.sl().ncnt);
  int32_t* bound = W.A(W.sl().bound);
  int32_t* stack = W.A(W.sl().stack);
  int32_t* lent = W.A(W.sl().lent);
  const uint64_t* ckey = W.A64(W.sl().ckey);
  const int32_t* coff = W.A(W.sl().coff);
  const int32_t* cadj = W.A(W.sl().cadj);
  const int32_t* aoff = W.A(W.sl().aoff);
  const int32_t* aadj = W.A(W.sl().aadj);
  const bool emitting = s_blk.emit != nullptr;
  const int t2max = W.gp->tier2_max_l;
  const int cwords = (t.nC + 31) >> 5;

  // The level bitmaps start clear (a task that ended early may leave bits).
  ROLLED for (int lv = 2; lv <= kLevelBits + 1; ++lv) {
    uint32_t* b = level_bits(W, lv);
    ROLLED for (int w = lane; w < cwords; w += 32) b[w] = 0u;
  }
  if (lane == 0) {
    stack[0] = t.nq;
    lent[0] = aoff[t.nL];
    W.dead = 0;
  }
  __syncwarp();
  int level = 1;
  unsigned steps = 0;
  while (level != 0) {
    // The stop flag is a global load the whole warp waits for: look at it on
    // the first step and every 64th after.
    if ((steps++ & 63u) == 0u && must_stop()) return;
    if (level == 1) {
      const int total = lent[0];
      if (total >= kCompactMin && 4 * W.dead > (unsigned long long)total) {
        t1_compact(t.nL);
        if (lane == 0) {
          lent[0] = aoff[t.nL];
          W.dead = 0;
        }
        __syncwarp();
      }
    }
    const int end = level == 1 ? t.nend : t.nC;  // the first level may push a part only
    int cur = t1_next_live(bound, ncnt, level_bits(W, level), stack[level - 1], end, level);
    if (cur >= 0) {
      // ---- finder_push (src/IterFinderGpu.h:206-264) ----
      acc(W.pushes, 1);
      int kept = 0;
      uint64_t sL = 0;
      long long kent = 0;                 // entries of the kept rows
      unsigned long long best = ~0ULL;    // (row length << 32) | position of the shortest kept row
      int first = INT_MAX, last = -1;     // the first and the last kept row
      int rb = coff[cur], re = coff[cur + 1];
      ROLLED for (int j = rb + lane; j < re; j += 32) {
        int l = cadj[j];
        if (llevel[l] == level - 1) {
          llevel[l] = level;
          ++kept;
          sL += W.gp->ukey[t.L[l]];
          const int len = aoff[l + 1] - aoff[l];
          kent += len;
          best = min(best, ((unsigned long long)(unsigned)len << 32) | (unsigned)l);
          last = max(last, l);
          first = min(first, l);
        }
      }
      kept = (int)__reduce_add_sync(kFull, (unsigned)kept);
      sL = warp_sum64(sL);
      if (s_blk.prune && kept <= min(t2max, 2)) {
        __syncwarp();
        first = __reduce_min_sync(kFull, first);
        last = __reduce_max_sync(kFull, last);
        t1_narrow_push(t, cur, level, first, kept == 2 ? last : -1, sL);
        if (lane == 0) stack[level - 1] = cur + 1;
        __syncwarp();
        continue;
      }
      kent = warp_sum64(kent);
      best = warp_min_u64(best);
      __syncwarp();
      if (s_blk.prune && kept <= t2max) {
        t1_sparse_push(t, cur, level, kept, sL);
        if (lane == 0) stack[level - 1] = cur + 1;
        __syncwarp();
        continue;
      }
      // Counts over the kept rows: subtract the removed rows, or clear the
      // level's counts and add the kept rows, whichever walks less.
      const uint32_t* pbits = level_bits(W, level);
      const long long rent = (long long)lent[level - 1] - kent;
      const long long clear_cost = pbits ? (long long)cwords : (long long)t.nC;
      if (clear_cost + kent < rent) {
        if (pbits) {
          ROLLED for (int w = lane; w < cwords; w += 32) {
            uint32_t m = pbits[w];
            while (m) {
              ncnt[(w << 5) + __ffs(m) - 1] = 0;
              m &= m - 1;
            }
          }
        } else {
          ROLLED for (int i = lane; i < t.nC; i += 32) ncnt[i] = 0;
        }
        __syncwarp();
        t1_walk(t.nL, cur, level, kOpAdd, level, nullptr);
      } else {
        t1_walk(t.nL, -1, level - 1, kOpSub, level, nullptr);
      }
      __syncwarp();
      // Maximality (src/IterFinderGpu.h:252-261): a candidate covering the new
      // L is adjacent to every kept row, the shortest one included, so only
      // that row's candidates are examined.
      bool ism = true;
      uint64_t sR = 0;
      unsigned long long nR = 0;
      {
        const int lstar = (int)(best & 0xffffffffu);
        const int mb = aoff[lstar], me = aoff[lstar + 1];
        ROLLED for (int j = mb + lane; j < me; j += 32) {
          const int i = aadj[j];
          if (i >= 0 && ncnt[i] == kept) {
            sR += ckey[i];
            ++nR;
            int b = bound[i];
            if (i < cur && b >= level) ism = false;
            else if (b > level) bound[i] = level;
          }
        }
      }
      ism = __all_sync(kFull, ism);
      sR = warp_sum64(sR) + t.sRtask;
      nR = warp_sum64(nR) + t.nRtask;
      if (ism) {
        acc(W.cnt, 1);
        acc(W.hash, biclique_hash(*W.gp, sL, (uint64_t)kept, sR, nR));
        if (emitting)
          emit_level(s_blk.ctl, emit_dst(*s_blk.p), W.gid, kept, t.nL, llevel, level, t.L);
      } else {
        acc(W.nonmax, 1);
      }
      __syncwarp();
      if (ism && kept > 1) {
        if (kept <= t2max) {
          t1_handoff(t, cur, level, kept, sR, nR);
        } else {
          uint32_t* nbits = level_bits(W, level + 1);
          // The candidates the kept rows meet, as a bitmap: the next level's
          // own one, or (deeper levels) the warp's global touch bitmap, built
          // only when the child may be shared out.
          uint32_t* cbits = nbits;
          const bool want = t1_export_wanted(W, kept, kent);
          if (!cbits && want) cbits = W.gseen();
          if (cbits) {
            t1_walk(t.nL, cur, level, kOpSetBit, level, cbits);
            __threadfence_block();
            __syncwarp();
          }
          const bool exported =
              want && cbits && t1_try_export(t, cur, level, kept, sR, nR, cbits);
          if (cbits && (exported || cbits != nbits)) {
            // back to clear: a shared-out child's level bitmap, or the touch bitmap
            t1_walk(t.nL, cur, level, kOpClearBit, level, cbits);
            __syncwarp();
          }
          if (exported) {
            // shared out: pop x here
          } else {
            if (lane == 0) {
              stack[level - 1] = cur;
              stack[level] = cur + 1;
              lent[level] = (int32_t)kent;
            }
            __syncwarp();
            ++level;
            continue;
          }
        }
      }
      if (lane == 0) stack[level - 1] = cur + 1;
      __syncwarp();
      t1_pop(t.nL, cur, level);
    } else {
      --level;
      if (level > 0) {
        cur = stack[level - 1];
        __syncwarp();
        uint32_t* cbits = level_bits(W, level + 1);
        if (cbits) {  // the finished level's bitmap back to clear
          t1_walk(t.nL, cur, level, kOpClearBit, level, cbits);
          __syncwarp();
        }
        t1_pop(t.nL, cur, level);
        if (lane == 0) stack[level - 1] = cur + 1;
        __syncwarp();
      }
    }
  }
}

__device__ int lay_out_rows(const int32_t* L, int nL, int entries, bool count, bool keep);
__device__ void t1_transpose(int entries, int nC);

// Runs a counts-tier child exported by t1_try_export: the frame is rebuilt
// from the vertex lists (local adjacency from the graph's U -> V rows, the
// counts of each candidate inside L'), then the counts tier runs it from its
// first level.  The child's own biclique was counted by the exporter.
__device__ __noinline__ void tier1_from_slot(int slot) {
  Warp& W = this_warp();
  const int lane = (int)lane_id();
  int32_t* sp = slot_ptr(W, slot);
  volatile const int32_t* vh = sp;
  const int n = vh[0], m = vh[1], nq = vh[2];
  const int32_t gid = vh[3];
  const uint64_t sR = (uint64_t)(uint32_t)vh[4] | ((uint64_t)(uint32_t)vh[5] << 32);
  const uint64_t nR = (uint32_t)vh[6];
  int32_t* lv = W.A(W.sl().lv);
  int32_t* cv = W.A(W.sl().cv);
  const bool fits = n <= W.sl().capL && m <= W.sl().capC;
  if (fits) {
    const unsigned* src = reinterpret_cast<const unsigned*>(sp + kFrameHdr);
    ROLLED for (int i = lane; i < n; i += 32) lv[i] = (int32_t)__ldcg(src + i);
    ROLLED for (int i = lane; i < m; i += 32) cv[i] = (int32_t)__ldcg(src + n + i);
  }
  __syncwarp();
  if (lane == 0) slot_free(W, slot);
  __syncwarp();
  if (!fits) {
    set_status(s_blk.ctl, kStCapacity, ((unsigned long long)4 << 32) | (unsigned)m);
    return;
  }
  __syncwarp();
  W.gid = gid;
  W.gp = graph_at(W, gid);
  __syncwarp();
  const DevGraph& g = *W.gp;
  int32_t* map = W.A(W.sl().map);
  int32_t* aoff = W.A(W.sl().aoff);
  int32_t* aadj = W.A(W.sl().aadj);
  int32_t* ent = W.A(W.sl().ent);
  int32_t* ncnt = W.A(W.sl().ncnt);
  int32_t* bound = W.A(W.sl().bound);
  int32_t* coff = W.A(W.sl().coff);
  int32_t* fill = W.A(W.sl().fill);
  int32_t* cadj = W.A(W.sl().cadj);
  int32_t* sidx = W.A(W.sl().sidx);
  int32_t* llevel = W.A(W.sl().llevel);
  uint64_t* ckey = W.A64(W.sl().ckey);
  int run = 0;
  ROLLED for (int c0 = 0; c0 < n; c0 += 32) {
    const int l = c0 + lane;
    const int d = l < n ? g.rev_off[lv[l] + 1] - g.rev_off[lv[l]] : 0;
    int tot;
    const int ex = excl_scan(d, &tot);
    if (l < n) aoff[l] = run + ex;
    run += tot;
  }
  if (lane == 0) aoff[n] = run;
  if (run > W.sl().capS) {
    set_status(s_blk.ctl, kStCapacity, ((unsigned long long)5 << 32) | (unsigned)run);
    return;
  }
  ROLLED for (int i = lane; i < m; i += 32) {
    map[cv[i]] = i + 1;
    ncnt[i] = 0;
    bound[i] = kFree;
    fill[i] = 0;
    sidx[i] = -1;
    ckey[i] = g.vkey[cv[i]];
  }
  ROLLED for (int l = lane; l < n; l += 32) llevel[l] = 0;
  __threadfence_block();
  __syncwarp();
  lay_out_rows(lv, n, run, false, true);
  ROLLED for (int e = lane; e < run; e += 32) {
    const int p = map[aadj[e]] - 1;
    aadj[e] = p;
    if (p >= 0) atomicAdd(&ncnt[p], 1);
  }
  __threadfence_block();
  __syncwarp();
  t1_transpose(run, m);
  T1 t1;
  t1.L = lv;
  t1.nL = n;
  t1.nC = m;
  t1.nq = nq;
  t1.nend = m;
  t1.sRtask = sR;
  t1.nRtask = nR;
  const uint64_t t1s = globaltimer_ns();
  const uint64_t t2_before = W.ns_t2;
  tier1_run(t1);
  acc(W.ns_t1, (globaltimer_ns() - t1s) - (W.ns_t2 - t2_before));
  __syncwarp();
  ROLLED for (int i = lane; i < m; i += 32) map[cv[i]] = 0;
  __syncwarp();
}

// ---------------------------------------------------------------------------
// Queue (bounded MPMC ring; replaces WorkList<LargeTask>, src/WorkList.cuh).
//
// Position gp lives in slot gp % cap during round gp / cap.  A slot's state
// word is 2*round while it is free for that round's producer and 2*round+1
// once the task is written; the consumer of position h hands the slot to the
// next round by writing 2*(h/cap)+2.  q_used (reserved, not yet released
// positions) never exceeds cap, so a producer only ever waits for a consumer
// that has already claimed the older position and is reading it.
__device__ __forceinline__ unsigned long long slot_free_tag(unsigned long long gp, int cap) {
  return 2ULL * (gp / (unsigned long long)cap);
}

__device__ __noinline__ bool queue_pop(Task* out) {
  Warp& W = this_warp();
  // lane 0 only
  EnumCtl* ctl = s_blk.ctl;
  volatile unsigned long long* vh = &ctl->q_head;
  volatile unsigned long long* vt = &ctl->q_tail;
  unsigned long long h = *vh;
  if (h >= *vt) return false;
  if (atomicCAS(&ctl->q_head, h, h + 1) != h) return false;
  const int cap = s_blk.p->queue_cap;
  unsigned long long slot = h % (unsigned long long)cap;
  volatile unsigned long long* st = s_blk.q_seq + slot;
  const unsigned long long full = slot_free_tag(h, cap) + 1;
  int64_t spins = 0;
  while (*st != full) {
    if (++spins > s_blk.p->slot_spin_limit) {
      set_status(ctl, kStQueue, h);
      return false;
    }
    __nanosleep(64);
  }
  __threadfence();
  volatile int32_t* src = reinterpret_cast<volatile int32_t*>(s_blk.q_tasks + slot);
  out->v[0] = src[0];
  out->v[1] = src[1];
  out->v[2] = src[2];
  out->v[3] = src[3];
  out->graph = src[4];
  out->part = src[5];
  out->parts = src[6];
  __threadfence();
  atomicExch(s_blk.q_seq + slot, full + 1);  // free for round h/cap + 1
  atomicAdd(&ctl->q_used, (unsigned long long)-1LL);
  return true;
}

// Queues n tasks, task i (0 <= i < n) made by make(i); false if the ring is
// full (then nothing is queued).
template <typename Make>
__device__ bool queue_push_n(Warp& W, unsigned long long n, Make make) {
  const int lane = (int)lane_id();
  EnumCtl* ctl = s_blk.ctl;
  const int cap = s_blk.p->queue_cap;
  unsigned long long pos = 0;
  int ok = 0;
  if (lane == 0) {
    unsigned long long used = atomicAdd(&ctl->q_used, n);
    if (used + n > (unsigned long long)cap) {
      atomicAdd(&ctl->q_used, (unsigned long long)(-(long long)n));
    } else {
      atomicAdd(&ctl->pending, n);
      graph_spawned(W, n);
      pos = atomicAdd(&ctl->q_tail, n);
      ok = 1;
    }
  }
  ok = __shfl_sync(kFull, ok, 0);
  if (!ok) return false;
  pos = __shfl_sync(kFull, pos, 0);
  ROLLED for (unsigned long long i = lane; i < n; i += 32) {
    unsigned long long gp = pos + i;
    unsigned long long slot = gp % (unsigned long long)cap;
    volatile unsigned long long* st = s_blk.q_seq + slot;
    const unsigned long long free_tag = slot_free_tag(gp, cap);
    int64_t spins = 0;
    bool ready = true;
    while (*st != free_tag) {
      if (++spins > s_blk.p->slot_spin_limit) {
        set_status(ctl, kStQueue, gp);
        ready = false;
        break;
      }
      __nanosleep(64);
    }
    if (!ready) continue;  // the run is aborting; the slot stays unwritten
    s_blk.q_tasks[slot] = make((int)i);
    __threadfence();
    atomicExch(s_blk.q_seq + slot, free_tag + 1);
  }
  __syncwarp();
  return true;
}

// Pushes children task + {cv[i]} for i in [nq, nC); false if the ring is full.
__device__ __noinline__ bool queue_push_children(const Task& t, int k, int nq, int nC) {
  Warp& W = this_warp();
  const int32_t* cv = W.A(W.sl().cv);
  return queue_push_n(W, (unsigned long long)(nC - nq), [&](int i) {
    Task c = t;
    c.v[k] = cv[nq + i];
    c.part = c.parts = 0;
    return c;
  });
}

// Pushes parts 1 .. m-1 of root task t; false if the ring is full.
__device__ __noinline__ bool queue_push_parts(const Task& t, int m) {
  Warp& W = this_warp();
  return queue_push_n(W, (unsigned long long)(m - 1), [&](int i) {
    Task c = t;
    c.part = i + 1;
    c.parts = m;
    return c;
  });
}

// Parts 1 .. m-1 of a listed big root (lane-uniform): a part record that only
// big warps claim from (the other warps' scratch cannot hold the root).
// They count as pending before the record becomes visible.  False if the
// record list is full (the root then runs whole).
__device__ __noinline__ bool big_parts_push(int v, int m) {
  Warp& W = this_warp();
  int ok = 0;
  if (lane_id() == 0) {
    const unsigned long long i = atomicAdd(&s_blk.ctl->n_big_parts, 1ULL);
    if (i < (unsigned long long)s_blk.p->big_parts_cap) {
      atomicAdd(&s_blk.ctl->pending, (unsigned long long)(m - 1));
      int32_t* r = s_blk.p->big_parts + 4 * i;
      r[0] = v;
      r[1] = m;
      r[2] = 1;  // part 0 runs on this warp
      __threadfence();
      atomicExch(&r[3], 1);
      ok = 1;
    }
  }
  return __shfl_sync(kFull, ok, 0) != 0;
}

// Claims a part of a listed big root (lane 0 of a big warp).
__device__ __noinline__ bool big_parts_claim(Task* t) {
  Warp& W = this_warp();
  EnumCtl* c = s_blk.ctl;
  const unsigned long long n = min(*(volatile unsigned long long*)&c->n_big_parts,
                                   (unsigned long long)s_blk.p->big_parts_cap);
  ROLLED for (unsigned long long i = *(volatile unsigned long long*)&c->big_parts_head; i < n; ++i) {
    int32_t* r = s_blk.p->big_parts + 4 * i;
    if (*(volatile int32_t*)&r[3] == 0) continue;  // being written
    const int m = *(volatile int32_t*)&r[1];
    if (*(volatile int32_t*)&r[2] < m) {
      const int j = atomicAdd(&r[2], 1);
      if (j < m) {
        t->v[0] = *(volatile int32_t*)&r[0];
        t->v[1] = t->v[2] = t->v[3] = -1;
        t->graph = 0;
        t->part = j;
        t->parts = m;
        t->pad = 0;
        return true;
      }
    }
    // exhausted: move the head past it (another warp may have done so)
    atomicCAS(&c->big_parts_head, i, i + 1);
  }
  return false;
}

// Pushes one task (lane-uniform); false if the ring is full.
__device__ bool queue_push_one(Warp& W, const Task& t) {
  const int lane = (int)lane_id();
  EnumCtl* ctl = s_blk.ctl;
  const int cap = s_blk.p->queue_cap;
  int ok = 0;
  if (lane == 0) {
    unsigned long long used = atomicAdd(&ctl->q_used, 1ULL);
    if (used + 1 > (unsigned long long)cap) {
      atomicAdd(&ctl->q_used, (unsigned long long)-1LL);
    } else {
      atomicAdd(&ctl->pending, 1ULL);
      graph_spawned(W, 1ULL);
      unsigned long long gp = atomicAdd(&ctl->q_tail, 1ULL);
      unsigned long long slot = gp % (unsigned long long)cap;
      volatile unsigned long long* st = s_blk.q_seq + slot;
      const unsigned long long free_tag = slot_free_tag(gp, cap);
      int64_t spins = 0;
      ok = 1;
      while (*st != free_tag) {
        if (++spins > s_blk.p->slot_spin_limit) {
          set_status(ctl, kStQueue, gp);
          ok = 2;
          break;
        }
        __nanosleep(64);
      }
      if (ok == 1) {
        s_blk.q_tasks[slot] = t;
        __threadfence();
        atomicExch(s_blk.q_seq + slot, free_tag + 1);
      }
    }
  }
  ok = __shfl_sync(kFull, ok, 0);
  return ok != 0;  // 2: the run is aborting; the task counts as handed over
}

// Lays the two-hop multiset of L out in order: the V ids met into aadj, each
// one's L position into ent, nL rows of the graph's U -> V lists end to end.
// With `count`, counts every id in the dense map on the way and lists the ids
// met (each once, at most capC of them) in `touched`; returns their number.
// Without `keep`, only that.
__device__ __noinline__ int lay_out_rows(const int32_t* L, int nL, int entries, bool count,
                                         bool keep) {
  Warp& W = this_warp();
  const int lane = (int)lane_id();
  const DevGraph& g = *W.gp;
  int32_t* map = W.A(W.sl().map);
  int32_t* touched = W.A(W.sl().touched);
  int32_t* aadj = W.A(W.sl().aadj);
  int32_t* ent = W.A(W.sl().ent);
  const int capC = W.sl().capC;
  const int vwords = (g.nV + 31) >> 5;
  const int32_t* rev_off = g.rev_off;
  const int32_t* rev_col = g.rev_col;
  uint32_t* gseen = W.gseen();
  // Large set-up without the shared bitmap: fire-and-forget counts and touch
  // bits, then the touched list in id order from the bitmap.
  const bool scan = count && use_gseen(W, entries, vwords);
  if (count && !scan) clear_seen(W, vwords);
  const bool shared = W.seen;
  uint32_t* seen = this_smem();
  int nt = 0;
  flat_rows(
      nL,
      [&](int r, int& beg, int& len) {
        const int u = L[r];
        beg = rev_off[u];
        len = rev_off[u + 1] - beg;
      },
      [&](bool valid, int pos) { return valid ? __ldg(rev_col + pos) : 0; },
      [&](bool valid, int r, int k, int w) {
        bool isnew = false;
        if (valid) {
          if (keep) {
            aadj[k] = w;
            ent[k] = r;
          }
          if (scan) {
            atomicAdd(&map[w], 1);
            atomicOr(&gseen[w >> 5], 1u << (w & 31));
          } else if (count) {
            isnew = count_first(shared, seen, map, w);
          }
        }
        const unsigned bal = __ballot_sync(kFull, isnew);
        const int at = nt + __popc(bal & lanemask_lt());
        if (isnew && at < capC) touched[at] = w;
        nt += __popc(bal);
      });
  if (scan) {
    __threadfence_block();
    __syncwarp();
    nt = collect_bits(gseen, vwords, touched, capC);
  } else if (count) {
    counts_done(W, touched, min(nt, capC));
  }
  __syncwarp();
  return nt;
}

// The transpose of the local adjacency: cadj lists, from coff[i], the L
// positions of candidate i (aadj: candidate of each entry, ent: its position;
// fill: all-zero, and again so on return).  Every lane has four slot
// reservations in flight before it uses any.
__device__ __noinline__ void t1_transpose(int entries, int nC) {
  Warp& W = this_warp();
  const int lane = (int)lane_id();
  const int32_t* aadj = W.A(W.sl().aadj);
  const int32_t* ent = W.A(W.sl().ent);
  const int32_t* ncnt = W.A(W.sl().ncnt);
  int32_t* coff = W.A(W.sl().coff);
  int32_t* fill = W.A(W.sl().fill);
  int32_t* cadj = W.A(W.sl().cadj);
  int run = 0;
  ROLLED for (int c0 = 0; c0 < nC; c0 += 32) {
    const int i = c0 + lane;
    int tot;
    const int ex = excl_scan(i < nC ? ncnt[i] : 0, &tot);
    if (i < nC) coff[i] = run + ex;
    run += tot;
  }
  if (lane == 0) coff[nC] = run;
  __syncwarp();
  ROLLED for (int j0 = 0; j0 < entries; j0 += 128) {
    int pp[4], rr[4], ss[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int j = j0 + k * 32 + lane;
      pp[k] = j < entries ? aadj[j] : -1;
      rr[k] = j < entries ? ent[j] : 0;
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) ss[k] = pp[k] >= 0 ? atomicAdd(&fill[pp[k]], 1) : 0;
#pragma unroll
    for (int k = 0; k < 4; ++k)
      if (pp[k] >= 0) cadj[coff[pp[k]] + ss[k]] = rr[k];
  }
  __syncwarp();
  ROLLED for (int i = lane; i < nC; i += 32) fill[i] = 0;
  __syncwarp();
}

// Entries above which the set-up of a root on its way to the bitmap tier keeps
// no copy of them.  Whole calls, a copy of all of them kept / none above the
// line: 900 roots of about 33,000 entries 2.30 / 1.90 ms, 8,000 of 374,000 35.4 /
// 31.9 ms.  Lower lines cost small roots the second walk over short rows:
// 256 graphs of 20,000 to 40,000 edges 166 ms with none kept, 164.6 up to 1,024,
// 161.7 up to 4,096, 161.4 up to 16,384.
constexpr int kKeepEntries = 4096;

// ---------------------------------------------------------------------------
// Task set-up (IterFinderWithMultipleVertex) and dispatch.
__device__ __noinline__ void run_task(const Task& t) {
  Warp& W = this_warp();
  const int lane = (int)lane_id();
  const DevGraph& g = *W.gp;
  int k = 1;
  while (k < 4 && t.v[k] >= 0) ++k;
  const int last = t.v[k - 1];
  int32_t* map = W.A(W.sl().map);
  int32_t* touched = W.A(W.sl().touched);
  int32_t* lv = W.A(W.sl().lv);

  // ---- L = common neighbours of the task vertices ----
  const int32_t* L;
  int nL;
  if (k == 1) {
    L = g.col + g.row_off[last];
    nL = g.row_off[last + 1] - g.row_off[last];
  } else {
    // Intersect: probe the smallest row against the others.
    int best = 0, bestlen = 0x7fffffff;
    ROLLED for (int i = 0; i < k; ++i) {
      int len = g.row_off[t.v[i] + 1] - g.row_off[t.v[i]];
      if (len < bestlen) {
        bestlen = len;
        best = i;
      }
    }
    const int32_t* sm = g.col + g.row_off[t.v[best]];
    int n = 0;
    ROLLED for (int b0 = 0; b0 < bestlen; b0 += 32) {
      int j = b0 + lane;
      bool in = j < bestlen;
      int u = in ? __ldg(sm + j) : 0;
      ROLLED for (int i = 0; i < k && in; ++i) {
        if (i == best) continue;
        const int32_t* row = g.col + g.row_off[t.v[i]];
        in = contains_sorted(row, g.row_off[t.v[i] + 1] - g.row_off[t.v[i]], u);
      }
      unsigned bal = __ballot_sync(kFull, in);
      if (in) lv[n + __popc(bal & lanemask_lt())] = u;
      n += __popc(bal);
    }
    __syncwarp();
    L = lv;
    nL = n;
  }
  if (nL == 0) return;
  if (nL > W.sl().capL) {
    set_status(s_blk.ctl, kStCapacity, ((unsigned long long)1 << 32) | (unsigned)nL);
    return;
  }

  // ---- two-hop multiset: counts in the per-warp dense map ----
  int32_t* aoff = W.A(W.sl().aoff);
  {
    int run = 0;
    ROLLED for (int c0 = 0; c0 < nL; c0 += 32) {
      int l = c0 + lane;
      int d = 0;
      if (l < nL) {
        int u = L[l];
        d = g.rev_off[u + 1] - g.rev_off[u];
      }
      int tot;
      int ex = excl_scan(d, &tot);
      if (l < nL) aoff[l] = run + ex;
      run += tot;
    }
    if (lane == 0) aoff[nL] = run;
    if (run > W.sl().capS) {
      set_status(s_blk.ctl, kStCapacity, ((unsigned long long)2 << 32) | (unsigned)run);
      return;
    }
  }
  __syncwarp();
  const int entries = aoff[nL];
  // A root that goes to the bitmap tier reads its entries once more, to set
  // them as bits; many of them (every warp's together do not fit L2) come from
  // the graph's rows again, which all warps share, rather than by way of this
  // warp's scratch.
  const bool laid_out = nL > W.gp->tier2_max_l || entries <= kKeepEntries;
  const int nt = lay_out_rows(L, nL, entries, true, laid_out);
  if (nt > W.sl().capC) {
    // Vertices beyond the touched list's room keep counts: clear the whole
    // map (the launch is failing; this keeps the invariant for the record).
    set_status(s_blk.ctl, kStCapacity, ((unsigned long long)3 << 32) | (unsigned)nt);
    ROLLED for (int i = lane; i < g.nV; i += 32) map[i] = 0;
    __syncwarp();
    return;
  }

  // ---- classify: R (count == |L|), Q (w < last), P (w > last) ----
  int32_t* cv = W.A(W.sl().cv);
  int32_t* ncnt = W.A(W.sl().ncnt);
  int32_t* bound = W.A(W.sl().bound);
  uint64_t sR = 0;
  unsigned long long nR = 0;
  int nq = 0, np = 0, nend = 0;
  int viol_first = 0x7fffffff;  // smallest R vertex below `last` (maximality witnesses)
  int nC = 0;
  // C is laid out [Q | P before this part | P of this part | P after it]; a
  // task that is not a part has only the middle P group.  The first level
  // pushes the candidates of this part; those before it act as Q, those after
  // it stay candidates of the children.
  int part = t.part, parts = t.parts;
  int cntQ = 0, cntPre = 0, cntIn = 0;
  {
    int cntC = 0;
    bool r_below = false;
    ROLLED for (int b0 = 0; b0 < nt; b0 += 32) {
      int i = b0 + lane;
      bool valid = i < nt;
      int w = valid ? touched[i] : 0;
      int c = valid ? map[w] : 0;
      bool isC = valid && c != nL;
      cntC += __popc(__ballot_sync(kFull, isC));
      cntQ += __popc(__ballot_sync(kFull, isC && w < last));
      r_below |= __ballot_sync(kFull, valid && c == nL && w < last) != 0u;
    }
    nC = cntC;
    const int np_all = cntC - cntQ;
    // A heavy maximal root is split into parts before its C is laid out.
    // Its first level costs about |P| pushes, each a pass over all of C.
    if (k == 1 && parts == 0 && !r_below && s_blk.p->range_work > 0 &&
        np_all >= 2 * s_blk.p->range_chunk &&
        (long long)np_all * cntC > (long long)s_blk.p->range_work) {
      const int m = min((np_all + s_blk.p->range_chunk - 1) / s_blk.p->range_chunk, kMaxParts);
      // A listed big root's parts go to big warps only; other roots' parts
      // fit every warp and take the common queue.
      const bool big_root = s_blk.p->n_big_warps > 0 && s_blk.p->big_flag[last];
      if (big_root ? big_parts_push(last, m) : queue_push_parts(t, m)) {
        part = 0;
        parts = m;
        acc(W.splits, 1);
      }
    }
    if (parts > 1) {
      ROLLED for (int b0 = 0; b0 < nt; b0 += 32) {
        int i = b0 + lane;
        bool valid = i < nt;
        int w = valid ? touched[i] : 0;
        bool isP = valid && map[w] != nL && w > last;
        int b = isP ? part_of(w, parts) : 0;
        cntPre += __popc(__ballot_sync(kFull, isP && b < part));
        cntIn += __popc(__ballot_sync(kFull, isP && b == part));
      }
    } else {
      cntIn = np_all;
    }
  }
  {
    int oQ = 0, oPre = cntQ, oIn = cntQ + cntPre, oPost = cntQ + cntPre + cntIn;
    ROLLED for (int b0 = 0; b0 < nt; b0 += 32) {
      int i = b0 + lane;
      bool valid = i < nt;
      int w = valid ? touched[i] : 0;
      int c = valid ? map[w] : 0;
      bool isR = valid && c == nL;
      bool isQ = valid && !isR && w < last;
      bool isP = valid && !isR && w > last;
      int b = (isP && parts > 1) ? part_of(w, parts) : part;
      bool isPre = isP && b < part, isIn = isP && b == part, isPost = isP && b > part;
      if (isR) {
        sR += g.vkey[w];
        ++nR;
        if (w < last) viol_first = min(viol_first, w);
      }
      unsigned bq = __ballot_sync(kFull, isQ);
      unsigned bpre = __ballot_sync(kFull, isPre);
      unsigned bin = __ballot_sync(kFull, isIn);
      unsigned bpost = __ballot_sync(kFull, isPost);
      const unsigned lt = lanemask_lt();
      int pos = -1;
      if (isQ) pos = oQ + __popc(bq & lt);
      if (isPre) pos = oPre + __popc(bpre & lt);
      if (isIn) pos = oIn + __popc(bin & lt);
      if (isPost) pos = oPost + __popc(bpost & lt);
      if (pos >= 0) {
        cv[pos] = w;
        ncnt[pos] = c;
        bound[pos] = kFree;
        map[w] = pos + 1;
      } else if (valid) {
        map[w] = 0;
      }
      oQ += __popc(bq);
      oPre += __popc(bpre);
      oIn += __popc(bin);
      oPost += __popc(bpost);
    }
    nq = cntQ + cntPre;  // first P position this task pushes
    np = cntIn;
    nend = nq + cntIn;
    W.shape = (unsigned long long)(unsigned)nC | ((unsigned long long)(part & 0xffff) << 32) |
              ((unsigned long long)(parts & 0xffff) << 48);
  }
  sR = warp_sum64(sR);
  nR = warp_sum64(nR);
  viol_first = warp_min_i(viol_first);
  __syncwarp();

  // ---- maximality of the task (src/IterFinderGpu.cu:800-822) ----
  bool ism = true;
  if (viol_first != 0x7fffffff) {
    if (k == 1) {
      ism = false;  // R[0] != root
    } else {
      // Every R vertex below `last` must already cover L_parent.
      int32_t* lp = W.A(W.sl().lp);
      const int32_t* Lpar;
      int nLp;
      if (k == 2) {
        Lpar = g.col + g.row_off[t.v[0]];
        nLp = g.row_off[t.v[0] + 1] - g.row_off[t.v[0]];
      } else {
        const int32_t* r0 = g.col + g.row_off[t.v[0]];
        int len0 = g.row_off[t.v[0] + 1] - g.row_off[t.v[0]];
        int n = 0;
        ROLLED for (int b0 = 0; b0 < len0; b0 += 32) {
          int j = b0 + lane;
          bool in = j < len0;
          int u = in ? __ldg(r0 + j) : 0;
          ROLLED for (int i = 1; i < k - 1 && in; ++i)
            in = contains_sorted(g.col + g.row_off[t.v[i]],
                                 g.row_off[t.v[i] + 1] - g.row_off[t.v[i]], u);
          unsigned bal = __ballot_sync(kFull, in);
          if (in) lp[n + __popc(bal & lanemask_lt())] = u;
          n += __popc(bal);
        }
        __syncwarp();
        Lpar = lp;
        nLp = n;
      }
      ROLLED for (int b0 = 0; b0 < nt && ism; b0 += 32) {
        int i = b0 + lane;
        int w = i < nt ? touched[i] : 0;
        bool cand = i < nt && w < last && map[w] == 0;  // R vertex below last
        // (map[w] == 0 marks R after classification)
        unsigned bal = __ballot_sync(kFull, cand);
        while (bal && ism) {
          int src = __ffs(bal) - 1;
          bal &= bal - 1;
          int ww = __shfl_sync(kFull, w, src);
          bool trivially = false;
          ROLLED for (int q = 0; q < k - 1; ++q) trivially |= (t.v[q] == ww);
          if (trivially) continue;
          const int32_t* rw = g.col + g.row_off[ww];
          int dw = g.row_off[ww + 1] - g.row_off[ww];
          // ww covers L_parent only if it has at least |L_parent| neighbours;
          // otherwise it is a new R vertex below `last`: not maximal here.
          if (dw < nLp) {
            ism = false;
            break;
          }
          bool all = true;
          ROLLED for (int j0 = 0; j0 < nLp && all; j0 += 32) {
            int j = j0 + lane;
            bool in = j >= nLp || contains_sorted(rw, dw, Lpar[j]);
            all = __all_sync(kFull, in);
          }
          if (!all) ism = false;
        }
      }
    }
  }
  if (!ism) {
    acc(W.nonmax, 1);
    ROLLED for (int i = lane; i < nt; i += 32) map[touched[i]] = 0;
    __syncwarp();
    return;
  }
  // the task's own biclique (once: parts after the first skip it)
  if (part == 0) {
    uint64_t sL = 0;
    ROLLED for (int l = lane; l < nL; l += 32) sL += g.ukey[L[l]];
    sL = warp_sum64(sL);
    acc(W.cnt, 1);
    acc(W.hash, biclique_hash(g, sL, (uint64_t)nL, sR, nR));
    if (s_blk.emit) emit_list(s_blk.ctl, emit_dst(*s_blk.p), W.gid, nL, L, nullptr);
  }
  bool done = nL <= 1 || np == 0;
  // ---- split (src/IterFinderGpu.cu:835-858) ----
  // A heavy root splits the same way in the sub-problem sharing mode: its
  // first level alone would otherwise run on one warp for the whole launch.
  if (!done && k < 4) {
    long long rest = np;
    bool split;
    if (s_blk.p->vertex_split)
      split = (rest > W.gp->bound_height || nL > W.gp->bound_height) &&
              rest * (long long)nL > (long long)W.gp->bound_size;
    else
      split = k == 1 && parts <= 1 && s_blk.p->root_split > 0 &&
              rest * (long long)nL > (long long)s_blk.p->root_split;
    if (split) {
      if (queue_push_children(t, k, nq, nC)) {
        acc(W.splits, 1);
        done = true;
      }
    }
  }
  if (!done) {
    const int K = words_k(nL);
    if (nL <= W.gp->tier2_max_l && nC <= W.gp->direct_max_c) {
      // ---- tier 2 directly ----
      uint32_t* at = reinterpret_cast<uint32_t*>(W.A(W.sl().ar_root));
      uint64_t* lkey = reinterpret_cast<uint64_t*>(at);
      int32_t* lid = reinterpret_cast<int32_t*>(at + 64 * K);
      ROLLED for (int l = lane; l < nL; l += 32) lkey[l] = g.ukey[L[l]];
      if (s_blk.emit)
        ROLLED for (int l = lane; l < nL; l += 32) lid[l] = L[l];
      uint32_t* end = reinterpret_cast<uint32_t*>(W.A(W.sl().ar_end));
      const ClsList cl = cls_build(
          at + cls_key_words(K), end, nC, nq, K, nL, &nend, ncnt, g.vkey, cv,
          ClsEdges{laid_out ? W.A(W.sl().aadj) : nullptr, W.A(W.sl().ent), map,
                   laid_out ? entries : 0, 1, L, g.rev_off, g.rev_col},
          nullptr);
      cls_run(cl, first_bits(nL, lane), nend, lkey, lid, sR, nR,
              cl.m + cls_list_words(cl.n, cl.K), end);
    } else {
      // ---- tier 1: local adjacency ----
      {
        uint64_t* ckey = W.A64(W.sl().ckey);  // hash key per candidate, for the pushes
        ROLLED for (int i = lane; i < nC; i += 32) ckey[i] = g.vkey[cv[i]];
      }
      int32_t* llevel = W.A(W.sl().llevel);
      int32_t* aadj = W.A(W.sl().aadj);
      int32_t* fill = W.A(W.sl().fill);
      int32_t* sidx = W.A(W.sl().sidx);
      if (!laid_out) lay_out_rows(L, nL, entries, false, true);
      ROLLED for (int l = lane; l < nL; l += 32) llevel[l] = 0;
      // aadj: L row -> C index (or -1 for R)
#pragma unroll 4
      for (int e = lane; e < entries; e += 32) aadj[e] = map[aadj[e]] - 1;
      ROLLED for (int i = lane; i < nC; i += 32) {
        fill[i] = 0;
        sidx[i] = -1;
      }
      __syncwarp();
      // (fill doubles as the sparse push's child-count array: left all-zero)
      t1_transpose(entries, nC);
      T1 t1;
      t1.L = L;
      t1.nL = nL;
      t1.nC = nC;
      t1.nq = nq;
      t1.nend = nend;
      t1.sRtask = sR;
      t1.nRtask = nR;
      uint64_t t1s = globaltimer_ns();
      uint64_t t2_before = W.ns_t2;
      tier1_run(t1);
      acc(W.ns_t1, (globaltimer_ns() - t1s) - (W.ns_t2 - t2_before));
    }
  }
  __syncwarp();
  ROLLED for (int i = lane; i < nt; i += 32) map[touched[i]] = 0;
  __syncwarp();
}

}  // namespace

// ---------------------------------------------------------------------------
// Maps a global root position to (graph, root vertex): positions are the
// graphs' root lists laid end to end (root_prefix[i] = roots before graph i).
__device__ __forceinline__ int graph_of_position(const long long* prefix, int n, long long pos) {
  int lo = 0, hi = n - 1;
  while (lo < hi) {
    int mid = (lo + hi + 1) >> 1;
    if (prefix[mid] <= pos) lo = mid;
    else hi = mid - 1;
  }
  return lo;
}

// Serving: claims a root of the oldest published graph that has roots left
// (lane 0).  Graphs are drained in publication order; a warp that finds the
// head graph exhausted moves the head on.  As for a static launch, the
// launch-wide pending count is raised before a claim but only while some
// published graph may have roots left: idle warps polling an empty arrival
// ring must leave it at zero, or the launch could never see itself quiet.
// A warp that saw the head below the tail just before another moved it past
// its graph claims nothing (that graph was exhausted), so the quiet test
// (pending == 0, head >= tail) loses no root.
__device__ __noinline__ bool serve_claim_root(Task* t) {
  Warp& W = this_warp();
  const ServeLink& L = s_blk.p->serve;
  volatile ServeCtl* sc = L.sctl;
  if (sc->arr_head >= sc->arr_tail) return false;
  // A launch that is ending takes no new roots: the host relaunches for them.
  if (*(volatile int32_t*)&s_blk.ctl->closing) return false;
  atomicAdd(&s_blk.ctl->pending, 1ULL);
  ROLLED for (int tries = 0; tries < 64; ++tries) {
    const unsigned long long h = sc->arr_head;
    if (h >= sc->arr_tail) break;
    const uint32_t blk = *(volatile const uint32_t*)&L.arr_blk[h % (unsigned long long)L.arr_cap];
    ServeGraph* sg = serve_graph(W, (int32_t)blk);
    const unsigned long long r = atomicAdd(&sg->next_root, 1ULL);
    const DevGraph& g = sg->g;
    if (r < (unsigned long long)g.n_roots) {
      t->v[0] = g.root_end - 1 - (g.root_offset + (int)r * g.root_stride);
      t->v[1] = t->v[2] = t->v[3] = -1;
      t->graph = (int32_t)blk;
      t->part = t->parts = t->pad = 0;
      return true;
    }
    atomicCAS((unsigned long long*)&L.sctl->arr_head, h, h + 1);
  }
  atomicAdd(&s_blk.ctl->pending, (unsigned long long)-1LL);
  return false;
}

// Serving: one task of graph `gid` finished (lane 0, after its results were
// added).  The task that brings the graph's pending count to zero writes the
// graph's completion record for the host.
__device__ __noinline__ void serve_task_done(int32_t gid) {
  Warp& W = this_warp();
  const ServeLink& L = s_blk.p->serve;
  ServeGraph* sg = serve_graph(W, gid);
  if (atomicAdd(&sg->pending, (unsigned long long)-1LL) != 1ULL) return;
  __threadfence();
  volatile ServeGraph* vs = sg;
  const unsigned long long c = vs->res[0], h = vs->res[1], nm = vs->res[2], req = vs->request;
  const unsigned long long pos = atomicAdd(&L.sctl->done_pos, 1ULL);
  volatile ServeDone* d = L.done + (pos % (unsigned long long)L.done_cap);
  d->request = req;
  d->count = c;
  d->hash = h;
  d->non_maximal = nm;
  // Every task of the graph reserved its records before it finished, so the
  // reservation counter now lies past all of them.
  d->emit_end = *(volatile unsigned long long*)&s_blk.ctl->emit_pos;
  __threadfence_system();
  d->seq = pos + 1;
}

// The persistent loop.  kTiers: the launch has a big tier (p.n_big_warps >
// 0); without it every warp uses `sl` and the tier code compiles away.
template <bool kTiers>
__device__ __forceinline__ void enum_main(const DevGraph* graphs, const long long* root_prefix,
                                          unsigned long long* gres, const EnumParams& p,
                                          const ScratchLayout& sl, EnumCtl* ctl, Task* q_tasks,
                                          unsigned long long* q_seq, const SlotPool& pool,
                                          int32_t* scratch, unsigned long long* exit_ns) {
  uint64_t t_start = globaltimer_ns();
  const int lane = (int)lane_id();
  const int warp_global = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  // Two tiers: the first n_big_warps warps hold the big layout, then the
  // launch's layout follows for every other warp.
  const bool big = kTiers && warp_global < p.n_big_warps;
  Warp& W = this_warp();
  if (threadIdx.x == 0) {
    s_blk.p = &p;
    s_blk.ctl = ctl;
    s_blk.q_tasks = q_tasks;
    s_blk.q_seq = q_seq;
    s_blk.graphs = graphs;
    s_blk.slots = pool.slots;
    s_blk.slot_bits = pool.bits;
    s_blk.bigslots = pool.big;
    s_blk.big_bits = pool.big_bits;
    s_blk.emit = p.emit;
    s_blk.deadline = p.time_limit_ns > 0 ? t_start + (uint64_t)p.time_limit_ns : 0;
    s_blk.import_words = pool.import_words;
    s_blk.nslot = pool.nslot;
    s_blk.nbig = pool.nbig;
    s_blk.import_cap = pool.import_cap;
    s_blk.import_l = pool.import_l;
    s_blk.import_s = pool.import_s;
    s_blk.prune = p.prune;
    s_blk.server = p.server;
    s_blk.share_min_work = p.share_min_work;
    s_blk.slot_records = p.slot_records;
    s_blk.eager_share = p.eager_share;
    s_blk.share_counts = p.share_counts;
    s_blk.touch_scan = p.touch_scan;
    s_blk.smem_words = sl.smem_words;
    s_blk.lookout = 0;
    s_sl[0] = sl;
    if (kTiers) s_sl[1] = p.big_sl;
  }
  // Shared memory of a warp: the first-touch bitmap of counting passes and the
  // bitmap tier take turns in it (clear_seen).
  uint32_t* smem =
      reinterpret_cast<uint32_t*>(enum_smem4) + (size_t)(threadIdx.x >> 5) * sl.smem_words;
  ROLLED for (int i = lane; i < sl.smem_words; i += 32) smem[i] = 0u;
  if (lane == 0) {
    if (!kTiers)
      W.base = scratch + (size_t)warp_global * (size_t)sl.words_per_warp;
    else
      W.base = big ? scratch + (size_t)warp_global * (size_t)p.big_sl.words_per_warp
                   : scratch + (size_t)p.n_big_warps * (size_t)p.big_sl.words_per_warp +
                         (size_t)(warp_global - p.n_big_warps) * (size_t)sl.words_per_warp;
    W.tier = big ? 1 : 0;
    W.seen = sl.seen_words && p.touch_scan <= 0;
    W.gp = graphs;
    W.gid = 0;
    W.cnt = W.hash = W.nonmax = W.splits = 0;
    W.ns_t1 = W.ns_t2 = W.n_t2 = 0;
    W.pushes = W.shape = 0;
    W.dem = 0;
    W.dem_t = -(1LL << 62);
  }
  __syncthreads();
  uint64_t ns_idle = 0, n_tasks = 0, max_task = 0, max_info = 0, max_split = 0;
  uint64_t max_pushes = 0, max_shape = 0;
  int32_t max_gid = 0;
  const long long nroots = p.server ? 0 : root_prefix[p.n_graphs];
  uint64_t idle_since = 0;
  uint64_t busy_ns = 0, last_done_ns = 0, idle_last = 0;
  while (true) {
    int ab = 0;
    if (lane == 0 && p.server) ab = *(volatile int32_t*)&p.serve.sctl->stop;  // shutting down
    if (__shfl_sync(kFull, ab, 0) || must_stop()) break;
    Task t;
    int have = 0;
    if (lane == 0) {
      have = queue_pop(&t) ? 1 : 0;
      if (!have && p.server) {
        have = serve_claim_root(&t) ? 1 : 0;
      } else if (!have) {
        // A big warp first takes parts of big roots, then the roots no other
        // warp has room for.
        if (kTiers && big && p.big_parts_cap > 0) have = big_parts_claim(&t) ? 1 : 0;
        if (!have && kTiers && big &&
            *(volatile long long*)&ctl->next_big < (long long)p.n_big_roots) {
          atomicAdd(&ctl->pending, 1ULL);
          long long b = (long long)atomicAdd((unsigned long long*)&ctl->next_big, 1ULL);
          if (b < (long long)p.n_big_roots) {
            t.v[0] = p.big_roots[b];
            t.v[1] = t.v[2] = t.v[3] = -1;
            t.graph = 0;
            t.part = t.parts = t.pad = 0;
            have = 1;
          } else {
            atomicAdd(&ctl->pending, (unsigned long long)-1LL);
          }
        }
        if (!have && *(volatile long long*)&ctl->next_root < nroots) {
          atomicAdd(&ctl->pending, 1ULL);
          // Claims positions until one is not a listed big root (at most
          // every remaining position).
          while (true) {
            long long r = (long long)atomicAdd((unsigned long long*)&ctl->next_root, 1ULL);
            if (r >= nroots) {
              atomicAdd(&ctl->pending, (unsigned long long)-1LL);
              break;
            }
            int gi = graph_of_position(root_prefix, p.n_graphs, r);
            const DevGraph& gg = graphs[gi];
            long long k = r - root_prefix[gi];
            const int v = gg.root_end - 1 - (int)(gg.root_offset + k * gg.root_stride);
            if (kTiers && p.big_flag[v]) continue;
            t.v[0] = v;
            t.v[1] = t.v[2] = t.v[3] = -1;
            t.graph = gi;
            t.part = t.parts = t.pad = 0;
            have = 1;
            break;
          }
        }
      }
    }
    have = __shfl_sync(kFull, have, 0);
    if (have) {
#pragma unroll
      for (int i = 0; i < 4; ++i) t.v[i] = __shfl_sync(kFull, t.v[i], 0);
      t.graph = __shfl_sync(kFull, t.graph, 0);
      t.part = __shfl_sync(kFull, t.part, 0);
      t.parts = __shfl_sync(kFull, t.parts, 0);
      if (idle_since != 0 && lane == 0) atomicSub(&ctl->idle_warps, 1);
      uint64_t tb = globaltimer_ns();
      const unsigned long long t1_before = W.ns_t1, t2_before = W.ns_t2;
      const unsigned long long pushes_before = W.pushes;
      if (t.v[0] >= 0) {
        W.gid = t.graph;
        W.gp = graph_at(W, t.graph);
        run_task(t);
      } else if (t.v[1] == 1) {
        tier1_from_slot(-2 - t.v[0]);  // an exported counts-tier child (sets the graph)
      } else {
        tier2_from_slot(-2 - t.v[0]);  // an exported bitmap sub-problem (sets the graph)
      }
      __syncwarp();
      // Results go to the task's graph.
      if (lane == 0) {
        unsigned long long* r = p.server ? serve_graph(W, W.gid)->res : gres + 3 * (size_t)W.gid;
        if (W.cnt) atomicAdd(&r[0], W.cnt);
        if (W.hash) atomicAdd(&r[1], W.hash);
        if (W.nonmax) atomicAdd(&r[2], W.nonmax);
        W.cnt = W.hash = W.nonmax = 0;
      }
      uint64_t te = globaltimer_ns();
      busy_ns += te - tb;
      last_done_ns = te - t_start;
      ++n_tasks;
      if (te - tb > max_task) {
        max_task = te - tb;
        int nl = t.v[0] >= 0 ? W.gp->row_off[t.v[0] + 1] - W.gp->row_off[t.v[0]] : 0;
        max_info = ((unsigned long long)(unsigned)t.v[0] << 32) | (unsigned)nl;
        max_split = (W.ns_t1 - t1_before) / 1000 | ((W.ns_t2 - t2_before) / 1000 << 32);
        max_pushes = W.pushes - pushes_before;
        max_shape = t.v[0] >= 0 ? W.shape : 0;
        max_gid = W.gid;
      }
      if (lane == 0) {
        __threadfence();
        if (p.server) serve_task_done(W.gid);
        atomicAdd(&ctl->pending, (unsigned long long)-1LL);
      }
      idle_since = 0;
      continue;
    }
    // 1: leave now; 2 (serving): nothing in flight and no published roots left.
    // A serving launch ends as a whole: the first warp to see it quiet for
    // idle_exit_ns sets `closing`, after which no warp claims a new root and
    // every warp leaves once nothing is pending.  Graphs published meanwhile
    // wait for the host's next launch, which gets the whole grid.  (Warps
    // that left one by one would let arrivals keep a launch of a few
    // remaining warps alive indefinitely.)
    int finished = 0;
    if (lane == 0) {
      if (p.server) {
        volatile ServeCtl* sc = p.serve.sctl;
        const bool quiet = *(volatile unsigned long long*)&ctl->pending == 0ULL;
        if (sc->stop || (quiet && *(volatile int32_t*)&ctl->closing)) finished = 1;
        else if (quiet && sc->arr_head >= sc->arr_tail)
          finished = 2;
      } else {
        finished = (*(volatile long long*)&ctl->next_root >= nroots &&
                    (!kTiers ||
                     *(volatile long long*)&ctl->next_big >= (long long)p.n_big_roots) &&
                    *(volatile unsigned long long*)&ctl->pending == 0ULL)
                       ? 1
                       : 0;
      }
    }
    finished = __shfl_sync(kFull, finished, 0);
    if (finished == 1) break;
    uint64_t now = globaltimer_ns();
    if (idle_since != 0) ns_idle += now - idle_last;
    idle_last = now;
    if (idle_since == 0) {
      idle_since = now;
      if (lane == 0) atomicAdd(&ctl->idle_warps, 1);
    } else if (p.server && finished == 2 && now - idle_since > (uint64_t)p.serve.idle_exit_ns) {
      // A serving launch ends once it has had nothing to do for a while; the
      // host launches again when graphs arrive.
      if (lane == 0) {
        atomicExch(&ctl->closing, 1);
        atomicSub(&ctl->idle_warps, 1);
      }
      break;
    } else if (now - idle_since > (uint64_t)p.idle_ns_limit) {
      if (lane == 0) set_status(ctl, kStTimeout, now - idle_since);
      break;
    }
    // Until something may have changed.  One idle warp of the block looks at
    // the queue, the others at the block's own flag in shared memory until they
    // take the lookout over: thousands of warps reading the launch's counters
    // keep one L2 slice busy and hold up everyone's memory traffic (a shard of
    // eight of the medium graph, on which most warps idle: 139-148 ms, with
    // every idle warp looking 153 ms; the 256-graph batch 164 / 165 ms).
    if (lane == 0) {
      bool look = false;
      ROLLED for (int r = 0; r < 16; ++r) {
        if (!look) look = atomicCAS(&s_blk.lookout, 0, 1) == 0;
        if (look) {
          const unsigned long long h = *(volatile unsigned long long*)&ctl->q_head;
          const unsigned long long q = *(volatile unsigned long long*)&ctl->q_tail;
          if (h < q || *(volatile unsigned long long*)&ctl->pending == 0ULL) break;
          if (p.server) {
            volatile ServeCtl* sc = p.serve.sctl;
            if (sc->arr_head < sc->arr_tail) break;
          }
        }
        __nanosleep(look ? 200 : 400);
      }
      if (look) atomicExch(&s_blk.lookout, 0);
    }
    __syncwarp();
  }
  __syncwarp();
  if (lane == 0) {
    if (W.splits) atomicAdd(&ctl->tasks_split, W.splits);
    atomicAdd(&ctl->ns_setup, (unsigned long long)(busy_ns - W.ns_t1 - W.ns_t2));
    atomicAdd(&ctl->ns_tier1, (unsigned long long)W.ns_t1);
    atomicAdd(&ctl->ns_tier2, (unsigned long long)W.ns_t2);
    atomicAdd(&ctl->ns_idle, (unsigned long long)ns_idle);
    atomicAdd(&ctl->n_tasks, (unsigned long long)n_tasks);
    atomicAdd(&ctl->n_tier2, (unsigned long long)W.n_t2);
    unsigned long long old = atomicMax(&ctl->max_task_ns, (unsigned long long)max_task);
    if (old < max_task) {
      atomicExch(&ctl->max_task_info, (unsigned long long)max_info);
      // (counts-tier us) | (bitmap-tier us << 32), and the task's graph
      atomicExch(&ctl->max_task_split, (unsigned long long)max_split);
      atomicExch(&ctl->max_task_graph, (unsigned long long)max_gid);
      atomicExch(&ctl->max_task_pushes, (unsigned long long)max_pushes);
      atomicExch(&ctl->max_task_shape, (unsigned long long)max_shape);
    }
  }
  if (p.record_exit) {
    // Per block: when its last task finished, and its warps' summed busy time.
    if (threadIdx.x == 0) {
      s_blk.last_ns = 0;
      s_blk.busy_ns = 0;
    }
    __syncthreads();
    if (lane == 0) {
      atomicMax(&s_blk.last_ns, (unsigned long long)last_done_ns);
      atomicAdd(&s_blk.busy_ns, (unsigned long long)busy_ns);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      exit_ns[blockIdx.x] = s_blk.last_ns;
      exit_ns[gridDim.x + blockIdx.x] = s_blk.busy_ns;
    }
  }
}

__global__ void __launch_bounds__(kEnumThreads, kEnumMinBlocks)
    mbe_enum_kernel(const DevGraph* graphs, const long long* root_prefix,
                    unsigned long long* gres, const __grid_constant__ EnumParams p,
                    const __grid_constant__ ScratchLayout sl, EnumCtl* ctl, Task* q_tasks,
                    unsigned long long* q_seq, SlotPool pool, int32_t* scratch,
                    unsigned long long* exit_ns) {
  enum_main<false>(graphs, root_prefix, gres, p, sl, ctl, q_tasks, q_seq, pool, scratch, exit_ns);
}

__global__ void __launch_bounds__(kEnumThreads, kEnumMinBlocks)
    mbe_enum_kernel_tiers(const DevGraph* graphs, const long long* root_prefix,
                          unsigned long long* gres, const __grid_constant__ EnumParams p,
                          const __grid_constant__ ScratchLayout sl, EnumCtl* ctl, Task* q_tasks,
                          unsigned long long* q_seq, SlotPool pool, int32_t* scratch,
                          unsigned long long* exit_ns) {
  enum_main<true>(graphs, root_prefix, gres, p, sl, ctl, q_tasks, q_seq, pool, scratch, exit_ns);
}

}  // namespace gmbe
