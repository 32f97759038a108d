// Device-side view of a regex scan, shared by the DFA kernels (ws_dfa.cu) and
// the literal verify kernel (ws_literal.cu), which finds the candidates of
// regexes whose matches begin with known prefixes.
#pragma once
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include "ws_dfa.h"

namespace ws {

constexpr uint32_t F_MATCH = 0x80000000u;
constexpr uint32_t F_DEAD = 0x40000000u;
constexpr uint32_t F_MASK = 0x3FFFFFFFu;
// Leftmost-first walks in the parallel pass stop after kLfCap bytes; the
// chain kernel finishes such a walk only if it picks that start (picked
// matches do not overlap, so that work is bounded by the input).
constexpr uint64_t kLfCap = 1024;
constexpr uint32_t kLfNone = 0xFFFFFFFFu;  // no match from this start (or a duplicate start)
constexpr uint32_t kLfLong = 0xFFFFFFFEu;  // cut off after a match
constexpr uint32_t kLfOpen = 0xFFFFFFFDu;  // cut off before any match
constexpr uint32_t kLfTodo = 0xFFFFFFFCu;  // (in a sorted candidate) the walk is still to be done

// A candidate: regex, start, end of a match from there, and its rank among the
// regex's candidates, with kEndKnown when the end is the leftmost-first one (or
// kLfLong).
struct KCand { uint32_t r, s, e, rank; };
constexpr uint32_t kEndKnown = 0x80000000u;
struct Event { uint32_t e, state, q, tag; };

// counters block (unsigned long long[16]):
//  [0] K count  [1] event count  [2] error flags  [3..3+kFixRounds] round-changed flags
//  [8] chunk re-walks of the fix-up  [9] bytes those re-walks stepped
//  [10] boundary guesses that were the true state  [11] boundary guesses
//  [12] the prefix candidates were given up (the gated groups walk)
//  [13] steps of the walks from prefixes (weighted)  [14] finished verify blocks
//  [15] some regex's candidates are more than a block resolves alone
enum { C_K = 0, C_EV = 1, C_ERR = 2, C_ROUND = 3, C_FIX = 8, C_REWALK = 9, C_HITS = 10, C_GUESSES = 11, C_GATE = 12,
       C_WORK = 13, C_TICKET = 14, C_LONG = 15 };
// error bits in ctr[C_ERR]: 1 candidate overflow, 2 event overflow, 4 a
// bounded device-side wait ran out
constexpr unsigned long long kErrTimeout = 4;

struct DevTables {
  const GroupDev* groups;
  const uint32_t* fwd;
  const uint32_t* hot;
  const uint32_t* rev;
  const uint32_t* lf;
  const uint8_t* cls;
  const uint32_t* mptr;
  const uint32_t* mlist;
  const uint32_t* rmptr;
  const uint32_t* rmlist;
  const uint4* lfinfo;   // per regex: {lf_off, lf_start row, group, classes}
  const uint32_t* lfx;   // per regex: context DFA starts and end-step flags (8 words)
  const uint32_t* pid;
  uint32_t n_groups, n_regex, n_spec;
  // Groups whose candidates the prefix filter finds walk only when it gave up
  // (ctr[C_GATE]): the speculative groups from n_walk and the context groups
  // from n_ctx_walk on (n_spec and n_groups when the filter does not run).
  uint32_t n_walk, n_ctx_walk;
};

struct ScanPtrs {
  const uint8_t* data;
  uint64_t len;
  unsigned long long* ctr;
  KCand* k;
  uint64_t k_cap;
  Event* ev;
  uint64_t ev_cap;
  uint32_t* guess;
  uint32_t* used;
  uint32_t* end;
  uint32_t* spec;
  uint32_t* conv;
  uint32_t* round;
  uint32_t* ckpt;
  uint32_t* count;
  uint32_t* offs;
  unsigned long long* pair;     // candidates by regex: start << 32 | leftmost-first end
  unsigned long long* pair2;    // the same size, for merging
  unsigned long long* rmark;    // visited reverse-walk triples, or null (state numbers too large, or full K)
  uint32_t full_k;              // report every (start, end) of K, not only distinct starts (diagnostics)
  uint32_t count_guesses;       // profiled speculative scans: the speculative groups whose guesses are counted
  uint64_t n_chunks, chunk, nck;
  ws_match* out;
  uint64_t out_cap;
  unsigned long long* out_counter;
  const uint32_t* item_end;     // batch item ends (n_items), else null
  uint32_t n_items;
  unsigned long long* cursor64;  // stream: per-regex find_iter position, else null
  uint64_t base, frontier;
};

// One slot of an append buffer, one atomic per group of converged lanes.
__device__ __forceinline__ unsigned long long warp_append(unsigned long long* counter) {
  cooperative_groups::coalesced_group g = cooperative_groups::coalesced_threads();
  unsigned long long base = 0;
  if (g.thread_rank() == 0) base = atomicAdd(counter, (unsigned long long)g.size());
  base = g.shfl(base, 0);
  return base + g.thread_rank();
}

// Stores candidate i of K with its rank among its regex's candidates (the
// per-regex counts size the resolution's lists, the rank is its place in one).
__device__ __forceinline__ void store_k(const ScanPtrs& p, unsigned long long i, uint32_t r, uint32_t s, uint32_t e,
                                        uint32_t rank_known) {
  if (i < p.k_cap) p.k[i] = KCand{r, s, e, rank_known};
  else atomicOr(&p.ctr[C_ERR], 1ull);
}

__device__ __forceinline__ void emit_k(const ScanPtrs& p, uint32_t r, uint32_t s, uint32_t e, uint32_t known = 0) {
  const unsigned long long i = warp_append(&p.ctr[C_K]);
  if (i < p.k_cap) p.k[i] = KCand{r, s, e, atomicAdd(&p.count[r], 1u) | known};
  else atomicOr(&p.ctr[C_ERR], 1ull);
}

// The same where a thread may emit many in turn: a candidate is counted whether it
// fits or not, so that its two atomics do not wait for one another (1,000 regexes
// that match at the same places of 256 MiB: 3,000 -> 2,190 us a scan, 2,160 to
// 2,290 before candidates had ranks); the lists of a scan whose candidates did not
// fit are not read.  (In the loops of the plain and the context kernel that order
// cost more than it saved: 20 regexes with assertions over 32 MiB 138 -> 171 us.)
__device__ __forceinline__ void emit_k_ahead(const ScanPtrs& p, uint32_t r, uint32_t s, uint32_t e) {
  const uint32_t rank = atomicAdd(&p.count[r], 1u);
  store_k(p, warp_append(&p.ctr[C_K]), r, s, e, rank);
}

// Context of a byte for the assertions (byte_context in ws_regex.h).
__device__ __forceinline__ uint32_t ctx_of(uint32_t b) {
  if (b == '\n') return CTX_NL;
  const bool w = (b - '0' < 10u) || ((b | 0x20u) - 'a' < 26u) || b == '_';
  return w ? CTX_WORD : CTX_OTHER;
}

// Leftmost-first end of a match of regex r from start s: the walk of the
// regex's priority DFA from s, remembering the last match position, until the
// DFA dies or the item or input ends.  kLfNone when no match starts at s;
// kLfLong or kLfOpen when the walk was cut off after `cap` bytes, with or
// without a match so far.  `steps`: the bytes it stepped.
__device__ inline uint32_t lf_walk(const DevTables& t, const ScanPtrs& p, uint32_t r, uint32_t s, uint64_t cap,
                                   uint32_t* steps = nullptr) {
  const uint4 info = t.lfinfo[r];
  const uint8_t* cm = t.cls + info.z * 256;
  const uint32_t* tab = t.lf + info.x;
  uint32_t st = info.y;
  int64_t last = -1;
  const uint64_t stop = p.n_items ? min(p.len, (uint64_t)item_end_of(p.item_end, p.n_items, s)) : p.len;
  const uint32_t* x = t.lfx + 8 * (size_t)r;
  const bool context = __ldg(x) != 0;
  if (context) {
    // context DFA (build_context_lf_dfa): start row by the byte before s, a
    // match flag on the byte at pos ends a match at pos, the end step after
    // the last byte of the input or item
    const uint64_t lo = p.n_items ? item_start_of(p.item_end, p.n_items, s) : 0;
    st = __ldg(x + 1 + (s == lo ? CTX_BEGIN : ctx_of(__ldg(p.data + s - 1))));
  }
  // four bytes at a time: their classes are looked up together, so that a step
  // waits for its table load only
  const uint64_t cut = cap < stop - s ? s + cap : stop;  // (s < stop)
  uint64_t pos = s;
  bool dead = false;
  while (pos < cut && !dead) {
    const uint32_t n = cut - pos < 4 ? (uint32_t)(cut - pos) : 4u;
    uint32_t c[4];
#pragma unroll
    for (uint32_t k = 0; k < 4; ++k) c[k] = k < n ? __ldg(p.data + pos + k) : 0u;
#pragma unroll
    for (uint32_t k = 0; k < 4; ++k) c[k] = __ldg(cm + c[k]);
#pragma unroll
    for (uint32_t k = 0; k < 4; ++k) {
      if (k < n && !dead) {
        const uint32_t w = __ldg(tab + st * info.w + c[k]);
        if (context && (w & F_MATCH)) last = (int64_t)pos;
        if (w & F_DEAD) {
          dead = true;
        } else {
          st = w & F_MASK;
          ++pos;
          if (!context && (w & F_MATCH)) last = (int64_t)pos;
        }
      }
    }
  }
  if (steps) *steps = (uint32_t)(pos - s);
  if (!dead && pos < stop) return last < 0 ? kLfOpen : kLfLong;
  if (!dead && context && __ldg(t.lf + __ldg(x + 5) + st)) last = (int64_t)stop;
  return last < 0 ? kLfNone : (uint32_t)last;
}

// The device state of one regex scan between its stages (regex_begin, the
// literal scan that adds candidates, regex_finish).
struct RegexScan {
  ScanPtrs p;
  DevTables t;
  uint64_t k_cap = 0, n_q = 0;
  uint32_t clear_words = 0;  // u32 words from p.ctr on that start as zero
  const DeviceBuffer* walk_tables[4] = {};  // what lf_walk reads
  bool prefixes = false;  // the literal scan finds the covered groups' candidates
};

// Prefixes of the covered regexes: entries {first 4 bytes, next 4 bytes, their
// mask, regex} by bucket of the bytes' hash.
struct PrefixDev {
  const uint32_t* range;
  const uint4* entry;
  uint32_t shift, mul;
};

}  // namespace ws
