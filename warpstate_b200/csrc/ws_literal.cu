// Literal prefilter + verify for sm_100a.
//
// Replaces the reference's two WGSL passes, literal_prefilter
// (core/src/gpu/shader.rs:18-101) and literal_verify (core/src/gpu/shader.rs:106-236).
//
// Kernel 1, literal_filter_kernel (streams the input once, HBM-bound):
//   stage 1   every thread owns 16 input bytes per step (one 16-byte coalesced
//             load, issued one step ahead).  It looks up the 4-byte grams at the
//             P-aligned positions in a nibble table staged in shared memory and
//             forms a 16-bit mask of positions that may start a literal (see
//             LiteralPlan); the warp's 512-byte block is copied to shared memory.
//   compact   popc prefix sums put the flagged positions of the warp into a
//             shared-memory queue, so stage 1.5 runs with all 32 lanes busy.
//   stage 1.5 each queued position reads its 8-byte window from shared memory
//             and checks, at every prefix length that has literals, a
//             multiply-shift key of the first min(len, 8) bytes against a Bloom
//             bitmap of the literals' prefixes in shared memory.
//   survivors are appended to a compact position list with one atomic per warp
//             (ballot + popc).  If the list is full, the position is verified in
//             place instead, so results never depend on the list's capacity.
// Kernel 1 of most sets is literal_gram_kernel (see its comment): stage 1 only,
//             no compaction; stage 1.5 moves to kernel 2.  The kernel above is
//             for sets with literals of one or two bytes and for sets whose
//             grams crowd their alphabet.
// Kernel 2, literal_verify_kernel: the reference's per-position algorithm on the
//             surviving positions only: FNV-1a probe of the LiteralPrefilterTable
//             partition at each non-empty prefix length (shader.rs:59-98) and an
//             exact compare of every entry whose hash is equal (shader.rs:174-227).
//
// The output is contract L: every overlapping occurrence of every literal.
#include <cuda_runtime.h>


#include "ws_internal.h"
#include "ws_launch.h"
#include "ws_scan.h"

namespace ws {

namespace {

constexpr int kThreads = 1024;
constexpr int kWarps = kThreads / 32;
constexpr uint32_t kBloomBits = 18;  // 2^18-bit Bloom bitmap (32 KiB)

struct LitArgs {
  const uint8_t* data;
  uint64_t len;
  const uint32_t* filter;
  uint32_t filter_words;
  uint32_t bits;
  uint32_t period;
  uint32_t parts;            // bit i: prefix length i+1 has literals
  uint32_t bloom_parts;      // bit i: prefix length i+1 is in the prefix Bloom (literals, regex prefixes)
  const uint32_t* short_bits;
  const uint32_t* bloom;
  const uint4* info;
  const uint8_t* lit_bytes;
  uint2 meta[HASH_WINDOW];  // per prefix length: {first bucket, bucket mask} (LiteralPrefilterTable partition)
  const uint2* ranges;
  const uint4* entries;      // {hash, literal, its bytes 8..11, their mask}
  ws_match* out;
  uint64_t cap;
  unsigned long long* counter;
  uint32_t* survivors;       // candidate start positions (low 32 bits)
  unsigned long long* survivor_count;
  uint64_t survivor_cap;
  const uint32_t* item_end;  // batch: ascending item ends (n_items), else null
  uint32_t n_items;
  uint64_t min_end;          // stream: matches ending at or before it were reported
  uint64_t max_start;        // shard: matches starting at or after it belong to the next shard
  uint32_t gram_len;        // stage-1 gram bytes: 3, 4, 8 or 16 (8 and 16 with P = 4)
  uint32_t parts16;          // stage-1.5b key lengths (bit i: i+1 bytes)
  const uint32_t* bloom2;    // stage-1.5b bitmap (2^kBloom2Bits bits, L2), or null
  const uint8_t* big;        // stage-1b gram table (2^kBigBits bytes, L2), or null (compacting kernel)
  // gram kernel: stage 1 has 2^gram_word_bits words, the phase table
  // 2^(32 - phase_shift) bytes
  const uint32_t* gram_bloom;
  uint32_t gram_word_bits;
  uint32_t gram_bits;        // bits per gram in it; 0: the compacting kernel ran
  const uint8_t* phase;
  uint32_t phase_shift;
  uint32_t slot_chunk;       // survivor slots a warp reserves at a time
  uint32_t two;              // 2, unknown to the compiler: a sum of bits stays on the multiply pipe
  uint32_t fold;             // ASCII case-insensitive: input bytes A-Z read as a-z
};

__device__ __forceinline__ uint4 fold16(uint4 v) {
  return make_uint4(ascii_fold4(v.x), ascii_fold4(v.y), ascii_fold4(v.z), ascii_fold4(v.w));
}

__device__ __forceinline__ uint32_t nib(const uint32_t* tab, uint32_t gram, uint32_t bits) {
  uint32_t h = (gram * 0x9E3779B1u) >> (32 - bits);
  return (tab[h >> 3] >> ((h & 7) << 2)) & 0xFu;
}

// Loads the 16 bytes of vector v, zero-filling past the end of the input.
__device__ __forceinline__ uint4 load_vec(const uint8_t* data, uint64_t len, uint64_t v) {
  uint64_t off = v * 16;
  if (off + 16 <= len) return __ldg(reinterpret_cast<const uint4*>(data + off));
  uint32_t w[4] = {0, 0, 0, 0};
#pragma unroll
  for (int k = 0; k < 16; ++k) {
    uint64_t p = off + k;
    if (p < len) w[k >> 2] |= (uint32_t)__ldg(data + p) << ((k & 3) * 8);
  }
  return make_uint4(w[0], w[1], w[2], w[3]);
}

// Bytes [a, a + 4) of the input for a 4-aligned a, zero past its end.
__device__ __forceinline__ uint32_t word_at(const uint8_t* d, uint32_t len, uint32_t a) {
  if (a + 4 <= len) return __ldg(reinterpret_cast<const uint32_t*>(d + a));
  uint32_t x = 0;
  for (uint32_t k = 0; k < 4; ++k)
    if (a + k < len) x |= (uint32_t)__ldg(d + a + k) << (8 * k);
  return x;
}

// word_at for the scan's input, case-folded for case-insensitive sets.
__device__ __forceinline__ uint32_t input_word(const LitArgs& a, uint32_t len, uint32_t at) {
  const uint32_t w = word_at(a.data, len, at);
  return a.fold ? ascii_fold4(w) : w;
}

// The reference's per-position probe and exact verify (stage 2), in two parts
// so that a survivor's loads go out together: probe_literals hashes the
// position's first eight bytes and reads the bucket of every prefix length that
// has literals, verify_literals walks the buckets and compares.  Inputs of one
// launch are below 4 GiB.
struct Probe {
  uint32_t h[8];
  uint2 r[8];
};

__device__ __forceinline__ void probe_literals(const LitArgs& a, uint32_t lo, uint32_t hi, uint32_t rem, Probe& pr) {
  uint32_t h = 2166136261u;
#pragma unroll
  for (uint32_t i = 0; i < HASH_WINDOW; ++i) {
    h = (h ^ (((i < 4 ? lo : hi) >> (8 * (i & 3))) & 0xFFu)) * 16777619u;
    pr.h[i] = h;
    pr.r[i] = ((a.parts >> i) & 1u) && i < rem ? __ldg(a.ranges + a.meta[i].x + (h & a.meta[i].y)) : make_uint2(0, 0);
  }
}

// Compares literals of the probed buckets at s; x0 is the (folded) word at
// s & ~3, `next` the four bytes from s + 8 on: an entry tells by four more bytes
// whether its literal is worth looking at (k-mers share their first eight bytes
// with a quarter of all positions: 20,000 of them over 2 GiB 596 -> 580 us a scan).  Literal bytes start 4-aligned in a buffer padded to 16 bytes; four
// words of literal and input are read together.
template <class Sink>
__device__ __forceinline__ void verify_literals(const LitArgs& a, uint32_t s, uint32_t x0, uint32_t next, const Probe& pr, Sink&& sink) {
  const uint32_t len = (uint32_t)a.len, rem = len - s, w0 = s & ~3u, sh = (s & 3) * 8;
  uint32_t part = 0, e = 0;  // the next entry: bucket `part`, place e
  while (true) {
    uint32_t found = 0xFFFFFFFFu;
#pragma unroll
    for (uint32_t i = 0; i < HASH_WINDOW; ++i) {
      if (i < part || found != 0xFFFFFFFFu) continue;
      for (; e < pr.r[i].y && found == 0xFFFFFFFFu; ++e) {
        const uint4 ent = __ldg(a.entries + pr.r[i].x + e);
        if (ent.x == pr.h[i] && !((ent.z ^ next) & ent.w)) found = ent.y;
      }
      part = i;
      if (found == 0xFFFFFFFFu) e = 0;
    }
    if (found == 0xFFFFFFFFu) return;
    const uint4 info = __ldg(a.info + found);  // {offset, len, pattern id, 0}
    if (info.y > rem) continue;
    const uint32_t* lit = reinterpret_cast<const uint32_t*>(a.lit_bytes + info.x);
    uint32_t differ = 0, cur = x0;
    for (uint32_t k = 0; k < info.y && !differ; k += 16) {
      uint32_t l[4], d[5];
      d[0] = cur;
#pragma unroll
      for (uint32_t j = 0; j < 4; ++j) {
        const bool on = k + 4 * j < info.y;
        l[j] = on ? __ldg(lit + (k >> 2) + j) : 0u;
        d[j + 1] = on ? input_word(a, len, w0 + k + 4 * j + 4) : 0u;
      }
#pragma unroll
      for (uint32_t j = 0; j < 4; ++j) {
        const uint32_t left = info.y > k + 4 * j ? info.y - k - 4 * j : 0u;
        const uint32_t m = left >= 4 ? 0xFFFFFFFFu : ((1u << (8 * left)) - 1u);
        differ |= (l[j] ^ __funnelshift_r(d[j], d[j + 1], sh)) & m;
      }
      cur = d[4];
    }
    if (differ || s + info.y <= a.min_end) continue;
    if (a.n_items && s + info.y > item_end_of(a.item_end, a.n_items, s)) continue;  // crosses items
    sink(info.z, s, s + info.y);
  }
}

// A match straight to the output.
__device__ __forceinline__ void report_match(const LitArgs& a, uint32_t pid, uint32_t s, uint32_t e) {
  const unsigned long long idx = warp_append(a.counter);
  if (idx < a.cap) a.out[idx] = ws_match{pid, s, e};
}

// probe_literals and verify_literals one prefix length and one word at a time,
// for inputs whose survivors do not fit the list.  The probes in flight together
// are more code and registers: inlined in the compacting kernels they spilled
// the main loop (11-mers over 128 MiB 313 us a scan, this way 246).
template <class Sink>
__device__ __forceinline__ void verify_by_word(const LitArgs& a, uint32_t s, Sink&& sink) {
  if (s >= a.max_start) return;
  const uint32_t len = (uint32_t)a.len, rem = len - s, w0 = s & ~3u, sh = (s & 3) * 8;
  const uint32_t x0 = input_word(a, len, w0), x1 = input_word(a, len, w0 + 4), x2 = input_word(a, len, w0 + 8);
  const uint32_t lo = __funnelshift_r(x0, x1, sh), hi = __funnelshift_r(x1, x2, sh);
  const uint32_t window = rem < HASH_WINDOW ? rem : HASH_WINDOW;
  uint32_t h = 2166136261u;
#pragma unroll 1
  for (uint32_t i = 0; i < window; ++i) {
    h = (h ^ (((i < 4 ? lo : hi) >> (8 * (i & 3))) & 0xFFu)) * 16777619u;
    if (!((a.parts >> i) & 1u)) continue;
    const uint2 r = __ldg(a.ranges + a.meta[i].x + (h & a.meta[i].y));
#pragma unroll 1
    for (uint32_t e = 0; e < r.y; ++e) {
      const uint4 ent = __ldg(a.entries + r.x + e);
      if (ent.x != h) continue;
      const uint4 info = __ldg(a.info + ent.y);  // {offset, len, pattern id, 0}
      if (info.y > rem) continue;
      const uint32_t* lit = reinterpret_cast<const uint32_t*>(a.lit_bytes + info.x);
      bool eq = true;
      uint32_t cur = x0;
#pragma unroll 1
      for (uint32_t k = 0; k < info.y && eq; k += 4) {
        const uint32_t nxt = input_word(a, len, w0 + k + 4), left = info.y - k;
        const uint32_t m = left >= 4 ? 0xFFFFFFFFu : ((1u << (8 * left)) - 1u);
        eq = ((__ldg(lit + (k >> 2)) ^ __funnelshift_r(cur, nxt, sh)) & m) == 0;
        cur = nxt;
      }
      if (!eq || s + info.y <= a.min_end) continue;
      if (a.n_items && s + info.y > item_end_of(a.item_end, a.n_items, s)) continue;  // crosses items
      sink(info.z, s, s + info.y);
    }
  }
}

// 16-bit mask of owned positions that may start a literal (stage 1).  w[0..3]
// are the thread's own words; w[4..7] are the next thread's words (w[4] is
// needed by the P = 1 and P = 2 layouts and by lane 31, w[5..7] by grams
// longer than 4 bytes).  The layout is a compile-time choice (P = period,
// G = gram bytes, LONG / SHORT = literals of >= 4 / < 4 bytes present).
template <int P, int G, bool LONG, bool SHORT>
__device__ __forceinline__ uint32_t stage1(const uint32_t* filt, const uint32_t* shortb, const uint32_t (&w)[8],
                                           uint32_t lane, uint32_t bits, const uint8_t* big) {
  uint32_t mask = 0;
  if (LONG) {
    if (G > 4 || P == 4) {
      // P = 4: grams of G bytes starting at the four aligned words; full
      // 32-bit hashes, the shared-memory table indexed by their top `bits`
      // bits, the L2 table (when present) by their top kBigBits bits
      uint32_t h[5];
#pragma unroll
      for (int j = 0; j < 5; ++j) {
        if (j == 4 && lane != 31) { h[4] = 0; break; }
        if (G == 4) h[j] = w[j] * 0x9E3779B1u;
        else if (G == 8) h[j] = mix_words(w[j], w[j + 1], 0, 0, 8);
        else h[j] = mix_words(w[j], w[j + 1], w[j + 2], w[j + 3], 16);
      }
      // with the stage-1b table, shared memory holds its stage 1 (the
      // two-bit blocked Bloom filter of long grams, or the bitmap derived
      // from the table) and the phase bits come from stage 1b alone
      auto phases = [&](uint32_t hf) -> uint32_t {
        if (big && G > 4) {
          const uint32_t m = lean2_mask(hf);
          return (filt[lean2_word(hf)] & m) == m ? (uint32_t)__ldg(big + (hf >> (32 - kBigBits))) : 0u;
        }
        if (big) {
          const uint32_t b = hf >> (32 - kLeanBits);
          return ((filt[b >> 5] >> (b & 31)) & 1u) ? (uint32_t)__ldg(big + (hf >> (32 - kBigBits))) : 0u;
        }
        const uint32_t hs = hf >> (32 - bits);
        return (filt[hs >> 3] >> ((hs & 7) << 2)) & 0xFu;
      };
      uint32_t n[5];
#pragma unroll
      for (int j = 0; j < 4; ++j) n[j] = phases(h[j]);
      n[4] = __shfl_down_sync(0xFFFFFFFFu, n[0], 1);
      if (lane == 31) n[4] = phases(h[4]);
      const uint32_t m = n[0] | (n[1] << 4) | (n[2] << 8) | (n[3] << 12) | (n[4] << 16);
      mask |= (m >> 3) & 0xFFFFu;
    } else if (P == 2) {
      uint32_t m = 0;
#pragma unroll
      for (int j = 0; j < 9; ++j) {
        uint32_t g = (j & 1) ? __funnelshift_r(w[j >> 1], w[(j >> 1) + 1], 16) : w[j >> 1];
        uint32_t n;
        if (big) {  // the bitmap of the stage-1b table, then its phase bits
          const uint32_t hf = g * 0x9E3779B1u, b = hf >> (32 - kLeanBits);
          n = ((filt[b >> 5] >> (b & 31)) & 1u) ? (uint32_t)__ldg(big + (hf >> (32 - kBigBits))) : 0u;
        } else {
          n = nib(filt, g, bits);
        }
        m |= n << (2 * j);
      }
      mask |= (m >> 1) & 0xFFFFu;
    } else {
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        uint32_t g = __funnelshift_r(w[j >> 2], w[(j >> 2) + 1], 8 * (j & 3));
        mask |= (nib(filt, g, bits) & 1u) << j;
      }
    }
  }
  if (SHORT) {
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      uint32_t g = __funnelshift_r(w[j >> 2], w[(j >> 2) + 1], 8 * (j & 3)) & 0xFFFFu;
      mask |= ((shortb[g >> 5] >> (g & 31)) & 1u) << j;
    }
  }
  return mask;
}

// Stage 1.5 key of the first pl bytes of a window (the host builds the Bloom
// bitmap with the same function over each literal's first min(len, 8) bytes).
__device__ __forceinline__ uint32_t prefix_key(uint32_t lo, uint32_t hi, uint32_t pl) {
  uint32_t ml = pl >= 4 ? 0xFFFFFFFFu : ((1u << (8 * pl)) - 1u);
  uint32_t mh = pl >= 8 ? 0xFFFFFFFFu : pl <= 4 ? 0u : ((1u << (8 * (pl - 4))) - 1u);
  uint32_t h = (lo & ml) * 0x9E3779B1u + (hi & mh) * 0x85EBCA77u + pl * 0xC2B2AE3Du;
  return h >> (32 - kBloomBits);
}

constexpr int kBlockWords = 136;  // 512 B warp block + 16 B of the next block + slack
constexpr int kQueue = 512;       // u16 offsets: at most 16 per lane

// A warp block with at least one stage-1 candidate: the block is copied to
// shared memory, the candidates are compacted into the queue (popc prefix
// sums), stage 1.5 runs with all lanes busy, survivors are appended with one
// atomic per warp.
template <int G>
__device__ __forceinline__ void process_block(const LitArgs& a, uint32_t* blk, uint16_t* queue, const uint32_t* bloom,
                                              uint32_t lane, const uint4& cur, const uint4& tail, uint32_t mask,
                                              uint32_t blk_base) {
  reinterpret_cast<uint4*>(blk)[lane] = cur;
  if (lane == 31) {
    reinterpret_cast<uint4*>(blk)[32] = tail;
    blk[132] = 0;
    blk[133] = 0;
  }
  __syncwarp();
  // compact the candidates of the warp into the queue
  const uint32_t cnt = __popc(mask);
  uint32_t incl = cnt;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    uint32_t y = __shfl_up_sync(0xFFFFFFFFu, incl, d);
    if (lane >= (uint32_t)d) incl += y;
  }
  const uint32_t total = __shfl_sync(0xFFFFFFFFu, incl, 31);
  uint32_t pos = incl - cnt;
  while (mask) {
    uint32_t i = __ffs(mask) - 1;
    mask &= mask - 1;
    queue[pos++] = (uint16_t)(lane * 16 + i);
  }
  __syncwarp();
  // stage 1.5 with all lanes busy, then a warp-aggregated append of survivors
  for (uint32_t k0 = 0; k0 < total; k0 += 32) {
    const uint32_t k = k0 + lane;
    bool keep = false;
    uint32_t off = 0;
    if (k < total) {
      off = queue[k];
      const uint32_t wi = off >> 2, sh = (off & 3) * 8;
      const uint32_t x0 = blk[wi], x1 = blk[wi + 1], x2 = blk[wi + 2];
      const uint32_t lo = __funnelshift_r(x0, x1, sh), hi = __funnelshift_r(x1, x2, sh);
      for (uint32_t m = a.bloom_parts; m; m &= m - 1) {  // prefix lengths of the set
        const uint32_t key = prefix_key(lo, hi, __ffs(m));
        keep |= (bloom[key >> 5] >> (key & 31)) & 1u;
      }
      if (G > 4 && keep) {
        // stage 1.5b: the first min(len, 16) bytes against the L2 bitmap
        const uint32_t x3 = blk[wi + 3], x4 = blk[wi + 4];
        const uint32_t y2 = __funnelshift_r(x2, x3, sh), y3 = __funnelshift_r(x3, x4, sh);
        bool k2 = false;
        for (uint32_t m = a.parts16; m; m &= m - 1) {
          const uint32_t key = prefix16_key(lo, hi, y2, y3, __ffs(m));
          k2 |= (__ldg(a.bloom2 + (key >> 5)) >> (key & 31)) & 1u;
        }
        keep = k2;
      }
    }
    const uint32_t ball = __ballot_sync(0xFFFFFFFFu, keep);
    if (ball) {
      unsigned long long wbase = 0;
      if (lane == 0) wbase = atomicAdd(a.survivor_count, (unsigned long long)__popc(ball));
      wbase = __shfl_sync(0xFFFFFFFFu, wbase, 0);
      if (keep) {
        const unsigned long long slot = wbase + __popc(ball & ((1u << lane) - 1u));
        const uint32_t s = blk_base + off;
        if (slot < a.survivor_cap) a.survivors[slot] = s;
        else verify_by_word(a, s, [&](uint32_t pid, uint32_t at, uint32_t e) {  // list full
          // (not report_match, whose code held registers of the loop: 262 -> 246 us)
          const unsigned long long idx = atomicAdd(a.counter, 1ull);
          if (idx < a.cap) a.out[idx] = ws_match{pid, at, e};
        });
      }
    }
  }
  __syncwarp();
}

// Inputs of one launch are below 4 GiB, so block, vector and byte indices are
// 32-bit.
template <int P, int G, bool LONG, bool SHORT>
__global__ void __launch_bounds__(kThreads, 1) literal_filter_kernel(const __grid_constant__ LitArgs a) {
  pdl_wait();  // (the verify kernel is not let in early: its waiting blocks cost up to 60 us of 370)
  extern __shared__ __align__(16) uint32_t smem[];
  uint32_t* filt = smem;                                 // filter_words
  uint32_t* bloom = filt + a.filter_words;               // 2^kBloomBits / 32 words
  uint32_t* shortb = bloom + (1u << (kBloomBits - 5));   // 2048 words when SHORT
  uint32_t* warpmem = shortb + (SHORT ? 2048 : 0);

  {
    const uint4* src = reinterpret_cast<const uint4*>(a.filter);
    uint4* dst = reinterpret_cast<uint4*>(filt);
    const uint32_t n4 = LONG ? a.filter_words / 4 : 0;
    for (uint32_t k = threadIdx.x; k < n4; k += kThreads) dst[k] = __ldg(src + k);
    const uint4* bs = reinterpret_cast<const uint4*>(a.bloom);
    uint4* bd = reinterpret_cast<uint4*>(bloom);
    for (uint32_t k = threadIdx.x; k < (1u << (kBloomBits - 7)); k += kThreads) bd[k] = __ldg(bs + k);
    if (SHORT) {
      const uint4* s2 = reinterpret_cast<const uint4*>(a.short_bits);
      uint4* d2 = reinterpret_cast<uint4*>(shortb);
      for (uint32_t k = threadIdx.x; k < 512; k += kThreads) d2[k] = __ldg(s2 + k);
    }
  }
  __syncthreads();

  const uint32_t lane = threadIdx.x & 31;
  const uint32_t warp = threadIdx.x >> 5;
  uint32_t* blk = warpmem + warp * (kBlockWords + kQueue / 2);
  uint16_t* queue = reinterpret_cast<uint16_t*>(blk + kBlockWords);
  const uint32_t len = (uint32_t)a.len;
  const uint32_t nvec = (uint32_t)((a.len + 15) >> 4);
  const uint32_t full_vecs = len >> 4;                 // vectors entirely inside the input
  const uint32_t nblk = (nvec + 31) >> 5;              // 512-byte warp blocks
  const uint32_t nwarps = gridDim.x * kWarps;
  const uint32_t bits = a.bits;
  auto load = [&](uint32_t v) -> uint4 {
    const uint4 x = v < full_vecs ? __ldg(reinterpret_cast<const uint4*>(a.data) + v)
                    : v < nvec ? load_vec(a.data, a.len, v) : make_uint4(0, 0, 0, 0);
    return a.fold ? fold16(x) : x;
  };

  uint32_t b = blockIdx.x * kWarps + warp;
  uint4 cur = make_uint4(0, 0, 0, 0);
  if (b < nblk) cur = load(b * 32 + lane);
  for (; b < nblk; b += nwarps) {
    // software pipeline: the next block's load is in flight during this one
    const uint32_t bn = b + nwarps;
    const uint4 nxt = bn < nblk ? load(bn * 32 + lane) : make_uint4(0, 0, 0, 0);
    const uint32_t v = b * 32 + lane;
    const uint4 tail = lane == 31 ? load(v + 1) : make_uint4(0, 0, 0, 0);
    uint32_t w[8] = {cur.x, cur.y, cur.z, cur.w, __shfl_down_sync(0xFFFFFFFFu, cur.x, 1), 0, 0, 0};
    if (G > 4) {
      w[5] = __shfl_down_sync(0xFFFFFFFFu, cur.y, 1);
      w[6] = __shfl_down_sync(0xFFFFFFFFu, cur.z, 1);
      w[7] = __shfl_down_sync(0xFFFFFFFFu, cur.w, 1);
    }
    if (lane == 31) {
      w[4] = tail.x;
      w[5] = tail.y;
      w[6] = tail.z;
      w[7] = tail.w;
    }
    uint32_t mask = stage1<P, G, LONG, SHORT>(filt, shortb, w, lane, bits, a.big);
    const uint32_t blk_base = b * 512;
    if (v >= full_vecs) {  // the input's last, partial vector (or past the end)
      const uint32_t base = v * 16;
      const uint32_t valid = len > base ? len - base : 0;
      mask &= (valid >= 16) ? 0xFFFFu : ((1u << valid) - 1u);
    }
    // most warp blocks have no candidate at all once stage 1b is in place
    if (__ballot_sync(0xFFFFFFFFu, mask != 0) == 0) {
      cur = nxt;
      continue;
    }
    process_block<G>(a, blk, queue, bloom, lane, cur, tail, mask, blk_base);
    __syncwarp();
    cur = nxt;
  }
}

// Stage 1 of 4-byte grams at every fourth position with the stage-1b table, split
// in two so that the L2 loads of a block are in flight while the previous block
// finishes: grams_issue hashes the five aligned grams of a lane (the fifth only on
// lane 31), looks them up in shared memory and starts the L2 loads of the passing
// ones; grams_finish combines them into the 16-bit candidate mask.
struct Grams {
  uint32_t n[5], bw[5];
};

__device__ __forceinline__ void grams_issue(const uint32_t* filt, const uint8_t* big, const uint32_t (&w)[5],
                                            uint32_t lane, Grams& s) {
#pragma unroll
  for (int j = 0; j < 5; ++j) {
    if (j == 4 && lane != 31) {
      s.n[4] = 0;
      s.bw[4] = 0;
      break;
    }
    const uint32_t hf = w[j] * 0x9E3779B1u;
    // stage 1: the 2^kLeanBits-bit bitmap derived from the stage-1b table
    const uint32_t b = hf >> (32 - kLeanBits);
    s.n[j] = ((filt[b >> 5] >> (b & 31)) & 1u) ? 0xFu : 0u;
    s.bw[j] = s.n[j] ? __ldg(big + (hf >> (32 - kBigBits))) : 0u;
  }
}

__device__ __forceinline__ uint32_t grams_finish(const Grams& s, uint32_t lane) {
  uint32_t n[5];
#pragma unroll
  for (int j = 0; j < 5; ++j) n[j] = s.n[j] & s.bw[j];
  const uint32_t n4 = __shfl_down_sync(0xFFFFFFFFu, n[0], 1);
  const uint32_t m = n[0] | (n[1] << 4) | (n[2] << 8) | (n[3] << 12) | ((lane == 31 ? n[4] : n4) << 16);
  return (m >> 3) & 0xFFFFu;
}

// The words a lane needs: its own four and the next lane's first (the tail
// vector's on lane 31).
__device__ __forceinline__ void lane_words(const uint4& cur, const uint4& tail, uint32_t lane, uint32_t (&w)[5]) {
  w[0] = cur.x;
  w[1] = cur.y;
  w[2] = cur.z;
  w[3] = cur.w;
  w[4] = __shfl_down_sync(0xFFFFFFFFu, cur.x, 1);
  if (lane == 31) w[4] = tail.x;
}

constexpr int kBigThreads = 512;
constexpr int kBigWarps = kBigThreads / 32;

// 4-byte grams at every fourth position with the stage-1b table in L2, and literals
// of one to three bytes: the same work as literal_filter_kernel
// in a three-block software pipeline per warp -- the input of block i+2 is
// loaded, the grams of block i+1 are hashed and their L2 checks issued, then
// block i is finished -- so that the L2 latency overlaps useful work.
// 16 warps per CTA leave room for the pipeline's registers.
__global__ void __launch_bounds__(kBigThreads, 1) literal_filter_big_kernel(const __grid_constant__ LitArgs a) {
  pdl_wait();  // (as in literal_filter_kernel)
  extern __shared__ __align__(16) uint32_t smem[];
  uint32_t* filt = smem;
  uint32_t* bloom = filt + a.filter_words;
  uint32_t* shortb = bloom + (1u << (kBloomBits - 5));
  uint32_t* warpmem = shortb + 2048;
  {
    const uint4* src = reinterpret_cast<const uint4*>(a.filter);
    uint4* dst = reinterpret_cast<uint4*>(filt);
    for (uint32_t k = threadIdx.x; k < a.filter_words / 4; k += kBigThreads) dst[k] = __ldg(src + k);
    const uint4* bs = reinterpret_cast<const uint4*>(a.bloom);
    uint4* bd = reinterpret_cast<uint4*>(bloom);
    for (uint32_t k = threadIdx.x; k < (1u << (kBloomBits - 7)); k += kBigThreads) bd[k] = __ldg(bs + k);
    const uint4* s2 = reinterpret_cast<const uint4*>(a.short_bits);
    uint4* d2 = reinterpret_cast<uint4*>(shortb);
    for (uint32_t k = threadIdx.x; k < 512; k += kBigThreads) d2[k] = __ldg(s2 + k);
  }
  __syncthreads();

  const uint32_t lane = threadIdx.x & 31;
  const uint32_t warp = threadIdx.x >> 5;
  uint32_t* blk = warpmem + warp * (kBlockWords + kQueue / 2);
  uint16_t* queue = reinterpret_cast<uint16_t*>(blk + kBlockWords);
  const uint32_t len = (uint32_t)a.len;
  const uint32_t nvec = (uint32_t)((a.len + 15) >> 4);
  const uint32_t full_vecs = len >> 4;
  const uint32_t nblk = (nvec + 31) >> 5;
  const uint32_t nwarps = gridDim.x * kBigWarps;
  auto load = [&](uint32_t v) -> uint4 {
    const uint4 x = v < full_vecs ? __ldg(reinterpret_cast<const uint4*>(a.data) + v)
                    : v < nvec ? load_vec(a.data, a.len, v) : make_uint4(0, 0, 0, 0);
    return a.fold ? fold16(x) : x;
  };
  const uint4 zero = make_uint4(0, 0, 0, 0);

  uint32_t b = blockIdx.x * kBigWarps + warp;
  // pipeline registers: block b (cur, grams in flight), block b + nwarps (nxt)
  uint4 cur = zero, tail_c = zero, nxt = zero, tail_n = zero;
  Grams gc;
  if (b < nblk) {
    cur = load(b * 32 + lane);
    tail_c = lane == 31 ? load(b * 32 + 32) : zero;
    uint32_t w[5];
    lane_words(cur, tail_c, lane, w);
    grams_issue(filt, a.big, w, lane, gc);
  }
  if (b + nwarps < nblk) {
    nxt = load((b + nwarps) * 32 + lane);
    tail_n = lane == 31 ? load((b + nwarps) * 32 + 32) : zero;
  }
  for (; b < nblk; b += nwarps) {
    const uint32_t bn = b + nwarps, bn2 = bn + nwarps;
    // input of block b + 2 nwarps
    uint4 nxt2 = zero, tail2 = zero;
    if (bn2 < nblk) {
      nxt2 = load(bn2 * 32 + lane);
      tail2 = lane == 31 ? load(bn2 * 32 + 32) : zero;
    }
    // grams of block b + nwarps, L2 checks issued
    Grams gn;
    if (bn < nblk) {
      uint32_t w[5];
      lane_words(nxt, tail_n, lane, w);
      grams_issue(filt, a.big, w, lane, gn);
    }
    // finish block b
    uint32_t mask = grams_finish(gc, lane);
    uint32_t w[5];
    lane_words(cur, tail_c, lane, w);
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      const uint32_t g = __funnelshift_r(w[j >> 2], w[(j >> 2) + 1], 8 * (j & 3)) & 0xFFFFu;
      mask |= ((shortb[g >> 5] >> (g & 31)) & 1u) << j;
    }
    const uint32_t v = b * 32 + lane;
    if (v >= full_vecs) {
      const uint32_t base = v * 16;
      const uint32_t valid = len > base ? len - base : 0;
      mask &= (valid >= 16) ? 0xFFFFu : ((1u << valid) - 1u);
    }
    if (__ballot_sync(0xFFFFFFFFu, mask != 0) != 0)
      process_block<4>(a, blk, queue, bloom, lane, cur, tail_c, mask, b * 512);
    cur = nxt;
    tail_c = tail_n;
    gc = gn;
    nxt = nxt2;
    tail_n = tail2;
  }
}

// ------------------------------------------------------------- gram kernel
// Stage 1 for every set without literals of one or two bytes whose grams are
// sparse enough in their alphabet (LiteralPlan::gram_kernel).  The filter only
// hashes, looks up and appends; stage 1.5 moves to the verify kernel.
//   - a literal of at least P + G - 1 bytes holds, wherever it starts, one
//     G-byte gram at a position that is a multiple of P (G = 16 has P = 4), so
//     16 / P grams per 16 bytes are tested.  A lane's grams are those at
//     base - OFF + P * j (base the offset of its 16 bytes), all inside its own
//     bytes and the few bytes before them, which come from the lane below;
//   - stage 1 is a bitmap in shared memory (BITS = 1), or for crowded sets a
//     blocked Bloom filter of two bits of one word per gram (BITS = 2): the second
//     bit costs no second load and squares the pass rate (10,000 literals: 0.6% of
//     the grams pass where one bit let 3.4% pass).  Word and bits come from dot
//     products of the gram (gram_word, gram_bit);
//   - the warp takes kGramBits / NG vectors of 512 coalesced bytes in a row (a
//     run), one pass bit per gram in a 32-bit mask, and looks at the mask once:
//     the passing grams go into the warp's queue in shared memory;
//   - with 32 or more queued, every lane takes one: its phase bits (which
//     offsets of a literal have this gram, a byte of a table in L2) give the
//     start positions, which are appended to the warp's reserved slots of the
//     list, one global atomic per slot_chunk slots.
// One CTA of 1,024 threads per SM, four 512-byte loads in flight per warp.
// What bounds it: with few passing grams HBM for P = 4 (2,100 literals over 1 GiB
// 170 us a scan, a copy takes 164); each passing gram costs a warp 5 to 6 issue
// slots (10,000 literals 182, 20,000 216), and 16-byte grams three shuffles a
// vector (2,100 k-mers 197, 20,000 259).  P = 2 and P = 1 are bound by the shared
// memory lookups: a warp's 32 random words meet in 3.4 wavefronts of the data
// pipe, which is 0.88 busy with P = 2.  Measured, us per 256 MiB: 10,000 literals
// (P = 4) 57 -> 52, where the kernel before it (one bit, a vote and an append per
// 1 KiB step, its candidates' L2 loads in the main loop) took 65; 500 literals of
// 5 bytes and more (P = 2) 73; 20,000 k-mers (G = 16) 81 -> 74 against 164 for the
// compacting kernel; 1,000 caseless literals of 3 and more over 97 MiB 69 -> 63
// against 184.  (The arrows: hashes by multiplication and shifts, which kept the
// integer pipe 0.8 busy, and positions worked out when a gram was queued, 15 issue
// slots a passing gram, to the present ones.)
constexpr int kGramThreads = 1024;
constexpr uint32_t kGramWarps = kGramThreads / 32;
// u32 positions per warp.  (512 of them left less L1 for the flush, which reads
// the queued grams again: 10,000 literals over 1 GiB 204 -> 200 us a scan.)
constexpr uint32_t kGramQueue = 128;
constexpr uint32_t kGramBits = 32;    // grams per lane and mask
constexpr uint32_t kNoSurvivor = 0xFFFFFFFFu;  // no position: inputs are shorter than 2^32 bytes

// Bytes before its own that a lane's grams start at.
template <int P, int G>
__host__ __device__ constexpr int gram_off() { return G == 16 ? 12 : P == 4 ? 0 : P == 2 ? 2 : G == 3 ? 2 : 3; }

struct WarpSlots {
  unsigned long long next = 0, end = 0;  // the warp's reserved range [next, end)
};

// Marks the warp's unfilled reserved slots as holes.
__device__ __forceinline__ void mark_holes(const LitArgs& a, const WarpSlots& r, uint32_t lane) {
  for (unsigned long long k = r.next + lane; k < r.end && k < a.survivor_cap; k += 32) a.survivors[k] = kNoSurvivor;
}

// Key of the phase table for the gram at position at: a hash independent of
// stage 1's, so that what stage 1 lets through by chance does not pass again.  No
// word is read that holds none of the gram's bytes.  EDGE: the last one may reach
// past the input.
template <bool EDGE>
__device__ __forceinline__ uint32_t phase_key_at(const LitArgs& a, uint32_t at, int G) {
  const uint32_t len = (uint32_t)a.len, w0 = at & ~3u, sh = (at & 3) * 8;
  auto word = [&](uint32_t x) {
    if (EDGE) return input_word(a, len, x);
    const uint32_t w = __ldg(reinterpret_cast<const uint32_t*>(a.data + x));
    return a.fold ? ascii_fold4(w) : w;
  };
  if (G == 16) return phase_key(word(w0), word(w0 + 4), word(w0 + 8), word(w0 + 12), 16);  // aligned
  return phase_key(__funnelshift_r(word(w0), sh + 8 * G > 32 ? word(w0 + 4) : 0u, sh), 0, 0, 0, G);
}

// Position of a queued gram: bit i of lane l's mask in run r is r * 1024 + l * 32
// + i (a run is 32 grams of every lane, gram i of vector i / NG).
template <int P, int G>
__device__ __forceinline__ uint32_t gram_at(uint32_t code) {
  constexpr uint32_t NG = 16 / P, i_bits = kGramBits - 1;
  return (code >> 10) * (1024 * P) + ((code & i_bits) / NG) * 512 + ((code >> 5) & 31) * 16 + (code % NG) * P -
         gram_off<P, G>();
}

// Takes the queued grams [0, n), 32 at a time: phase bits, start positions,
// append.  EDGE: words may lie past the input.  True when the list was full
// before: the verify kernel then looks at every gram of the input again, and this
// kernel has nothing more to add.
template <int P, int G, bool EDGE>
__device__ __forceinline__ bool gram_flush(const LitArgs& a, const uint32_t* queue, uint32_t n, WarpSlots& r,
                                           uint32_t lane) {
  const uint32_t len = (uint32_t)a.len;
  for (uint32_t k0 = 0; k0 < n; k0 += 32) {
    uint32_t at = 0, bits = 0;
    if (!EDGE || k0 + lane < n) {
      at = gram_at<P, G>(queue[k0 + lane]);
      bits = (uint32_t)__ldg(a.phase + (phase_key_at<EDGE>(a, at, G) >> a.phase_shift));
    }
    if (__ballot_sync(0xFFFFFFFFu, bits != 0) == 0) continue;  // the usual group
#pragma unroll
    for (int k = 0; k < P; ++k)  // bit P - 1 - k: the literal starts k bytes before the gram
      if (at < (uint32_t)k || at - k >= len) bits &= ~(1u << (P - 1 - k));
    const uint32_t cnt = __popc(bits);
    uint32_t incl = cnt;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, incl, d);
      if (lane >= (uint32_t)d) incl += y;
    }
    const uint32_t total = __shfl_sync(0xFFFFFFFFu, incl, 31);
    if (r.next + total > r.end) {  // warp-uniform: reserve more slots
      mark_holes(a, r, lane);
      const unsigned long long want = total > a.slot_chunk ? total : a.slot_chunk;
      unsigned long long wb = 0;
      if (lane == 0) wb = atomicAdd(a.survivor_count, want);
      wb = __shfl_sync(0xFFFFFFFFu, wb, 0);
      r.next = wb;
      r.end = wb + want;
      if (wb >= a.survivor_cap) return true;
    }
    unsigned long long slot = r.next + incl - cnt;
    r.next += total;
    for (; bits; bits &= bits - 1) {
      // (verifying here when the list is full cost the loop its registers)
      if (slot < a.survivor_cap) a.survivors[slot] = at - (P - 1) + (__ffs(bits) - 1);
      ++slot;
    }
  }
  return false;
}

// Queues the passing grams of a run (bit 31 - i of `pass`: the lane's gram i), the
// run's codes from `code` on, and flushes whole groups of 32; kListFull when the
// list was.
constexpr uint32_t kListFull = 0xFFFFFFFFu;

template <int P, int G, bool EDGE>
__device__ __forceinline__ uint32_t gram_queue(const LitArgs& a, uint32_t* queue, uint32_t queued, uint32_t pass,
                                               uint32_t code, WarpSlots& slots, uint32_t lane) {
  uint32_t ball = __ballot_sync(0xFFFFFFFFu, pass != 0);
  while (ball) {
    if (pass) {  // one gram of every lane that has one left
      const uint32_t i = __clz(pass);
      pass ^= 0x80000000u >> i;
      queue[queued + __popc(ball & ((1u << lane) - 1u))] = code + i;
    }
    queued += __popc(ball);
    ball = __ballot_sync(0xFFFFFFFFu, pass != 0);
    if (queued >= (ball ? kGramQueue - 31 : 32)) {
      __syncwarp();
      const uint32_t whole = queued & ~31u, left = queued & 31u;
      if (gram_flush<P, G, EDGE>(a, queue, whole, slots, lane)) return kListFull;
      const uint32_t keep = lane < left ? queue[whole + lane] : 0u;
      __syncwarp();
      if (lane < left) queue[lane] = keep;
      queued = left;
    }
  }
  return queued;
}

// Pass bits of one vector: gram j shifts into the bottom of `pass`.  w[k] is word
// k - NPRE of the lane's bytes; `below` holds the words before the vector for
// lane 0 and receives those of the next one.
template <int P, int G, int BITS, int NPRE>
__device__ __forceinline__ uint32_t gram_test(const uint32_t* filt, uint32_t mask, uint32_t two, uint32_t lane, const uint4& v,
                                              uint32_t (&below)[NPRE ? NPRE : 1], uint32_t pass) {
  constexpr int NG = 16 / P, OFF = gram_off<P, G>();
  uint32_t w[NPRE + 4];
  w[NPRE] = v.x;
  w[NPRE + 1] = v.y;
  w[NPRE + 2] = v.z;
  w[NPRE + 3] = v.w;
#pragma unroll
  for (int k = 0; k < NPRE; ++k) {
    // lane 31's word goes to lane 0, which keeps it for the next vector
    const uint32_t x = __shfl_sync(0xFFFFFFFFu, k == 0 ? v.w : k == 1 ? v.z : v.y, (lane + 31) & 31);
    w[NPRE - 1 - k] = lane == 0 ? below[k] : x;
    below[k] = x;
  }
  uint32_t g[NG], x[NG];
#pragma unroll
  for (int j = 0; j < NG; ++j) {
    const int o = P * j - OFF + 4 * NPRE, i = o / 4;  // byte offset of gram j in w
    g[j] = (o & 3) ? __funnelshift_r(w[i], w[i + 1 < NPRE + 4 ? i + 1 : i], 8 * (o & 3)) : w[i];
    const uint32_t at = G == 16 ? gram_word(w[i], w[i + 1], w[i + 2], w[i + 3], G) : gram_word(g[j], 0, 0, 0, G);
    x[j] = *reinterpret_cast<const uint32_t*>(reinterpret_cast<const char*>(filt) + (at & mask));
  }
#pragma unroll
  for (int j = 0; j < NG; ++j) {
    const int i = (P * j - OFF + 4 * NPRE) / 4;
    auto bit_of = [&](int k) {
      return __funnelshift_r(x[j], x[j], gram_bit(g[j], G == 16 ? w[i + 1] : 0, G == 16 ? w[i + 2] : 0, G, k));
    };
    uint32_t bit = bit_of(0);
    if (BITS == 2) bit &= bit_of(1);
    pass = pass * two + (bit & 1u);
  }
  return pass;
}

template <int P, int G, int BITS>
__global__ void __launch_bounds__(kGramThreads, 1) literal_gram_kernel(const __grid_constant__ LitArgs a) {
  constexpr int NG = 16 / P, OFF = gram_off<P, G>(), NPRE = (OFF + 3) / 4;
  constexpr uint32_t VECS = kGramBits / NG;                // 512-byte vectors of a run
  constexpr uint32_t RING = VECS < 4 ? VECS : 4;           // vectors loaded ahead
  const bool fold = a.fold != 0;
  extern __shared__ __align__(16) uint32_t gsm[];
  uint32_t* queue = gsm + (1u << a.gram_word_bits) + (threadIdx.x >> 5) * kGramQueue;
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  {
    const uint4* src = reinterpret_cast<const uint4*>(a.gram_bloom);
    uint4* dst = reinterpret_cast<uint4*>(gsm);
    for (uint32_t k = threadIdx.x; k < (1u << a.gram_word_bits) / 4; k += kGramThreads) dst[k] = __ldg(src + k);
  }
  __syncthreads();
  // (the tables above are no kernel's output; the verify kernel is not let in
  // early, its waiting blocks cost the last runs 1%)
  pdl_wait();
  const uint32_t mask = gram_mask(a.gram_word_bits);
  const uint32_t len = (uint32_t)a.len;
  const uint32_t nvec = (uint32_t)((a.len + 15) >> 4);
  const uint32_t runs = len / (VECS * 512);                // runs entirely inside the input
  // neighbouring runs go to different SMs, so that a small input spreads out
  const uint32_t first = warp * gridDim.x + blockIdx.x, nw = gridDim.x * kGramWarps;
  WarpSlots slots;
  uint32_t queued = 0;
  uint32_t below[NPRE ? NPRE : 1];
  auto run_ptr = [&](uint32_t r) { return reinterpret_cast<const uint4*>(a.data + (uint64_t)r * (VECS * 512)) + lane; };
  auto before = [&](uint32_t at, uint32_t (&x)[NPRE ? NPRE : 1]) {  // the words before byte `at` (lane 0)
#pragma unroll
    for (int k = 0; k < NPRE; ++k)
      x[k] = lane == 0 && at ? __ldg(reinterpret_cast<const uint32_t*>(a.data + at) - 1 - k) : 0u;
  };
  auto folded = [&](uint32_t (&x)[NPRE ? NPRE : 1]) {
#pragma unroll
    for (int k = 0; k < NPRE; ++k) x[k] = ascii_fold4(x[k]);
  };
  uint4 ring[RING];
  uint32_t ahead[NPRE ? NPRE : 1];
  if (first < runs) {
    const uint4* p = run_ptr(first);
#pragma unroll
    for (uint32_t i = 0; i < RING; ++i) ring[i] = __ldg(p + i * 32);
    before(first * (VECS * 512), ahead);
  }
  for (uint32_t r = first; r < runs; r += nw) {
    const uint4* p = run_ptr(r);
    const bool more = r + nw < runs;
    const uint4* pn = more ? run_ptr(r + nw) : p;
#pragma unroll
    for (int k = 0; k < NPRE; ++k) below[k] = ahead[k];
    if (NPRE && more) before((r + nw) * (VECS * 512), ahead);
    if (fold) folded(below);
    uint32_t pass = 0;
#pragma unroll
    for (uint32_t i = 0; i < VECS; ++i) {
      uint4 v = ring[i % RING];
      if (i + RING < VECS) ring[i % RING] = __ldg(p + (i + RING) * 32);
      else if (more) ring[i % RING] = __ldg(pn + (i + RING - VECS) * 32);
      if (fold) v = fold16(v);
      pass = gram_test<P, G, BITS, NPRE>(gsm, mask, a.two, lane, v, below, pass);
    }
    if (OFF && r == 0 && lane == 0) pass &= 0xFFFFFFFFu >> ((OFF + P - 1) / P);  // grams that begin before the input
    queued = gram_queue<P, G, false>(a, queue, queued, pass, r * 1024 + lane * 32, slots, lane);
    if (queued == kListFull) return;
  }
  // the vectors after the last whole run, one warp each
  const uint32_t v0 = runs * VECS, nv = (nvec + 31) >> 5;
  if (first < nv - v0) {
    const uint32_t b = v0 + first, vec = b * 32 + lane;
    uint4 v = vec < nvec ? load_vec(a.data, a.len, vec) : make_uint4(0, 0, 0, 0);
    before(b * 512, below);
    if (fold) {
      v = fold16(v);
      folded(below);
    }
    uint32_t pass = gram_test<P, G, BITS, NPRE>(gsm, mask, a.two, lane, v, below, 0u) << (32 - NG);
    if (OFF && b == 0 && lane == 0) pass &= 0xFFFFFFFFu >> ((OFF + P - 1) / P);
    queued = gram_queue<P, G, true>(a, queue, queued, pass, (b / VECS) * 1024 + lane * 32 + (b % VECS) * NG, slots, lane);
    if (queued == kListFull) return;
  }
  __syncwarp();
  if (queued) gram_flush<P, G, true>(a, queue, queued, slots, lane);
  mark_holes(a, slots, lane);
}

// A position where a covered regex's prefix may start: every regex of which one
// does (entries of different regexes may share it) runs its leftmost-first walk
// from there, and a match makes a candidate.  A walk still open after kLfCap
// bytes gives the prefix candidates up: the regexes' groups are walked instead
// (ctr[C_GATE]), whose cost does not depend on the input.  So do walks of more
// steps than kWorkPerByte per input byte, entries looked at included; a long
// walk, which keeps its whole warp waiting, counts for more.  A warp reports its
// work in pieces of at least kWorkReport.
constexpr uint32_t kWorkPerByte = 8, kLongWalk = 64, kLongWeight = 8, kWorkReport = 16384;
template <class Sink>
__device__ __forceinline__ void verify_prefixes(const LitArgs& a, const DevTables& t, const ScanPtrs& p,
                                                const PrefixDev& pf, uint32_t s, uint32_t lo, uint32_t hi, uint32_t k,
                                                uint32_t k1, bool gate, uint32_t& work, Sink&& sink) {
  // every lane finds its next entry, then the lanes that have one walk together
  while (true) {
    uint32_t r = 0xFFFFFFFFu;
    while (k < k1 && r == 0xFFFFFFFFu) {
      const uint4 e = __ldg(pf.entry + k++);
      ++work;
      if (e.x == lo && !((e.y ^ hi) & e.z)) r = e.w;
    }
    if (__ballot_sync(0xFFFFFFFFu, r != 0xFFFFFFFFu) == 0) return;
    if (r != 0xFFFFFFFFu && !gate) {
      uint32_t steps = 0;
      const uint32_t end = lf_walk(t, p, r, s, kLfCap, &steps);
      work += steps > kLongWalk ? kLongWeight * steps : steps;
      if (end == kLfOpen) {
        atomicOr(&p.ctr[C_GATE], 1ull);
        gate = true;
      } else if (end != kLfNone) {
        sink(r, s, end);
      }
    }
    __syncwarp();
  }
}

// Stage 1 of the grams that start in the 16 bytes of vector v, by tables in
// global memory: bit j of the result is the gram at byte j.
template <int G>
__device__ __forceinline__ uint32_t grams_pass(const LitArgs& a, uint32_t v) {
  const uint32_t len = (uint32_t)a.len, at = v * 16, mask = gram_mask(a.gram_word_bits);
  uint32_t w[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  const uint4 x = load_vec(a.data, a.len, v);
  w[0] = x.x, w[1] = x.y, w[2] = x.z, w[3] = x.w;
#pragma unroll
  for (uint32_t k = 0; k < 4; ++k) {
    if (a.fold) w[k] = ascii_fold4(w[k]);
    if ((k == 0 || G == 16) && at + 16 + 4 * k < len) w[4 + k] = input_word(a, len, at + 16 + 4 * k);
  }
  uint32_t pass = 0;
#pragma unroll
  for (uint32_t j = 0; j < 16; ++j) {
    if ((G == 16 && (j & 3)) || (j & (a.period - 1))) continue;
    const uint32_t i = j >> 2, g = G == 16 ? w[i] : __funnelshift_r(w[i], w[i + 1], 8 * (j & 3));
    const uint32_t word = G == 16 ? gram_word(g, w[i + 1], w[i + 2], w[i + 3], G) : gram_word(g, 0, 0, 0, G);
    const uint32_t x = __ldg(a.gram_bloom + ((word & mask) >> 2));
    uint32_t bit = __funnelshift_r(x, x, gram_bit(g, w[i + 1], w[i + 2], G, 0));
    if (a.gram_bits == 2) bit &= __funnelshift_r(x, x, gram_bit(g, w[i + 1], w[i + 2], G, 1));
    pass |= (bit & 1u) << j;
  }
  const uint32_t left = len - at;
  return left < 16 ? pass & ((1u << left) - 1u) : pass;
}

// Tables of the verify kernel to be brought into L2 at its start: the filter has
// just streamed the whole input through L2, and a walk or a bucket's chain that
// finds its tables gone waits for HBM at each of its steps, all walks at the
// same ones.  The gain is small, the tables having mostly stayed (us a scan: 160
// regexes over 1 GiB 323.0 -> 321.9, 60 over 200 MiB 94.9 -> 94.1, 10,000 literals
// over 1 GiB 191.9 -> 191.2), and so is the cost.
struct WarmDev {
  const char* p[10];
  uint32_t lines[10];  // of 128 bytes
};

__device__ __forceinline__ void warm_tables(const WarmDev& wd) {
#pragma unroll
  for (int q = 0; q < 10; ++q)
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < wd.lines[q]; i += gridDim.x * blockDim.x)
      asm volatile("prefetch.global.L2 [%0];" ::"l"(wd.p[q] + (size_t)i * 128));
}

// Kernel 2.  When the gram kernel's list was full (it then stopped early), every
// gram of the input is tested again here: a warp takes 16 bytes per lane, queues
// the grams that pass in shared memory and verifies their literals with all its
// lanes busy.  (One gram per thread, verified where it was found, took 2,300 us
// for the 4 M literals of 64 MiB; a queue per block, with its barriers, 340.)  RX: the survivors are also looked up
// among the regex prefixes.  A full list (more than one survivor per 64 bytes)
// gives the prefix candidates up, like long walks do; the last block then drops
// the candidates found so far, so that the gated groups start from none.
//
// Matches and candidates collect in shared memory, a buffer per warp that is
// written out with one atomic when half full, and what is left at the end with
// one per block (an atomic per match on the one counter: 35 us for 65,536 of
// them).  No barrier before the end: a warp whose walks are long delays no other
// (with block buffers and a barrier a step, 40,000 items took 40 us here, with
// these 34).
constexpr uint32_t kVerifyThreads = 256, kVerifyWarps = kVerifyThreads / 32;
constexpr uint32_t kVerifyBuf = 64;  // per warp

template <bool RX>
__global__ void __launch_bounds__(kVerifyThreads, 4) literal_verify_kernel(const __grid_constant__ LitArgs a,
                                                             const __grid_constant__ DevTables t,
                                                             const __grid_constant__ ScanPtrs p, PrefixDev pf,
                                                             const __grid_constant__ WarmDev wd) {
  warm_tables(wd);
  pdl_begin();
  __shared__ uint3 mbuf[kVerifyWarps][kVerifyBuf];
  __shared__ uint3 kbuf[kVerifyWarps][kVerifyBuf];  // (or the grams of the dense pass: a full list makes no candidates)
  __shared__ uint32_t held[2][kVerifyWarps];
  const uint32_t lane = threadIdx.x & 31, wi = threadIdx.x >> 5;
  if (lane < 2) held[lane][wi] = 0;
  __syncwarp();
  auto match = [&](uint32_t pid, uint32_t s, uint32_t e) {
    const uint32_t i = atomicAdd(&held[0][wi], 1u);
    if (i < kVerifyBuf) mbuf[wi][i] = make_uint3(pid, s, e);
    else report_match(a, pid, s, e);
  };
  auto candidate = [&](uint32_t r, uint32_t s, uint32_t e) {
    const uint32_t i = atomicAdd(&held[1][wi], 1u);
    if (i < kVerifyBuf) kbuf[wi][i] = make_uint3(r, s, e);
    else emit_k(p, r, s, e, kEndKnown);
  };
  // the warp's first `nm` matches and `nk` candidates to places at and kat
  auto write_out = [&](uint32_t nm, unsigned long long at, uint32_t nk, unsigned long long kat) {
    for (uint32_t i = lane; i < nm; i += 32)
      if (at + i < a.cap) a.out[at + i] = ws_match{mbuf[wi][i].x, mbuf[wi][i].y, mbuf[wi][i].z};
    for (uint32_t i = lane; RX && i < nk; i += 32)
      store_k(p, kat + i, kbuf[wi][i].x, kbuf[wi][i].y, kbuf[wi][i].z, atomicAdd(&p.count[kbuf[wi][i].x], 1u) | kEndKnown);
  };
  auto drain = [&]() {  // by the warp, after each step
    __syncwarp();
    const uint32_t nm = min(held[0][wi], kVerifyBuf), nk = RX ? min(held[1][wi], kVerifyBuf) : 0u;
    if (nm > kVerifyBuf / 2 || nk > kVerifyBuf / 2) {
      unsigned long long at = 0;
      if (lane == 0 && nm) at = atomicAdd(a.counter, (unsigned long long)nm);
      if (RX && lane == 1 && nk) at = atomicAdd(&p.ctr[C_K], (unsigned long long)nk);
      write_out(nm, __shfl_sync(0xFFFFFFFFu, at, 0), nk, __shfl_sync(0xFFFFFFFFu, at, 1));
      __syncwarp();
      if (lane < 2) held[lane][wi] = 0;
    }
    __syncwarp();
  };
  unsigned long long n = *a.survivor_count;
  const bool full = n > a.survivor_cap;
  if (full) n = a.survivor_cap;
  // the gram kernel drops what does not fit (the compacting kernel verifies it)
  const bool dense = full && a.gram_bits;
  // Neighbouring survivors go to different warps: a short list (the usual one)
  // then has a survivor per warp, whose chains of dependent loads do not wait
  // for one another.
  const uint32_t warps = gridDim.x * (blockDim.x >> 5);
  const uint32_t w = blockIdx.x + gridDim.x * wi;
  uint32_t warp_work = 0;
  for (unsigned long long k0 = 0; k0 < n && !dense; k0 += 32ull * warps) {  // the same for all lanes
    const unsigned long long k = k0 + (unsigned long long)lane * warps + w;
    const uint32_t s = k < n ? a.survivors[k] : kNoSurvivor;
    const bool in = s != kNoSurvivor;  // (else a slot the gram kernel reserved but did not fill)
    // the first words, then the buckets of the literals' table and of the
    // prefixes', in flight together
    const uint32_t len = (uint32_t)a.len, w0 = s & ~3u, sh = (s & 3) * 8;
    uint32_t x0 = 0, x1 = 0, x2 = 0, x3 = 0;
    if (in) {
      x0 = word_at(a.data, len, w0);
      x1 = word_at(a.data, len, w0 + 4);
      x2 = word_at(a.data, len, w0 + 8);
      if (a.parts) x3 = word_at(a.data, len, w0 + 12);
    }
    const uint32_t lo = __funnelshift_r(x0, x1, sh), hi = __funnelshift_r(x1, x2, sh);
    const bool literals = in && a.parts && s < a.max_start;
    uint32_t pk = 0, pk1 = 0;
    bool gate = true;
    if (RX && in && !full) {
      const uint32_t* rg = pf.range + ((lo * 0x9E3779B1u + hi * pf.mul) >> pf.shift);
      pk = __ldg(rg);
      pk1 = __ldg(rg + 1);
      gate = *(volatile unsigned long long*)&p.ctr[C_GATE] != 0;
    }
    if (literals) {
      Probe pr;
      const uint32_t next = __funnelshift_r(x2, x3, sh);
      if (a.fold) probe_literals(a, ascii_fold4(lo), ascii_fold4(hi), len - s, pr);
      else probe_literals(a, lo, hi, len - s, pr);
      verify_literals(a, s, a.fold ? ascii_fold4(x0) : x0, a.fold ? ascii_fold4(next) : next, pr, match);
    }
    if (RX) {
      uint32_t work = 0;
      verify_prefixes(a, t, p, pf, s, lo, hi, pk, pk1, gate, work, candidate);
      warp_work += __reduce_add_sync(0xFFFFFFFFu, work);
      if (warp_work >= kWorkReport) {
        if (lane == 0 && atomicAdd(&p.ctr[C_WORK], (unsigned long long)warp_work) + warp_work > kWorkPerByte * a.len)
          atomicOr(&p.ctr[C_GATE], 1ull);
        warp_work = 0;
      }
    }
    drain();
  }
  if (dense && a.parts) {
    const uint32_t len = (uint32_t)a.len, nvec = (uint32_t)((a.len + 15) >> 4);
    uint32_t* grams = reinterpret_cast<uint32_t*>(kbuf[wi]);
    auto verify_grams = [&](uint32_t n) {  // grams[0, n), n <= 32
      if (lane < n) {
        const uint32_t at = grams[lane];
        uint32_t bits = __ldg(a.phase + (phase_key_at<true>(a, at, (int)a.gram_len) >> a.phase_shift));
        for (; bits; bits &= bits - 1) {
          const uint32_t k = a.period - __ffs(bits);  // bit period - 1 - k: the literal starts k bytes before
          if (at >= k && at - k < len) verify_by_word(a, at - k, match);
        }
      }
      drain();
    };
    uint32_t queued = 0;
    for (uint64_t v0 = (uint64_t)w * 32; v0 < nvec; v0 += (uint64_t)warps * 32) {
      const uint32_t v = (uint32_t)v0 + lane;
      uint32_t pass = 0;
      if (v < nvec) pass = a.gram_len == 16 ? grams_pass<16>(a, v) : a.gram_len == 3 ? grams_pass<3>(a, v) : grams_pass<4>(a, v);
      for (uint32_t ball; (ball = __ballot_sync(0xFFFFFFFFu, pass != 0)) != 0;) {
        if (pass) {  // one gram of every lane that has one left
          grams[queued + __popc(ball & ((1u << lane) - 1u))] = v * 16 + __ffs(pass) - 1;
          pass &= pass - 1;
        }
        queued += __popc(ball);
        __syncwarp();
        if (queued >= 32) {
          verify_grams(32);
          queued -= 32;
          const uint32_t keep = lane < queued ? grams[32 + lane] : 0u;
          __syncwarp();
          if (lane < queued) grams[lane] = keep;
          __syncwarp();
        }
      }
    }
    verify_grams(queued);
  }
  // what the warps still hold
  __shared__ unsigned long long first[2];
  __syncthreads();
  uint32_t before[2] = {0, 0}, sum[2] = {0, 0};
#pragma unroll
  for (uint32_t i = 0; i < kVerifyWarps; ++i)
    for (uint32_t q = 0; q < (RX ? 2u : 1u); ++q) {
      if (i == wi) before[q] = sum[q];
      sum[q] += min(held[q][i], kVerifyBuf);
    }
  if (threadIdx.x == 0 && sum[0]) first[0] = atomicAdd(a.counter, (unsigned long long)sum[0]);
  if (RX && threadIdx.x == 32 && sum[1]) first[1] = atomicAdd(&p.ctr[C_K], (unsigned long long)sum[1]);
  if (sum[0] | sum[1]) {
    __syncthreads();
    write_out(min(held[0][wi], kVerifyBuf), first[0] + before[0], RX ? min(held[1][wi], kVerifyBuf) : 0u,
              first[1] + before[1]);
  }
  if (RX) {
    __shared__ bool last;
    __syncthreads();
    if (threadIdx.x == 0) {
      __threadfence();
      last = atomicAdd(&p.ctr[C_TICKET], 1ull) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    if (!full && *(volatile unsigned long long*)&p.ctr[C_GATE] == 0) return;
    for (uint32_t r = threadIdx.x; r < t.n_regex; r += blockDim.x) p.count[r] = 0;
    if (threadIdx.x == 0) {
      p.ctr[C_K] = 0;
      p.ctr[C_ERR] = 0;
      p.ctr[C_GATE] = 1;
    }
  }
}

}  // namespace

size_t literal_smem_bytes(const LiteralPlan& plan) {
  const size_t filter_words = plan.has_big ? ((size_t)1 << (kLeanBits - 5)) : plan.filter.size();
  return (filter_words + (1u << (kBloomBits - 5)) + (plan.has_short ? 2048 : 0) +
          (size_t)kWarps * (kBlockWords + kQueue / 2)) * 4;
}

size_t literal_scratch_bytes(uint64_t survivor_cap) { return 64 + survivor_cap * 4; }

void launch_literal_scan(const LiteralPlan& plan, const LiteralLaunch& l, cudaStream_t st, int sm_count) {
  if (plan.n_strings == 0 || l.len == 0) return;
  LitArgs a;
  a.data = l.data;
  a.len = l.len;
  // with a stage-1b table, stage 1 in shared memory is its bitmap
  a.filter = plan.has_big ? plan.d_lean_bits.as<uint32_t>() : plan.d_filter.as<uint32_t>();
  a.filter_words = plan.has_big ? (1u << (kLeanBits - 5)) : (uint32_t)plan.filter.size();
  a.bits = plan.table_bits;
  a.period = plan.period;
  a.parts = l.literals ? plan.parts : 0;  // (no prefix length, no literal)
  a.short_bits = plan.d_short.as<uint32_t>();
  a.bloom = plan.d_bloom.as<uint32_t>();
  a.info = plan.d_info.as<uint4>();
  a.lit_bytes = plan.d_bytes.as<uint8_t>();
  for (uint32_t i = 0; i < HASH_WINDOW; ++i) a.meta[i] = make_uint2(plan.meta[4 * i], plan.meta[4 * i + 1]);
  a.ranges = plan.d_ranges.as<uint2>();
  a.entries = plan.d_entries.as<uint4>();
  a.out = l.out;
  a.cap = l.cap;
  a.counter = l.counter;
  a.survivor_count = reinterpret_cast<unsigned long long*>(l.scratch);
  a.survivors = reinterpret_cast<uint32_t*>(static_cast<uint8_t*>(l.scratch) + 64);
  a.survivor_cap = l.survivor_cap;
  a.item_end = l.item_end;
  a.n_items = l.n_items;
  a.min_end = l.min_end;
  a.max_start = l.max_start;
  a.gram_len = plan.gram_len;
  a.parts16 = plan.parts16;
  a.bloom2 = plan.gram_len > 4 ? plan.d_bloom2.as<uint32_t>() : nullptr;
  a.big = plan.has_big ? plan.d_big.as<uint8_t>() : nullptr;
  a.bloom_parts = plan.bloom_parts;
  a.gram_bloom = plan.d_gram.as<uint32_t>();
  a.gram_word_bits = plan.gram_word_bits;
  a.gram_bits = plan.gram_kernel ? plan.gram_bits : 0;
  a.phase = plan.d_phase.as<uint8_t>();
  a.phase_shift = 32 - plan.phase_bits;
  a.two = 2;
  a.fold = plan.fold ? 1 : 0;
  if (!l.cleared) check_cuda(cudaMemsetAsync(a.survivor_count, 0, 8, st), "memset survivors");
  if (l.len > 0xFFFFFFFFull) raise(WS_ERR_INPUT_TOO_LARGE, "literal scan launch beyond 32-bit offsets", 0, l.len,
                                   0xFFFFFFFFull);
  const size_t smem = literal_smem_bytes(plan);
  uint64_t nblk = ((l.len + 15) / 16 + 31) / 32;
  uint64_t want = (nblk + kWarps - 1) / kWarps;
  int grid = (int)std::min<uint64_t>((uint64_t)sm_count, std::max<uint64_t>(want, 1));
  // the filter layout is a compile-time choice of the kernel
  auto run = [&](auto kernel, int threads = kThreads) {
    check_cuda(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem),
               "cudaFuncSetAttribute(literal)");
    launch_scan(!l.cleared, kernel, grid, threads, smem, st, a);
    check_cuda(cudaGetLastError(), "literal_filter_kernel launch");
  };
  const bool lg = plan.has_long != 0, sh = plan.has_short != 0;
  auto run_gram = [&](auto kernel, uint32_t run_bytes) {
    // a warp per run of run_bytes, or per 512-byte vector after the last one
    const uint64_t units = l.len / run_bytes + (l.len % run_bytes + 511) / 512;
    const int blocks = (int)std::min<uint64_t>((uint64_t)sm_count, units);
    // a warp reserves 32 list slots at a time when it has many runs (one
    // atomic in place of several), else what it appends: the unfilled slots
    // of all warps stay well below the list's capacity
    a.slot_chunk = l.len >= 16384ull * blocks * kGramWarps ? 32 : 1;
    const size_t gsmem = ((size_t)4 << plan.gram_word_bits) + (size_t)kGramWarps * kGramQueue * 4;
    check_cuda(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)gsmem),
               "cudaFuncSetAttribute(literal gram)");
    launch_scan(!l.cleared, kernel, blocks, kGramThreads, gsmem, st, a);
    check_cuda(cudaGetLastError(), "literal_gram_kernel launch");
  };
  // sparse sets: the gram kernel; else with literals shorter than 4 bytes and
  // a stage-1b table the pipelined compacting kernel; long grams, whose hashing
  // dominates, keep 32 warps per SM
  if (plan.gram_kernel) {
    const bool two = plan.gram_bits == 2;
    if (plan.gram_len == 16) run_gram(two ? literal_gram_kernel<4, 16, 2> : literal_gram_kernel<4, 16, 1>, 4096);
    else if (plan.gram_len == 3) run_gram(two ? literal_gram_kernel<1, 3, 2> : literal_gram_kernel<1, 3, 1>, 1024);
    else if (plan.period == 4) run_gram(two ? literal_gram_kernel<4, 4, 2> : literal_gram_kernel<4, 4, 1>, 4096);
    else if (plan.period == 2) run_gram(two ? literal_gram_kernel<2, 4, 2> : literal_gram_kernel<2, 4, 1>, 2048);
    else run_gram(two ? literal_gram_kernel<1, 4, 2> : literal_gram_kernel<1, 4, 1>, 1024);
  } else if (lg && sh && a.big && plan.period == 4 && plan.gram_len == 4) {
    run(literal_filter_big_kernel, kBigThreads);
  } else if (!lg) {
    run(literal_filter_kernel<4, 4, false, true>);
  } else if (plan.gram_len == 16) {
    run(literal_filter_kernel<4, 16, true, true>);  // (without short literals the gram kernel has it)
  } else if (plan.gram_len == 8) {
    sh ? run(literal_filter_kernel<4, 8, true, true>) : run(literal_filter_kernel<4, 8, true, false>);
  } else if (plan.period == 4) {
    sh ? run(literal_filter_kernel<4, 4, true, true>) : run(literal_filter_kernel<4, 4, true, false>);
  } else if (plan.period == 2) {
    sh ? run(literal_filter_kernel<2, 4, true, true>) : run(literal_filter_kernel<2, 4, true, false>);
  } else {
    sh ? run(literal_filter_kernel<1, 4, true, true>) : run(literal_filter_kernel<1, 4, true, false>);
  }
  // the verify pass is a chain of dependent loads per survivor: as many threads
  // as are resident at once (four blocks per SM; a second wave doubled the
  // latency: 40,000 items 65 -> 39 us in this kernel), and for a short list no
  // more blocks than it can fill
  const uint64_t vgrid = std::min<uint64_t>((uint64_t)sm_count * 4, (l.survivor_cap + 255) / 256);
  // (a set whose tables are more than two lines a thread leaves them where they are)
  WarmDev wd{};
  uint64_t lines = 0;
  uint32_t n_warm = 0;
  auto warm = [&](const DeviceBuffer& b) {
    const uint64_t n = (b.bytes + 127) / 128;
    if (!b.ptr || lines + n > 2 * 256 * vgrid) return;
    wd.p[n_warm] = b.as<char>();
    wd.lines[n_warm++] = (uint32_t)n;
    lines += n;
  };
  if (l.literals)
    for (const DeviceBuffer* b : {&plan.d_ranges, &plan.d_entries, &plan.d_info, &plan.d_bytes}) warm(*b);
  if (l.rx) {
    for (const DeviceBuffer* b : {&plan.d_prefix_range, &plan.d_prefix_entry}) warm(*b);
    for (const DeviceBuffer* b : l.rx->walk_tables)
      if (b) warm(*b);
    const PrefixDev pf{plan.d_prefix_range.as<uint32_t>(), plan.d_prefix_entry.as<uint4>(), plan.prefix_shift,
                       plan.prefix_mul};
    launch_pdl(literal_verify_kernel<true>, (unsigned)vgrid, 256, 0, st, a, l.rx->t, l.rx->p, pf, wd);
  } else {
    launch_pdl(literal_verify_kernel<false>, (unsigned)vgrid, 256, 0, st, a, DevTables{}, ScanPtrs{}, PrefixDev{}, wd);
  }
  check_cuda(cudaGetLastError(), "literal_verify_kernel launch");
}

}  // namespace ws
