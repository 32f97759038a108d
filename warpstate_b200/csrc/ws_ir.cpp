// Pattern IR: the host half of PatternSetBuilder::build that the GPU path needs,
// and the literal-scan plan derived from it.
#include <algorithm>
#include <cmath>
#include <cstring>

#include "ws_internal.h"

namespace ws {

void raise(ws_status s, const std::string& msg, uint64_t index, uint64_t count, uint64_t max) {
  Failure f;
  f.status = s;
  f.message = msg;
  f.index = index;
  f.count = count;
  f.max = max;
  throw WsError(std::move(f));
}

void check_cuda(cudaError_t e, const char* what) {
  if (e == cudaSuccess) return;
  cudaGetLastError();  // a failed call's error is not left behind for the caller's next check
  if (e == cudaErrorNoDevice || e == cudaErrorInsufficientDriver)
    raise(WS_ERR_NO_DEVICE, std::string(what) + ": " + cudaGetErrorString(e));
  raise(WS_ERR_DEVICE, std::string(what) + ": " + cudaGetErrorString(e));
}

uint32_t fnv1a(const uint8_t* p, size_t len, size_t window) {
  // core/src/pattern/compiler.rs:343-350: bytes.iter().take(window.max(1))
  uint32_t h = FNV_BASIS;
  size_t n = std::min(len, std::max<size_t>(window, 1));
  for (size_t k = 0; k < n; ++k) { h ^= p[k]; h *= FNV_PRIME; }
  return h;
}

void build_prefilter_table(const std::vector<uint32_t>& offsets, const std::vector<uint32_t>& hashes,
                           uint32_t window, std::vector<uint32_t>& meta,
                           std::vector<uint32_t>& ranges, std::vector<uint32_t>& entries) {
  // core/src/literal_prefilter.rs:23-88: one partition per effective prefix
  // length min(len, window), each a power-of-two bucket table (2n rounded up)
  // with contiguous collision chains.
  const size_t n = hashes.size();
  std::vector<std::vector<uint32_t>> groups(window);  // literal indices
  for (size_t li = 0; li < n; ++li) {
    uint32_t len = offsets[2 * li + 1];
    uint32_t pl = std::max<uint32_t>(std::min(len, window), 1);
    groups[pl - 1].push_back((uint32_t)li);
  }
  meta.assign(4 * (size_t)window, 0);
  ranges.clear();
  entries.clear();
  entries.reserve(2 * n);
  for (uint32_t g = 0; g < window; ++g) {
    const auto& grp = groups[g];
    if (grp.empty()) continue;
    uint64_t buckets = 1;
    while (buckets < 2 * (uint64_t)grp.size()) buckets <<= 1;
    if (buckets > 0xFFFFFFFFull) raise(WS_ERR_PATTERN_SET_TOO_LARGE, "literal prefilter bucket count overflow");
    uint32_t first_bucket = (uint32_t)(ranges.size() / 2);
    // counting sort of the group's literals by bucket keeps insertion order in a chain
    std::vector<uint32_t> count(buckets + 1, 0);
    for (uint32_t li : grp) ++count[(hashes[li] & (buckets - 1)) + 1];
    for (uint64_t b = 0; b < buckets; ++b) count[b + 1] += count[b];
    std::vector<uint32_t> order(grp.size());
    std::vector<uint32_t> fill(count.begin(), count.end() - 1);
    for (uint32_t li : grp) order[fill[hashes[li] & (buckets - 1)]++] = li;
    uint32_t base = (uint32_t)(entries.size() / 2);
    for (uint64_t b = 0; b < buckets; ++b) {
      ranges.push_back(base + count[b]);
      ranges.push_back(count[b + 1] - count[b]);
    }
    for (uint32_t li : order) { entries.push_back(hashes[li]); entries.push_back(li); }
    meta[4 * g + 0] = first_bucket;
    meta[4 * g + 1] = (uint32_t)buckets - 1;
    meta[4 * g + 2] = (uint32_t)buckets;
    meta[4 * g + 3] = 0;
  }
}

DeviceBuffer::~DeviceBuffer() {
  if (ptr) cudaFree(ptr);
}

void DeviceBuffer::alloc(size_t n) {
  if (ptr) { cudaFree(ptr); ptr = nullptr; }
  bytes = n;
  if (n == 0) return;
  check_cuda(cudaMalloc(&ptr, n), "cudaMalloc");
}

void DeviceBuffer::upload(const void* src, size_t n) {
  alloc(n + 16);  // 16 spare bytes: vector loads of the tail stay inside the allocation
  check_cuda(cudaMemset(ptr, 0, n + 16), "cudaMemset");
  // a null source (an empty table given a minimum size) leaves zeros
  if (n && src) check_cuda(cudaMemcpy(ptr, src, n, cudaMemcpyHostToDevice), "cudaMemcpy H2D");
}

namespace {

struct FilterString {
  const uint8_t* p;
  uint32_t len;
};

// Distinct G-byte grams of the strings at offsets 0..P-1, as a share of all
// G-byte grams over the bytes the strings use (G <= 4).
double gram_coverage(const std::vector<FilterString>& strings, uint32_t P, uint32_t G) {
  bool seen[256] = {};
  std::vector<uint32_t> grams;
  for (const FilterString& f : strings) {
    for (uint32_t k = 0; k < f.len; ++k) seen[f.p[k]] = true;
    for (uint32_t k = 0; f.len >= G && k < P && k + G <= f.len; ++k) {
      uint32_t g = 0;
      std::memcpy(&g, f.p + k, G);
      grams.push_back(g);
    }
  }
  std::sort(grams.begin(), grams.end());
  const double distinct = (double)(std::unique(grams.begin(), grams.end()) - grams.begin());
  double alphabet = 0, all = 1;
  for (bool b : seen) alphabet += b ? 1.0 : 0.0;
  for (uint32_t k = 0; k < G; ++k) all *= alphabet;
  return distinct / std::min(std::max(all, 1.0), 4294967296.0);
}

// Tables of the gram kernel.  Stage 1 has 1,024 bits a gram (0.1% of other
// grams pass), from 4 KiB for small sets (it is staged per block) up to
// 128 KiB; from 8,192 grams on, where one bit of that would let 0.8% pass, two
// bits per gram.  The phase table has 64 bytes a gram, up to 32 MiB.
void build_gram_tables(const std::vector<FilterString>& strings, LiteralPlan& plan) {
  const uint32_t P = plan.period, G = plan.gram_len;
  struct Gram {
    uint32_t word, bit[2], key;
    uint8_t phase;
  };
  std::vector<Gram> grams;
  for (const FilterString& f : strings)
    for (uint32_t k = 0; k < P; ++k) {
      uint32_t g[4] = {0, 0, 0, 0};
      std::memcpy(g, f.p + k, G);
      grams.push_back({gram_word(g[0], g[1], g[2], g[3], (int)G),
                       {gram_bit(g[0], g[1], g[2], (int)G, 0), gram_bit(g[0], g[1], g[2], (int)G, 1)},
                       phase_key(g[0], g[1], g[2], g[3], (int)G), (uint8_t)(1u << (P - 1 - k))});
    }
  uint32_t bits = 0;
  while (bits < 25 && ((size_t)1 << bits) < grams.size()) ++bits;
  plan.gram_bits = grams.size() >= 8192 ? 2 : 1;
  plan.gram_word_bits = std::min<uint32_t>(std::max<uint32_t>(bits + 5, 10), kGramWords);
  std::vector<uint32_t> words((size_t)1 << plan.gram_word_bits, 0u);
  for (const Gram& g : grams)
    for (uint32_t b = 0; b < plan.gram_bits; ++b)
      words[(g.word & gram_mask(plan.gram_word_bits)) >> 2] |= 1u << (g.bit[b] & 31u);
  plan.d_gram.upload(words.data(), words.size() * 4);
  plan.phase_bits = std::min<uint32_t>(std::max<uint32_t>(bits + 6, 12), kBigBits);
  std::vector<uint8_t> phase((size_t)1 << plan.phase_bits, 0);
  for (const Gram& g : grams) phase[g.key >> (32 - plan.phase_bits)] |= g.phase;
  plan.d_phase.upload(phase.data(), phase.size());
}

// P grams at offsets 0..P-1 must fit inside every string: P + 3 <= len.
uint32_t period_of(uint32_t min_len) { return min_len >= 7 ? 4 : min_len >= 5 ? 2 : 1; }

// Share of its alphabet's 4-byte grams that a set covers before longer grams are
// the better choice.
constexpr double kLowEntropy = 0.25;

// Share of its alphabet's G-byte grams that a set of the gram kernel may cover.
// That kernel passes on every position whose gram is in the set; on an input over
// the set's own alphabet that is coverage / P of all positions, and the list holds
// one of 64.  Beyond it every gram is looked up a second time; the compacting
// kernel, which checks prefixes inside the filter, is then the better one.
// Measured over 128 MiB of uniform letters, us a scan with the gram and with the
// compacting kernel, by coverage: P = 4 4.4% 107 and 123 (26 letters), 102 and 107
// (8 letters), 4.8% 117 and 126, 5.0% 113 and 108 (12 letters), 7% 269 and 132, 10%
// (8 letters) 269 and 110; P = 1 1.26% 202 and 322, 1.31% 619 and 340; 3-byte grams
// 1.08% 185 and 260, 1.14% 346 and 259.  P = 2: 1.5% 109 and 184.
double gram_limit(uint32_t P, uint32_t G) {
  return P == 4 ? 0.05 : P == 2 ? 1.0 / 64 : G == 3 ? 0.0105 : 0.0125;
}

struct Layout {
  bool has_long = false, has_short = false;  // strings of at least, of fewer than 4 bytes
  bool gram_kernel = false;
  uint32_t period = 4, gram_len = 4;
};

// (fewer literals say little about the alphabet of the input)
constexpr size_t kOwnAlphabet = 16;

// `n_literals` of the strings, the first, are literals.  Their grams count by
// their own alphabet too: a few other bytes in the prefixes make the alphabet of
// all larger, not the input.
Layout choose_layout(const std::vector<FilterString>& strings, size_t n_literals) {
  Layout l;
  const std::vector<FilterString> literals(strings.begin(), strings.begin() + n_literals);
  auto coverage = [&](uint32_t P, uint32_t G) {
    const double all = gram_coverage(strings, P, G);
    return n_literals >= kOwnAlphabet && n_literals < strings.size() ? std::max(all, gram_coverage(literals, P, G)) : all;
  };
  uint32_t min_len = UINT32_MAX, min_long = UINT32_MAX;
  for (const FilterString& f : strings) {
    min_len = std::min(min_len, f.len);
    if (f.len >= 4) { l.has_long = true; min_long = std::min(min_long, f.len); }
    else l.has_short = true;
  }
  l.period = !l.has_long ? 4 : period_of(min_long);
  // A low-entropy set (a small alphabet whose 4-grams the strings mostly
  // cover, e.g. nucleotide k-mers) lets most input positions through 4-byte
  // grams: it takes the longest gram every long string holds at all P phases.
  const bool low_entropy =
      l.has_long && l.period == 4 && min_long >= 11 && coverage(4, 4) > kLowEntropy;
  if (low_entropy) l.gram_len = min_long >= 19 ? 16 : 8;
  // Crowded sets take the compacting kernel, which checks prefixes inside the
  // filter.  Shortest string of three bytes: 3-byte grams at every position.
  if (low_entropy) {
    l.gram_kernel = l.gram_len == 16 && !l.has_short;
  } else if (min_len == 3) {
    l.gram_kernel = coverage(1, 3) <= gram_limit(1, 3);
    if (l.gram_kernel) {
      l.period = 1;
      l.gram_len = 3;
    }
  } else if (min_len >= 4) {
    l.gram_kernel = coverage(l.period, 4) <= gram_limit(l.period, 4);
  }
  return l;
}

}  // namespace

bool filter_crowded(const ws_pattern_tables& t, const std::vector<std::string>& prefixes) {
  std::vector<FilterString> strings;
  for (uint32_t li = 0; li < t.n_literals; ++li)
    strings.push_back({t.packed_bytes + t.offsets[2 * li], t.offsets[2 * li + 1]});
  const Layout alone = choose_layout(strings, strings.size());
  for (const std::string& x : prefixes)
    strings.push_back({reinterpret_cast<const uint8_t*>(x.data()), (uint32_t)x.size()});
  const Layout l = choose_layout(strings, t.n_literals);
  if (l.gram_kernel) return false;  // (its list holds, or it would not run)
  // the literals' long grams are worth more than the walks (4-byte ones let nearly
  // every position of such an input through)
  if (t.n_literals && alone.gram_len > l.gram_len) return true;
  // The compacting kernel lets a position through whose first bytes (8 of them, 16
  // with longer grams) a string begins with: as a share of all positions of an
  // input over the strings' alphabet, and over the literals' for theirs.
  const uint32_t most = l.gram_len > 4 ? 16 : 8;
  auto share = [&](size_t n) {
    bool seen[256] = {};
    double alphabet = 0, sum = 0;
    std::vector<std::string> heads;
    for (size_t k = 0; k < n; ++k) {
      heads.emplace_back(reinterpret_cast<const char*>(strings[k].p), std::min(strings[k].len, most));
      for (uint32_t j = 0; j < strings[k].len; ++j) seen[strings[k].p[j]] = true;
    }
    for (bool x : seen) alphabet += x ? 1 : 0;
    std::sort(heads.begin(), heads.end());
    heads.erase(std::unique(heads.begin(), heads.end()), heads.end());
    for (const std::string& h : heads) sum += std::pow(alphabet, -(double)h.size());
    return sum;
  };
  return std::max(share(strings.size()), t.n_literals >= kOwnAlphabet ? share(t.n_literals) : 0.0) > 1.0 / 80;
}

double filter_ms_per_gib(const LiteralPlan& plan) {
  if (plan.n_strings == 0) return 0;
  if (plan.gram_kernel) return plan.period == 4 ? (plan.gram_len == 16 ? 0.25 : 0.18) : plan.period == 2 ? 0.27 : 0.55;
  return plan.period == 4 ? 0.9 : plan.period == 2 ? 1.5 : 2.6;
}

double literals_ms_per_gib(const ws_pattern_tables& t) {
  std::vector<FilterString> strings;
  for (uint32_t li = 0; li < t.n_literals; ++li)
    strings.push_back({t.packed_bytes + t.offsets[2 * li], t.offsets[2 * li + 1]});
  const Layout l = choose_layout(strings, strings.size());
  LiteralPlan plan;
  plan.n_strings = t.n_literals;
  plan.gram_kernel = l.gram_kernel;
  plan.period = l.period;
  plan.gram_len = l.gram_len;
  return filter_ms_per_gib(plan);
}

void plan_literals(const ws_pattern_tables& given, LiteralPlan& plan, const std::vector<std::string>& prefixes) {
  plan.n_literals = given.n_literals;
  plan.n_strings = given.n_literals + (uint32_t)prefixes.size();
  if (plan.n_strings == 0) return;
  // ASCII case-insensitive sets (PatternSetBuilder::case_insensitive,
  // core/src/pattern/compiler.rs:66-76, an Aho-Corasick automaton with
  // ascii_case_insensitive): every table below is planned on the literals
  // with A-Z folded to a-z, the prefilter table rebuilt on their FNV-1a
  // hashes, and the kernels fold the input the same way.
  ws_pattern_tables t = given;
  std::vector<uint8_t> folded;
  std::vector<std::string> pre = prefixes;
  std::vector<uint32_t> foffsets, fhashes, fmeta, franges, fentries;
  plan.fold = given.case_insensitive != 0;
  if (plan.fold) {
    folded.assign(given.packed_bytes, given.packed_bytes + given.packed_len);
    for (uint8_t& c : folded) c = ascii_fold(c);
    for (std::string& x : pre)
      for (char& c : x) c = (char)ascii_fold((uint8_t)c);
    foffsets.assign(given.offsets, given.offsets + 2 * (size_t)given.n_literals);
    for (uint32_t li = 0; li < given.n_literals; ++li)
      fhashes.push_back(fnv1a(folded.data() + foffsets[2 * li], foffsets[2 * li + 1], HASH_WINDOW));
    build_prefilter_table(foffsets, fhashes, HASH_WINDOW, fmeta, franges, fentries);
    t.packed_bytes = folded.data();
    t.hash_window_len = HASH_WINDOW;
    t.prefix_meta = fmeta.data();
    t.bucket_ranges = franges.data();
    t.n_buckets = (uint32_t)(franges.size() / 2);
    t.entries = fentries.data();
  }
  std::vector<FilterString> strings;
  for (uint32_t li = 0; li < t.n_literals; ++li)
    strings.push_back({t.packed_bytes + t.offsets[2 * li], t.offsets[2 * li + 1]});
  for (const std::string& x : pre) strings.push_back({reinterpret_cast<const uint8_t*>(x.data()), (uint32_t)x.size()});
  plan.max_len = 0;
  for (const FilterString& f : strings) plan.max_len = std::max(plan.max_len, f.len);
  const Layout layout = choose_layout(strings, t.n_literals);
  plan.has_long = layout.has_long;
  plan.has_short = layout.has_short;
  plan.period = layout.period;
  plan.gram_len = layout.gram_len;
  plan.gram_kernel = layout.gram_kernel;
  plan.table_bits = 18;
  const uint32_t P = plan.period, G = plan.gram_len, bits = plan.table_bits;
  plan.parts = plan.bloom_parts = 0;
  plan.lit_info.assign(4 * (size_t)t.n_literals, 0);
  plan.lit_bytes.clear();
  plan.bloom.assign((size_t)1 << (18 - 5), 0);
  for (size_t k = 0; k < strings.size(); ++k) {
    const uint32_t len = strings[k].len;
    const uint8_t* lit = strings[k].p;
    // Bloom bitmap of the first min(len, 8) bytes (the kernel's prefix_key)
    const uint32_t pl = std::max<uint32_t>(std::min<uint32_t>(len, HASH_WINDOW), 1);
    uint32_t x[2] = {0, 0};
    std::memcpy(x, lit, pl);
    const uint32_t key = (x[0] * 0x9E3779B1u + x[1] * 0x85EBCA77u + pl * 0xC2B2AE3Du) >> (32 - 18);
    plan.bloom[key >> 5] |= 1u << (key & 31);
    plan.bloom_parts |= 1u << (pl - 1);
    if (k >= t.n_literals) continue;
    plan.parts |= 1u << (pl - 1);
    while (plan.lit_bytes.size() % 4) plan.lit_bytes.push_back(0);
    plan.lit_info[4 * k + 0] = (uint32_t)plan.lit_bytes.size();
    plan.lit_info[4 * k + 1] = len;
    plan.lit_info[4 * k + 2] = t.literal_pattern_ids[k];
    plan.lit_bytes.insert(plan.lit_bytes.end(), lit, lit + len);
  }
  while (plan.lit_bytes.size() % 16) plan.lit_bytes.push_back(0);
  if (plan.gram_kernel) {
    build_gram_tables(strings, plan);
  } else {
    // the compacting kernel's tables
    plan.filter.assign((size_t)1 << (bits - 3), 0);
    plan.short_bits.assign(65536 / 32, 0);
    if (G > 4) plan.bloom2.assign((size_t)1 << (kBloom2Bits - 5), 0u);
    plan.parts16 = 0;
    for (const FilterString& f : strings) {
      for (uint32_t k = 0; f.len >= 4 && k < P; ++k) {
        uint32_t g[4] = {0, 0, 0, 0};
        std::memcpy(g, f.p + k, G);
        const uint32_t h = G == 4 ? gram_hash(g[0], bits) : long_gram_hash(g[0], g[1], g[2], g[3], G, bits);
        plan.filter[h >> 3] |= (1u << (P - 1 - k)) << ((h & 7) * 4);
      }
      if (f.len < 4) {
        const uint32_t b0 = f.p[0];
        for (uint32_t b1 = f.len == 1 ? 0 : f.p[1]; b1 < (f.len == 1 ? 256u : f.p[1] + 1u); ++b1) {
          const uint32_t key = b0 | (b1 << 8);
          plan.short_bits[key >> 5] |= 1u << (key & 31);
        }
      }
      plan.parts16 |= 1u << (std::min<uint32_t>(std::max<uint32_t>(f.len, 1), 16) - 1);
      if (G > 4) {  // every string (short ones too) is in the 16-byte-prefix Bloom
        uint32_t x[4] = {0, 0, 0, 0};
        const uint32_t pl = std::min<uint32_t>(f.len, 16);
        std::memcpy(x, f.p, pl);
        const uint32_t key = prefix16_key(x[0], x[1], x[2], x[3], pl);
        plan.bloom2[key >> 5] |= 1u << (key & 31);
      }
    }
    if (G > 4) plan.d_bloom2.upload(plan.bloom2.data(), plan.bloom2.size() * 4);
  }
  // Stage 1b of the compacting kernel: when more than 0.5% (P = 4) or 0.1%
  // (P = 2: nine grams per 16 bytes, each passing one sends the warp block to
  // compaction) of the shared table's phase bits are set, a 2^kBigBits-byte
  // table in L2 (the same full 32-bit gram hashes, more of their bits)
  // re-checks each passing gram.
  if (!plan.gram_kernel && plan.has_long && (P == 4 || P == 2)) {
    uint64_t set = 0;
    for (uint32_t w : plan.filter) set += (uint64_t)__builtin_popcount(w);
    if ((double)set / (double)((uint64_t)plan.filter.size() * 32) > (P == 4 ? 0.005 : 0.001)) {
      plan.big.assign((size_t)1 << kBigBits, 0);
      std::vector<uint32_t> lean2(G > 4 ? (size_t)1 << (kLeanBits - 5) : 0, 0u);
      for (const FilterString& f : strings) {
        if (f.len < 4) continue;
        for (uint32_t k = 0; k < P; ++k) {
          uint32_t g[4] = {0, 0, 0, 0};
          std::memcpy(g, f.p + k, G);
          const uint32_t hf = G == 4 ? g[0] * 0x9E3779B1u
                              : G == 8 ? mix_words(g[0], g[1], 0, 0, 8)
                                       : mix_words(g[0], g[1], g[2], g[3], 16);
          const uint32_t h = hf >> (32 - kBigBits);
          plan.big[h] |= (uint8_t)(1u << (P - 1 - k));
          if (G > 4) lean2[lean2_word(hf)] |= lean2_mask(hf);
        }
      }
      plan.d_big.upload(plan.big.data(), plan.big.size());
      plan.lean_bits.assign((size_t)1 << (kLeanBits - 3), 0);
      if (G > 4) {
        std::memcpy(plan.lean_bits.data(), lean2.data(), plan.lean_bits.size());
      } else {
        for (size_t h = 0; h < plan.big.size(); ++h)
          if (plan.big[h]) {
            const size_t b = h >> (kBigBits - kLeanBits);
            plan.lean_bits[b >> 3] |= (uint8_t)(1u << (b & 7));
          }
      }
      plan.d_lean_bits.upload(plan.lean_bits.data(), plan.lean_bits.size());
      plan.has_big = true;
      std::vector<uint8_t>().swap(plan.big);
    }
  }
  plan.n_buckets = t.n_buckets;
  plan.d_filter.upload(plan.filter.data(), plan.filter.size() * 4);
  plan.d_bloom.upload(plan.bloom.data(), plan.bloom.size() * 4);
  plan.d_short.upload(plan.short_bits.data(), plan.short_bits.size() * 4);
  plan.d_info.upload(plan.lit_info.data(), plan.lit_info.size() * 4);
  plan.d_bytes.upload(plan.lit_bytes.data(), plan.lit_bytes.size());
  plan.meta.assign(4 * HASH_WINDOW, 0u);
  if (t.prefix_meta)
    std::copy(t.prefix_meta, t.prefix_meta + 4 * std::min(t.hash_window_len, HASH_WINDOW), plan.meta.begin());
  plan.d_ranges.upload(t.bucket_ranges, 2 * (size_t)t.n_buckets * 4);
  // entries {hash, literal} with bytes 8..11 of the literal and their mask
  std::vector<uint32_t> entries(4 * (size_t)t.n_literals, 0u);
  for (size_t e = 0; e < t.n_literals; ++e) {
    const uint32_t li = t.entries[2 * e + 1], len = li < t.n_literals ? t.offsets[2 * li + 1] : 0;
    entries[4 * e] = t.entries[2 * e];
    entries[4 * e + 1] = li;
    if (len <= 8) continue;
    std::memcpy(&entries[4 * e + 2], t.packed_bytes + t.offsets[2 * li] + 8, std::min<uint32_t>(len - 8, 4));
    std::memset(&entries[4 * e + 3], 0xFF, std::min<uint32_t>(len - 8, 4));
  }
  plan.d_entries.upload(entries.data(), entries.size() * 4);
}

}  // namespace ws

using namespace ws;

namespace {

void fill_err(ws_error_info* err, const Failure& f) {
  if (!err) return;
  err->index = f.index;
  err->count = f.count;
  err->max = f.max;
  std::snprintf(err->message, sizeof(err->message), "%s", f.message.c_str());
}

}  // namespace

extern "C" ws_status ws_ir_build(const ws_pattern_spec* patterns, uint64_t n, int case_insensitive,
                                 ws_ir** out, ws_error_info* err) {
  if (err) std::memset(err, 0, sizeof(*err));
  if (!out || (n && !patterns)) {
    if (err) std::snprintf(err->message, sizeof(err->message), "null argument");
    return WS_ERR_INVALID_ARGUMENT;
  }
  *out = nullptr;
  try {
    // core/src/pattern/compiler.rs:97-340
    if (n == 0) raise(WS_ERR_EMPTY_PATTERN_SET, "pattern set is empty. Fix: add at least one literal pattern before building.");
    if (n > 0xFFFFFFFFull) raise(WS_ERR_PATTERN_SET_TOO_LARGE, "too many patterns", 0, n, 0xFFFFFFFFull);
    auto ir = std::make_unique<ws_ir>();
    IrData& d = ir->d;
    d.n_patterns = (uint32_t)n;
    d.case_insensitive = case_insensitive != 0;
    auto add_literal = [&](uint64_t i, const uint8_t* b, uint64_t len) {
      if (len > 0xFFFFFFFFull) raise(WS_ERR_PATTERN_TOO_LARGE, "pattern too large", i, len, 0xFFFFFFFFull);
      if (d.packed_bytes.size() + len > 0xFFFFFFFFull)
        raise(WS_ERR_PATTERN_SET_TOO_LARGE, "packed literal bytes exceed u32", 0, d.packed_bytes.size(), 0xFFFFFFFFull);
      d.offsets.push_back((uint32_t)d.packed_bytes.size());
      d.offsets.push_back((uint32_t)len);
      d.literal_hashes.push_back(fnv1a(b, len, HASH_WINDOW));
      d.literal_pattern_ids.push_back((uint32_t)i);
      d.packed_bytes.insert(d.packed_bytes.end(), b, b + len);
    };
    for (uint64_t i = 0; i < n; ++i) {
      const ws_pattern_spec& p = patterns[i];
      if (p.len == 0) raise(WS_ERR_EMPTY_PATTERN, "pattern " + std::to_string(i) + " is empty. Fix: provide a non-empty byte sequence for every pattern.", i);
      if (!p.bytes) raise(WS_ERR_INVALID_ARGUMENT, "null pattern bytes", i);
      if (p.kind == WS_PATTERN_LITERAL) {
        add_literal(i, p.bytes, p.len);
      } else if (p.kind == WS_PATTERN_REGEX) {
        std::string src((const char*)p.bytes, (size_t)p.len);
        ReTree tree;
        try {
          tree = parse_regex(src);
        } catch (const CompileError& e) {
          raise(WS_ERR_COMPILE, "invalid regex at index " + std::to_string(i) + ": " + e.what(), i);
        }
        if (tree_pathological(tree)) raise(WS_ERR_PATHOLOGICAL, "regex pattern " + std::to_string(i) + " contains nested repetitions (pathological)", i);
        std::vector<uint8_t> lit;
        if (tree_literal(tree, &lit)) {  // compiler.rs:181-212: literal demotion
          add_literal(i, lit.data(), lit.size());
          continue;
        }
        d.regex_sources.push_back(src);
        d.regex_pattern_ids.push_back((uint32_t)i);
      } else {
        raise(WS_ERR_INVALID_ARGUMENT, "unknown pattern kind", i);
      }
    }
    build_prefilter_table(d.offsets, d.literal_hashes, HASH_WINDOW, d.prefix_meta, d.bucket_ranges, d.entries);
    for (auto& s : d.regex_sources) d.regex_ptrs.push_back(s.c_str());
    *out = ir.release();
    return WS_OK;
  } catch (const WsError& e) {
    fill_err(err, e.f);
    return e.f.status;
  } catch (const std::exception& e) {
    if (err) std::snprintf(err->message, sizeof(err->message), "%s", e.what());
    return WS_ERR_COMPILE;
  }
}

extern "C" void ws_ir_destroy(ws_ir* ir) { delete ir; }

extern "C" ws_status ws_ir_tables(const ws_ir* ir, ws_pattern_tables* t) {
  if (!ir || !t) return WS_ERR_INVALID_ARGUMENT;
  const IrData& d = ir->d;
  std::memset(t, 0, sizeof(*t));
  t->packed_bytes = d.packed_bytes.data();
  t->packed_len = d.packed_bytes.size();
  t->offsets = d.offsets.data();
  t->literal_pattern_ids = d.literal_pattern_ids.data();
  t->n_literals = (uint32_t)d.literal_pattern_ids.size();
  t->hash_window_len = HASH_WINDOW;
  t->prefix_meta = d.prefix_meta.data();
  t->bucket_ranges = d.bucket_ranges.data();
  t->n_buckets = (uint32_t)(d.bucket_ranges.size() / 2);
  t->entries = d.entries.data();
  t->regex_sources = d.regex_ptrs.data();
  t->regex_pattern_ids = d.regex_pattern_ids.data();
  t->n_regex = (uint32_t)d.regex_pattern_ids.size();
  t->n_patterns = d.n_patterns;
  t->case_insensitive = d.case_insensitive ? 1 : 0;
  return WS_OK;
}

// Test hook: the literal filter's layout for the literals of a pattern set: bytes
// between the positions it looks at, bytes of a gram, whether the gram kernel runs.
extern "C" void ws_testing_literal_layout(const ws_ir* ir, unsigned* out) {
  std::vector<FilterString> strings;
  for (size_t k = 0; k < ir->d.literal_pattern_ids.size(); ++k)
    strings.push_back({ir->d.packed_bytes.data() + ir->d.offsets[2 * k], ir->d.offsets[2 * k + 1]});
  const Layout l = choose_layout(strings, strings.size());
  out[0] = l.period, out[1] = l.gram_len, out[2] = l.gram_kernel ? 1 : 0;
}
