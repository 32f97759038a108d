// Regex prefixes in the literal filter.
//
// A regex whose every match begins with one of a few strings needs no walk of
// its group's DFA over the whole input: the literal filter, which passes over
// the input at several times the walk's rate and once for all groups, finds
// where those strings occur, and the verify kernel runs the regex's
// leftmost-first DFA from there.  The candidates are the same distinct
// (regex, start) pairs the walk finds.
//
// The walk takes one shared-memory lookup per input byte and group, 1.8 T
// lookups/s over the chip; the filter one per second or fourth byte, once for
// the literals and all groups.  Measured, us a pass with the walk (as it was
// before there were prefixes) and with the filter: 500 regexes (9 groups) over 64
// MiB 483 -> 116, 160 regexes (1 group) over 1 GiB 939 -> 474, 60 unbounded
// regexes over 200 MiB 740 -> 221, 40 anchored ones over 32 MiB 304 -> 98, 40,000
// items with 1,500 literals and 200 regexes 1734 -> 336, 20,000 k-mers and 100
// motifs over 2 GiB 3105 -> 715.
// Where prefixes are dense the filter gives up at run time (ws_literal.cu,
// literal_verify_kernel) and the walk does what it did before.
#include <algorithm>
#include <cstring>
#include <map>

#include "ws_dfa.h"

namespace ws {

namespace {

// All covered regexes' prefixes of one length; false when some regex has none
// listed there or there are more than `most`.
bool collect(const RegexPlan& P, int k, size_t most, std::vector<std::pair<std::string, uint32_t>>& out) {
  out.clear();
  for (uint32_t r = 0; r < P.n_regex; ++r) {
    if (!P.covered[r]) continue;
    if (P.prefixes[k][r].empty()) return false;
    for (const std::string& x : P.prefixes[k][r]) out.emplace_back(x, r);
    if (out.size() > most) return false;
  }
  return !out.empty();
}

// The verify kernel's table needs no more of a regex's prefixes than tell most
// false positions apart, the walk decides: the longest listed with at most 16
// different beginnings of up to 8 bytes, else those of 4 bytes (a class after a
// short word makes hundreds with the same beginning, and a bucket is read one
// entry after another).
std::vector<std::string> heads_of(const RegexPlan& P, uint32_t r) {
  std::vector<std::string> heads;
  for (int k = 0; k < kPrefixLens; ++k) {
    if (P.prefixes[k][r].empty()) continue;
    heads.clear();
    for (const std::string& x : P.prefixes[k][r]) heads.push_back(x.substr(0, 8));
    heads.erase(std::unique(heads.begin(), heads.end()), heads.end());  // (sorted)
    if (heads.size() <= 16) break;
  }
  return heads;
}

// Most regexes that may share a beginning, and most entries of one bucket.
//   - A position where a shared beginning occurs is walked by all of its regexes,
//     one after the other: 3.4 us a regex for beginnings of 19 bytes, whatever the
//     input's size, where the walk of their group takes one lookup a byte.
//     Measured, us a scan with the filter and before there were prefixes: 24
//     regexes over 4 KiB 113 and 171, over 64 MiB 135 and 254; 48 regexes 193 and
//     170, 222 and 254; 300 regexes 1,016 and 176, 1,136 and 258.  24 are the same
//     time where 40 bytes are shared.
//   - Unless all beginnings have 8 bytes, buckets go by the first 4, and a bucket
//     is read to its end at every position that falls to it.
constexpr size_t kSharedMost = 24, kBucketMost = 64;

// Leaves the regexes that would be walked for too many at a position uncovered.
void drop_shared(RegexPlan& P) {
  std::map<std::string, std::vector<uint32_t>> by_head;
  std::map<std::string, size_t> by_word;
  bool all8 = true;
  for (uint32_t r = 0; r < P.n_regex; ++r) {
    if (!P.covered[r]) continue;
    for (const std::string& h : heads_of(P, r)) {
      by_head[h].push_back(r);
      all8 &= h.size() == 8;
    }
  }
  std::vector<uint8_t> drop(P.n_regex, 0);
  for (const auto& h : by_head) {  // a position with this beginning has every shorter one of it too
    size_t n = 0;
    for (size_t l = 4; l <= h.first.size(); ++l) {
      const auto it = by_head.find(h.first.substr(0, l));
      n += it == by_head.end() ? 0 : it->second.size();
    }
    for (size_t l = 4; n > kSharedMost && l <= h.first.size(); ++l) {
      const auto it = by_head.find(h.first.substr(0, l));
      if (it != by_head.end())
        for (uint32_t r : it->second) drop[r] = 1;
    }
  }
  size_t longest = 0;
  for (const auto& h : by_head)
    for (uint32_t r : h.second)
      if (!drop[r]) longest = std::max(longest, ++by_word[h.first.substr(0, 4)]);
  if (!all8 && longest > kBucketMost)
    for (const auto& h : by_head)
      if (h.first.size() < 8)
        for (uint32_t r : h.second) drop[r] = 1;
  for (uint32_t r = 0; r < P.n_regex; ++r)
    if (drop[r]) P.covered[r] = 0;
}

}  // namespace

// The length is the one that lets the filter look at the fewest positions that
// the literals allow too: 7 bytes for every fourth, 5 for every second.  Longer
// prefixes are more strings (a class in the prefix multiplies them): at most
// 4,096 at 7 bytes and 16,384 at 5, beyond which the crowded filter costs more
// than the lookups it saves.  A set whose strings would fill the survivor list on
// an input over their alphabet, or whose literals would lose their long grams
// (filter_crowded), takes 20 bytes (16-byte grams), and there one short string
// would choose the layout of all: 4-byte grams, nearly all of which a nucleotide
// input passes.  So a regex is covered there only if each of its strings has the
// 19 bytes that 16-byte grams at every fourth position need; the others are walked
// (20,000 k-mers and 100 motifs over 512 MiB, us a scan: with one motif more of 8
// bases 19,600 -> 1,190, of 12 bases 1,810 -> 640).  Where no length is possible,
// every regex is walked.
void choose_prefixes(const ws_pattern_tables& t, RegexPlan& P) {
  P.prefix_len = -1;
  drop_shared(P);
  uint32_t shortest = UINT32_MAX;
  for (uint32_t i = 0; i < t.n_literals; ++i) shortest = std::min(shortest, t.offsets[2 * i + 1]);
  // (a literal of one byte fills the survivor list by itself: the filter would
  // give the prefixes up on most inputs)
  if (shortest < 2) std::fill(P.covered.begin(), P.covered.end(), 0);
  std::vector<std::pair<std::string, uint32_t>> pre;
  const size_t most[kPrefixLens] = {65536, 4096, 16384, 65536};
  for (int k = 1; k < kPrefixLens && P.prefix_len < 0; ++k)
    if ((kPrefixLen[k] <= shortest || kPrefixLen[k] == 4) && collect(P, k, most[k], pre)) P.prefix_len = k;
  if (P.prefix_len > 0) {
    std::vector<std::string> strings;
    for (const auto& x : pre) strings.push_back(x.first);
    if (filter_crowded(t, strings)) {
      P.prefix_len = -1;
      for (uint32_t r = 0; r < P.n_regex; ++r) {
        const auto& list = P.prefixes[0][r];
        bool fits = P.covered[r] && !list.empty();
        for (const std::string& x : list) fits &= x.size() >= 19;
        P.covered[r] = fits ? 1 : 0;
      }
      if (shortest >= 19 && collect(P, 0, most[0], pre)) P.prefix_len = 0;
    }
  }
  if (P.prefix_len < 0) std::fill(P.covered.begin(), P.covered.end(), 0);
}

void plan_filter(const ws_pattern_tables& t, const RegexPlan& P, LiteralPlan& plan) {
  std::vector<std::pair<std::string, uint32_t>> pre;
  if (P.n_regex && P.prefix_len >= 0) collect(P, P.prefix_len, SIZE_MAX, pre);
  std::vector<std::string> strings;
  for (const auto& x : pre) strings.push_back(x.first);
  std::sort(strings.begin(), strings.end());
  strings.erase(std::unique(strings.begin(), strings.end()), strings.end());
  plan_literals(t, plan, strings);
  if (pre.empty()) return;
  // The verify kernel's table: entries by bucket of the first 4 bytes' hash (of
  // all 8 where every entry has 8).
  struct Entry {
    uint32_t bucket, w0, w1, mask, r;
  };
  std::vector<Entry> es;
  bool all8 = true;
  for (uint32_t r = 0; r < P.n_regex; ++r) {
    if (!P.covered[r]) continue;
    for (const std::string& x : heads_of(P, r)) {
      uint32_t w[2] = {0, 0}, m[2] = {0, 0};
      std::memcpy(w, x.data(), x.size());
      std::memset(m, 0xFF, x.size());
      es.push_back({0, w[0], w[1], m[1], r});
      all8 &= x.size() == 8;
    }
  }
  uint32_t bits = 6;
  while (bits < 16 && ((size_t)1 << bits) < es.size()) ++bits;
  plan.prefix_mul = all8 ? 0x85EBCA77u : 0u;
  for (Entry& e : es) e.bucket = (e.w0 * 0x9E3779B1u + e.w1 * plan.prefix_mul) >> (32 - bits);
  std::sort(es.begin(), es.end(), [](const Entry& a, const Entry& b) { return a.bucket < b.bucket; });
  std::vector<uint32_t> range(((size_t)1 << bits) + 1, 0), entry;
  for (const Entry& e : es) {
    ++range[e.bucket + 1];
    entry.insert(entry.end(), {e.w0, e.w1, e.mask, e.r});
  }
  for (size_t k = 1; k < range.size(); ++k) range[k] += range[k - 1];
  // A pass of the compacting kernels takes longer than a walk of one group, 0.55
  // ms per GiB (a group with assertions 6): there the filter serves inputs up to
  // the size where that eats the 0.15 ms that a small walk and its reverse walks
  // take at least.
  const double extra = filter_ms_per_gib(plan) - literals_ms_per_gib(t) -
                       (0.55 * (P.n_spec - P.n_walk) + 6.0 * (P.n_groups - P.n_ctx_walk));
  plan.prefix_most = plan.gram_kernel || extra <= 0 ? UINT64_MAX : (uint64_t)(0.15 / extra * (1ull << 30));
  plan.prefix_shift = 32 - bits;
  plan.n_prefixes = (uint32_t)es.size();
  plan.d_prefix_range.upload(range.data(), range.size() * 4);
  plan.d_prefix_entry.upload(entry.data(), entry.size() * 4);
}

}  // namespace ws

// Test hook: the prefixes of one regex at `len` bytes, as lines of hex.
// Returns their number, -1 when there are too many or one is shorter than 4
// bytes, -2 for a regex that does not parse; the text is cut at `cap` bytes.
extern "C" long ws_testing_regex_prefixes(const char* source, unsigned len, unsigned long most, char* out,
                                          unsigned long cap) {
  using namespace ws;
  try {
    const ReTree tree = parse_regex(source);
    const bool ctx = tree_has_look(tree);
    const Nfa n = build_nfa({&tree}, false);
    const ByteClasses bc = compute_classes({&n});
    const Dfa d = ctx ? build_context_all_dfa(n, bc, 1 << 16) : build_all_dfa(n, bc, true, 1 << 16);
    std::vector<std::string> found;
    if (d.too_big || !regex_prefixes(d, bc, ctx, len, most, found)) return -1;
    std::string text;
    for (const std::string& x : found) {
      for (char c : x) {
        const char* hex = "0123456789abcdef";
        text += hex[(uint8_t)c >> 4];
        text += hex[(uint8_t)c & 15];
      }
      text += '\n';
    }
    const size_t k = std::min<size_t>(text.size(), cap ? cap - 1 : 0);
    std::memcpy(out, text.data(), k);
    if (cap) out[k] = 0;
    return (long)found.size();
  } catch (const std::exception&) {
    return -2;
  }
}

// Test hook: the host part of a matcher's plan for a pattern set.  Writes per
// regex whether the literal filter covers it; returns the length of the prefixes
// it looks for, 0 when it looks for none, -1 on an error.
extern "C" int ws_testing_prefix_plan(const ws_ir* ir, unsigned dfa_max_states, unsigned char* covered, unsigned long n) {
  using namespace ws;
  try {
    ws_pattern_tables t;
    ws_config c;
    if (ws_ir_tables(ir, &t) != WS_OK || t.n_regex > n) return -1;
    ws_config_default(&c);
    if (dfa_max_states) c.dfa_max_states = dfa_max_states;
    RegexPlan plan;
    read_regexes(t, c, plan);
    choose_prefixes(t, plan);
    std::copy(plan.covered.begin(), plan.covered.end(), covered);
    return plan.prefix_len < 0 ? 0 : (int)kPrefixLen[plan.prefix_len];
  } catch (const std::exception&) {
    return -1;
  }
}
