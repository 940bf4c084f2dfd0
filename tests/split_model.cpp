// Every call that the entry points accept (their conditions in brackets) fits the words of its workspace, and the split
// covers all sub-tiles with CTAs that fit the exchange; offsets inside a CTA beyond 32 bits.  Prints what does not; "ok <calls>" at the end.
#include <stdio.h>

#include <random>

#include "hc_split.h"

static long g_calls = 0, g_bad = 0;
static void expect(bool ok, const char* what, size_t max_elems, size_t n, unsigned k, unsigned sms) {
  ++g_calls;
  if (!ok && ++g_bad < 20) printf("%s: handle for %zu, n %zu, streams %u, %u SMs\n", what, max_elems, n, k, sms);
}
static uint32_t subs_of(size_t n) { return (uint32_t)((n + 1023) / 1024); }

static void encode(const char* what, size_t max_elems, const uint32_t* subs, unsigned n_seg, unsigned n_in, unsigned sms, size_t n) {
  for (unsigned warps : {15u, 23u}) {
    const hc::EncodeSplit s = hc::split_encode(subs, n_seg, sms, warps);
    bool ok = hc::encode_words(s, n_seg, n_in) <= hc::workspace_words(max_elems);
    ok = ok && s.warps >= 4 && s.warps <= warps && s.grid <= sms && s.grid <= (unsigned)hc::kMaxCtas;
    for (unsigned g = 0; g < n_seg; ++g) {
      const uint64_t chunks = s.first[g + 1] - s.first[g];
      ok = ok && chunks * s.warps >= subs[g] && (chunks == 0 || (chunks - 1) * s.warps < subs[g]);
    }
    expect(ok, what, max_elems, n, n_in, sms);
  }
}
static void decode(const char* what, size_t max_elems, size_t n, unsigned k, unsigned sms) {
  for (unsigned warps : {16u, 20u}) {
    const hc::RunSplit s = hc::split_runs(subs_of(n), sms, warps);
    const uint64_t all = (uint64_t)s.grid * s.warps, run = subs_of(n) / all;
    expect(hc::run_words(s, k) <= hc::workspace_words(max_elems) && s.grid <= (unsigned)hc::kMaxCtas && s.warps <= warps &&
               (s.pool == 0 || s.pool < run),
           what, max_elems, n, k, sms);
  }
}

// the lanes' shares of the runs before a warp, with runs as long as they can be: 60 GB in a CTA
static void offsets() {
  uint32_t totals[16][hc::kMaxDst];
  for (unsigned w = 0; w < 16; ++w)
    for (unsigned q = 0; q < (unsigned)hc::kMaxDst; ++q) totals[w][q] = 0xffffffffu - 1000u * w - q;
  for (unsigned q = 0; q < (unsigned)hc::kMaxDst; ++q) {
    uint64_t want = 0;
    for (unsigned warp = 0; warp < 16; ++warp) {
      uint64_t sum = 0;
      for (unsigned part = 0; part < 8; ++part) sum += hc::runs_before(totals, q, warp, part);
      expect(sum == want, "runs before a warp", warp, q, 0, 0);
      want += totals[warp][q];
    }
  }
}

int main() {
  offsets();
  std::mt19937_64 rng(1);
  auto size = [&](size_t most) {  // spread over the logarithm, edges of sub-tiles, tiles and chunks among them
    const double e = std::uniform_real_distribution<double>(0, 1)(rng);
    size_t n = (size_t)__builtin_pow((double)most, e);
    if (rng() % 3 == 0) n = n / 32768 * 32768 + rng() % 3;
    if (rng() % 3 == 0) n = n / 1024 * 1024 + rng() % 3;
    return n < 1 ? (size_t)1 : n > most ? most : n;
  };
  for (int it = 0; it < 200000; ++it) {
    const unsigned sms = it % 4 ? 148u : (unsigned)(1 + rng() % 160);
    const size_t max_elems = size((size_t)1 << 33);
    const size_t n = it % 3 ? size(max_elems) : max_elems;  // [n <= max_elems]
    const uint32_t subs = subs_of(n);
    encode("compress", max_elems, &subs, 1, 0, sms, n);
    encode("add", max_elems, &subs, 1, 1, sms, n);
    encode("add of two streams", max_elems, &subs, 1, 2, sms, n);
    decode("decompress", max_elems, n, 1, sms);
    for (unsigned k = 1; k <= 8; ++k) {
      if (k * hc::rate_bytes(n) > hc::rate_bytes(max_elems) + 64) break;  // [hc_hom_add_multi, hc_decompress_sum]
      encode("add of several streams", max_elems, &subs, 1, k, sms, n);
      decode("sum", max_elems, n, k, sms);
    }
    uint32_t seg[8];
    size_t total = 0;
    unsigned n_seg = 0;
    for (; n_seg < 8; ++n_seg) {
      const size_t m = rng() % 8 ? size(n) : 0;
      if (total + hc::rate_bytes(m) * 32 > hc::rate_bytes(max_elems) * 32) break;  // [hc_compress_batch]
      total += hc::rate_bytes(m) * 32;
      seg[n_seg] = subs_of(m);
    }
    uint64_t any = 0;
    for (unsigned g = 0; g < n_seg; ++g) any += seg[g];
    if (any) encode("batch", max_elems, seg, n_seg, 0, sms, n);
  }
  if (g_bad) printf("%ld of %ld\n", g_bad, g_calls);
  else printf("ok %ld\n", g_calls);
  return g_bad != 0;
}
