// Host arithmetic that shapes the launches: plain C++, no CUDA.
#pragma once

namespace fta {

// Row groups of the forward pass are dealt round-robin to grid.y CTAs per (query block, head); `per` is the number of
// (query block, head) pairs. Picks the smallest grid.y whose schedule (waves of one CTA per SM, the longest CTA setting
// the pace) is within 3 % of the best: few long-lived CTAs amortise their start-up and keep the pipeline full across
// row groups. At most 96, or what one wave holds if that is more: with one pair a wave has room for 148 (L1 1024 L2 128
// D64: 17.2 us with 128 CTAs of four groups, 23.5 with 86 of six), but short CTAs in several waves pay their start-up
// each time, more than this model says (B1 H3 L1 592 L2 128 D32: 26.4 us with 3 x 148 CTAs of one group, 23.2 with
// 3 x 37 of four).
// Only the smallest grid.y of each length of the longest CTA is looked at: more CTAs of the same length fill no fewer
// waves. That is the answer of a search over all grid.y in about 2 sqrt(ngroups) steps.
inline int fwd_grid_rows(int ngroups, long long per, int sms) {
  const int most = sms / per > 96 ? static_cast<int>(sms / per) : 96;
  auto efficiency = [&](int gy) {
    const long long waves = (per * gy + sms - 1) / sms;
    const int longest = (ngroups + gy - 1) / gy;
    // fixed cost per CTA of about a third of a row group
    return static_cast<double>(per) * ngroups / (static_cast<double>(waves) * sms * (longest + 0.35));
  };
  auto next = [&](int gy) {  // the smallest grid.y with a shorter longest CTA, or 0
    const int longest = (ngroups + gy - 1) / gy;
    const int n = longest > 1 ? (ngroups + longest - 2) / (longest - 1) : 0;
    return n <= most ? n : 0;
  };
  double best = 0.0;
  for (int gy = 1; gy; gy = next(gy)) {
    const double e = efficiency(gy);
    best = e > best ? e : best;
  }
  for (int gy = 1; gy; gy = next(gy))
    if (efficiency(gy) >= 0.97 * best) return gy;
  return 1;
}

}  // namespace fta
