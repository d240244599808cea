// gb_msm_rules.h as host code, for test_msm_rules.py
#include "gb_msm_rules.h"

extern "C" {
int r_choose_window(size_t n, int precomputed) { return gb::choose_window(n, precomputed != 0); }
int r_windows(int c) { return gb::windows_for(c); }
int r_rounds(uint64_t digits, uint64_t G, uint64_t slots, uint64_t most)
{
    return gb::affine_rounds(digits, (double)digits / (double)G, G, slots, most);
}
uint64_t r_scratch(uint64_t digits, uint64_t G, int rounds, uint64_t slots)
{
    return gb::rounds_scratch(gb::padded_entries(digits, G, rounds), rounds, slots);
}
double r_typical(const size_t *sizes, size_t n, int c, int precomputed)
{
    gb::typical_bucket b;
    for (size_t i = 0; i < n; i++) b.add(sizes[i]);
    return b.entries(c, precomputed != 0);
}
uint32_t r_short_span(double mean, double typical, uint32_t L) { return gb::short_span(mean, typical, L); }
size_t r_table_items(size_t K, size_t n) { return gb::table_items(K, n); }
uint32_t r_sum_groups(uint64_t sums, uint32_t n, int sms) { return gb::sum_groups(sums, n, sms); }
uint32_t r_pairs_per_thread(uint64_t pairs, uint64_t slots) { return gb::pairs_per_thread(pairs, slots); }
uint64_t r_rounds_limit() { return gb::kRoundsScratch; }
// the groups' first items and the end into out (n + 1 places at most); how many
size_t r_groups(const size_t *sizes, size_t n, int c, int precomputed, size_t *out)
{
    size_t k = 0, at = 0;
    for (; at < n; at += gb::group_items(at, n, [&](size_t i) { return sizes[i]; }, c, precomputed != 0)) out[k++] = at;
    out[k++] = at;
    return k;
}
}
