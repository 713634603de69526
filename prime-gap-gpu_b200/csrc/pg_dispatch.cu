// pg_dispatch.cu -- maps a runtime operand layout to its compiled kernels.
//
// A layout code is L (one thread per number, L words) or (T << 16) | L (a
// group of T lanes per number, L/T words per lane); see pg_limbs.h.
#include "pg_limbs.h"
#include "pg_search.cuh"
#include "pg_search_group.cuh"
#include "pg_tc_search.cuh"

#include <algorithm>
#include <cmath>

namespace pg {

#define PG_DECL(n) PG_DECLARE_LIMBS(n)
PG_LIMB_LIST(PG_DECL)
#undef PG_DECL
#define PG_GDECL(t, lt) PG_GDECLARE(t, lt)
PG_GROUP_LIST(PG_GDECL)
#undef PG_GDECL
#define PG_TDECL(n) PG_TC_DECLARE(n)
PG_TC_LIST(PG_TDECL)
#undef PG_TDECL

bool supported_limbs(uint32_t L) {
#define PG_CASE(n) \
    if (L == n) return true;
    PG_LIMB_LIST(PG_CASE)
#undef PG_CASE
#define PG_GCASE(t, lt) \
    if (L == PG_LAYOUT_GROUP(t, (t) * (lt))) return true;
    PG_GROUP_LIST(PG_GCASE)
#undef PG_GCASE
    return false;
}

uint32_t pick_layout(uint32_t bits, uint32_t tpi) {
    uint32_t best = 0;
    if (tpi <= 1) {
#define PG_CASE(n) \
    if (best == 0 && 32u * (n) >= bits) best = n;
        PG_LIMB_LIST(PG_CASE)
#undef PG_CASE
        if (best || tpi == 1) return best;
    }
    uint32_t bestL = 0;
#define PG_GCASE(t, lt)                                                                                 \
    if ((tpi == 0 || tpi == (uint32_t)(t)) && 32u * (t) * (lt) >= bits + 2 &&                           \
        (bestL == 0 || (uint32_t)((t) * (lt)) < bestL)) {                                               \
        bestL = (t) * (lt);                                                                             \
        best = PG_LAYOUT_GROUP(t, (t) * (lt));                                                          \
    }
    PG_GROUP_LIST(PG_GCASE)
#undef PG_GCASE
    return best;
}

uint32_t pick_limbs(uint32_t words) { return pick_layout(32 * words, 0); }

// A batch that does not fill the device takes the time of its longest chain:
// the bases of a number one after the other, and the words of a squaring.
// Bases run side by side while 16 lanes (or groups) per number still finish in
// the time of one test: up to 16 384 tests of one thread each (22 words:
// 2.05 ms for 16 and for 16 384 tests), or 18 944 lanes in groups (one warp per
// SM quarter).  They also do for as many numbers of more than 20 words as base 2
// alone tests in groups, for those take the other bases in turn slower than one
// thread does (1 025 primes of 25 words, 16 bases: 63.5 ms in turn in groups, 52 on
// one thread each, 7.2 with base 2 in groups and the others side by side).  Few tests of more than 20 words take a group of lanes per
// number; the layouts were timed against one thread per number:
//   21 words 8 x 3: 1.58, 1.60, 1.79 ms at 64, 2 048, 4 096 tests (1.85 to 1.95)
//   22 words 8 x 3: 1.66, 1.87, 2.53 ms at 2 048, 4 096, 8 192 tests (2.05 at each)
//   32 words 16 x 3: 3.58, 4.19, 6.27 ms at 512, 2 048, 4 096 (5.8)
//   40 words 16 x 3: 4.37, 5.13, 7.72 ms at 512, 2 048, 4 096 (10.8)
//   48 words 8 x 8: 8.08, 10.8, 20.1 ms at 2 048, 4 096, 8 192 (18.7)
// Longer operands are in groups already; 16 lanes instead of 8 halve a row's
// products on a lane, for twice the warps:
//   95 words 16 x 6: 19.2, 25.8, 36.3, 47.5 ms at 1 184, 2 368, 3 072, 4 096
//            8 x 12: 27.5, 27.5, 39.7, 39.7
//  135 words 16 x 9: 45.8, 66.9, 101.2 ms at 1 184, 2 368, 3 072
//            8 x 17: 70.8, 70.8, 101.6
// Other bases than 2 multiply where base 2 is doubled, which groups fold into
// the squaring, so side by side they start at 17 words (64 primes, 16 bases: 17
// words 1.4 ms, 26 in turn).  17 to 20 and 24 words stop where base 2 has no warp
// of its own per number any more (launch_prp_bases_t), from where a batch of
// composites would take longer than on one thread.  Base 2 alone keeps to one
// thread per number at the sizes that its kernel fills and a group pads: 16 words
// (0.85 ms, 1.27 in groups), 17 to 20 (17 words: 1.31 to 1.38 ms at 64 to 4 096
// tests, 1.35 to 1.51 on 8 x 3; 20: 1.48 to 1.56, 1.52 to 1.71) and 24 (2.50 to 2.57 ms
// at 64 to 1 536, 2.77 to 3.23 on 16 x 3).
uint32_t pick_batch(uint32_t words, uint32_t n, uint32_t rounds, bool *side_by_side) {
    const uint32_t L = pick_limbs(words);
    *side_by_side = false;
    if (!L) return 0;
    if (L >> 16) {
        *side_by_side = rounds > 1 && (uint64_t)n * 16 * (L >> 16) <= 18944;
        const uint32_t tests = *side_by_side ? 16 * n : n;
        if (L == PG_LAYOUT_GROUP(8, 96) && tests <= 3072) return PG_LAYOUT_GROUP(16, 96);
        if (L == PG_LAYOUT_GROUP(8, 136) && tests <= 2368) return PG_LAYOUT_GROUP(16, 144);
        return L;
    }
    // numbers that base 2 alone tests in groups
    const uint32_t few = words > 23 ? (words == 48 ? 4096 : words > 24 ? 64 * words : 0) : words > 20 ? 4096 : 0;
    *side_by_side = rounds > 1 && n <= std::max(1024u, few);
    const uint32_t tests = *side_by_side ? 16 * n : n;
    // lanes of base 2 at a warp per number, the other bases in groups of T lanes
    const auto apart = [&](uint32_t T) { return *side_by_side && n * (32 + (rounds - 1) * T) <= 18944; };
    if (words > 16 && words <= 23 && (few ? tests <= few : apart(8))) return PG_LAYOUT_GROUP(8, 24);
    if (words > 23 && words <= 47 && (few ? tests <= few : apart(16))) return PG_LAYOUT_GROUP(16, 48);
    if (words == 48 && tests <= few) return PG_LAYOUT_GROUP(8, 64);
    return L;
}

uint32_t layout_words(uint32_t layout) { return layout & 0xffffu; }

cudaError_t launch_prp_batch(uint32_t L, const uint32_t *cand, uint32_t words, uint32_t n, uint32_t rounds,
                             int32_t *out, bool side_by_side, cudaStream_t st) {
    if (n == 0) return cudaSuccess;
    // Base 2 first, in a launch of its own and in the layout of a batch of it alone,
    // where it would wait for the other bases: the code of base 2 and that of the
    // others, each too long for the instruction cache, slow each other down.  One
    // thread per number from 25 words on: from a warp an SM (1 024 composites, 16
    // bases: 32 words 5.7 ms in turn, 6.6 side by side, 40 words 10.9 and 14.8; at 48
    // words the two spill); the widest groups: from two (74 composites of 144 words
    // 101.8 and 109.9 ms).  The others run beside it as fast as after it.  More than
    // 1 024 numbers on one thread are those whose base 2 runs in groups.
    const uint32_t lanes = L >> 16 ? L >> 16 : 1, warps = n * ((rounds - 1) * lanes + (lanes > 1 ? 32 : 1)) / 32;
    const bool tested = side_by_side && (L == 48 || (L >= 28 && lanes == 1 && warps > 148) || (lanes == 1 && n > 1024) ||
                                         (L == PG_LAYOUT_GROUP(8, 160) && warps > 2 * 148));
    if (tested) {
        bool one = false;
        const cudaError_t e = launch_prp_batch(pick_batch(words, n, 1, &one), cand, words, n, 1, out, one, st);
        if (e != cudaSuccess) return e;
    }
#define PG_CASE(nl)                                                                                              \
    if (L == nl)                                                                                                 \
        return side_by_side                                                                                      \
                   ? launch_prp_bases_t<OneThread<nl>>(cand, words, n, rounds, out, tested, st)                  \
                   : launch_prp_batch_t<nl>(cand, words, n, rounds, out, st);
    PG_LIMB_LIST(PG_CASE)
#undef PG_CASE
#define PG_GCASE(t, lt)                                                                                              \
    if (L == PG_LAYOUT_GROUP(t, (t) * (lt)))                                                                         \
        return side_by_side                                                                                          \
                   ? launch_prp_bases_t<LaneGroup<t, lt>>(cand, words, n, rounds, out, tested, st)                    \
                   : glaunch_prp_batch<t, lt>(cand, words, n, rounds, out, st);
    PG_GROUP_LIST(PG_GCASE)
#undef PG_GCASE
    return cudaErrorInvalidValue;
}

int search_grid(uint32_t L, int device) {
    int sms = 0, per = 0;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
#define PG_CASE(nl) \
    if (L == nl) per = search_occupancy_t<nl>();
    PG_LIMB_LIST(PG_CASE)
#undef PG_CASE
#define PG_GCASE(t, lt) \
    if (L == PG_LAYOUT_GROUP(t, (t) * (lt))) per = gsearch_occupancy<t, lt>();
    PG_GROUP_LIST(PG_GCASE)
#undef PG_GCASE
    if (per < 1) per = 1;
    return sms * per;
}

cudaError_t launch_search_persistent(uint32_t L, const SearchArgs &a, int grid, cudaStream_t st) {
    if (a.n_act == 0) return cudaSuccess;
#define PG_CASE(nl) \
    if (L == nl) return launch_search_persistent_t<nl>(a, grid, st);
    PG_LIMB_LIST(PG_CASE)
#undef PG_CASE
#define PG_GCASE(t, lt) \
    if (L == PG_LAYOUT_GROUP(t, (t) * (lt))) return glaunch_search_persistent<t, lt>(a, grid, st);
    PG_GROUP_LIST(PG_GCASE)
#undef PG_GCASE
    return cudaErrorInvalidValue;
}

// The sizes the error bounds of pg_tc.cuh's step are stated for, with
// n <= 2^n_log2, |X| < 2^x_log2, y < 2.22 n (2^1.16), T < 2^2.31 n^2, L words:
//   y fits L words, z = m*T/n fits L + 1;
//   the words of T and z left out (T_hi = T >> 32 (L-4); the correction reads
//   z above 2^(32 (L-4))) weigh less than 2^-8: 2^(32 (L-4)) * |X| / K < 2^-8;
//   the correction, at most |X| * m * 2^2.31 with relative error 2^-51.4, is
//   off by less than 2^-5;
//   m * 2 and |X| * 2 leave the 64-bit sums of the last line without a carry.
uint32_t pick_tc(uint32_t kbits, double k_log2, uint64_t max_m, uint64_t max_x) {
    if (max_m == 0 || max_m >= (1ull << 30) || max_x >= (1ull << 24)) return 0;
    const double m_log2 = std::log2((double)max_m), x_log2 = std::log2((double)max_x);
    const double n_log2 = std::log2((double)max_m + 1) + k_log2;
    if (m_log2 + x_log2 > 44) return 0;
    uint32_t best = 0;
#define PG_TCASE(n) \
    if (!best && 32.0 * (n) >= n_log2 + 1.17) best = n;
    PG_TC_LIST(PG_TCASE)
#undef PG_TCASE
    if (!best) return 0;
    if (n_log2 + m_log2 + 2.4 > 32.0 * (best + 1)) return 0;
    if (kbits < 32 * (best - 4) + 25) return 0;  // mu no longer than its column offset + 1 (tc_mma)
    if ((double)kbits - 1 < 32.0 * (best - 4) + x_log2 + 8) return 0;
    return best;
}

int tc_blocks_per_sm(uint32_t tcL) {
    int per = 0;
#define PG_TCASE(n) \
    if (tcL == n) per = tc_occupancy_t<n>();
    PG_TC_LIST(PG_TCASE)
#undef PG_TCASE
    return per < 1 ? 1 : per;
}

cudaError_t launch_search_tc(uint32_t tcL, const SearchArgs &a, int grid, cudaStream_t st) {
    if (a.n_act == 0) return cudaSuccess;
#define PG_TCASE(n) \
    if (tcL == n) return launch_search_tc_t<n>(a, grid, st);
    PG_TC_LIST(PG_TCASE)
#undef PG_TCASE
    return cudaErrorInvalidValue;
}

cudaError_t launch_search_plain(uint32_t L, const SearchArgs &a, uint32_t *k_next, cudaStream_t st) {
    if (a.n_act == 0) return cudaSuccess;
#define PG_CASE(nl) \
    if (L == nl) return launch_search_plain_t<nl>(a, k_next, st);
    PG_LIMB_LIST(PG_CASE)
#undef PG_CASE
#define PG_GCASE(t, lt) \
    if (L == PG_LAYOUT_GROUP(t, (t) * (lt))) return glaunch_search_plain<t, lt>(a, k_next, st);
    PG_GROUP_LIST(PG_GCASE)
#undef PG_GCASE
    return cudaErrorInvalidValue;
}

cudaError_t launch_finalize(uint32_t L, const SearchArgs &a, uint32_t nsides, uint32_t *gaps, uint32_t *redo,
                            uint32_t *n_redo, unsigned long long *confirm_tests, uint32_t *k_start_rw,
                            cudaStream_t st) {
    if (a.n_act == 0) return cudaSuccess;
#define PG_CASE(nl) \
    if (L == nl) return launch_finalize_t<nl>(a, nsides, gaps, redo, n_redo, confirm_tests, k_start_rw, st);
    PG_LIMB_LIST(PG_CASE)
#undef PG_CASE
#define PG_GCASE(t, lt)                                                                                    \
    if (L == PG_LAYOUT_GROUP(t, (t) * (lt)))                                                               \
        return glaunch_finalize<t, lt>(a, nsides, gaps, redo, n_redo, confirm_tests, k_start_rw, st);
    PG_GROUP_LIST(PG_GCASE)
#undef PG_GCASE
    return cudaErrorInvalidValue;
}

cudaError_t launch_confirm(uint32_t L, const SearchArgs &a, uint32_t *gaps, uint32_t *conf, uint32_t *redo,
                           uint32_t *n_redo, unsigned long long *confirm_tests, uint32_t *k_start_rw,
                           cudaStream_t st) {
    if (a.n_act == 0) return cudaSuccess;
#define PG_CASE(nl) \
    if (L == nl) return launch_confirm_t<nl>(a, gaps, conf, redo, n_redo, confirm_tests, k_start_rw, st);
    PG_LIMB_LIST(PG_CASE)
#undef PG_CASE
#define PG_GCASE(t, lt)                                                                                    \
    if (L == PG_LAYOUT_GROUP(t, (t) * (lt)))                                                               \
        return glaunch_confirm<t, lt>(a, gaps, conf, redo, n_redo, confirm_tests, k_start_rw, st);
    PG_GROUP_LIST(PG_GCASE)
#undef PG_GCASE
    return cudaErrorInvalidValue;
}

}  // namespace pg
