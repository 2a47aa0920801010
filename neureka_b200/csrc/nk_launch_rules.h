// Rules of launch shapes that are plain arithmetic on sizes. No CUDA header is needed: tests compile this file for the host.
#pragma once
#include <cstdint>

// ---- F64 products: parts along k -------------------------------------------------------------------------------------
// Every part of a 64 x 64 tile is left in scratch and read back (64 KB in all), so parts cost what there are of them. Estimated
// cycles of the busiest SM, r CTAs on it: one, two, three resident CTAs need 2100, 2950, 4240 cycles per 16-deep k panel (the FP64
// pipe is full at three; one alone waits for its own loads), more CTAs run in groups of three; a part adds 1250 cycles of
// traffic, a split 4000 + 600 per part for the last one's additions. Measured with 1 to 16 parts over 20 products of 1 to 4096 tiles:
// the rule's choice is within 4 % of the best everywhere (4096 x 1000 x 4096: 1 part 1197 us, 7 parts 1310; 640 x 4096 x 768: 6
// parts 166, 1 part 281). The parts of a call never take more than 64 MB.
struct NkDgemmParts {
    int splits;
    int64_t kb_per;   // k panels per part
};
constexpr int NK_DGEMM_MAX_SPLITS = 16;
constexpr int64_t NK_DGEMM_PART_BYTES = 64 * 64 * 8, NK_DGEMM_SCRATCH_LIMIT = int64_t(64) << 20;

inline NkDgemmParts nk_dgemm_parts(int64_t tiles, int64_t k_panels, int64_t sms) {
    const double resident[3] = {0, 2100, 2950};
    NkDgemmParts best = {1, k_panels};
    double best_est = 0;
    for (int s = 1; s <= NK_DGEMM_MAX_SPLITS; s++) {
        if (s > 1 && (s > k_panels / 4 || tiles > NK_DGEMM_SCRATCH_LIMIT / NK_DGEMM_PART_BYTES / s)) break;
        const int64_t per = (k_panels + s - 1) / s, r = (tiles * s + sms - 1) / sms;
        const double est = (double(r / 3) * 4240 + resident[r % 3]) * double(per) + (s > 1 ? 4000 + 600.0 * s + 1250.0 * double(r) : 0);
        if (s == 1 || est < best_est) {
            best_est = est;
            best.splits = s;
            best.kb_per = per;
        }
    }
    best.splits = int((k_panels + best.kb_per - 1) / best.kb_per);   // rounding may leave the last part empty
    return best;
}
