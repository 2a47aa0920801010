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

// ---- gradient of a fused expression: which form of the kernel ----------------------------------------------------------
// vectors: 128-bit vectors of the target (0 where its operands do not allow them), positions: extent of the lowest dim it is summed
// along (1: nothing is summed). A vector per thread costs the fewest instructions per element and wins where the vectors alone fill the
// chip (2048 resident threads per SM), and for less than a group of positions down to about one CTA per SM. Otherwise a thread takes
// one element and eight positions at a time or, where half a group is not reached, one element and one position.
// silu(a*b+b), F32 / F64, us: 2844 x 1024 elements, 9 positions: vectors 82 / 121, steps 101 / 161, single 147 / 156; 400 x 1024, 64
// positions: 89 / 139, 72 / 117, 135 / 144; 256 x 1024, 7 positions: 10 / 12, 12 / 15, 12 / 12; 25600 x 1023 (no vectors), nothing
// summed: steps 611 / 745, single 296 / 321.
enum : int { NK_GRAD_ONE = 0, NK_GRAD_VEC = 1, NK_GRAD_STEPS = 2 };
constexpr int NK_GRAD_POSITIONS = 8;

inline int nk_fused_grad_form(int64_t vectors, int64_t positions, int64_t sms) {
    if (vectors >= sms * 2048) return NK_GRAD_VEC;
    if (positions >= NK_GRAD_POSITIONS) return NK_GRAD_STEPS;
    if (vectors >= sms * 256) return NK_GRAD_VEC;
    return positions > NK_GRAD_POSITIONS / 2 ? NK_GRAD_STEPS : NK_GRAD_ONE;
}
