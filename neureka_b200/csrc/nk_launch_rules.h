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

// ---- sums: what adds the tiles of 128 elements ----------------------------------------------------------------------------
constexpr int64_t NK_SUM_LAST = 4096;   // elements that one CTA adds by itself: a tile per warp (16384, four tiles per warp: 18 us, two launches 10)

// Contiguous and 16-byte aligned: 32 tiles per warp through asynchronous copies where a warp per tile would take more than 40 warps per SM.
// F32, us, rows / warps: 300000 elements 10.3 / 8.2, 600000 14.3 / 12.3, 2^20 13.3 / 14.4, 2^21 13.3 / 16.4, 2^23 18.5 / 33.
inline bool nk_sum_by_rows(int64_t tiles, int64_t sms) { return tiles >= sms * 40; }

// A view that 16-byte copies do not fit: 32 tiles per warp with an adder per lane (true), or a tile per warp with one adder. A group takes
// 60 to 100 us of dependent loads however few there are, a warp (64 per SM) about 8 us per tile, more where several dims have to be
// taken apart. F32, us, groups / warps: 2^20 elements from an odd address 68 / 18, 12.6 M 74 / 72, 16.8 M 78 / 90, 33.6 M 154 / 208; a slice of
// 1000 x 1000 83 / 21; 300 x 300 x 300 turned 268 / 242 (F64 405 / 270), 400 x 400 x 400 turned 545 / 627 (734 / 742).
inline bool nk_sum_by_groups(int64_t tiles, int merged_dims, int64_t sms) { return tiles >= sms * 64 * (merged_dims <= 2 ? 12 : 24); }
