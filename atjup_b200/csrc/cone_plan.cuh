// How the projection around the obstacle (cone.cu) lays its levels' boxes out over blocks: host code, no CUDA.
#pragma once
#include <algorithm>
#include <climits>
#include <cstddef>
#include <cstdint>
#include <vector>

namespace atjup {

constexpr int CONE_CLUSTER = 4;          // blocks per level (fewer when the GPU cannot hold them)
// Dynamic shared memory of a block, of the 227 KB a block may have. The bands' constants (a wall cell's eight
// doubles, a row's eight) take up to some 24 KB more than two doubles a special cell and six a row would: a box whose
// bands fit 200 KB so must not leave shared memory for them (two levels of 299 x 179, a call from cold: 1150 ms on
// HBM, 246 so, 347 with the former kernel).
constexpr size_t CONE_SMEM_CAP = 224 * 1024;
constexpr int CONE_NROW = 8;             // doubles of constants per box row
constexpr int CONE_ROWS = 28, CONE_WORDS = 64;   // the most rows of a band a warp per row takes, and its words

// A level's box: rows, meridians, slots of its ring, doubles of its special cells' constants
struct ConeBox {
    int NJ, NK, ring, n_tab;
};
// Blocks per level; a warp per row (else words over the block's warps); the bands in shared memory (else one
// block per level on HBM); threads and dynamic shared memory of a block (0: does not fit)
struct ConePlan {
    int C;
    bool row, smem;
    int threads;
    size_t bytes;
};

// Words per row and colour, halo included. The lanes of a warp per row have all their words in every row; the
// other form takes the words a row has: padded to CONE_WORDS, half its warps have nothing to do on a box of up to
// 61 meridians (two levels of 117 x 31, a call from cold: 11.2 ms padded, 7.2 as it is; of 117 x 59 12.0 and 7.8).
inline int cone_words(const ConeBox& b, bool row) { return row ? CONE_WORDS : (b.NK + 3) / 2; }

inline size_t cone_bytes(const std::vector<ConeBox>& boxes, int C, bool row) {
    size_t most = 0, ring = 1;
    for (const ConeBox& b : boxes) {
        const size_t rows = (size_t)(b.NJ + C - 1) / C, words = cone_words(b, row);
        most = std::max(most, sizeof(double) * (2 * (rows + 2) * words + CONE_NROW * (size_t)b.NJ + (size_t)b.n_tab) +
                                  sizeof(uint32_t) * 2 * rows * words);
        ring = std::max(ring, (size_t)b.ring);
    }
    return most + sizeof(double) * 2 * ring;
}

// The form for C blocks a level: a warp per row where every band allows it
inline ConePlan cone_form(const std::vector<ConeBox>& boxes, int C) {
    int rows = 1, least = INT_MAX, words = 1;
    for (const ConeBox& b : boxes) {
        rows = std::max(rows, (b.NJ + C - 1) / C);
        least = std::min(least, b.NJ / C);
        words = std::max(words, cone_words(b, false));
    }
    const bool row = least >= 2 && rows <= CONE_ROWS && words <= CONE_WORDS && cone_bytes(boxes, C, true) <= CONE_SMEM_CAP;
    const size_t bytes = cone_bytes(boxes, C, row);
    return ConePlan{C, row, true, row ? 32 * rows : 1024, bytes <= CONE_SMEM_CAP ? bytes : 0};
}

// The largest cluster for which the GPU holds every level's cluster at once (resident(plan)), each block a band of
// at least one row; boxes that shared memory does not hold run as one block each on HBM.
template <class F>
ConePlan cone_plan(const std::vector<ConeBox>& boxes, F resident) {
    int C = CONE_CLUSTER;
    size_t ring = 1;
    for (const ConeBox& b : boxes) {
        C = std::min(C, b.NJ);
        ring = std::max(ring, (size_t)b.ring);
    }
    const ConePlan hbm{1, false, false, 1024, sizeof(double) * 2 * ring};
    if (boxes.empty() || cone_form(boxes, C).bytes == 0) return hbm;
    for (; C > 1; C--) {
        const ConePlan p = cone_form(boxes, C);
        if (p.bytes && resident(p)) return p;
    }
    const ConePlan p = cone_form(boxes, 1);
    return p.bytes ? p : hbm;
}

}  // namespace atjup
