// Sizes of the digit splits' workspace (mlf_split64.cu), host code without CUDA.
#pragma once
#include <algorithm>
#include <cstddef>

namespace mlf {

constexpr int OZ_C = 12;           // complex columns per CTA
constexpr int OZ_DENSE_COLS = 48;  // columns at a time of the dense operator
constexpr int OZ_MAX_SPLIT = 4, OZ_MAX_DENSE_SPLIT = 8;

// Parts of the terms: enough CTAs for about four waves of one per SM
inline int oz_split(int tiles, int nsm, int nrhs, bool dense) {
    const int ctas = tiles * ((nrhs + OZ_C - 1) / OZ_C);
    return std::max(1, std::min(dense ? OZ_MAX_DENSE_SPLIT : OZ_MAX_SPLIT, (4 * nsm + ctas - 1) / ctas));
}

// What blocks of up to nrhs columns need of the two buffers: the parts' sums (not
// monotone in the columns: the split falls where a further 12 begin, so the
// maximum over them) and the exponents, `fixed` and `per_col` a column.  The one
// may be long enough where the other is not.
struct OzSizes {
    size_t sums = 0, exps = 0;
};
inline OzSizes oz_sizes(int tiles, int nsm, int N, bool dense, size_t fixed, size_t per_col, int nrhs) {
    OzSizes z;
    for (int n = 2; n <= nrhs; ++n) z.sums = std::max(z.sums, (size_t)oz_split(tiles, nsm, n, dense) * n * N);
    z.exps = fixed + per_col * nrhs;
    return z;
}
inline bool oz_short(const OzSizes& have, const OzSizes& need) { return have.sums < need.sums || have.exps < need.exps; }

}  // namespace mlf
