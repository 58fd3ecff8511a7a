// Memory and index ranges of the grouped M2L (m2l_gemm.cu): where it may run and
// where the pairs go one by one, which needs no memory per pair.  Host
// arithmetic only.
#pragma once

#include <algorithm>
#include <cstdint>

namespace fmm {

// Result rows are padded to units of kRowUnit entries (32 bytes in FP32, one DRAM
// sector) and numbered in them by 32-bit integers.
constexpr int kRowUnit = 8;
inline bool m2l_rows_fit(int64_t units) { return units <= INT32_MAX; }

// Split operators of one batch of groups, and the memory that the grouped
// products may take where the per-pair kernel is an alternative of the same kind
// (reference coefficients, periodic images, groups of a few pairs): of 280 GB, so
// that several threads' calls fit beside what else a program holds.
constexpr double kOperatorBytes = 16e9, kGroupedBytes = 64e9;

struct M2lSize {
    int64_t pairs, groups;
    int row;           // entries of a result row at the call's order
    int tensor;        // entries of a group's tensor
    int64_t operator_bytes;  // of a group's split operator and its exponents
    int entry;         // bytes of an entry
};

// Device memory of the grouped products beyond the nodes' weights: per pair its
// row, two keys, two values, target, run key, count and start; per group its
// tensor and (a batch's) operator.
inline double m2l_bytes(const M2lSize& s) {
    const double per_pair = (double)s.row * s.entry + 44.0;
    return (double)s.pairs * per_pair + (double)s.groups * s.tensor * s.entry +
           std::min(kOperatorBytes, (double)s.groups * (double)s.operator_bytes);
}

}  // namespace fmm
