// mw_opplan.hpp -- how the lists of a group of operators are built (mw_optab.cu): together, one operator at a
// time, or not at all.  Host arithmetic only.
#pragma once

namespace mwb {

// Operators share a build while their records' scratch stays at 1.2 GB or less: 72 bytes a record (key in three copies,
// bound and place in two each, term, head and its sum, the sorts' own).  A root of 10 boxes a side, 19^3 offsets for each
// of 8 x 134 terms, has 7.4 million records; beyond the limit one operator at a time costs little against the lists
constexpr long long kOpGroupRecords = 1ll << 24;
// positions within one operator's lists are 32-bit, rounded up to whole blocks of threads
constexpr long long kOpMaxRecords = (1ll << 31) - 1024, kOpMaxRows = 1ll << 30;
// offsets of the bands that one operator's lists are picked from: 4e10 take 2.5 s on the device, 1e12 took 44
constexpr double kOpMaxScan = 1e11;

enum class OpPlan { together, singly, refuse };

// rows: (term, dx, dy) rows of the whole group; scan: the offsets of all rows; records: those above the cut (each row
// has up to 1023, so their sum needs 64 bits)
inline OpPlan op_plan_rows(int nop, long long rows, double scan) {
    if (nop > 1 && (rows > kOpGroupRecords || scan > kOpMaxScan)) return OpPlan::singly;
    return rows > kOpMaxRows || scan > kOpMaxScan ? OpPlan::refuse : OpPlan::together;
}
inline OpPlan op_plan_records(int nop, long long records) {
    if (nop > 1 && records > kOpGroupRecords) return OpPlan::singly;
    return records > kOpMaxRecords ? OpPlan::refuse : OpPlan::together;
}

}  // namespace mwb
