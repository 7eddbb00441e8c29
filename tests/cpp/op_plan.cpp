// How operator lists of given sizes are built (mw_opplan.hpp): prints one word per case of tests/test_op_plan.py.
#include <cstdio>
#include <cstdlib>

#include "mw_opplan.hpp"

int main(int argc, char** argv) {  // nop rows scan records
    const int nop = std::atoi(argv[1]);
    const long long rows = std::atoll(argv[2]), records = std::atoll(argv[4]);
    const double scan = std::atof(argv[3]);
    const char* names[] = {"together", "singly", "refuse"};
    mwb::OpPlan p = mwb::op_plan_rows(nop, rows, scan);
    if (p == mwb::OpPlan::together) p = mwb::op_plan_records(nop, records);
    std::puts(names[(int)p]);
    return argc == 5 ? 0 : 1;
}
