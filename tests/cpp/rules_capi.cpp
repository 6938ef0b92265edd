// csrc/ss_rules.hpp for tests/test_rules.py
#include "ss_rules.hpp"

extern "C" double rule_sweep_wide_rows(int fp32, int complex_values, int G, int batch) {
    return ssg::sweep_wide_rows(fp32 != 0, complex_values != 0, G, batch != 0);
}
