// csrc/ss_rules.hpp for tests/test_rules.py
#include "ss_rules.hpp"

extern "C" double rule_sweep_wide_rows(int fp32, int complex_values, int G, int batch) {
    return ssg::sweep_wide_rows(fp32 != 0, complex_values != 0, G, batch != 0);
}

// 1: persistent; levels, rows and entries of one instance, all instances alike
extern "C" int rule_batch_persists(double instances, double n, double nnz, double levels, int complex_values, int tiles) {
    ssg::BatchShape b{};
    b.instances = instances;
    b.rows = instances * n;
    b.nnz = instances * nnz;
    b.max_rows = n;
    b.max_nnz = nnz;
    b.levels = levels;
    b.sms = 152;
    b.complex_values = complex_values != 0;
    b.tiles = tiles != 0;
    return ssg::batch_persists(b);
}
