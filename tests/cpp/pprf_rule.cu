// The PPRF's rule for threads per tree, for a CPU test.
#include "../../cuot_b200/csrc/pprf_kernel.cuh"

extern "C" int pprf_rule(uint64_t trees, int h, uint64_t ctas) { return cuot::pprf_group_size(trees, h, ctas); }
