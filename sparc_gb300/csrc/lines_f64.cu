// The line transforms of lines.cuh for double.
#include "lines_impl.cuh"

INST_LINES(double, double2)
