// The line transforms of lines.cuh for float.
#include "lines_impl.cuh"

INST_LINES(float, float2)
