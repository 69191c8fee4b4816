// fs_lines32.cu -- the periodic Stokes solve by line transforms (fs_lines.cuh), FP32:
// forward real transform, projection of flow_solve (FCMfunctions.cpp:648-736) and
// inverse real transform in five passes over the grid.
#include <cmath>
#include <vector>
#include "fs_lines.cuh"

fs_status lines_init32(fs_ctx *c) { return lines_init_t<F2>(c); }
fs_status lines_prepare32(fs_ctx *c) { return lines_prepare_t<F2>(c); }
fs_status lines_flow_solve32(fs_ctx *c) { return lines_flow_solve_t<F2>(c); }
