// fs_lines64.cu -- the periodic Stokes solve by line transforms (fs_lines.cuh), FP64:
// forward real transform, projection of flow_solve (FCMfunctions.cpp:648-736) and
// inverse real transform in five passes over the grid.
#include <cmath>
#include <vector>
#include "fs_lines.cuh"

fs_status lines_init64(fs_ctx *c) { return lines_init_t<double>(c); }
fs_status lines_prepare64(fs_ctx *c) { return lines_prepare_t<double>(c); }
fs_status lines_flow_solve64(fs_ctx *c) { return lines_flow_solve_t<double>(c); }
