// tiles_f32_pipe.cu -- float pipelined tile kernels (tiles_pipe.cuh): the
// column and row passes of the four-step split and the column FFTs of the
// 2D and column transforms, lengths 2^8 .. 2^12.
#include "tiles_impl.cuh"

namespace gfft {
// (length, columns or rows a tile, points a thread, groups, stages)
#define P(V, L, C, E, NG, NB) static PipeReg<V, L, C, E, NG, NB> pipe_##V##_##L##_##C;
#define P2(L, C, E, NG, NB) P(TILE_COL_TWP, L, C, E, NG, NB) P(TILE_ROW_PIPE, L, C, E, NG, NB)
P2(8, 16, 32, 4, 4) P2(9, 16, 32, 2, 2) P2(10, 8, 32, 2, 2) P2(11, 8, 64, 1, 1) P2(12, 4, 64, 1, 1)
#undef P2
#undef P
}  // namespace gfft
