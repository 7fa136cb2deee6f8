// tiles_f32_pipecol.cu -- float pipelined column FFTs (tiles_pipe.cuh) of
// the 2D and column transforms, lengths 2^9 .. 2^12.
#include "tiles_impl.cuh"

namespace gfft {
// (length, columns a tile, points a thread, groups, stages, stages of the
// version for rows off 16-byte boundaries)
#define P2(L, C, E, NG, NB, NBU) static PipeReg<TILE_COL_PLAIN, L, C, E, NG, NB, NBU> pipe_plain_##L##_##C;
P2(9, 16, 32, 2, 3, 3) P2(10, 8, 32, 2, 3, 2) P2(11, 8, 64, 1, 1, 1) P2(12, 4, 64, 1, 1, 1)
#undef P2
}  // namespace gfft
