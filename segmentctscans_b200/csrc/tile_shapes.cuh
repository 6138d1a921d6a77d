// Tile shapes of the fused kernel compiled per K and state width (rows x
// slices x slices per thread; W = 4 for FP32, 2 for the 16-bit formats), each in
// the exact and the fast arithmetic (fused_*.cu).  Options can name the first
// `named` entries.  exact / fast: time per voxel of a full tile relative to the
// best shape's (per cent), measured on a 448 x 448 x 256 core of radius 215 over
// the iterations 2 to 24; choose_tile weighs a volume's ragged tiles with them.
// Best shapes per iteration: K = 3 FP32 exact 0.844 ms (8 x 128 x 4; 16 x 64 x 2 0.871,
// but 15 % faster where few voxels run the projection loop, 0.89 against 1.05 ms
// at 4 % of them on 512 x 512 x 256: its weight is below), fast 0.593, bf16 0.882
// and 0.605; K = 4 1.36 and 0.978; K = 5 2.09 and 1.24; K = 2 (512 x 512 x 256,
// iterations 2 to 40, 8 x 64 x 4 with two blocks per multiprocessor) 0.589 and
// 0.452.  A K = 3 tile of 8 x 64 x 4 with two blocks measured 0.840 against 0.806
// ms fast and 1.33 against 1.17 exact there.
#pragma once

namespace potts {

template <int K, int W>
struct TileShapes;
template <int W> struct TileShapes<2, W> { static constexpr int n = 2, named = 2; static constexpr int r[n] = {8, 8}, t[n] = {128, 64}, v[n] = {2, 4}, exact[n] = {104, 100}, fast[n] = {108, 100}; };
template <> struct TileShapes<3, 4> { static constexpr int n = 4, named = 4; static constexpr int r[n] = {16, 8, 8, 8}, t[n] = {64, 128, 64, 128}, v[n] = {2, 2, 2, 4}, exact[n] = {100, 109, 106, 104}, fast[n] = {107, 113, 123, 100}; };
template <> struct TileShapes<3, 2> { static constexpr int n = 3, named = 2; static constexpr int r[n] = {16, 8, 8}, t[n] = {64, 128, 128}, v[n] = {2, 2, 4}, exact[n] = {100, 112, 108}, fast[n] = {109, 120, 100}; };
template <> struct TileShapes<4, 4> { static constexpr int n = 3, named = 3; static constexpr int r[n] = {8, 8, 4}, t[n] = {64, 64, 128}, v[n] = {2, 4, 4}, exact[n] = {100, 170, 162}, fast[n] = {100, 116, 110}; };
template <> struct TileShapes<4, 2> { static constexpr int n = 1, named = 1; static constexpr int r[n] = {8}, t[n] = {64}, v[n] = {2}, exact[n] = {100}, fast[n] = {100}; };
template <int W> struct TileShapes<5, W> { static constexpr int n = 2, named = 2; static constexpr int r[n] = {4, 8}, t[n] = {64, 64}, v[n] = {4, 2}, exact[n] = {261, 100}, fast[n] = {201, 100}; };
template <> struct TileShapes<6, 4> { static constexpr int n = 1, named = 1; static constexpr int r[n] = {4}, t[n] = {64}, v[n] = {4}, exact[n] = {100}, fast[n] = {100}; };
template <> struct TileShapes<6, 2> { static constexpr int n = 2, named = 2; static constexpr int r[n] = {4, 8}, t[n] = {64, 64}, v[n] = {4, 2}, exact[n] = {250, 100}, fast[n] = {200, 100}; };

template <int K, typename ST>
using ShapesOf = TileShapes<K, (int)sizeof(ST) == 4 ? 4 : 2>;

}  // namespace potts
