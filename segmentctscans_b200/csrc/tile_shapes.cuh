// Tile shapes of the fused kernel compiled per K and state width (rows x
// slices x slices per thread; W = 4 for FP32, 2 for the 16-bit formats), each in
// the exact and the fast arithmetic (fused_*.cu).  Options can name the first
// `named` entries.  exact / fast: time per voxel of a full tile relative to the
// best shape's (per cent); choose_tile weighs a volume's ragged tiles with them.
// Which shape is best depends on the share of voxels in the projection loop.  K = 2,
// K = 4 FP32 and K = 3: measured on a 448 x 448 x 256 core of radius 215 with small grains
// (16-bit K = 2: FP32's).  K = 3 FP32 exact: 8 x 64 x 2 measured 106 there, but 112 to 126
// on smoother fields, and cores of 300^3 and 440^3 took it at 1.11 against 0.91 ms
// (smooth 440^3); 109 is the least weight that avoids those, and over 112 runs on 28 cores
// (grains of 12 to 160 voxels, 40 to 600 iterations) none is slower than with 106, the best
// by 24 %.  16 x 64 x 2 is 4 % slower than 8 x 128 x 4 on small grains, 10 % faster on large
// ones late (512 x 512 x 256, 600 iterations: 0.874 against 0.961 ms): its weight is the
// least.  K = 5 and K = 6: means over cubic grains of 200, 56 and 14 voxels on a 512 x
// 512 x 256 core.
// Best shapes per iteration on the 14-voxel grains of that core, exact and fast: K = 2 0.546 and
// 0.428 ms, K = 3 1.334 (8 x 128 x 4; 16 x 64 x 2 1.387) and 0.880, 16-bit 1.452 and 0.933, K = 4
// 2.99 and 1.66, K = 5 6.22 and 2.91, K = 6 24.6 and 9.2 (4 x 64 x 4; 16-bit with 8 x 64 x 2:
// 11.7 and 4.7).  A K = 3 tile of 8 x 64 x 4 with two blocks per multiprocessor measured
// 0.840 against 0.806 ms fast and 1.33 against 1.17 exact on 512 x 512 x 256.
#pragma once

namespace potts {

template <int K, int W>
struct TileShapes;
template <int W> struct TileShapes<2, W> { static constexpr int n = 2, named = 2; static constexpr int r[n] = {8, 8}, t[n] = {128, 64}, v[n] = {2, 4}, exact[n] = {104, 100}, fast[n] = {108, 100}; };
template <> struct TileShapes<3, 4> { static constexpr int n = 4, named = 4; static constexpr int r[n] = {16, 8, 8, 8}, t[n] = {64, 128, 64, 128}, v[n] = {2, 2, 2, 4}, exact[n] = {100, 109, 109, 104}, fast[n] = {107, 113, 123, 100}; };
template <> struct TileShapes<3, 2> { static constexpr int n = 3, named = 2; static constexpr int r[n] = {16, 8, 8}, t[n] = {64, 128, 128}, v[n] = {2, 2, 4}, exact[n] = {100, 112, 108}, fast[n] = {109, 120, 100}; };
template <> struct TileShapes<4, 4> { static constexpr int n = 3, named = 3; static constexpr int r[n] = {8, 8, 4}, t[n] = {64, 64, 128}, v[n] = {2, 4, 4}, exact[n] = {100, 170, 162}, fast[n] = {100, 116, 110}; };
template <> struct TileShapes<4, 2> { static constexpr int n = 1, named = 1; static constexpr int r[n] = {8}, t[n] = {64}, v[n] = {2}, exact[n] = {100}, fast[n] = {100}; };
template <> struct TileShapes<5, 4> { static constexpr int n = 2, named = 2; static constexpr int r[n] = {4, 8}, t[n] = {64, 64}, v[n] = {4, 2}, exact[n] = {214, 100}, fast[n] = {162, 100}; };
template <> struct TileShapes<5, 2> { static constexpr int n = 2, named = 2; static constexpr int r[n] = {4, 8}, t[n] = {64, 64}, v[n] = {4, 2}, exact[n] = {172, 100}, fast[n] = {142, 100}; };
template <> struct TileShapes<6, 4> { static constexpr int n = 1, named = 1; static constexpr int r[n] = {4}, t[n] = {64}, v[n] = {4}, exact[n] = {100}, fast[n] = {100}; };
template <> struct TileShapes<6, 2> { static constexpr int n = 2, named = 2; static constexpr int r[n] = {4, 8}, t[n] = {64, 64}, v[n] = {4, 2}, exact[n] = {179, 100}, fast[n] = {167, 100}; };

template <int K, typename ST>
using ShapesOf = TileShapes<K, (int)sizeof(ST) == 4 ? 4 : 2>;

}  // namespace potts
