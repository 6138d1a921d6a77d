// Tile shapes of the fused kernel compiled per K and state width (rows x
// slices x slices per thread; W = 4 for FP32, 2 for the 16-bit formats), each in
// the exact and the fast arithmetic (fused_*.cu).  Entries `exact` and `fast` are
// the defaults of the two; options can name the first `named` entries.
// Measured per iteration on a 448 x 448 x 256 core (radius 215, iterations 2 to 24):
//   K = 3, FP32   exact 8 x 128 x 4 0.844 ms, 16 x 64 x 2 0.871; fast 0.593, 0.636
//   K = 3, bf16   exact 16 x 64 x 2 0.882 ms, 8 x 128 x 4 0.950; fast 0.659, 0.605
//   K = 2, FP32   exact 8 x 128 x 2 0.476 ms, 8 x 64 x 4 0.673; fast 0.375, 0.345
//   K = 4, FP32   exact 8 x 64 x 2 1.36 ms, 4 x 128 x 4 2.19; fast 0.978, 1.08
//   K = 5, FP32   exact 8 x 64 x 2 2.09 ms, 4 x 64 x 4 5.46; fast 1.24, 2.50
#pragma once

namespace potts {

template <int K, int W>
struct TileShapes;
template <int W> struct TileShapes<2, W> { static constexpr int n = 2, named = 2, exact = 0, fast = 1; static constexpr int r[n] = {8, 8}, t[n] = {128, 64}, v[n] = {2, 4}; };
template <> struct TileShapes<3, 4> { static constexpr int n = 4, named = 4, exact = 3, fast = 3; static constexpr int r[n] = {16, 8, 8, 8}, t[n] = {64, 128, 64, 128}, v[n] = {2, 2, 2, 4}; };
template <> struct TileShapes<3, 2> { static constexpr int n = 3, named = 2, exact = 0, fast = 2; static constexpr int r[n] = {16, 8, 8}, t[n] = {64, 128, 128}, v[n] = {2, 2, 4}; };
template <> struct TileShapes<4, 4> { static constexpr int n = 3, named = 3, exact = 0, fast = 0; static constexpr int r[n] = {8, 8, 4}, t[n] = {64, 64, 128}, v[n] = {2, 4, 4}; };
template <> struct TileShapes<4, 2> { static constexpr int n = 1, named = 1, exact = 0, fast = 0; static constexpr int r[n] = {8}, t[n] = {64}, v[n] = {2}; };
template <int W> struct TileShapes<5, W> { static constexpr int n = 2, named = 2, exact = 1, fast = 1; static constexpr int r[n] = {4, 8}, t[n] = {64, 64}, v[n] = {4, 2}; };
template <> struct TileShapes<6, 4> { static constexpr int n = 1, named = 1, exact = 0, fast = 0; static constexpr int r[n] = {4}, t[n] = {64}, v[n] = {4}; };
template <> struct TileShapes<6, 2> { static constexpr int n = 2, named = 2, exact = 1, fast = 1; static constexpr int r[n] = {4, 8}, t[n] = {64, 64}, v[n] = {4, 2}; };

template <int K, typename ST>
using ShapesOf = TileShapes<K, (int)sizeof(ST) == 4 ? 4 : 2>;

}  // namespace potts
