// Constants and plain structs shared by the host runtime and the device kernels.
#pragma once
#include <cstdint>

namespace fslbm {

constexpr int kTX = 32;                 // step tile width along x (one warp per tile row)
constexpr int kTY = 8;                  // step tile height along y
constexpr int kThreads = kTX * kTY;
constexpr uint8_t kWall = 125;          // mask value of a wall cell (pipe.m:45-47)
constexpr uint8_t kGhost = 2;           // periodic image cell of a cross-section periodic in x, y

// Per cross-section column: static wall sums of the predictor and the fluid flag.
template <class TC> struct ColCoef {
  TC ws0, wsx, wsy, fluid;
};

// Per cell, for masks that vary along z: wall sums of the predictor over the 3x3x3
// neighbourhood, including the streamwise moment (zero for extruded masks).
template <class TC> struct CellCoef {
  TC ws0, wsx, wsy, wsz;
};

// Masks per plane, FP32: a cell's wall sums in one word. Times 216 the D3Q27 weights are 64, 16, 4
// and 1, so the sums are whole numbers: bits 0-7 the sum of the weights over the cell's wall
// neighbours (at most 152), then three signed 7-bit fields with the sums of weight times cx, cy, cz
// (at most 36 in size), bit 31 set for a wall cell. A fluid cell away from walls holds 0.
constexpr uint32_t kSolidCell = 1u << 31;
inline uint32_t pack_wall_sums(int s0, int sx, int sy, int sz) {
  return uint32_t(s0) | (uint32_t(sx) & 127u) << 8 | (uint32_t(sy) & 127u) << 15 | (uint32_t(sz) & 127u) << 22;
}

}  // namespace fslbm
