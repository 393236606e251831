// What both forms of the sweep share: frames, label rows and cell tests.
#pragma once

#include <cstdint>

#include "lattice_common.cuh"

namespace apgar_b200 {
namespace {

constexpr int16_t kNever = -32000;
constexpr int kMaxRowPasses = 4096;

// Geometry of one net in its frame.
struct Frame {
  int transposed;
  int R, K, pitch;
  int x0, y0;
};

// C consecutive labels of a row from cell xs on (the pitch is a multiple of 4).
template <int C>
__device__ __forceinline__ void load_cells(const uint32_t* src, int pitch, int xs, uint32_t (&v)[C]) {
  static_assert(C % 4 == 0, "16-byte loads");
#pragma unroll
  for (int q = 0; q < C / 4; ++q) {
    const int x = xs + 4 * q;
    if (x < pitch) {
      const uint4 t = *reinterpret_cast<const uint4*>(src + x);
      v[4 * q + 0] = t.x;
      v[4 * q + 1] = t.y;
      v[4 * q + 2] = t.z;
      v[4 * q + 3] = t.w;
    } else {
      v[4 * q + 0] = v[4 * q + 1] = v[4 * q + 2] = v[4 * q + 3] = kLabelInf;
    }
  }
}

template <int C>
__device__ __forceinline__ void store_cells(uint32_t* dst, int pitch, int xs, const uint32_t (&v)[C]) {
#pragma unroll
  for (int q = 0; q < C / 4; ++q) {
    const int x = xs + 4 * q;
    if (x < pitch) {
      *reinterpret_cast<uint4*>(dst + x) = make_uint4(v[4 * q + 0], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
    }
  }
}

__device__ __forceinline__ bool cell_free(const LatticeDeviceView& lat,
                                          const apgar_b200_lattice_net& n, int l, int x, int y) {
  if (l < 0 || l >= lat.layers || x < 0 || y < 0 || x >= static_cast<int>(n.win_w) ||
      y >= static_cast<int>(n.win_h)) {
    return false;
  }
  const int gx = static_cast<int>(n.win_x0) + x, gy = static_cast<int>(n.win_y0) + y;
  const uint32_t word =
      __ldg(lat.blocked + (static_cast<size_t>(l) * lat.height + gy) * lat.words + (gx >> 5));
  return ((word >> (gx & 31)) & 1u) == 0;
}

__device__ __forceinline__ bool via_bit_at(const LatticeDeviceView& lat,
                                           const apgar_b200_lattice_net& n, int lower, int x,
                                           int y) {
  if (lat.via_ok == nullptr) return true;
  const int gx = static_cast<int>(n.win_x0) + x, gy = static_cast<int>(n.win_y0) + y;
  const uint32_t word =
      __ldg(lat.via_ok + (static_cast<size_t>(lower) * lat.height + gy) * lat.words + (gx >> 5));
  return ((word >> (gx & 31)) & 1u) != 0;
}

__constant__ int kDxc[8] = {1, 1, 0, -1, -1, -1, 0, 1};
__constant__ int kDyc[8] = {0, 1, 1, 1, 0, -1, -1, -1};

}  // namespace
}  // namespace apgar_b200
