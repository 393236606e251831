// What both forms of the sweep share: frames, label rows, and the result with
// its canonical path.
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

// The net's record and, from exact labels, its path (one warp).
__device__ __forceinline__ void write_sweep_result(const SweepLaunch& p, const NetPlan& plan, const Frame& f,
                                                   const apgar_b200_lattice_net& net, const uint32_t* slab,
                                                   uint32_t layer_stride, const int16_t* modified, uint32_t completion,
                                                   uint32_t sweeps_done, uint32_t stat_rows, uint32_t stat_stores,
                                                   uint32_t stat_loads, int lane) {
  const LatticeDeviceView& lat = p.lat;
  const uint32_t orth = lat.orth, diag = lat.diag, via = lat.via;
  const int lsx = static_cast<int>(net.start_x) - f.x0, lsy = static_cast<int>(net.start_y) - f.y0;
  const int lgx = static_cast<int>(net.goal_x) - f.x0, lgy = static_cast<int>(net.goal_y) - f.y0;
  const int s_layer = static_cast<int>(net.start_layer), g_layer = static_cast<int>(net.goal_layer);
  apgar_b200_lattice_result res{};
  res.cost = APGAR_B200_UNREACHABLE;
  res.completion = completion;
  res.sweeps = sweeps_done;
  res.row_steps = stat_rows;
  res.row_stores = stat_stores;
  res.row_loads = stat_loads;
  auto label_at = [&](int l, int x, int y) -> uint32_t {
    const int r = f.transposed ? x : y, q = f.transposed ? y : x;
    const uint32_t label = slab[static_cast<uint32_t>(l) * layer_stride +
                                static_cast<uint32_t>(r) * static_cast<uint32_t>(f.pitch) + static_cast<uint32_t>(q)];
    return modified[r] == kNever ? kLabelInf : label;  // a row never stored holds no labels
  };
  if (completion == APGAR_B200_COMPLETION_REACHED) {
    const uint32_t goal = label_at(g_layer, lgx, lgy);
    if (goal >= kLabelInf) {
      res.completion = APGAR_B200_COMPLETION_DISCONNECTED;
    } else {
      res.cost = goal;
      const uint32_t min_move = min(orth, min(diag, via));
      const unsigned long long bound = goal / min_move + 1ull;
      unsigned long long base = 0;
      if (lane == 0) base = atomicAdd(p.arena_cursor, bound);
      base = __shfl_sync(0xFFFFFFFFu, base, 0);
      if (base + bound > p.path_arena_capacity) {
        res.completion = APGAR_B200_COMPLETION_REJECTED;
        res.cost = APGAR_B200_UNREACHABLE;
      } else {
        const int Ln = lat.layers;
        int cl = g_layer, cx = lgx, cy = lgy;
        uint32_t here = goal;
        uint32_t n = 0;
        bool ok = false;
        while (n < bound) {
          if (lane == 0) {
            p.path_arena[base + n] = static_cast<uint32_t>(
                (static_cast<size_t>(cl) * lat.height + (f.y0 + cy)) * lat.width + (f.x0 + cx));
          }
          ++n;
          if (cl == s_layer && cx == lsx && cy == lsy) {
            ok = true;
            break;
          }
          // One round of independent loads per cell (0.45 us a cell with the
          // bit planes read first and the labels after).  The labels tell
          // what is free: at the fixed point every free cell next to a
          // reached one is reached, so an unreached side cell is blocked.
          int pl = cl, px = cx, py = cy;
          bool via_legal = true;
          if (lane < 8) {
            px = cx - kDxc[lane];
            py = cy - kDyc[lane];
          } else if (lane == 8 || lane == 9) {
            pl = (lane == 8) ? cl - 1 : cl + 1;
            if (pl >= 0 && pl < Ln) via_legal = via_bit_at(lat, net, min(pl, cl), cx, cy);
          }
          uint32_t pd = kLabelInf;
          if (lane < 10 && pl >= 0 && pl < Ln && px >= 0 && px < static_cast<int>(net.win_w) && py >= 0 &&
              py < static_cast<int>(net.win_h)) {
            pd = label_at(pl, px, py);
          }
          // the side cells of diagonal h are the neighbours at h - 1 and h + 1
          const uint32_t side_a = __shfl_sync(0xFFFFFFFFu, pd, (lane + 7) & 7);
          const uint32_t side_b = __shfl_sync(0xFFFFFFFFu, pd, (lane + 1) & 7);
          const bool diagonal = lane < 8 && (lane & 1);
          const uint32_t move = lane >= 8 ? via : diagonal ? diag : orth;
          const bool legal = via_legal && (!diagonal || (side_a < kLabelInf && side_b < kLabelInf));
          const bool cand = legal && pd < kLabelInf && pd + move == here;
          const unsigned ballot = __ballot_sync(0xFFFFFFFFu, cand);
          if (ballot == 0u) break;
          const int hsel = __ffs(ballot) - 1;
          cl = __shfl_sync(0xFFFFFFFFu, pl, hsel);
          cx = __shfl_sync(0xFFFFFFFFu, px, hsel);
          cy = __shfl_sync(0xFFFFFFFFu, py, hsel);
          here = __shfl_sync(0xFFFFFFFFu, pd, hsel);
        }
        if (ok) {
          res.path_len = n;
          res.arena_offset = base;
        } else {
          res.completion = APGAR_B200_COMPLETION_REJECTED;
          res.cost = APGAR_B200_UNREACHABLE;
        }
      }
    }
  }
  if (lane == 0) p.results[plan.net] = res;
}

}  // namespace
}  // namespace apgar_b200
