// The sweep's other form (the first is lattice_sweep.cu, which states the frame,
// the row step, the schedule and the path rule): a lane holds its C consecutive
// cells of every layer, G warps of one CTA cover the frame row.  It serves the
// wide rows of few layers.
//
// There a step costs two barriers (the scan's warp sums, the vote), where the
// form with a warp a layer needs a third to exchange labels and to find out
// whether the row changed at all, which a wide row nearly always does; and a
// net has a third to half of the warps, so an SM holds more nets.  With many
// layers the cells of a lane would be few, and with narrow rows most lanes idle:
// those rows are the other form's.
#include <cuda_runtime.h>

#include <cstdint>

#include "lattice_sweep.cuh"

namespace apgar_b200 {
namespace {

// Per-lane view of the guard-padded sweep planes for one net: the two words
// holding the lane's span (frame positions xs-1 .. xs+C) of frame row r on
// layer l sit at base + l*layer_stride + r*row_stride.
struct BitSpan {
  const uint32_t* blocked;
  const uint32_t* via;  // nullptr without a via mask
  size_t layer_stride;
  int row_stride;
  int shift;
  uint32_t valid;  // span positions inside the frame (bit j <-> position xs-1+j)
};

template <int C>
__device__ __forceinline__ BitSpan make_span(const LatticeDeviceView& lat, const Frame& f, int xs) {
  static_assert(C + 2 <= 32, "a lane's span must fit one word");
  BitSpan s;
  const int origin = f.transposed ? f.y0 : f.x0;
  const int limit = (f.transposed ? lat.height : lat.width) - 1;
  const int first_row = f.transposed ? f.x0 : f.y0;
  const int rows_in_plane = f.transposed ? lat.width : lat.height;
  s.row_stride = (f.transposed ? lat.words_t : lat.words) + 2;
  s.layer_stride = static_cast<size_t>(rows_in_plane) * s.row_stride;
  // a lane wholly outside the frame clamps its position; its valid mask is 0
  const int pos = min(origin + xs - 1, limit);
  const int wi = pos >> 5;  // -1 for pos == -1: the leading guard word
  s.shift = pos & 31;
  const size_t base = static_cast<size_t>(first_row) * s.row_stride + 1 + wi;
  s.blocked = (f.transposed ? lat.sweep_cols : lat.sweep_rows) + base;
  const uint32_t* via_plane = f.transposed ? lat.sweep_via_cols : lat.sweep_via_rows;
  s.via = via_plane == nullptr ? nullptr : via_plane + base;
  const int lo = 1 - xs;        // j >= lo  <=> p >= 0
  const int hi = f.K - xs + 1;  // j <  hi  <=> p <  K
  uint32_t valid = 0;
  if (hi > lo) {
    const uint32_t hi_mask = hi >= 32 ? 0xFFFFFFFFu : ((1u << (hi > 0 ? hi : 0)) - 1u);
    const uint32_t lo_mask = lo <= 0 ? 0u : ((1u << lo) - 1u);
    valid = hi_mask & ~lo_mask;
  }
  s.valid = valid & ((1u << (C + 2)) - 1u);
  return s;
}

// Free bits of the lane's span (bit j+1 is the lane's cell j).
__device__ __forceinline__ uint32_t span_free(const BitSpan& s, int l, int r) {
  const uint32_t* w = s.blocked + l * s.layer_stride + static_cast<size_t>(r) * s.row_stride;
  return ~__funnelshift_r(__ldg(w), __ldg(w + 1), s.shift) & s.valid;
}

// Via bits of layer pair (l, l+1) for the span; all ones without a via mask.
__device__ __forceinline__ uint32_t span_via(const BitSpan& s, int l, int r) {
  if (s.via == nullptr) return 0xFFFFFFFFu;
  const uint32_t* w = s.via + l * s.layer_stride + static_cast<size_t>(r) * s.row_stride;
  return __funnelshift_r(__ldg(w), __ldg(w + 1), s.shift);
}

// Per-group shared memory carve-up (shared by the kernel and the host).
struct GroupSmem {
  size_t modified, edges, sums, flags, total;
};

__host__ __device__ inline GroupSmem group_smem(int L, int G, int max_rows) {
  GroupSmem s{};
  size_t off = 0;
  s.modified = off;
  off += (static_cast<size_t>(max_rows) * sizeof(int16_t) + 15) & ~size_t(15);
  s.edges = off;  // [2 buffers][G][L][first, last] of the previous row
  off += 2 * static_cast<size_t>(G) * L * 2 * sizeof(uint32_t);
  s.sums = off;  // [G][L][aE, bE, aW, bW]
  off += static_cast<size_t>(G) * L * 4 * sizeof(uint32_t);
  s.flags = off;  // [2 parities][G]: bit 0 via improved, bit 1 changed, bit 8+l layer l changed
  off += 2 * static_cast<size_t>(G) * sizeof(uint32_t);
  s.total = (off + 15) & ~size_t(15);
  return s;
}

// The net's record and path (one warp).  A function here: in the kernel's body
// the same text made its steps up to 3% longer (1 layer of 1,030 cells: 3.55 and
// 3.67 ms).
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
#include "lattice_sweep_walk.cuh"
}

template <int L, int C, int G>
__global__ void __launch_bounds__(G * 32)
    lattice_sweep_rows_kernel(SweepLaunch p, int max_rows) {
  const int g = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const NetPlan plan = p.plans[blockIdx.x];
  const apgar_b200_lattice_net net = p.nets[plan.net];
  const LatticeDeviceView& lat = p.lat;
  const int xs = (g * 32 + lane) * C;  // frame position of this lane's first cell
  Frame f;
  f.transposed = static_cast<int>(plan.transposed);
  f.R = static_cast<int>(plan.rows);
  f.K = static_cast<int>(plan.width);
  f.pitch = static_cast<int>(plan.pitch);
  f.x0 = static_cast<int>(net.win_x0);
  f.y0 = static_cast<int>(net.win_y0);
  uint32_t* slab = p.dist_pool + plan.dist_offset;
  const size_t layer_stride = static_cast<size_t>(f.R) * f.pitch;
  const BitSpan span = make_span<C>(lat, f, xs);

  extern __shared__ __align__(16) unsigned char smem_raw[];
  const GroupSmem gs = group_smem(L, G, max_rows);
  int16_t* modified = reinterpret_cast<int16_t*>(smem_raw + gs.modified);
  uint32_t* const sh_edges = reinterpret_cast<uint32_t*>(smem_raw + gs.edges);
  constexpr int kEdgeBuf = G * L * 2;  // entries of one edge buffer
  uint32_t* sh_sum = reinterpret_cast<uint32_t*>(smem_raw + gs.sums);
  uint32_t* sh_flags = reinterpret_cast<uint32_t*>(smem_raw + gs.flags);

  const uint32_t orth = p.lat.orth, diag = p.lat.diag, via = p.lat.via;
  const int lsx = static_cast<int>(net.start_x) - f.x0, lsy = static_cast<int>(net.start_y) - f.y0;
  const int lgx = static_cast<int>(net.goal_x) - f.x0, lgy = static_cast<int>(net.goal_y) - f.y0;
  const int s_layer = static_cast<int>(net.start_layer), g_layer = static_cast<int>(net.goal_layer);
  const int sr = f.transposed ? lsx : lsy, sp = f.transposed ? lsy : lsx;

  for (int y = g * 32 + lane; y < f.R; y += G * 32) modified[y] = kNever;
  const bool endpoints_free =
      cell_free(lat, net, s_layer, lsx, lsy) && cell_free(lat, net, g_layer, lgx, lgy);
  // counters live in registers (every warp of a group follows the same
  // control flow; warp 0's copy is reported)
  uint32_t stat_rows = 0, stat_stores = 0, stat_loads = 0;
  bool fault = false;
  __syncthreads();

  uint32_t completion = APGAR_B200_COMPLETION_DISCONNECTED;
  uint32_t sweeps_done = 0;
  if (endpoints_free) {
    {  // initial row: INF except the start cell
#pragma unroll
      for (int l = 0; l < L; ++l) {
        uint32_t v0[C];
#pragma unroll
        for (int j = 0; j < C; ++j) v0[j] = (l == s_layer && xs + j == sp) ? 0u : kLabelInf;
        store_cells<C>(slab + l * layer_stride + static_cast<size_t>(sr) * f.pitch, f.pitch, xs, v0);
      }
      modified[sr] = 0;  // same value from every thread
      stat_stores += L;
    }
    __syncthreads();

    bool converged = false, cancelled = false;
    int parity = 0;
    // The row step reads its predecessor row's warp-edge labels from buffer
    // eb and publishes its own into the other buffer before its last group
    // vote, which therefore also ends the step (no barrier of its own).
    int eb = 0;
    uint32_t prv[L][C], nxt[L][C];
    uint32_t pf[L], nf[L], nvb[L];
    for (uint32_t k = 1; k <= p.max_sweeps; ++k) {
      // The host-mapped flag is read by one thread and broadcast, so every
      // thread of the group takes the same branch.
      uint32_t cancel_now = 0;
      if (g == 0 && lane == 0) cancel_now = (p.cancel != nullptr && *p.cancel != 0u) ? 1u : 0u;
      if (g == 0 && lane == 0) sh_flags[parity * G] = cancel_now;
      __syncthreads();
      cancel_now = sh_flags[parity * G];
      __syncthreads();
      if (cancel_now != 0u) {
        cancelled = true;
        break;
      }
      sweeps_done = k;
      const bool fwd = (k & 1u) != 0;
      const int dr = fwd ? 1 : -1;
      const int ki = static_cast<int>(k);
      bool any_change = false;
      bool have_prev = false;
      bool have_next = false;  // nxt/nf/nvb hold this step's row
      bool next_loaded = false;
      for (int step = 0; step < f.R; ++step) {
        const int r = fwd ? step : f.R - 1 - step;
        const int pr = r - dr;
        const int16_t mp = (pr >= 0 && pr < f.R) ? modified[pr] : kNever;
        const int16_t my = modified[r];
        const bool skip = (ki <= 2) ? (mp == kNever && my == kNever)
                                    : (mp <= ki - 2 && my <= ki - 2);
        if (skip) {
          have_prev = false;
          have_next = false;
          continue;
        }
        // ---- previous row (registers, or reloaded after a skipped row) ----
        if (!have_prev) {
#pragma unroll
          for (int l = 0; l < L; ++l) {
            if (mp != kNever) {
              load_cells<C>(slab + l * layer_stride + static_cast<size_t>(pr) * f.pitch, f.pitch,
                            xs, prv[l]);
              pf[l] = span_free(span, l, pr);
            } else {
#pragma unroll
              for (int j = 0; j < C; ++j) prv[l][j] = kLabelInf;
              pf[l] = 0;
            }
          }
          if (mp != kNever) stat_loads += L;
          if (lane == 0 || lane == 31) {
#pragma unroll
            for (int l = 0; l < L; ++l) {
              sh_edges[eb * kEdgeBuf + (g * L + l) * 2 + (lane == 0 ? 0 : 1)] =
                  lane == 0 ? prv[l][0] : prv[l][C - 1];
            }
          }
          __syncthreads();
        }
        // ---- current row ----
        uint32_t v[L][C];
        uint32_t cf[L], vb[L];
        if (have_next) {
#pragma unroll
          for (int l = 0; l < L; ++l) {
#pragma unroll
            for (int j = 0; j < C; ++j) v[l][j] = next_loaded ? nxt[l][j] : kLabelInf;
            cf[l] = nf[l];
            vb[l] = nvb[l];
          }
          if (next_loaded) stat_loads += L;
        } else {
#pragma unroll
          for (int l = 0; l < L; ++l) {
            if (my != kNever) {
              load_cells<C>(slab + l * layer_stride + static_cast<size_t>(r) * f.pitch, f.pitch, xs,
                            v[l]);
            } else {
#pragma unroll
              for (int j = 0; j < C; ++j) v[l][j] = kLabelInf;
            }
            cf[l] = span_free(span, l, r);
            vb[l] = (l + 1 < L) ? span_via(span, l, r) : 0u;
          }
          if (my != kNever) stat_loads += L;
        }
        // ---- prefetch the next row when the schedule guarantees it runs ----
        {
          const int nr = r + dr;
          have_next = false;
          next_loaded = false;
          if (nr >= 0 && nr < f.R) {
            const int16_t mn = modified[nr];
            const bool sure = (ki <= 2) ? (my != kNever || mn != kNever)
                                        : (my >= ki - 1 || mn >= ki - 1);
            if (sure) {
              have_next = true;
              next_loaded = mn != kNever;
#pragma unroll
              for (int l = 0; l < L; ++l) {
                if (next_loaded) {
                  load_cells<C>(slab + l * layer_stride + static_cast<size_t>(nr) * f.pitch,
                                f.pitch, xs, nxt[l]);
                }
                nf[l] = span_free(span, l, nr);
                nvb[l] = (l + 1 < L) ? span_via(span, l, nr) : 0u;
              }
            }
          }
        }
        uint32_t orig[L][C];
        uint32_t blk[L][C];  // 0 where free, INF where blocked
#pragma unroll
        for (int l = 0; l < L; ++l) {
#pragma unroll
          for (int j = 0; j < C; ++j) {
            orig[l][j] = v[l][j];
            blk[l][j] = ((cf[l] >> (j + 1)) & 1u) ? 0u : kLabelInf;
          }
        }
        // ---- 1. relax from the previous row ----
#pragma unroll
        for (int l = 0; l < L; ++l) {
          // diagonal side cells: (p in the previous row, p-1 / p+1 in this row)
          const uint32_t side_l = (pf[l] >> 1) & cf[l];
          const uint32_t side_r = (pf[l] >> 1) & (cf[l] >> 2);
          uint32_t left = __shfl_up_sync(0xFFFFFFFFu, prv[l][C - 1], 1);
          uint32_t right = __shfl_down_sync(0xFFFFFFFFu, prv[l][0], 1);
          const uint32_t* const sh_edge = sh_edges + eb * kEdgeBuf;
          if (lane == 0) left = (g > 0) ? sh_edge[((g - 1) * L + l) * 2 + 1] : kLabelInf;
          if (lane == 31) right = (g + 1 < G) ? sh_edge[((g + 1) * L + l) * 2 + 0] : kLabelInf;
#pragma unroll
          for (int j = 0; j < C; ++j) {
            const uint32_t pl = (j == 0) ? left : prv[l][j - 1];
            const uint32_t prr = (j == C - 1) ? right : prv[l][j + 1];
            const uint32_t cl = ((side_l >> j) & 1u) ? diag : kLabelInf;
            const uint32_t cr = ((side_r >> j) & 1u) ? diag : kLabelInf;
            uint32_t t = __viaddmin_u32(prv[l][j], orth, v[l][j]);
            t = __viaddmin_u32(pl, cl, t);
            t = __viaddmin_u32(prr, cr, t);
            v[l][j] = max(t, blk[l][j]);
          }
        }
        // Lanes whose whole chunk is free pass a carry straight through; the
        // nearest non-free lane at or below (east scan) / at or above (west
        // scan) bounds the segment a lane's scan value can come from.
        const uint32_t stepC = orth * C;
        const uint32_t below_me = (lane == 31) ? 0xFFFFFFFFu : ((2u << lane) - 1u);
        const uint32_t above_me = ~((1u << lane) - 1u);
        int segE[L], segW[L];
        bool through_below[L], through_above[L];
        uint32_t warp_free[L];
#pragma unroll
        for (int l = 0; l < L; ++l) {
          const uint32_t m = (1u << C) - 1u;
          const uint32_t free_lanes = __ballot_sync(0xFFFFFFFFu, ((cf[l] >> 1) & m) == m);
          const uint32_t blocked_lanes = ~free_lanes;
          const uint32_t lo = blocked_lanes & below_me;
          const uint32_t hi = blocked_lanes & above_me;
          segE[l] = lo ? 31 - __clz(lo) : 0;
          segW[l] = hi ? __ffs(hi) - 1 : 31;
          through_below[l] = (blocked_lanes & ((1u << lane) - 1u)) == 0u;   // lanes < me all free
          through_above[l] = (blocked_lanes & ~below_me) == 0u;             // lanes > me all free
          warp_free[l] = free_lanes;
        }
        // via hop costs of the row (INF where the via bit forbids the hop)
        uint32_t hopc[L > 1 ? L - 1 : 1][C];
#pragma unroll
        for (int l = 0; l + 1 < L; ++l) {
#pragma unroll
          for (int j = 0; j < C; ++j) hopc[l][j] = ((vb[l] >> (j + 1)) & 1u) ? via : kLabelInf;
        }
        // via cascade inside the lane: upwards then downwards through
        // consecutive legal vias (blocked cells clamp the cascade); returns
        // whether any label changed
        auto via_cascade = [&]() -> uint32_t {
          uint32_t diff = 0;
          if constexpr (L > 1) {
#pragma unroll
            for (int j = 0; j < C; ++j) {
              uint32_t d = v[0][j];
#pragma unroll
              for (int l = 1; l < L; ++l) {
                const uint32_t t = max(__viaddmin_u32(d, hopc[l - 1][j], v[l][j]), blk[l][j]);
                diff |= t ^ v[l][j];
                v[l][j] = t;
                d = t;
              }
#pragma unroll
              for (int l = L - 2; l >= 0; --l) {
                const uint32_t t = max(__viaddmin_u32(d, hopc[l][j], v[l][j]), blk[l][j]);
                diff |= t ^ v[l][j];
                v[l][j] = t;
                d = t;
              }
            }
          }
          return diff;
        };
        // a path that switches layer as it arrives needs no second pass
        via_cascade();
        // ---- 2./3. row-local fixed point ----
        // Each pass lowers at least one label, so the loop is finite; the cap
        // only guards against a broken invariant (reported, never silent).
        uint32_t row_flags = 0;  // group-wide: bit 1 changed, bit 8+l layer l changed
        for (int pass = 0;; ++pass) {
          if (pass == kMaxRowPasses) {
            fault = true;
            break;
          }
          uint32_t inclE[L], inclW[L];
#pragma unroll
          for (int l = 0; l < L; ++l) {
            // lane-local one-sided scans: value at the far cell with no carry
            uint32_t ce = v[l][0];
#pragma unroll
            for (int j = 1; j < C; ++j) ce = max(__viaddmin_u32(ce, orth, v[l][j]), blk[l][j]);
            uint32_t cw = v[l][C - 1];
#pragma unroll
            for (int j = C - 2; j >= 0; --j) cw = max(__viaddmin_u32(cw, orth, v[l][j]), blk[l][j]);
            // segmented min scans over lanes of lane-offset values: a chunk's
            // far-cell value reaches lane i through free chunks at C*orth each
            inclE[l] = ce + static_cast<uint32_t>(31 - lane) * stepC;
            inclW[l] = cw + static_cast<uint32_t>(lane) * stepC;
          }
#pragma unroll
          for (int sft = 1; sft < 32; sft <<= 1) {
#pragma unroll
            for (int l = 0; l < L; ++l) {
              const uint32_t oE = __shfl_up_sync(0xFFFFFFFFu, inclE[l], sft);
              const uint32_t oW = __shfl_down_sync(0xFFFFFFFFu, inclW[l], sft);
              if (lane - sft >= segE[l]) inclE[l] = min(inclE[l], oE);
              if (lane + sft <= segW[l]) inclW[l] = min(inclW[l], oW);
            }
          }
#pragma unroll
          for (int l = 0; l < L; ++l) {
            inclE[l] = min(inclE[l] - static_cast<uint32_t>(31 - lane) * stepC, kLabelInf);
            inclW[l] = min(inclW[l] - static_cast<uint32_t>(lane) * stepC, kLabelInf);
          }
          uint32_t warp_cE[L], warp_cW[L];
#pragma unroll
          for (int l = 0; l < L; ++l) warp_cE[l] = warp_cW[l] = kLabelInf;
          // warp summaries: far-cell value without outside carry, and the
          // cost to cross the whole warp (INF unless every chunk is free)
          if (lane == 31) {
#pragma unroll
            for (int l = 0; l < L; ++l) sh_sum[(g * L + l) * 4 + 0] = inclE[l];
          }
          if (lane == 0) {
#pragma unroll
            for (int l = 0; l < L; ++l) {
              sh_sum[(g * L + l) * 4 + 1] = warp_free[l] == 0xFFFFFFFFu ? 32u * stepC : kLabelInf;
              sh_sum[(g * L + l) * 4 + 2] = inclW[l];
            }
          }
          __syncthreads();
#pragma unroll
          for (int l = 0; l < L; ++l) {
            for (int q = 0; q < g; ++q) {
              warp_cE[l] = __viaddmin_u32(warp_cE[l], sh_sum[(q * L + l) * 4 + 1],
                                          sh_sum[(q * L + l) * 4 + 0]);
            }
            for (int q = G - 1; q > g; --q) {
              warp_cW[l] = __viaddmin_u32(warp_cW[l], sh_sum[(q * L + l) * 4 + 1],
                                          sh_sum[(q * L + l) * 4 + 2]);
            }
          }
#pragma unroll
          for (int l = 0; l < L; ++l) {
            // carry into the lane: the neighbour lane's far-cell value, or the
            // warp carry when every chunk between is free
            uint32_t carryE = __shfl_up_sync(0xFFFFFFFFu, inclE[l], 1);
            uint32_t carryW = __shfl_down_sync(0xFFFFFFFFu, inclW[l], 1);
            if (lane == 0) carryE = kLabelInf;
            if (lane == 31) carryW = kLabelInf;
            if (through_below[l]) carryE = __viaddmin_u32(warp_cE[l], static_cast<uint32_t>(lane) * stepC, carryE);
            if (through_above[l]) carryW = __viaddmin_u32(warp_cW[l], static_cast<uint32_t>(31 - lane) * stepC, carryW);
            uint32_t e[C];
#pragma unroll
            for (int j = 0; j < C; ++j) {
              carryE = max(__viaddmin_u32(carryE, orth, v[l][j]), blk[l][j]);
              e[j] = carryE;
            }
#pragma unroll
            for (int j = C - 1; j >= 0; --j) {
              carryW = max(__viaddmin_u32(carryW, orth, v[l][j]), blk[l][j]);
              v[l][j] = min(e[j], carryW);
            }
          }
          const uint32_t via_diff = via_cascade();
          // group vote: did a via lower a label (another pass needed), and
          // which layers changed since the row was loaded
          uint32_t lane_flags = via_diff != 0u ? 1u : 0u;
#pragma unroll
          for (int l = 0; l < L; ++l) {
            uint32_t diff = 0;
#pragma unroll
            for (int j = 0; j < C; ++j) diff |= v[l][j] ^ orig[l][j];
            if (diff != 0u) lane_flags |= 2u | (1u << (8 + l));
          }
          uint32_t warp_flags = __reduce_or_sync(0xFFFFFFFFu, lane_flags);
          // this pass's row edges for the next step (final if the vote ends
          // the row): buffer eb ^ 1 is read by no warp until the next step,
          // and every read of it by the previous step came before this
          // step's first barrier
          if (lane == 0 || lane == 31) {
#pragma unroll
            for (int l = 0; l < L; ++l) {
              sh_edges[(eb ^ 1) * kEdgeBuf + (g * L + l) * 2 + (lane == 0 ? 0 : 1)] =
                  lane == 0 ? v[l][0] : v[l][C - 1];
            }
          }
          if (lane == 0) sh_flags[parity * G + g] = warp_flags;
          __syncthreads();
          warp_flags = 0;
          for (int q = 0; q < G; ++q) warp_flags |= sh_flags[parity * G + q];
          parity ^= 1;
          row_flags = warp_flags;
          if ((warp_flags & 1u) == 0u || L == 1) break;
        }
        // ---- 4. write-back ----
        if (row_flags & 2u) {
          const bool materialise = (my == kNever);
#pragma unroll
          for (int l = 0; l < L; ++l) {
            if (materialise || (row_flags & (1u << (8 + l)))) {
              store_cells<C>(slab + l * layer_stride + static_cast<size_t>(r) * f.pitch, f.pitch,
                             xs, v[l]);
              ++stat_stores;
            }
          }
          modified[r] = static_cast<int16_t>(k);  // same value from every thread
          any_change = true;
        }
        ++stat_rows;
#pragma unroll
        for (int l = 0; l < L; ++l) {
#pragma unroll
          for (int j = 0; j < C; ++j) prv[l][j] = v[l][j];
          pf[l] = cf[l];
        }
        have_prev = true;
        eb ^= 1;
        // The step's last vote barrier published the edges; every thread
        // wrote modified[r] itself (the same value) and reads only its own
        // lane's cells of the slab.  A faulted row left the pass loop before
        // its vote, so it ends with a barrier of its own.
        if (fault) __syncthreads();
      }
      if (!any_change && k >= 2) {
        converged = true;
        break;
      }
    }
    __syncthreads();
    if (fault) {
      completion = APGAR_B200_COMPLETION_REJECTED;
    } else if (cancelled) {
      completion = APGAR_B200_COMPLETION_CANCELLED;
    } else if (!converged) {
      completion = APGAR_B200_COMPLETION_BUDGET_EXHAUSTED;
    } else {
      completion = APGAR_B200_COMPLETION_REACHED;  // refined below from the goal label
    }
  }

  // ----------------------------- result + walk -----------------------------
  if (g != 0) return;
  write_sweep_result(p, plan, f, net, slab, static_cast<uint32_t>(layer_stride), modified, completion, sweeps_done,
                     stat_rows, stat_stores, stat_loads, lane);
}

template <int L, int C, int G>
cudaError_t launch_one(const SweepLaunch& launch, int max_rows, cudaStream_t stream) {
  const size_t smem = group_smem(L, G, max_rows).total;
  cudaError_t e = cudaFuncSetAttribute(lattice_sweep_rows_kernel<L, C, G>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
  if (e != cudaSuccess) return e;
  lattice_sweep_rows_kernel<L, C, G><<<launch.plan_count, G * 32, smem, stream>>>(launch, max_rows);
  return cudaGetLastError();
}

template <int L, int C, int kFewest, int G = 16>
cudaError_t launch_warps(int warps, const SweepLaunch& launch, int max_rows, cudaStream_t stream) {
  if constexpr (G < kFewest) {
    return cudaErrorInvalidValue;
  } else {
    return warps == G ? launch_one<L, C, G>(launch, max_rows, stream)
                      : launch_warps<L, C, kFewest, G - 1>(warps, launch, max_rows, stream);
  }
}

}  // namespace

size_t sweep_rows_smem_bytes(int layers, int warps, int max_rows) { return group_smem(layers, warps, max_rows).total; }

// Every number of warps: a net takes the fewest that cover its row.
cudaError_t launch_sweep_rows(int layers, int warps, const SweepLaunch& launch, int max_rows, cudaStream_t stream) {
  switch (layers) {
    case 1: return launch_warps<1, 16, 3>(warps, launch, max_rows, stream);
    case 2: return launch_warps<2, 8, 3>(warps, launch, max_rows, stream);
    case 4: return launch_warps<4, 4, 13>(warps, launch, max_rows, stream);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace apgar_b200
