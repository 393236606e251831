// Lattice-mode batched search: exact single-source labels over each net's
// window by alternating forward/backward row sweeps, then the canonical
// reverse path.
//
// Frame: a net is swept along its window's shorter side.  Frame rows are
// lattice rows, or lattice columns when the window is taller than wide (the
// column-major bit planes uploaded with the lattice serve that case); the
// move model is symmetric under the swap.
//
// Work split: a net is a CTA, a warp holds one layer of 32 * C consecutive
// cells of the frame row (C labels per lane in registers), and G warps side by
// side cover the row on each of the L layers.  The sweep of one net is a chain
// of dependent row steps and a batch ends with its longest chains, so what
// counts is the latency of a step: up to 512 cells the warps' instructions one
// after the other, beyond that the integer throughput of the net's one SM.  Two
// things keep instructions out of a step: a row that the relaxation leaves
// alone ends there, and a warp whose labels nothing changed skips its scan and
// its via cascade.  With all layers of a chunk in one warp a warp had 4 x C
// cells to go through and no way to skip any: 1,024 nets of 4 x 1024^2, median
// row 162 cells, took 11.1 ms, 8.6 now; 96 planar nets, where the gain is
// fewer cells a lane and the rows that end early, 0.89 ms and 0.56.  Where that
// other form is the better one, wide rows of few layers keep it
// (lattice_sweep_rows.cu).
//
// A row step:
//   1. relaxes the row from the previous row in sweep order (straight plus
//      both diagonals; the previous row stays in registers between steps) and
//      applies the via cascade across layers;
//   2. runs, for every layer, a two-sided row scan: the east and west
//      one-sided scans of the same input combined by min (equal to an east
//      scan followed by a west scan on every connected segment).  Each is a
//      lane-serial add-min chain, a 5-step warp shuffle scan of lane summaries
//      and a fold over the row's preceding warps;
//   3. applies the via cascade again and repeats 2-3 until no via lowers a
//      label.  The layers meet in shared memory: every warp publishes its
//      labels, and each lane folds the column of its cells from the lowest
//      layer up and from the highest down to its own;
//   4. writes back only the layers whose labels changed.
// Blocked cells hold INF and a move into one costs INF, so orthogonal moves
// need no legality test; diagonal moves test their two side cells.  The next
// row's labels and mask bits are loaded while the current row is processed.
//
// Schedule (restated on the CPU by the oracle, lo_sweep_schedule): a row is
// skipped when neither it nor its predecessor row changed since the previous
// sweep in the same direction (first sweep per direction: when both are still
// all-INF); a sweep that changes nothing, after one sweep in each direction,
// proves the labels are the exact shortest-path fixed point.  Rows that never
// held a finite label are never read or written.
//
// Canonical path (reference gpu/cuda/planar_router.cu :977-1009 goal state,
// :1084-1165 reverse walk) on exact labels: from the goal, step to the
// predecessor through the smallest legal incoming heading whose label plus
// move cost equals the current label.  Headings 0..7 are the planar
// directions (geometry_compiler::Direction order), 8 = via from the layer
// below, 9 = via from the layer above.
#include <cuda_runtime.h>

#include <cstdint>

#include "lattice_sweep.cuh"

namespace apgar_b200 {

size_t sweep_rows_smem_bytes(int layers, int warps, int max_rows);
cudaError_t launch_sweep_rows(int layers, int warps, const SweepLaunch& launch, int max_rows, cudaStream_t stream);

namespace {

// Per-lane view of one layer's guard-padded sweep planes for one net: the two
// words holding the lane's span (frame positions xs-1 .. xs+C) of frame row r
// sit at base + r*row_stride.
struct BitSpan {
  const uint32_t* blocked;
  const uint32_t* via;  // nullptr without a via mask; layer pair (layer, layer + 1)
  uint32_t row_stride;
  int shift;
  uint32_t valid;  // span positions inside the frame (bit j <-> position xs-1+j)
};

template <int C>
__device__ __forceinline__ BitSpan make_span(const LatticeDeviceView& lat, const Frame& f, int xs, int layer) {
  static_assert(C + 2 <= 32, "a lane's span must fit one word");
  BitSpan s;
  const int origin = f.transposed ? f.y0 : f.x0;
  const int limit = (f.transposed ? lat.height : lat.width) - 1;
  const int first_row = f.transposed ? f.x0 : f.y0;
  const int rows_in_plane = f.transposed ? lat.width : lat.height;
  s.row_stride = (f.transposed ? lat.words_t : lat.words) + 2;
  // a lane wholly outside the frame clamps its position; its valid mask is 0
  const int pos = min(origin + xs - 1, limit);
  const int wi = pos >> 5;  // -1 for pos == -1: the leading guard word
  s.shift = pos & 31;
  const size_t base =
      (static_cast<size_t>(layer) * rows_in_plane + static_cast<size_t>(first_row)) * s.row_stride + 1 + wi;
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

// The two words of a plane that hold the lane's span of frame row r.  They are
// kept as loaded until the row is processed, so that nothing waits for a
// prefetch when it is issued.
__device__ __forceinline__ uint2 span_words(const BitSpan& s, const uint32_t* plane, int r) {
  const uint32_t* w = plane + static_cast<uint32_t>(r) * s.row_stride;
  return make_uint2(__ldg(w), __ldg(w + 1));
}

// Free bits of the lane's span (bit j+1 is the lane's cell j).
__device__ __forceinline__ uint32_t span_free(const BitSpan& s, uint2 w) {
  return ~__funnelshift_r(w.x, w.y, s.shift) & s.valid;
}

// 0 where bit j is set, INF where it is clear.
__device__ __forceinline__ uint32_t inf_unless(uint32_t bits, int j) {
  return ((bits >> j) & 1u) ? 0u : kLabelInf;
}

// Shuffles that stop at a lane of the caller's choice: a lane whose source
// lies beyond `stop` gets its own value back.
__device__ __forceinline__ uint32_t shfl_up_to(uint32_t v, int by, int stop) {
  uint32_t d;
  asm volatile("shfl.sync.up.b32 %0, %1, %2, %3, 0xFFFFFFFF;" : "=r"(d) : "r"(v), "r"(by), "r"(stop));
  return d;
}
__device__ __forceinline__ uint32_t shfl_down_to(uint32_t v, int by, int stop) {
  uint32_t d;
  asm volatile("shfl.sync.down.b32 %0, %1, %2, %3, 0xFFFFFFFF;" : "=r"(d) : "r"(v), "r"(by), "r"(stop));
  return d;
}

// Shared memory of a CTA (shared by the kernel and the host).
struct SweepSmem {
  size_t modified, labels, bits, edges, sums, flags, total;
};

__host__ __device__ inline SweepSmem sweep_smem(int L, int C, int G, int max_rows) {
  SweepSmem s{};
  size_t off = 0;
  s.modified = off;
  off += (static_cast<size_t>(max_rows) * sizeof(int16_t) + 15) & ~size_t(15);
  s.labels = off;  // [2][L][G][C / 4][32 lanes] uint4: the exchanged labels
  if (L > 1) off += 2 * static_cast<size_t>(L) * G * 32 * C * sizeof(uint32_t);
  s.bits = off;  // [L][G][32 lanes]: free cells, and via bits to the layer above << 16
  if (L > 1) off += static_cast<size_t>(L) * G * 32 * sizeof(uint32_t);
  s.edges = off;  // [2 buffers][L][G][first, last] of the previous row
  off += 2 * static_cast<size_t>(L) * G * 2 * sizeof(uint32_t);
  off = (off + 15) & ~size_t(15);
  s.sums = off;  // [L][G]: east far-cell value, crossing cost, west far-cell value
  off += static_cast<size_t>(L) * G * sizeof(uint4);
  s.flags = off;  // [2 parities][L * G]: bit l: layer l changed
  off += 2 * static_cast<size_t>(L) * G * sizeof(uint32_t);
  s.total = (off + 15) & ~size_t(15);
  return s;
}

// All warps of the net (a barrier of the whole CTA; kOne: its only warp).
template <bool kOne>
__device__ __forceinline__ void net_sync() {
  if constexpr (kOne) {
    __syncwarp();
  } else {
    __syncthreads();
  }
}

// G = p.row_warps <= kMost warps side by side; an SM holds kNets nets or more.
template <int L, int C, int kMost, int kNets>
__global__ void __launch_bounds__(32 * L * kMost, kNets)
    lattice_sweep_kernel(SweepLaunch p, int max_rows) {
  constexpr bool kMulti = kMost > 1;
  constexpr bool kOne = L == 1 && !kMulti;  // the CTA is one warp
  const uint32_t plan_index = blockIdx.x;
  const int G = kMulti ? p.row_warps : 1;
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int my_layer = L > 1 ? warp / G : 0;
  const int g = warp - my_layer * G;  // warp within the row
  const NetPlan plan = p.plans[plan_index];
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
  // a window's labels are fewer than 2^31: 32-bit offsets into its slab
  const uint32_t layer_stride = static_cast<uint32_t>(f.R) * static_cast<uint32_t>(f.pitch);
  uint32_t* const my_slab = slab + static_cast<uint32_t>(my_layer) * layer_stride;
  const auto row_at = [&](int r) { return my_slab + static_cast<uint32_t>(r) * static_cast<uint32_t>(f.pitch); };
  const BitSpan span = make_span<C>(lat, f, xs, my_layer);
  const bool via_words = L > 1 && span.via != nullptr && my_layer + 1 < L;

  extern __shared__ __align__(16) unsigned char smem_raw[];
  const SweepSmem gs = sweep_smem(L, C, G, max_rows);
  int16_t* modified = reinterpret_cast<int16_t*>(smem_raw + gs.modified);
  uint4* const sh_labels = reinterpret_cast<uint4*>(smem_raw + gs.labels);
  uint32_t* const sh_bits = reinterpret_cast<uint32_t*>(smem_raw + gs.bits);
  uint32_t* const sh_edges = reinterpret_cast<uint32_t*>(smem_raw + gs.edges);
  uint4* const sh_sum = reinterpret_cast<uint4*>(smem_raw + gs.sums) + my_layer * G;
  uint32_t* const sh_flags = reinterpret_cast<uint32_t*>(smem_raw + gs.flags);
  const int warps = L * G;
  const int edge_buf = warps * 2;                  // entries of one edge buffer
  const int layer_quads = G * (C / 4) * 32;        // uint4 of one layer of exchanged labels
  const int my_quads = g * (C / 4) * 32 + lane;    // this lane's first quad within a layer

  const uint32_t orth = p.lat.orth, diag = p.lat.diag, via = p.lat.via;
  const int lsx = static_cast<int>(net.start_x) - f.x0, lsy = static_cast<int>(net.start_y) - f.y0;
  const int lgx = static_cast<int>(net.goal_x) - f.x0, lgy = static_cast<int>(net.goal_y) - f.y0;
  const int s_layer = static_cast<int>(net.start_layer), g_layer = static_cast<int>(net.goal_layer);
  const int sr = f.transposed ? lsx : lsy, sp = f.transposed ? lsy : lsx;

  for (int y = threadIdx.x; y < f.R; y += blockDim.x) modified[y] = kNever;
  const bool endpoints_free =
      cell_free(lat, net, s_layer, lsx, lsy) && cell_free(lat, net, g_layer, lgx, lgy);
  // counters live in registers (every warp of a net follows the same control
  // flow; warp 0's copy is reported)
  uint32_t stat_rows = 0, stat_stores = 0, stat_loads = 0;
  bool fault = false;
  net_sync<kOne>();

  uint32_t completion = APGAR_B200_COMPLETION_DISCONNECTED;
  uint32_t sweeps_done = 0;
  if (endpoints_free) {
    {  // initial row: INF except the start cell
      uint32_t v0[C];
#pragma unroll
      for (int j = 0; j < C; ++j) v0[j] = (my_layer == s_layer && xs + j == sp) ? 0u : kLabelInf;
      store_cells<C>(row_at(sr), f.pitch, xs, v0);
      modified[sr] = 0;  // same value from every thread
      stat_stores += L;
    }
    net_sync<kOne>();

    bool converged = false, cancelled = false;
    int parity = 0;
    int xb = 0;  // exchange buffer
    // The row step reads its predecessor row's warp-edge labels from buffer
    // eb and publishes its own into the other buffer before its last vote,
    // which therefore also ends the step (no barrier of its own).
    int eb = 0;
    uint32_t prv[C], nxt[C];
    uint32_t pf = 0;    // free bits of the previous row
    uint2 nf{}, nvb{};  // the next row's plane words, as loaded
    // The carries of the row scan: what a crossing of C cells costs, and of
    // the chunks to the warp's last and first lane.
    const uint32_t stepC = orth * C;
    const uint32_t to_last = static_cast<uint32_t>(31 - lane) * stepC;
    const uint32_t to_first = static_cast<uint32_t>(lane) * stepC;
    for (uint32_t k = 1; k <= p.max_sweeps; ++k) {
      // The host-mapped flag is read by one thread and broadcast, so every
      // thread of the net takes the same branch.
      int cancel_now = 0;
      if (threadIdx.x == 0) cancel_now = (p.cancel != nullptr && *p.cancel != 0u) ? 1 : 0;
      if constexpr (kOne) {
        cancel_now = __shfl_sync(0xFFFFFFFFu, cancel_now, 0);
      } else {
        cancel_now = __syncthreads_or(cancel_now);
      }
      if (cancel_now != 0) {
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
      int16_t mp = kNever, my = kNever, mn = modified[fwd ? 0 : f.R - 1];  // of rows r - dr, r, r + dr
      for (int step = 0; step < f.R; ++step) {
        const int r = fwd ? step : f.R - 1 - step;
        const int pr = r - dr, nr = r + dr;
        mp = my;
        my = mn;
        mn = (step + 1 < f.R) ? modified[nr] : kNever;
        const bool skip = (ki <= 2) ? (mp == kNever && my == kNever)
                                    : (mp <= ki - 2 && my <= ki - 2);
        if (skip) {
          have_prev = false;
          have_next = false;
          continue;
        }
        // ---- previous row (registers, or reloaded after a skipped row) ----
        if (!have_prev) {
          if (mp != kNever) {
            load_cells<C>(row_at(pr), f.pitch, xs, prv);
            pf = span_free(span, span_words(span, span.blocked, pr));
            stat_loads += L;
          } else {
#pragma unroll
            for (int j = 0; j < C; ++j) prv[j] = kLabelInf;
            pf = 0;
          }
          if constexpr (kMulti) {
            if (lane == 0) sh_edges[eb * edge_buf + warp * 2] = prv[0];
            if (lane == 31) sh_edges[eb * edge_buf + warp * 2 + 1] = prv[C - 1];
            net_sync<kOne>();
          }
        }
        // ---- current row ----
        uint32_t v[C];
        uint2 cw, vw;
        if (have_next) {
#pragma unroll
          for (int j = 0; j < C; ++j) v[j] = my != kNever ? nxt[j] : kLabelInf;
          cw = nf;
          vw = nvb;
        } else {
          if (my != kNever) {
            load_cells<C>(row_at(r), f.pitch, xs, v);
          } else {
#pragma unroll
            for (int j = 0; j < C; ++j) v[j] = kLabelInf;
          }
          cw = span_words(span, span.blocked, r);
          vw = via_words ? span_words(span, span.via, r) : make_uint2(0xFFFFFFFFu, 0xFFFFFFFFu);
        }
        if (my != kNever) stat_loads += L;
        // ---- prefetch the next row: it runs if this one changes, which the
        // step learns only after the loads would be due (waiting for that
        // left one step in four with its loads exposed)
        have_next = step + 1 < f.R;
        if (have_next) {
          if (mn != kNever) load_cells<C>(row_at(nr), f.pitch, xs, nxt);
          nf = span_words(span, span.blocked, nr);
          nvb = via_words ? span_words(span, span.via, nr) : make_uint2(0xFFFFFFFFu, 0xFFFFFFFFu);
        }
        const uint32_t cf = span_free(span, cw);
        uint32_t diff = 0;     // labels that changed since the row was loaded
        uint32_t into[C];      // cost of a straight move into the cell: INF where blocked
        // ---- 1. relax from the previous row ----
        {
          // A diagonal step from (p -+ 1) of the previous row needs two free
          // side cells: the one below its source (this row), and the one
          // above its target (previous row).
          uint32_t src[C], slant[C];
#pragma unroll
          for (int j = 0; j < C; ++j) {
            const bool open = (cf >> (j + 1)) & 1u;
            into[j] = open ? orth : kLabelInf;
            slant[j] = open ? diag : kLabelInf;
            src[j] = open ? prv[j] : kLabelInf;
          }
          uint32_t left = __shfl_up_sync(0xFFFFFFFFu, src[C - 1], 1);
          uint32_t right = __shfl_down_sync(0xFFFFFFFFu, src[0], 1);
          if (lane == 0) {
            left = kLabelInf;
            if (kMulti && g > 0 && (cf & 1u)) left = sh_edges[eb * edge_buf + (warp - 1) * 2 + 1];
          }
          if (lane == 31) {
            right = kLabelInf;
            if (kMulti && g + 1 < G && ((cf >> (C + 1)) & 1u)) right = sh_edges[eb * edge_buf + (warp + 1) * 2];
          }
          uint32_t across[C];
#pragma unroll
          for (int j = 0; j < C; ++j) {
            across[j] = min(j == 0 ? left : src[j - 1], j == C - 1 ? right : src[j + 1]);
          }
          if (diag >= orth) {
            // The previous row is at its fixed point: a free cell there is at
            // most one straight move above its neighbours, and one that holds
            // INF (blocked, or as unreached as they are) leaves at least INF.
#pragma unroll
            for (int j = 0; j < C; ++j) {
              across[j] = static_cast<uint32_t>(__viaddmax_s32(
                  static_cast<int>(prv[j]), -static_cast<int>(orth), static_cast<int>(across[j])));
            }
          } else {
#pragma unroll
            for (int j = 0; j < C; ++j) across[j] = max(across[j], inf_unless(pf, j + 1));
          }
#pragma unroll
          for (int j = 0; j < C; ++j) {
            const uint32_t t = __viaddmin_u32(across[j], slant[j], __viaddmin_u32(prv[j], into[j], v[j]));
            diff |= t ^ v[j];
            v[j] = t;
          }
        }
        // Lanes whose whole chunk is free pass a carry straight through; the
        // nearest non-free lane at or below (east scan) / at or above (west
        // scan) bounds the segment a lane's scan value can come from.
        constexpr uint32_t kChunk = (1u << C) - 1u;
        const uint32_t free_lanes = __ballot_sync(0xFFFFFFFFu, ((cf >> 1) & kChunk) == kChunk);
        const uint32_t below_me = (lane == 31) ? 0xFFFFFFFFu : ((2u << lane) - 1u);
        const uint32_t lo = ~free_lanes & below_me, hi = ~free_lanes & ~((1u << lane) - 1u);
        const int segE = lo ? 31 - __clz(lo) : 0;
        const int segW = hi ? __ffs(hi) - 1 : 31;
        const bool through_below = (~free_lanes & ((1u << lane) - 1u)) == 0u;  // lanes < me all free
        const bool through_above = (~free_lanes & ~below_me) == 0u;            // lanes > me all free
        // Legal via hops of the lane's cells between layers q and q + 1,
        // known after the row's first exchange.
        uint32_t hop[L > 1 ? L - 1 : 1];
        if constexpr (L > 1) {
          const uint32_t vb = __funnelshift_r(vw.x, vw.y, span.shift);
          sh_bits[warp * 32 + lane] = ((cf >> 1) & kChunk) | ((vb >> 1) << 16);
        }
        // Via cascade: upwards then downwards through consecutive legal vias,
        // to this warp's layer; returns the bits that changed.
        // Only what layers `lo` .. `hi` changed can lower a label.
        const auto via_cascade = [&](const uint4* x, int lo, int hi) -> uint32_t {
          uint32_t changed = 0;
#pragma unroll
          for (int q = 0; q < C / 4; ++q) {
            uint32_t up[4], down[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) up[i] = down[i] = kLabelInf;
#pragma unroll
            for (int l = 0; l + 1 < L; ++l) {
              if (l >= lo && l < my_layer) {  // warp-uniform
                const uint4 t = x[l * layer_quads + q * 32];
                const uint32_t c[4] = {t.x, t.y, t.z, t.w};
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                  up[i] = __viaddmin_u32(min(up[i], c[i]), (hop[l] >> (4 * q + i)) & 1u ? via : kLabelInf, kLabelInf);
                }
              }
            }
#pragma unroll
            for (int l = L - 1; l > 0; --l) {
              if (l <= hi && l > my_layer) {
                const uint4 t = x[l * layer_quads + q * 32];
                const uint32_t c[4] = {t.x, t.y, t.z, t.w};
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                  down[i] =
                      __viaddmin_u32(min(down[i], c[i]), (hop[l - 1] >> (4 * q + i)) & 1u ? via : kLabelInf, kLabelInf);
                }
              }
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const uint32_t t = __vimin3_u32(up[i], down[i], v[4 * q + i]);
              changed |= t ^ v[4 * q + i];
              v[4 * q + i] = t;
            }
          }
          return changed;
        };
        // Publishes this warp's labels (L > 1) and meets the net's other
        // warps: whether any of them reports `changed`; the labels to read.
        const uint4* x = nullptr;
        const auto exchange = [&](bool changed) -> bool {
          if constexpr (kOne) {
            return __any_sync(0xFFFFFFFFu, changed);
          } else {
            if constexpr (L > 1) {
              uint4* const out = sh_labels + xb * (L * layer_quads) + my_quads;
#pragma unroll
              for (int q = 0; q < C / 4; ++q) {
                out[my_layer * layer_quads + q * 32] = make_uint4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
              }
              x = out;
              xb ^= 1;
            }
            return __syncthreads_or(changed) != 0;
          }
        };
        // The votes of a row: did a label change since the row was loaded (bit
        // l for layer l, for the write-back) and since the last exchange (bit
        // 8), and this row's edges for the next step.  Buffer eb ^ 1 is read by
        // no warp until the next step, and every read of it by the previous
        // step came before this step's first barrier.
        const auto publish_flags = [&](bool recent) {
          if constexpr (kMulti) {
            if (lane == 0) sh_edges[(eb ^ 1) * edge_buf + warp * 2] = v[0];
            if (lane == 31) sh_edges[(eb ^ 1) * edge_buf + warp * 2 + 1] = v[C - 1];
          }
          if constexpr (!kOne) {
            const uint32_t flags = __reduce_or_sync(
                0xFFFFFFFFu, (diff != 0u ? 1u << my_layer : 0u) | (recent ? 1u << 8 : 0u));
            if (lane == 0) sh_flags[parity * warps + warp] = flags;
          }
        };
        // The layers of this warp's cells that changed before the last
        // exchange (bit l); no via can lower a label unless another's did.
        const auto changed_layers = [&]() -> uint32_t {
          return __ballot_sync(0xFFFFFFFFu, lane < L && (sh_flags[parity * warps + lane * G + g] & (1u << 8)));
        };
        uint32_t row_layers = 0;  // layers that changed
        // A row that the relaxation does not lower is at its fixed point
        // already (the start's row is not until it has run): nearly half of
        // the steps end here.
        bool dirty = diff != 0u || my == 0;  // this warp's labels are not as a scan left them
        publish_flags(dirty);
        if (exchange(dirty)) {
          dirty = __any_sync(0xFFFFFFFFu, dirty);
          if constexpr (L > 1) {
            uint32_t b[L];
#pragma unroll
            for (int l = 0; l < L; ++l) b[l] = sh_bits[(l * G + g) * 32 + lane];
#pragma unroll
            for (int l = 0; l + 1 < L; ++l) hop[l] = b[l] & b[l + 1] & (b[l] >> 16);
            // a path that switches layer as it arrives needs no second pass
            const uint32_t from = changed_layers();
            if (from & ~(1u << my_layer)) {
              const uint32_t lowered = via_cascade(x, __ffs(from) - 1, 31 - __clz(from));
              diff |= lowered;
              dirty = __any_sync(0xFFFFFFFFu, dirty || lowered != 0u);
            }
          }
          // ---- 2./3. row-local fixed point ----
          // Each pass lowers at least one label, so the loop is finite; the
          // cap only guards against a broken invariant (reported, never
          // silent).
          for (int pass = 0;; ++pass) {
            if (pass == kMaxRowPasses) {
              fault = true;
              break;
            }
            // What reaches the chunk from outside, and the far cells' values.
            // A chunk that is as a scan left it has nothing to scan: its
            // labels are the far-cell values, and only a carry from another
            // warp can lower them.
            uint32_t inclE = v[C - 1], inclW = v[0];
            uint32_t carryE = kLabelInf, carryW = kLabelInf;
            if (dirty) {
              // lane-local one-sided scans: value at the far cell with no carry
              inclE = v[0];
              inclW = v[C - 1];
#pragma unroll
              for (int j = 1; j < C; ++j) {
                inclE = __viaddmin_u32(inclE, into[j], v[j]);
                inclW = __viaddmin_u32(inclW, into[C - 1 - j], v[C - 1 - j]);
              }
              // segmented min scans over lanes of lane-offset values: a chunk's
              // far-cell value reaches lane i through free chunks at C*orth each
              inclE += to_last;
              inclW += to_first;
#pragma unroll
              for (int sft = 1; sft < 32; sft <<= 1) {
                inclE = min(inclE, shfl_up_to(inclE, sft, segE));
                inclW = min(inclW, shfl_down_to(inclW, sft, segW));
              }
              inclE = min(inclE - to_last, kLabelInf);
              inclW = min(inclW - to_first, kLabelInf);
              // carry into the lane: the neighbour lane's far-cell value, or the
              // warp carry when every chunk between is free
              carryE = __shfl_up_sync(0xFFFFFFFFu, inclE, 1);
              carryW = __shfl_down_sync(0xFFFFFFFFu, inclW, 1);
              if (lane == 0) carryE = kLabelInf;
              if (lane == 31) carryW = kLabelInf;
            }
            bool chain = dirty;
            if constexpr (kMulti) {
              // warp summaries: far-cell value without outside carry, and the
              // cost to cross the whole warp (INF unless every chunk is free)
              if (lane == 31) sh_sum[g].x = inclE;
              if (lane == 0) {
                sh_sum[g].y = free_lanes == 0xFFFFFFFFu ? 32u * stepC : kLabelInf;
                sh_sum[g].z = inclW;
              }
              __syncthreads();
              uint32_t warp_cE = kLabelInf, warp_cW = kLabelInf;
              for (int q = 0; q < g; ++q) {
                const uint4 t = sh_sum[q];
                warp_cE = __viaddmin_u32(warp_cE, t.y, t.x);
              }
              for (int q = G - 1; q > g; --q) {
                const uint4 t = sh_sum[q];
                warp_cW = __viaddmin_u32(warp_cW, t.y, t.z);
              }
              if (through_below) carryE = __viaddmin_u32(warp_cE, to_first, carryE);
              if (through_above) carryW = __viaddmin_u32(warp_cW, to_last, carryW);
              // a carry that lowers any cell lowers the first one it enters
              const bool enters = (lane == 0 && __viaddmin_u32(carryE, into[0], v[0]) != v[0]) ||
                                  (lane == 31 && __viaddmin_u32(carryW, into[C - 1], v[C - 1]) != v[C - 1]);
              chain = __any_sync(0xFFFFFFFFu, enters) || dirty;
            }
            uint32_t scanned = 0;
            if (chain) {
              uint32_t e[C];
#pragma unroll
              for (int j = 0; j < C; ++j) {
                carryE = __viaddmin_u32(carryE, into[j], v[j]);
                e[j] = carryE;
              }
#pragma unroll
              for (int j = C - 1; j >= 0; --j) {
                carryW = __viaddmin_u32(carryW, into[j], v[j]);
                const uint32_t t = min(e[j], carryW);
                scanned |= t ^ v[j];
                v[j] = t;
              }
            }
            diff |= scanned;
            if constexpr (!kOne) {
              parity ^= 1;
              publish_flags(scanned != 0u);
              // vote: labels that no scan lowered are at the cascade's fixed
              // point already
              if (!exchange(scanned != 0u)) break;
            }
            if constexpr (L > 1) {
              const uint32_t from = changed_layers();
              const uint32_t lowered =
                  (from & ~(1u << my_layer)) ? via_cascade(x, __ffs(from) - 1, 31 - __clz(from)) : 0u;
              diff |= lowered;
              dirty = __any_sync(0xFFFFFFFFu, lowered != 0u);
              parity ^= 1;
              publish_flags(false);
              if (__syncthreads_or(lowered != 0u) == 0) break;
            } else {
              break;
            }
          }
          if constexpr (kOne) {
            row_layers = __any_sync(0xFFFFFFFFu, diff != 0u) ? 1u : 0u;
          } else {
            row_layers = __reduce_or_sync(0xFFFFFFFFu, lane < warps ? sh_flags[parity * warps + lane] & 0xFFu : 0u);
          }
        }
        parity ^= 1;
        // ---- 4. write-back ----
        if (row_layers != 0u) {
          const bool materialise = (my == kNever);
          if (materialise || ((row_layers >> my_layer) & 1u)) store_cells<C>(row_at(r), f.pitch, xs, v);
          stat_stores += materialise ? L : __popc(row_layers);
          modified[r] = my = static_cast<int16_t>(k);  // same value from every thread
          any_change = true;
        }
        ++stat_rows;
#pragma unroll
        for (int j = 0; j < C; ++j) prv[j] = v[j];
        pf = cf;
        have_prev = true;
        eb ^= 1;
        // The step's last vote published the edges; every thread
        // wrote modified[r] itself (the same value) and reads only its own
        // lane's cells of the slab.  A faulted row left the pass loop before
        // its vote, so it ends with a barrier of its own.
        if (fault) net_sync<kOne>();
      }
      if (!any_change && k >= 2) {
        converged = true;
        break;
      }
    }
    net_sync<kOne>();
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
  if (warp != 0) return;
#include "lattice_sweep_walk.cuh"
}

// Deterministic packing of the reverse paths in caller net order: one block
// computes exclusive offsets, then every block copies its nets' paths.
__global__ void pack_offsets_kernel(apgar_b200_lattice_result* results, uint32_t count,
                                    unsigned long long* total) {
  __shared__ unsigned long long warp_sums[32];
  __shared__ unsigned long long base;
  if (threadIdx.x == 0) base = 0;
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (uint32_t chunk = 0; chunk < count; chunk += blockDim.x) {
    const uint32_t i = chunk + threadIdx.x;
    const unsigned long long len = i < count ? results[i].path_len : 0ull;
    unsigned long long x = len;
#pragma unroll
    for (int k = 1; k < 32; k <<= 1) {
      const unsigned long long y = __shfl_up_sync(0xFFFFFFFFu, x, k);
      if (lane >= k) x += y;
    }
    if (lane == 31) warp_sums[warp] = x;
    __syncthreads();
    if (warp == 0) {
      unsigned long long s = lane < static_cast<int>(blockDim.x >> 5) ? warp_sums[lane] : 0ull;
#pragma unroll
      for (int k = 1; k < 32; k <<= 1) {
        const unsigned long long y = __shfl_up_sync(0xFFFFFFFFu, s, k);
        if (lane >= k) s += y;
      }
      warp_sums[lane] = s;
    }
    __syncthreads();
    const unsigned long long warp_base = warp == 0 ? 0ull : warp_sums[warp - 1];
    if (i < count) results[i].path_offset = base + warp_base + x - len;
    __syncthreads();
    if (threadIdx.x == 0) base += warp_sums[(blockDim.x >> 5) - 1];
    __syncthreads();
  }
  if (threadIdx.x == 0) *total = base;
}

__global__ void pack_copy_kernel(apgar_b200_lattice_result* results, uint32_t count,
                                 const uint32_t* arena, uint32_t* paths) {
  for (uint32_t i = blockIdx.x; i < count; i += gridDim.x) {
    const apgar_b200_lattice_result r = results[i];
    for (uint32_t j = threadIdx.x; j < r.path_len; j += blockDim.x) {
      paths[r.path_offset + j] = arena[r.arena_offset + j];
    }
    // the staging offset depends on the order nets finished; clear it so the
    // returned records are deterministic
    __syncthreads();
    if (threadIdx.x == 0) results[i].arena_offset = 0;
  }
}

template <int L, int C, int kMost, int kNets>
cudaError_t launch_one(const SweepLaunch& launch, int max_rows, cudaStream_t stream) {
  const size_t smem = sweep_smem(L, C, launch.row_warps, max_rows).total;
  cudaError_t e = cudaFuncSetAttribute(lattice_sweep_kernel<L, C, kMost, kNets>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       static_cast<int>(smem));
  if (e != cudaSuccess) return e;
  lattice_sweep_kernel<L, C, kMost, kNets>
      <<<launch.plan_count, L * launch.row_warps * 32, smem, stream>>>(launch, max_rows);
  return cudaGetLastError();
}

// Row width classes of a layer count, narrowest first (width 0 past the last).
// `crowded`: the class has more nets than the device has SMs.
//
// One warp a row up to 512 cells: a second one brings a barrier and a fold into
// every scan (4 layers of 424 cells: 2.2 us a step with 4 x 1 warps of 16 cells
// a lane, 3.0 with 4 x 4 of 4; 1 layer of 310: 0.88 us with one warp, 1.58 with
// three).  Twelve cells a lane save registers where sixteen leave room for too
// few nets on an SM (1,500 nets of 380 cells: 3 layers 10.7 -> 8.9 ms, 6 layers
// 30.6 -> 15.9); on four layers a class more, with a launch and a stream of its
// own, cost a batch of many widths up to 4%.
//
// Past that, a class alone on its SMs takes the shape whose step is shortest,
// and a crowded one the shape of which two nets fit on an SM (a register limit
// of 8 or 12 warps a net): 4 layers of 645 cells, 8 nets 5.2 ms with 3 warps a
// row and 6.0 with 2 x 12 cells, 592 nets 22.0 and 16.7.  Up to 1,024 cells on
// three and four layers the kernel's bound on the warps stays above their
// number: compiled for 3 warps a row the 8 nets took 4.8 ms, but each held an
// SM's registers, and a batch of many widths had no room for other nets beside
// them (1,024 nets of 4 x 1024^2, five seeds of 16: 6.7 to 7.5 -> 7.3 to 7.8 ms).
//
// Rows of one layer past 1,024 cells, of two past 512, and the widest of three
// and four take the other form, a lane with its cells of every layer
// (lattice_sweep_rows.cu): it has half the barriers a step, and at two layers a
// third of the warps, so an SM holds more nets (2 layers of 645 cells: 592 nets
// 7.5 ms, 15.1 with a warp a layer, 8 nets 3.5 and 3.6; 1 layer of 1,500: 592
// nets 10.8 and 15.4 ms, 8 nets 4.9 and 5.8).
constexpr SweepShape row_lanes(int cells, int warps) { return {32 * cells * warps, cells, warps, warps, 1, true}; }

constexpr SweepShape sweep_shape_at(int layers, int index, bool crowded) {
  const SweepShape none{};
  // width, cells a lane, warps a row, the kernel's bound on these, nets an SM holds
  switch (layers) {
    case 1: {
      const SweepShape t[] = {{128, 4, 1, 1, 20}, {256, 8, 1, 1, 16}, {512, 16, 1, 1, 1}, {768, 8, 3, 16, 1}, {1024, 8, 4, 16, 1}};
      return index < 5 ? t[index] : index < 19 ? row_lanes(16, index - 2) : none;
    }
    case 2: {
      const SweepShape t[] = {{128, 4, 1, 1, 10}, {256, 8, 1, 1, 8}, {512, 16, 1, 1, 1}};
      return index < 3 ? t[index] : index < 17 ? row_lanes(8, index) : none;
    }
    case 3: {
      const SweepShape t[] = {{128, 4, 1, 1, 6}, {256, 8, 1, 1, 5}, {384, 12, 1, 1, 1}, {512, 16, 1, 1, crowded ? 4 : 1},
                              crowded ? SweepShape{768, 12, 2, 2, 2} : SweepShape{768, 8, 3, 5, 1},
                              crowded ? SweepShape{1024, 16, 2, 2, 2} : SweepShape{1024, 8, 4, 5, 1},
                              {1280, 8, 5, 5, 1}, {1536, 12, 4, 4, 1}, {2048, 16, 4, 4, 1}};
      return index < 9 ? t[index] : none;
    }
    case 4: {
      const SweepShape t[] = {{128, 4, 1, 1, 5}, {256, 8, 1, 1, 4}, {512, 16, 1, 1, 1},
                              crowded ? SweepShape{768, 12, 2, 2, 2} : SweepShape{768, 8, 3, 4, 1},
                              crowded ? SweepShape{1024, 16, 2, 2, 2} : SweepShape{1024, 8, 4, 4, 1},
                              {1152, 12, 3, 3, 1}, {1536, 16, 3, 3, 1}};
      return index < 7 ? t[index] : index < 11 ? row_lanes(4, index + 6) : none;
    }
    case 6: {
      const SweepShape t[] = {{128, 4, 1, 1, 3}, {256, 8, 1, 1, 2}, {384, 12, 1, 1, crowded ? 2 : 1}, {512, 16, 1, 1, 1},
                              {768, 12, 2, 2, 1}, {1024, 16, 2, 2, 1}};
      return index < 6 ? t[index] : none;
    }
    case 8: {
      const SweepShape t[] = {{128, 4, 1, 1, 2}, {256, 8, 1, 1, 2}, {512, 16, 1, 1, 1}, {768, 12, 2, 2, 1}, {1024, 16, 2, 2, 1}};
      return index < 5 ? t[index] : none;
    }
    default: return none;
  }
}

template <int L, int kIndex = 0, bool kCrowded = false>
cudaError_t launch_shape(const SweepShape& shape, const SweepLaunch& launch, int max_rows, cudaStream_t stream) {
  constexpr SweepShape t = sweep_shape_at(L, kIndex, kCrowded);
  if constexpr (t.width == 0) {
    return cudaErrorInvalidValue;
  } else {
    if constexpr (!t.lanes) {
      if (shape.cells == t.cells && shape.warps == t.warps && shape.nets == t.nets) {
        return launch_one<L, t.cells, t.most, t.nets>(launch, max_rows, stream);
      }
    }
    return launch_shape<L, kCrowded ? kIndex + 1 : kIndex, !kCrowded>(shape, launch, max_rows, stream);
  }
}

}  // namespace

SweepShape lattice_sweep_shape(int layers, int index, bool crowded) {
  return index < 0 ? SweepShape{} : sweep_shape_at(layers, index, crowded);
}

size_t lattice_sweep_smem_bytes(int layers, const SweepShape& shape, int max_rows) {
  return shape.lanes ? sweep_rows_smem_bytes(layers, shape.warps, max_rows)
                     : sweep_smem(layers, shape.cells, shape.warps, max_rows).total;
}

cudaError_t launch_lattice_sweep(int layers, const SweepShape& shape, SweepLaunch launch, int max_rows,
                                 cudaStream_t stream) {
  if (launch.plan_count == 0) return cudaSuccess;
  launch.row_warps = shape.warps;
  if (shape.lanes) return launch_sweep_rows(layers, shape.warps, launch, max_rows, stream);
  switch (layers) {
    case 1: return launch_shape<1>(shape, launch, max_rows, stream);
    case 2: return launch_shape<2>(shape, launch, max_rows, stream);
    case 3: return launch_shape<3>(shape, launch, max_rows, stream);
    case 4: return launch_shape<4>(shape, launch, max_rows, stream);
    case 6: return launch_shape<6>(shape, launch, max_rows, stream);
    case 8: return launch_shape<8>(shape, launch, max_rows, stream);
    default: return cudaErrorInvalidValue;
  }
}

cudaError_t launch_lattice_pack(apgar_b200_lattice_result* results, uint32_t count,
                                unsigned long long* total, const uint32_t* arena, uint32_t* paths,
                                int sm_count, cudaStream_t stream) {
  if (count == 0) return cudaSuccess;
  pack_offsets_kernel<<<1, 1024, 0, stream>>>(results, count, total);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  const uint32_t cap = static_cast<uint32_t>(sm_count > 0 ? sm_count * 8 : 1024);
  const unsigned grid = count < cap ? count : cap;
  pack_copy_kernel<<<grid, 128, 0, stream>>>(results, count, arena, paths);
  return cudaGetLastError();
}

}  // namespace apgar_b200
