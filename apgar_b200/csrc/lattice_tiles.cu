// Lattice-mode frontier search over tiles: label-correcting A* whose unit of
// work is a 32 x 32 block of one layer, relaxed to its own fixed point in
// shared memory by one warp.
//
// A net's window is cut into units (32 x 32 cells of one layer, from the
// window's corner).  A unit is pending when a neighbouring unit (eight in the
// plane, one above, one below) lowered a cell that can lower one of its own;
// its key is the least f = g + h over those lowerings, h the admissible,
// consistent octile-plus-via bound.  Units whose key lies below the level's
// limit thr are queued, the others wait in the far list, which opens when
// nothing is queued or being relaxed (thr then becomes the least waiting key
// plus the level width).  A warp that takes a unit loads its labels and their
// one-cell rim, sweeps it down, up, right and left until nothing changes,
// stores the changed rows and makes the neighbours it can lower pending.
//
// A sweep line is 32 cells, one per lane; a step relaxes the three moves from
// the previous line (straight, and both diagonals through lane shuffles).  An
// octile-optimal path in the open is straight moves and diagonals of one
// 90-degree wedge, so one sweep carries a label across the whole unit in its
// wedge; the four sweeps repeat only around obstacles.  Lines are processed
// in chunks of eight, and only from a chunk whose source line changed.
//
// Exactness.  Labels are costs of real paths, so never below the distance.
// Let C* be the optimum, G >= C* the goal's current label.  Along an optimal
// path f never exceeds C*; take its first inexact cell v, its predecessor u
// exact.  In one unit, the unit was swept to its fixed point after u became
// exact, so v is exact.  Across units, u's unit made v's unit pending with
// key f(v) <= C*, and a pending unit with a key at most G is neither dropped
// nor left when the search stops.  So every cell of every optimal path is
// exact at the stop, and the canonical walk, which accepts a predecessor only
// on label + move == label, returns the full-window canonical path
// (reference tie-break, gpu/cuda/planar_router.cu:977-1009, :1084-1165).
//
// Corridor mode first keeps to the net's corridor (only its cells are
// entered; a diagonal's side cells need not lie in it).  Every legal move from
// a labelled corridor cell to a free cell outside is an exit with key g + cost
// + h; the result is certified when the goal's label is strictly below the
// least exit key (the proof is lattice_frontier.cu's: every exit whose exact
// key is at most the goal label starts at a cell that is exact here).  If not,
// the corridor's labels stay, as they are costs of real paths, and the search
// goes on from every labelled unit without the corridor.
//
// What bounds it, and why this split.  One expansion per queued cell
// (lattice_frontier.cu) costs some 22 scattered 8-byte requests, and its
// wavefront advances one cell per round of about 10,000 cycles.  Here a
// unit's labels move as whole 128-byte lines, a unit carries labels across 32
// cells, and a step is about 15 instructions for 32 cells (8 of them on the
// half-rate integer pipe: about 34 cycles of an SM quarter, which bounds a
// full SM).  A unit takes about 35,000 cycles alone (13,000 of them sweeps,
// the rest dependent L2 accesses) and 80,000 with 24 warps on the SM.
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cstdint>

#include "lattice_common.cuh"

namespace apgar_b200 {
namespace {

constexpr uint32_t kFull = 0xFFFFFFFFu;
constexpr int kPitch = 35;                  // odd: rows and columns are both conflict-free
constexpr int kTileWords = 34 * kPitch + 2;  // 32 x 32 labels with their rim
constexpr int kQuadWords = 66;              // 33 rows of 64-bit 2 x 2 freedom bits (path walk)
constexpr int kWarpWords = kTileWords + kQuadWords;
constexpr int kPricePitch = 33;
constexpr int kPriceWords = 32 * kPricePitch;  // prices of the unit's cells
// Prices and labels below this cannot reach the 32-bit limit in a move; a net
// that meets one above it is searched by the cell form instead.
constexpr uint32_t kPriceLimit = 1u << 29;
constexpr uint32_t kNoLimit = 0xFFFFFFFDu;
constexpr uint32_t kTileInf = kTileLabelLimit;  // no label yet
constexpr uint32_t kNoKey = 0xFFFFFFFFu;     // pending key of an idle unit
constexpr uint32_t kBusyKey = 0xFFFFFFFEu;   // of a unit being relaxed
constexpr uint32_t kSourceBits = 0x3FFu;    // unit flags: sides that lowered something
constexpr uint32_t kInFar = 1u << 16;       // the unit stands in the far list
constexpr uint32_t kTouched = 1u << 17;     // the unit's labels have been written
constexpr uint32_t kWhole = 1u << 18;       // every cell of the unit may lower others (the corridor was lifted)
// Cancellation is looked for when a net starts and after every so many turns of
// its owner.
constexpr uint32_t kCancelPollTurns = 256;
// The host's flag is read across the bus, about 1 us a read and one after the
// other (at every net's start: 600 nets of 12 x 12 cells took 0.6 ms, nearly all
// of it waiting for these), so one warp of the grid reads it at most this
// often, and the others its copy on the device.
constexpr uint32_t kCancelLookNs = 20000;
// Guards against a broken invariant only: reported, never silent.  Each pass
// makes the labels exact whose least path within the unit has one move more,
// and such a path has at most 1,023 moves, so 1,024 passes do.  A pass is at
// most 128 steps of 34 cycles, 204 with 24 warps on the SM: at the limit a
// unit takes 54 million cycles, which a waiting owner outlasts (kIdleLimit).
constexpr int kMaxUnitPasses = 1 << 11;
// An idle warp naps between looks at its net's queue: its looks take issue
// slots from the warps at work.
constexpr uint32_t kNapNs = 300;
// Naps without any unit finished in the net before its owner gives it up, and
// without work before a helper does.  Between two naps come three dependent
// reads of the L2, 750 cycles or more: 200 million cycles in all.
constexpr uint32_t kIdleLimit = 1u << 18;
// Guests of a net at a time, a guest's looks at an empty queue before it
// leaves, and SM clocks between a CTA's searches for a net to visit.
constexpr uint32_t kGuestsPerNet = 48, kGuestMisses = 16, kProbeClocks = 1500, kProbeClocksMost = 24000;
constexpr int kTileThreads = 256, kTileBlocks = 3;  // per CTA, CTAs per SM

struct Win {
  int x0, y0, w, h;
  int gl, gx, gy;
  int tx, ty;  // units per row and per column
};

__device__ __forceinline__ uint32_t bound_to_goal(const LatticeDeviceView& lat, const Win& win, int l,
                                                  int x, int y) {
  const uint32_t dx = static_cast<uint32_t>(abs(x - win.gx));
  const uint32_t dy = static_cast<uint32_t>(abs(y - win.gy));
  const uint32_t lo = min(dx, dy), hi = max(dx, dy);
  const uint32_t planar = lat.diag >= lat.orth
                              ? lo * min(lat.diag, 2u * lat.orth) + (hi - lo) * lat.orth
                              : hi * lat.diag;
  return planar + static_cast<uint32_t>(abs(l - win.gl)) * lat.via;
}

__device__ __forceinline__ bool free_at(const LatticeDeviceView& lat, const Win& win, int l, int x, int y) {
  if (l < 0 || l >= lat.layers || x < 0 || y < 0 || x >= win.w || y >= win.h) return false;
  const int X = win.x0 + x, Y = win.y0 + y;
  const uint32_t word = __ldg(lat.blocked + (static_cast<size_t>(l) * lat.height + Y) * lat.words + (X >> 5));
  return ((word >> (X & 31)) & 1u) == 0u;
}

// A label that no cell can take when bit k of `closed` is set, else the
// label: sums with a move cost (at most 16 bits) stay above kTileInf and do
// not wrap.  One shift and one three-input logic operation.
__device__ __forceinline__ uint32_t unless(uint32_t closed, int k, uint32_t label) {
  return label | ((closed << (31 - k)) & 0x80000000u);
}

// One unit's place.  Lists hold units packed as layer << 28 | row << 14 | column.
struct Unit {
  int id, l, bx, by;  // bx, by: window coordinates of its first cell
};

__device__ __forceinline__ uint32_t pack_unit(int l, int ty, int tx) {
  return (static_cast<uint32_t>(l) << 28) | (static_cast<uint32_t>(ty) << 14) | static_cast<uint32_t>(tx);
}

__device__ __forceinline__ int unit_id(int tx, int ty, uint32_t packed) {
  return (static_cast<int>(packed >> 28) * ty + static_cast<int>((packed >> 14) & 0x3FFFu)) * tx +
         static_cast<int>(packed & 0x3FFFu);
}

__device__ __forceinline__ Unit unpack_unit(const Win& win, uint32_t packed) {
  Unit u;
  u.l = static_cast<int>(packed >> 28);
  const int ty = static_cast<int>((packed >> 14) & 0x3FFFu), tx = static_cast<int>(packed & 0x3FFFu);
  u.id = (u.l * win.ty + ty) * win.tx + tx;
  u.bx = tx * 32;
  u.by = ty * 32;
  return u;
}

// The unit's neighbours that exist: above, below (rows), left, right, the
// four corners (top left, top right, bottom left, bottom right), the layers
// below and above.
__device__ __forceinline__ uint32_t neighbours(const Win& win, const Unit& u, int layers) {
  uint32_t m = 0x3FFu;
  if (u.by == 0) m &= ~0x31u;
  if (u.by + 32 >= win.h) m &= ~0xC2u;
  if (u.bx == 0) m &= ~0x54u;
  if (u.bx + 32 >= win.w) m &= ~0xA8u;
  if (u.l == 0) m &= ~0x100u;
  if (u.l + 1 >= layers) m &= ~0x200u;
  return m;
}

// Distance in units to neighbour k, and the side this unit is on as seen from
// it (bits in the order of the neighbours).
__device__ __forceinline__ int neighbour_offset(const Win& win, int k) {
  const int row = (k == 0 || k == 4 || k == 5) ? -1 : (k == 1 || k == 6 || k == 7) ? 1 : 0;
  const int col = (k == 2 || k == 4 || k == 6) ? -1 : (k == 3 || k == 5 || k == 7) ? 1 : 0;
  const int lay = k == 8 ? -1 : k == 9 ? 1 : 0;
  return (lay * win.ty + row) * win.tx + col;
}

__device__ __forceinline__ uint32_t neighbour_packed(int k) {  // added to a packed unit
  const int row = (k == 0 || k == 4 || k == 5) ? -1 : (k == 1 || k == 6 || k == 7) ? 1 : 0;
  const int col = (k == 2 || k == 4 || k == 6) ? -1 : (k == 3 || k == 5 || k == 7) ? 1 : 0;
  const int lay = k == 8 ? -1 : k == 9 ? 1 : 0;
  return (static_cast<uint32_t>(lay) << 28) + (static_cast<uint32_t>(row) << 14) + static_cast<uint32_t>(col);
}

__device__ __forceinline__ uint32_t seen_from(int k) {
  return k < 4 ? 1u << (k ^ 1) : (k < 8 ? 1u << (11 - k) : 1u << (17 - k));
}

// 33 bits of a guard-padded plane line from bit `pos` (>= 0) on: the low 32
// and, in `next`, the one after them.  words: the line's trailing guard.
__device__ __forceinline__ uint32_t line_word(const uint32_t* line, int words, int pos, uint32_t& next) {
  const int wi = pos >> 5, s = pos & 31;
  const uint32_t lo = __ldg(line + wi), hi = __ldg(line + min(wi + 1, words));
  next = (hi >> s) & 1u;
  return __funnelshift_r(lo, hi, s);
}

__device__ __forceinline__ uint32_t low_bits(int n) { return n >= 32 ? kFull : (1u << n) - 1u; }

// Free cells of window column x over rows by .. by + 31, and whether the cell
// below them is; zero outside the window.
__device__ __forceinline__ uint32_t column_word(const LatticeDeviceView& lat, const Win& win, int l, int x, int by,
                                                uint32_t& next) {
  const int xc = min(max(x, 0), win.w - 1);
  const uint32_t* line =
      lat.sweep_cols + (static_cast<size_t>(l) * lat.width + (win.x0 + xc)) * (lat.words_t + 2) + 1;
  uint32_t after;
  const uint32_t v = ~line_word(line, lat.words_t, win.y0 + by, after) & low_bits(win.h - by);
  const bool in = x == xc;
  next = in && by + 32 < win.h ? after ^ 1u : 0u;
  return in ? v : 0u;
}

// The same for window row y over columns bx .. bx + 31.
__device__ __forceinline__ uint32_t row_word(const LatticeDeviceView& lat, const Win& win, int l, int y, int bx,
                                             uint32_t& next) {
  const int yc = min(max(y, 0), win.h - 1);
  const uint32_t* line =
      lat.sweep_rows + (static_cast<size_t>(l) * lat.height + (win.y0 + yc)) * (lat.words + 2) + 1;
  uint32_t after;
  const uint32_t v = ~line_word(line, lat.words, win.x0 + bx, after) & low_bits(win.w - bx);
  const bool in = y == yc;
  next = in && bx + 32 < win.w ? after ^ 1u : 0u;
  return in ? v : 0u;
}

// Rows (bit r) of window column x whose via between `lower` and the layer
// above it is allowed; whether the two cells are free is not included.
__device__ __forceinline__ uint32_t via_word(const LatticeDeviceView& lat, const Win& win, int lower, int x, int by) {
  if (lat.sweep_via_cols == nullptr) return kFull;
  const uint32_t* line =
      lat.sweep_via_cols + (static_cast<size_t>(lower) * lat.width + (win.x0 + min(x, win.w - 1))) * (lat.words_t + 2) + 1;
  uint32_t next;
  return line_word(line, lat.words_t, win.y0 + by, next);
}

// Freedom masks of a unit.
struct Masks {
  uint32_t col_free;  // lane = column: free rows
  uint32_t row_free;  // lane = row: free columns
  // across the sides (top, bottom, left, right), for this lane's cell of the
  // side: bits 2 k and 2 k + 1 the moves to and from the rim cells one lane
  // before and after are legal (the 2 x 2 block they cross is free), bit
  // 8 + k the rim cell is free
  uint32_t rim;
};

// A line of 34 cells: one before, 32, one after.
__device__ __forceinline__ uint64_t line34(uint32_t before, uint32_t cells, uint32_t after) {
  return static_cast<uint64_t>(before & 1u) | (static_cast<uint64_t>(cells) << 1) |
         (static_cast<uint64_t>(after & 1u) << 33);
}

// Bit j: the 2 x 2 block of cells j and j + 1 of two neighbouring lines is free.
__device__ __forceinline__ uint64_t quads34(uint64_t a, uint64_t b) {
  const uint64_t both = a & b;
  return both & (both >> 1);
}

// The four rim lines and the cell words of a unit (lines top, left, bottom,
// right hold the corners at both ends).
struct Rims {
  uint64_t top, bottom, left, right;
};

__device__ __forceinline__ void unit_free(const LatticeDeviceView& lat, const Win& win, const Unit& u, int lane,
                                          Masks& m, Rims& rims) {
  uint32_t below, beyond, top_next, left_next;
  m.col_free = column_word(lat, win, u.l, u.bx + lane, u.by, below);
  m.row_free = row_word(lat, win, u.l, u.by + lane, u.bx, beyond);
  const uint32_t top = row_word(lat, win, u.l, u.by - 1, u.bx, top_next);  // the same in every lane
  const uint32_t left = column_word(lat, win, u.l, u.bx - 1, u.by, left_next);
  const uint32_t bottom = __ballot_sync(kFull, below != 0u), right = __ballot_sync(kFull, beyond != 0u);
  const uint32_t corner = __ballot_sync(
      kFull, lane < 2 && free_at(lat, win, u.l, u.bx + (lane == 0 ? -1 : 32), u.by + (lane == 0 ? -1 : 32)));
  rims.top = line34(corner, top, top_next);
  rims.left = line34(corner, left, left_next);
  rims.bottom = line34(left_next, bottom, corner >> 1);
  rims.right = line34(top_next, right, corner >> 1);
}

__device__ __forceinline__ void unit_masks(const LatticeDeviceView& lat, const Win& win, const Unit& u, int lane,
                                           Masks& m) {
  Rims rims;
  unit_free(lat, win, u, lane, m, rims);
  const uint32_t row0 = __shfl_sync(kFull, m.row_free, 0), row31 = __shfl_sync(kFull, m.row_free, 31);
  const uint32_t col0 = __shfl_sync(kFull, m.col_free, 0), col31 = __shfl_sync(kFull, m.col_free, 31);
  const auto side = [&](uint64_t rim, uint64_t line, int k) {
    const uint32_t legal = static_cast<uint32_t>(quads34(rim, line) >> lane) & 3u;
    const uint32_t open = static_cast<uint32_t>(rim >> (lane + 1)) & 1u;
    return (legal << (2 * k)) | (open << (8 + k));
  };
  m.rim = side(rims.top, line34(static_cast<uint32_t>(rims.left >> 1), row0, static_cast<uint32_t>(rims.right >> 1)), 0);
  m.rim |= side(rims.bottom, line34(static_cast<uint32_t>(rims.left >> 32), row31, static_cast<uint32_t>(rims.right >> 32)), 1);
  m.rim |= side(rims.left, line34(static_cast<uint32_t>(rims.top >> 1), col0, static_cast<uint32_t>(rims.bottom >> 1)), 2);
  m.rim |= side(rims.right, line34(static_cast<uint32_t>(rims.top >> 32), col31, static_cast<uint32_t>(rims.bottom >> 32)), 3);
}

// Labels of a unit and its rim into the warp's tile.  touched: bit k set when
// neighbour k (the order of `neighbours`) has labels; own: this unit has.
__device__ __forceinline__ void load_unit(const uint32_t* labels, const Win& win, const Unit& u,
                                          uint32_t touched, bool own, uint32_t* tile, int lane) {
  const uint32_t* mine = labels + static_cast<size_t>(u.id) * 1024u;
  uint32_t top = kTileInf, bottom = kTileInf, left = kTileInf, right = kTileInf, corner = kTileInf;
  if (touched & 1u) top = __ldcg(mine - static_cast<ptrdiff_t>(win.tx) * 1024 + 992 + lane);
  if (touched & 2u) bottom = __ldcg(mine + static_cast<ptrdiff_t>(win.tx) * 1024 + lane);
  if (touched & 4u) left = __ldcg(mine - 1024 + lane * 32 + 31);
  if (touched & 8u) right = __ldcg(mine + 1024 + lane * 32);
  if (lane < 4 && ((touched >> (4 + lane)) & 1u)) {
    const ptrdiff_t unit = (lane < 2 ? -win.tx : win.tx) + ((lane & 1) ? 1 : -1);
    corner = __ldcg(mine + unit * 1024 + (lane < 2 ? 992 : 0) + ((lane & 1) ? 0 : 31));
  }
  if (own) {
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      uint32_t v[8];
#pragma unroll
      for (int k = 0; k < 8; ++k) v[k] = __ldcg(mine + (q * 8 + k) * 32 + lane);
#pragma unroll
      for (int k = 0; k < 8; ++k) tile[(q * 8 + k + 1) * kPitch + 1 + lane] = v[k];
    }
  } else {
#pragma unroll 8
    for (int r = 1; r <= 32; ++r) tile[r * kPitch + 1 + lane] = kTileInf;
  }
  tile[1 + lane] = top;
  tile[33 * kPitch + 1 + lane] = bottom;
  tile[(lane + 1) * kPitch] = left;
  tile[(lane + 1) * kPitch + 33] = right;
  if (lane < 4) tile[(lane < 2 ? 0 : 33 * kPitch) + ((lane & 1) ? 33 : 0)] = corner;
}


// Lines (and lanes) a sweep changed, as the masks the other directions need.
struct Swept {
  uint32_t lines;  // changed lines, rounded up to chunks
  uint32_t back;   // lines whose next line changed (rounded likewise)
  uint32_t lanes;
};

// One directional sweep over the lines of a unit, in the order of the line
// index i (0..31): cell + i * stride is this lane's cell of line i, bit i of
// `blocked` set when it is not free.  Chunks of eight lines run when `need`
// has a line in them or the line before them changed; the rim is not a source
// here.  A diagonal move needs four free cells: its source (a blocked cell
// has no label), the lane's own cells of both lines (`pair`), and the
// source's lane's cell of this line, which that lane checks before it hands
// its label over.  The outermost lanes get their own label back from a
// shuffle; p + diag is then no better than the straight p + orth, unless a
// diagonal is cheaper than a straight move (kCheapDiagonal).  Priced, every
// move into a cell also costs price[i * price_stride].  In a corridor
// (kCorr), `blocked` has the cells outside it too and `sides`, for the
// diagonals' side cells, only the blocked ones; else both are the same.
template <bool kCheapDiagonal, bool kPriced, bool kCorr>
__device__ __forceinline__ Swept sweep_lines(uint32_t* cell, int stride, const uint32_t* price, int price_stride,
                                             uint32_t blocked, uint32_t sides, uint32_t need, uint32_t orth,
                                             uint32_t diag, int lane, uint32_t& steps) {
  Swept out{0u, 0u, 0u};
  uint32_t pair = blocked | (sides << 1);
#pragma unroll 1
  for (int c = 0; c < 32; c += 8) {
    if (((need >> c) & 0xFFu) != 0u) {
      uint32_t p = c == 0 ? kTileInf : cell[-stride];
      uint32_t v[8];
#pragma unroll
      for (int k = 0; k < 8; ++k) v[k] = cell[k * stride];
      uint32_t diff = 0, first = 0, last = 0;
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const uint32_t given = unless(kCorr ? sides : blocked, k, p);
        const uint32_t straight = kCorr ? unless(blocked, k, p) : given;
        uint32_t before = __shfl_up_sync(kFull, given, 1), after = __shfl_down_sync(kFull, given, 1);
        if constexpr (kCheapDiagonal) {
          if (lane == 0) before = kTileInf;
          if (lane == 31) after = kTileInf;
        }
        uint32_t t;
        if constexpr (kPriced) {
          t = __viaddmin_u32(unless(pair, k, min(before, after)), diag, straight + orth);
          t = __viaddmin_u32(min(t, kTileInf), price[k * price_stride], v[k]);
        } else {
          t = __viaddmin_u32(straight, orth, v[k]);
          t = __viaddmin_u32(unless(pair, k, min(before, after)), diag, t);
        }
        cell[k * stride] = t;
        diff |= t ^ v[k];
        if (k == 0) first = diff;
        if (k == 7) last = t ^ v[k];
        p = t;
      }
      const uint32_t lanes = __ballot_sync(kFull, diff != 0u);
      const bool first_changed = __any_sync(kFull, first != 0u), last_changed = __any_sync(kFull, last != 0u);
      out.lanes |= lanes;
      out.lines |= lanes != 0u ? 0xFFu << c : 0u;
      out.back |= lanes != 0u ? 0x7Fu << c : 0u;
      out.back |= first_changed ? (1u << c) >> 1 : 0u;
      need |= last_changed ? (0x80u << c) << 1 : 0u;
      steps += 8;
    }
    cell += 8 * stride;
    price += 8 * price_stride;
    blocked >>= 8;
    sides >>= 8;
    pair >>= 8;
  }
  return out;
}

// The moves from one side's rim into its line of cells: line and rim are this
// lane's cells, lane_step the distance to the next lane's; price is that of
// entering the lane's cell.
template <bool kPriced>
__device__ __forceinline__ bool enter_side(uint32_t* line, const uint32_t* rim, int lane_step, uint32_t legal,
                                           bool is_free, uint32_t price, uint32_t orth, uint32_t diag) {
  const uint32_t v = *line;
  uint32_t t = __viaddmin_u32(unless(~legal, 0, rim[-lane_step]), diag, rim[0] + orth);
  t = __viaddmin_u32(unless(~legal, 1, rim[lane_step]), diag, t);
  if constexpr (kPriced) t = min(t, kTileInf) + price;
  t = min(t, v);
  if (is_free) *line = t;
  return is_free && t != v;
}

// Workspace of a net: labels [unit][32][32], then per unit the pending key,
// the flags and two far lists, and the pending queue's ring.
//
// A unit is idle (key kNoKey), waiting in the far list (a key, kInFar), queued
// (a key, one ring entry), or being relaxed by one warp (kBusyKey, or the key
// of a lowering that arrived meanwhile: that warp queues it again when it is
// done).  Whoever lowers the key of an idle unit queues it or puts it in the
// far list; whoever clears kInFar of a waiting unit queues it; so a unit never
// has two ring entries and never two warps.
struct Space {
  uint32_t* labels;
  uint32_t* pend;
  uint32_t* flags;
  uint32_t* far[2];
  uint32_t* ring;
  uint32_t ring_mask;
  uint32_t far_cap;
  uint32_t* own;  // own-route bits, a word per unit row; nullptr without rip-up pricing
};

// Slots of a net's ring: a power of two that holds every unit once.
__host__ __device__ __forceinline__ uint32_t ring_slots(uint32_t units) {
  uint32_t n = 32u;
  while (n < units) n <<= 1;
  return n;
}

__device__ __forceinline__ Space space_at(uint32_t* base, uint32_t units) {
  Space ws;
  ws.labels = base;
  ws.pend = base + static_cast<size_t>(units) * 1024u;
  ws.flags = ws.pend + units;
  ws.far[0] = ws.flags + units;
  ws.far[1] = ws.far[0] + units;
  ws.ring = ws.far[1] + units;
  ws.ring_mask = ring_slots(units) - 1u;
  ws.far_cap = units;
  ws.own = nullptr;
  return ws;
}

template <typename T>
__device__ __forceinline__ T peek(const T* p) {
  return *reinterpret_cast<const volatile T*>(p);
}

constexpr uint32_t kEmptySlot = 0xFFFFFFFFu;  // no packed unit (at most 8 layers)
// Waits are short (a slot between its reservation and its write); the limits
// only end the search with an error if that ever fails.
constexpr int kSlotWaits = 1 << 20;

// Takes the queue's next unit, or returns kEmptySlot (the same in every lane).
// All loops here and below are the whole warp's: a loop that one lane runs
// alone left the warp split in the sweeps that follow (each shuffle then
// waits for both parts).
__device__ __forceinline__ uint32_t pop_unit(TileNetState* st, const Space& ws, int lane) {
  uint32_t at = 0, got = 0;
  if (lane == 0) {
    at = peek(&st->head);
    got = static_cast<int32_t>(peek(&st->tail) - at) > 0 && atomicCAS(&st->head, at, at + 1u) == at ? 1u : 0u;
  }
  __syncwarp();
  if (__shfl_sync(kFull, got, 0) == 0u) return kEmptySlot;
  volatile uint32_t* slot = ws.ring + (__shfl_sync(kFull, at, 0) & ws.ring_mask);
  uint32_t unit = kEmptySlot;
  for (int i = 0; i < kSlotWaits; ++i) {
    unit = __shfl_sync(kFull, *slot, 0);
    if (unit != kEmptySlot) break;
  }
  __syncwarp();
  if (lane == 0) {
    if (unit == kEmptySlot) {
      atomicMax(&st->stop, 2u);  // (still active: nobody reuses the net's workspace)
    } else {
      *slot = kEmptySlot;
    }
  }
  __syncwarp();
  return unit;
}

// Appends the lanes' units (where `take`) to the queue; `active` already
// counts them.
__device__ __forceinline__ void push_units(TileNetState* st, const Space& ws, bool take, uint32_t unit, int lane) {
  const unsigned lanes = __ballot_sync(kFull, take);
  if (lanes == 0u) return;
  uint32_t at = 0;
  if (lane == 0) at = atomicAdd(&st->tail, __popc(lanes));
  at = __shfl_sync(kFull, at, 0) + __popc(lanes & ((1u << lane) - 1u));
  volatile uint32_t* slot = ws.ring + (at & ws.ring_mask);
  for (int i = 0; __any_sync(kFull, take && *slot != kEmptySlot); ++i) {
    if (i == kSlotWaits) {
      if (lane == 0) atomicMax(&st->stop, 2u);
      break;
    }
  }
  __syncwarp();
  if (take) *slot = unit;
  __syncwarp();
}

// What a lane keeps for its net: lanes 0..9 stand for a unit's neighbours.
struct LanePart {
  int offset;       // in units
  uint32_t packed;  // added to a packed unit
  uint32_t seen;    // the side this unit is on, as seen from the neighbour
};

// Which neighbours have labels.
__device__ __forceinline__ uint32_t touched_neighbours(const Space& ws, const LanePart& part, int id, uint32_t exist,
                                                       int lane) {
  bool t = false;
  if ((exist >> lane) & 1u) {
    t = (*reinterpret_cast<volatile uint32_t*>(ws.flags + id + part.offset) & kTouched) != 0u;
  }
  return __ballot_sync(kFull, t);
}

// Not certified: the net goes on without its corridor, from every labelled
// unit (one warp; nothing is queued or being relaxed).  True when nothing is
// left active.
__device__ __noinline__ bool lift_corridor(int tx, int ty, Space ws, TileNetState* st, int lane) {
  const uint32_t units = ws.far_cap;
  if (lane == 0) {
    st->corridor = peek(&st->goal) < kTileInf ? APGAR_B200_CORRIDOR_FALLBACK_EXIT : APGAR_B200_CORRIDOR_FALLBACK_UNREACHED;
    st->confined = 0u;
    st->far_count[0] = st->far_count[1] = 0u;
    atomicAdd(&st->active, 1u);  // this warp, until every unit is queued
  }
  const Win shape{0, 0, tx * 32, ty * 32, 0, 0, 0, tx, ty};
  const int plane = tx * ty, layers = static_cast<int>(units) / plane;
  const auto unit_at = [&](uint32_t i) {
    const int l = static_cast<int>(i) / plane, rest = static_cast<int>(i) - l * plane, y = rest / tx;
    return pack_unit(l, y, rest - y * tx);
  };
  for (uint32_t i = lane; i < units; i += 32) {
    // (kTouched stays as it is, so a neighbour that is already rewritten reads the same)
    const bool touched = (__ldcg(ws.flags + i) & kTouched) != 0u;
    uint32_t sides = 0;
    if (touched) {  // a side bit means a neighbour with labels
      const uint32_t exist = neighbours(shape, unpack_unit(shape, unit_at(i)), layers);
#pragma unroll 1
      for (int k = 0; k < 10; ++k) {
        if (((exist >> k) & 1u) != 0u && (__ldcg(ws.flags + static_cast<int>(i) + neighbour_offset(shape, k)) & kTouched) != 0u) {
          sides |= 1u << k;
        }
      }
    }
    __stcg(ws.flags + i, touched ? kTouched | kWhole | sides : 0u);
    __stcg(ws.pend + i, touched ? 0u : kNoKey);
  }
  __threadfence();
  __syncwarp();
  for (uint32_t base = 0; base < units; base += 32) {
    const uint32_t i = base + lane;
    // a unit that others have queued since has no kWhole: it was not labelled
    const bool take = i < units && (__ldcg(ws.flags + i) & kWhole) != 0u;
    const unsigned lanes = __ballot_sync(kFull, take);
    if (lane == 0 && lanes != 0u) atomicAdd(&st->active, __popc(lanes));
    __threadfence();
    __syncwarp();
    push_units(st, ws, take, unit_at(i), lane);
  }
  uint32_t left = 1;
  if (lane == 0) {
    __threadfence();
    left = atomicSub(&st->active, 1u) - 1u;
  }
  __syncwarp();
  return __shfl_sync(kFull, left, 0) == 0u;
}

// Nothing is queued or being relaxed: opens the next level from the far list,
// or ends the search (one warp, the one that finished the last unit).
template <bool kCorr>
__device__ __noinline__ void open_level(int tx, int ty, Space ws, TileNetState* st, int lane) {
  for (;;) {
    __threadfence();
    const uint32_t par = peek(&st->far_par), waiting = min(peek(&st->far_count[par]), ws.far_cap), limit = peek(&st->limit);
    uint32_t least = kNoKey;
    for (uint32_t i = lane; i < waiting; i += 32) {
      least = min(least, __ldcg(ws.pend + unit_id(tx, ty, __ldcg(ws.far[par] + i))));
    }
    least = __reduce_min_sync(kFull, least);
    if (least > limit || peek(&st->stop) != 0u) {  // every cell whose key still matters is final
      __syncwarp();
      if constexpr (kCorr) {
        const uint32_t goal = peek(&st->goal);
        if (peek(&st->stop) == 0u && peek(&st->confined) != 0u && (goal >= kTileInf || goal >= peek(&st->exit_key))) {
          if (!lift_corridor(tx, ty, ws, st, lane)) return;
          continue;  // its units are already done
        }
      }
      __syncwarp();
      if (lane == 0) {
        __threadfence();
        *reinterpret_cast<volatile uint32_t*>(&st->phase) = 2u;
      }
      return;
    }
    const uint32_t thr = least + min(peek(&st->level_width), kNoKey - least);
    if (lane == 0) {
      st->thr = thr;
      st->far_par = par ^ 1u;
      st->far_count[par] = 0u;
      st->levels += 1u;
      atomicAdd(&st->active, 1u);  // this warp, until the level is open
    }
    __syncwarp();
    __threadfence();
    for (uint32_t base = 0; base < waiting; base += 32) {
      const uint32_t i = base + lane;
      const bool valid = i < waiting;
      uint32_t unit = 0, key = kNoKey;
      int id = 0;
      if (valid) {
        unit = __ldcg(ws.far[par] + i);
        id = unit_id(tx, ty, unit);
        key = __ldcg(ws.pend + id);
      }
      // (a unit queued since it entered the list has no kInFar, or a second
      // entry: the first claims it)
      const bool keep = valid && key <= limit && key >= thr;
      bool take = false;
      if (valid && !keep && (atomicAnd(ws.flags + id, ~kInFar) & kInFar) != 0u) {
        take = key <= limit || atomicCAS(ws.pend + id, key, kNoKey) != key;
      }
      const unsigned take_lanes = __ballot_sync(kFull, take), keep_lanes = __ballot_sync(kFull, keep);
      uint32_t kept = 0;
      if (lane == 0) {
        if (take_lanes != 0u) atomicAdd(&st->active, __popc(take_lanes));
        if (keep_lanes != 0u) kept = atomicAdd(&st->far_count[par ^ 1u], __popc(keep_lanes));
      }
      kept = __shfl_sync(kFull, kept, 0) + __popc(keep_lanes & ((1u << lane) - 1u));
      // the kept entries and this level's own never exceed the list: one that
      // would is queued at once
      if (keep) {
        if (kept < ws.far_cap) {
          __stcg(ws.far[par ^ 1u] + kept, unit);
        } else if ((atomicAnd(ws.flags + id, ~kInFar) & kInFar) != 0u) {
          take = true;
          atomicAdd(&st->active, 1u);
        }
      }
      __threadfence();
      push_units(st, ws, take, unit, lane);
    }
    __syncwarp();
    uint32_t left = 1;
    if (lane == 0) {
      __threadfence();
      left = atomicSub(&st->active, 1u) - 1u;
    }
    if (__shfl_sync(kFull, left, 0) != 0u) return;
  }
}

// Price of entering window cell (l, x, y): without the net's own use on a cell
// of its previous route.
__device__ __forceinline__ uint32_t price_of(const TileLaunch& p, const Win& win, int l, int x, int y, bool mine) {
  const size_t i = (static_cast<size_t>(l) * p.lat.height + (win.y0 + y)) * p.lat.width + (win.x0 + x);
  return __ldg((mine ? p.cell_cost_own : p.cell_cost) + i);
}

__device__ __forceinline__ uint32_t price_of(const TileLaunch& p, const Win& win, const Space& ws, int l, int x, int y) {
  bool mine = false;
  if (ws.own != nullptr) {
    const int id = (l * win.ty + (y >> 5)) * win.tx + (x >> 5);
    mine = ((__ldcg(ws.own + static_cast<size_t>(id) * 32u + (y & 31)) >> (x & 31)) & 1u) != 0u;
  }
  return price_of(p, win, l, x, y, mine);
}

// Prices of a unit's cells into shared memory (at most kPriceLimit each);
// returns whether a free cell's reaches the limit.
__device__ __forceinline__ bool load_prices(const TileLaunch& p, const Win& win, const Space& ws, const Unit& u,
                                            uint32_t col_free, uint32_t* prices, int lane) {
  uint32_t own = 0;  // lane = row
  if (ws.own != nullptr) own = __ldcg(ws.own + static_cast<size_t>(u.id) * 32u + lane);
  bool high = false;
#pragma unroll 1
  for (int c = 0; c < 32; c += 8) {
    uint32_t v[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const uint32_t word = __shfl_sync(kFull, own, c + i);
      const bool in = u.bx + lane < win.w && u.by + c + i < win.h;
      v[i] = in ? price_of(p, win, u.l, u.bx + lane, u.by + c + i, ((word >> lane) & 1u) != 0u) : 0u;
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      high = high || (v[i] >= kPriceLimit && ((col_free >> (c + i)) & 1u) != 0u);
      prices[(c + i) * kPricePitch + lane] = min(v[i], kPriceLimit);
    }
  }
  return high;
}

// A net's corridor: the 64 x 64 coarse bitmap over its window.
struct Corridor {
  const uint32_t* bits;
  int shift;
};

__device__ __forceinline__ bool in_corridor(const Corridor& corr, const Win& win, int x, int y) {
  const uint32_t cx = static_cast<uint32_t>(min(max(x, 0), win.w - 1)) >> corr.shift;
  const uint32_t cy = static_cast<uint32_t>(min(max(y, 0), win.h - 1)) >> corr.shift;
  return ((__ldg(corr.bits + cy * 2u + (cx >> 5)) >> (cx & 31u)) & 1u) != 0u;
}

// The corridor cells (bit i) of column x over rows by .. by + 31, or of row y
// over columns bx .. bx + 31: coarse cells are 4 or more cells a side, and a
// unit's corner is a corner of one or lies inside it.
__device__ __forceinline__ uint32_t corridor_column(const Corridor& corr, const Win& win, int x, int by) {
  const int side = min(32, 1 << corr.shift);
  uint32_t m = 0;
  for (int r = 0; r < 32; r += side) m |= in_corridor(corr, win, x, by + r) ? low_bits(side) << r : 0u;
  return m;
}

__device__ __forceinline__ uint32_t corridor_row(const Corridor& corr, const Win& win, int y, int bx) {
  const int side = min(32, 1 << corr.shift);
  uint32_t m = 0;
  for (int c = 0; c < 32; c += side) m |= in_corridor(corr, win, bx + c, y) ? low_bits(side) << c : 0u;
  return m;
}

// The least key of the moves that leave the corridor from the labelled cells
// of the given rows of a unit (its labels in the tile).
__device__ __noinline__ uint32_t exit_key(const LatticeDeviceView& lat, Win win, Corridor corr, Unit u,
                                          const uint32_t* tile, uint32_t rows, int lane) {
  Masks m;
  Rims rims;
  unit_free(lat, win, u, lane, m, rims);
  // free cells, and those of them outside the corridor, of this lane's column
  // and the columns beside it: bit r + 1 is row r, from -1 to 32
  const auto outside = [&](int x, uint64_t open) {
    uint64_t in = static_cast<uint64_t>(corridor_column(corr, win, x, u.by)) << 1;
    if (in_corridor(corr, win, x, u.by - 1)) in |= 1ull;
    if (in_corridor(corr, win, x, u.by + 32)) in |= 1ull << 33;
    return open & ~in;
  };
  const auto column = [&](int at, uint32_t cells) {  // at: the column's place in the rim lines
    return line34(static_cast<uint32_t>(rims.top >> at), cells, static_cast<uint32_t>(rims.bottom >> at));
  };
  uint64_t open[3], out[3];
  open[1] = column(lane + 1, m.col_free);
  out[1] = outside(u.bx + lane, open[1]);
  open[0] = __shfl_up_sync(kFull, open[1], 1);
  out[0] = __shfl_up_sync(kFull, out[1], 1);
  open[2] = __shfl_down_sync(kFull, open[1], 1);
  out[2] = __shfl_down_sync(kFull, out[1], 1);
  if (lane == 0) {
    open[0] = column(0, static_cast<uint32_t>(rims.left >> 1));
    out[0] = outside(u.bx - 1, open[0]);
  }
  if (lane == 31) {
    open[2] = column(33, static_cast<uint32_t>(rims.right >> 1));
    out[2] = outside(u.bx + 32, open[2]);
  }
  __syncwarp();
  uint32_t least = kNoKey;
  if (!__any_sync(kFull, (out[0] | out[1] | out[2]) != 0ull)) return least;
  for (uint32_t rest = rows; rest != 0u; rest &= rest - 1u) {
    const int r = __ffs(rest) - 1;
    const uint32_t label = tile[(r + 1) * kPitch + 1 + lane];
    if (label < kTileInf && (((out[0] | out[1] | out[2]) >> r) & 7ull) != 0ull) {
      const int x = u.bx + lane, y = u.by + r;
#pragma unroll
      for (int d = 0; d < 9; ++d) {
        const int dx = d % 3 - 1, dy = d / 3 - 1;
        if (dx == 0 && dy == 0) continue;
        bool leaves = ((out[dx + 1] >> (r + 1 + dy)) & 1ull) != 0ull;
        if (dx != 0 && dy != 0) {
          leaves = leaves && ((open[dx + 1] >> (r + 1)) & 1ull) != 0ull && ((open[1] >> (r + 1 + dy)) & 1ull) != 0ull;
        }
        if (leaves) {
          least = min(least, label + (dx != 0 && dy != 0 ? lat.diag : lat.orth) + bound_to_goal(lat, win, u.l, x + dx, y + dy));
        }
      }
    }
  }
  __syncwarp();
  return __reduce_min_sync(kFull, least);
}

// Relaxes one pending unit to its fixed point and makes the neighbours it
// lowers pending.  Ends by handing its place in `active` to the units it
// queued.
template <bool kCheapDiagonal, bool kPriced, bool kCorr>
__device__ __forceinline__ void relax_unit(const TileLaunch& p, const Win& win, const Space& ws, uint32_t packed,
                                           const LanePart& part, uint32_t start_unit, int start_cell,
                                           uint32_t goal_unit, int goal_cell, TileNetState* st, const Corridor& corr,
                                           uint32_t* tile, uint32_t* prices, int lane) {
  const LatticeDeviceView& lat = p.lat;
  const Unit u = unpack_unit(win, packed);
  uint32_t key = 0, flags = 0, steps = 0;
  // Ends the unit: queues the lanes' neighbours (`near`), puts others in the
  // far list (`far`) and, if its own key was lowered meanwhile, itself
  // (lane 31).  Its place in `active` goes to what it queued.
  const auto finish = [&](bool near, bool far, uint32_t unit) {
    __syncwarp();
    if (lane == 31) {
      const uint32_t again = atomicCAS(ws.pend + u.id, kBusyKey, kNoKey);
      if (again != kBusyKey) {
        near = again < peek(&st->thr);
        far = !near;
        unit = packed;
        if (far) atomicOr(ws.flags + u.id, kInFar);
      }
    }
    const unsigned far_lanes = __ballot_sync(kFull, far);
    if (far_lanes != 0u) {
      const uint32_t par = peek(&st->far_par);
      uint32_t at = 0;
      if (lane == 0) at = atomicAdd(&st->far_count[par], __popc(far_lanes));
      at = __shfl_sync(kFull, at, 0) + __popc(far_lanes & ((1u << lane) - 1u));
      if (far) {
        if (at < ws.far_cap) {
          __stcg(ws.far[par] + at, unit);
        } else {  // no room: queued at once
          near = (atomicAnd(ws.flags + unpack_unit(win, unit).id, ~kInFar) & kInFar) != 0u;
        }
      }
    }
    const unsigned lanes = __ballot_sync(kFull, near);
    __threadfence();  // keys, flags and lists before the unit stops counting as active
    __syncwarp();
    uint32_t left = 1;
    if (lane == 0) {
      if (steps != 0u) atomicAdd(&st->steps, steps);
      atomicAdd(&st->units, 1u);
      left = atomicAdd(&st->active, __popc(lanes) - 1u) + __popc(lanes) - 1u;
    }
    __syncwarp();
    left = __shfl_sync(kFull, left, 0);
    push_units(st, ws, near, unit, lane);
    if (left == 0u) open_level<kCorr>(win.tx, win.ty, ws, st, lane);
    __syncwarp();
  };
  if (lane == 0) {
    key = atomicExch(ws.pend + u.id, kBusyKey);
    // a key above the limit can no longer matter; its side bits stay set,
    // because a source sets its bit before it lowers the key
    if (key <= peek(&st->limit) && peek(&st->stop) == 0u) {
      flags = atomicAnd(ws.flags + u.id, kCorr ? ~(kSourceBits | kWhole) : ~kSourceBits);
      __threadfence();  // the sources' labels are read after their bits
    } else {
      key = kNoKey;
    }
  }
  __syncwarp();
  Masks m;
  unit_masks(lat, win, u, lane, m);
  key = __shfl_sync(kFull, key, 0);
  flags = __shfl_sync(kFull, flags, 0);
  if (key == kNoKey) {
    finish(false, false, packed);
    return;
  }
  const bool own = (flags & kTouched) != 0u;
  const uint32_t col_open = m.col_free, row_open = m.row_free;
  bool confined = false;
  if constexpr (kCorr) {
    confined = __shfl_sync(kFull, peek(&st->confined), 0) != 0u;
    if (confined) {
      m.col_free &= corridor_column(corr, win, u.bx + lane, u.by);
      m.row_free &= corridor_row(corr, win, u.by + lane, u.bx);
    }
  }
  const uint32_t exist = neighbours(win, u, lat.layers);
  // (a side bit also says that the neighbour has labels: its kTouched may land later)
  const uint32_t touched = touched_neighbours(ws, part, u.id, exist, lane) | (flags & exist);
  load_unit(ws.labels, win, u, touched, own, tile, lane);
  bool high = false;  // a price or label near the 32-bit limit
  if constexpr (kPriced) high = load_prices(p, win, ws, u, m.col_free, prices, lane);
  __syncwarp();
  const auto price_at = [&](int r, int c) { return kPriced ? prices[r * kPricePitch + c] : 0u; };

  uint32_t down = 0, up = 0, right = 0, left = 0;  // lines whose source line changed
  uint32_t rows = 0, cols = 0;                     // changed rows and columns
  // kept in registers: the launch parameters are indexed by the width class,
  // so the compiler would read them again on every step
  uint32_t orth = lat.orth, diag = lat.diag, via = lat.via;
  asm("" : "+r"(orth), "+r"(diag), "+r"(via));
  if (!own && packed == start_unit) {
    const int r = start_cell >> 5, c = start_cell & 31;
    if (lane == c) tile[(r + 1) * kPitch + 1 + c] = 0u;
    rows = 1u << r;
    cols = 1u << c;
  }
  // lowerings from the layers below and above
  uint32_t* const mine = ws.labels + static_cast<size_t>(u.id) * 1024u + lane;
  const size_t plane = static_cast<size_t>(win.tx) * win.ty * 1024u;
  const uint32_t from = flags & touched;
#pragma unroll 1
  for (int k = 8; k < 10; ++k) {
    if (((from >> k) & 1u) == 0u) continue;
    uint32_t closed = ~(via_word(lat, win, k == 8 ? u.l - 1 : u.l, u.bx + lane, u.by) & m.col_free);
    const uint32_t* other = k == 8 ? mine - plane : mine + plane;
    uint32_t* cell = tile + kPitch + 1 + lane;
#pragma unroll 1
    for (int c = 0; c < 32; c += 8) {
      uint32_t o[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) o[i] = __ldcg(other + i * 32);
      uint32_t diff = 0;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const uint32_t v = cell[i * kPitch];
        uint32_t t = unless(closed, i, o[i]) + via;
        if constexpr (kPriced) t = min(t, kTileInf) + price_at(c + i, lane);
        t = min(t, v);
        cell[i * kPitch] = t;
        diff |= t ^ v;
      }
      const uint32_t hit = __ballot_sync(kFull, diff != 0u);
      rows |= hit != 0u ? 0xFFu << c : 0u;
      cols |= hit;
      other += 8 * 32;
      cell += 8 * kPitch;
      closed >>= 8;
    }
  }
  __syncwarp();
  // moves from the rim: the top and bottom rows (lane = column), then the
  // left and right columns (lane = row)
  if ((flags & 0x31u) != 0u) {
    const unsigned hit = __ballot_sync(kFull, enter_side<kPriced>(tile + kPitch + 1 + lane, tile + 1 + lane, 1, m.rim,
                                                                  (m.col_free & 1u) != 0u, price_at(0, lane), orth, diag));
    if (hit != 0u) rows |= 1u, cols |= hit;
  }
  if ((flags & 0xC2u) != 0u) {
    const unsigned hit = __ballot_sync(kFull, enter_side<kPriced>(tile + 32 * kPitch + 1 + lane, tile + 33 * kPitch + 1 + lane, 1,
                                                                  m.rim >> 2, (m.col_free >> 31) != 0u, price_at(31, lane), orth, diag));
    if (hit != 0u) rows |= 0x80000000u, cols |= hit;
  }
  __syncwarp();
  if ((flags & 0x4u) != 0u) {
    const unsigned hit = __ballot_sync(kFull, enter_side<kPriced>(tile + (lane + 1) * kPitch + 1, tile + (lane + 1) * kPitch,
                                                                  kPitch, m.rim >> 4, (m.row_free & 1u) != 0u, price_at(lane, 0), orth, diag));
    if (hit != 0u) cols |= 1u, rows |= hit;
  }
  if ((flags & 0x8u) != 0u) {
    const unsigned hit = __ballot_sync(kFull, enter_side<kPriced>(tile + (lane + 1) * kPitch + 32, tile + (lane + 1) * kPitch + 33,
                                                                  kPitch, m.rim >> 6, (m.row_free >> 31) != 0u, price_at(lane, 31), orth, diag));
    if (hit != 0u) cols |= 0x80000000u, rows |= hit;
  }
  if (kCorr && (flags & kWhole) != 0u) rows = cols = kFull;
  down = rows << 1;
  up = rows >> 1;
  right = cols << 1;
  left = cols >> 1;

  uint32_t* const first_row = tile + kPitch + 1 + lane;         // lane = column, line = row
  uint32_t* const first_col = tile + (lane + 1) * kPitch + 1;   // lane = row, line = column
  int passes = 0;
  while ((down | up | right | left) != 0u) {
    if (++passes > kMaxUnitPasses) {
      if (lane == 0) atomicMax(&st->stop, 2u);
      break;
    }
    // Down, up, right, left: one copy of the sweep's code for the four, with
    // the stride in a register, so that it stays in the instruction cache
    // while an SM's warps are at different places of a unit (four copies:
    // waits for instructions were the top stall, 3.2 cycles an instruction;
    // medium batch 11.9 ms, 10.7 with one, priced rounds 50 ms and 44).
#pragma unroll 1
    for (int dir = 0; dir < 4; ++dir) {
      const bool across = dir >= 2, reverse = (dir & 1) != 0;
      uint32_t need = across ? (reverse ? left : right) : (reverse ? up : down);
      if (need == 0u) continue;
      __syncwarp();
      uint32_t blocked = ~(across ? m.row_free : m.col_free), sides = ~(across ? row_open : col_open);
      uint32_t* cell = across ? first_col : first_row;
      const uint32_t* price = across ? prices + lane * kPricePitch : prices + lane;
      int stride = across ? 1 : kPitch, price_stride = across ? 1 : kPricePitch;
      if (reverse) {
        need = __brev(need);
        blocked = __brev(blocked);
        sides = __brev(sides);
        cell += 31 * stride;
        price += 31 * price_stride;
        stride = -stride;
        price_stride = -price_stride;
      }
      const Swept w = sweep_lines<kCheapDiagonal, kPriced, kCorr>(cell, stride, price, price_stride, blocked, sides, need,
                                                                  orth, diag, lane, steps);
      const uint32_t back = reverse ? __brev(w.back) : w.back, lines = reverse ? __brev(w.lines) : w.lines;
      const uint32_t after = w.lanes << 1, before = w.lanes >> 1;
      if (across) {
        right = reverse ? right | back : 0u;
        left = reverse ? 0u : left | back;
        down |= after;
        up |= before;
        cols |= lines;
        rows |= w.lanes;
      } else {
        down = reverse ? down | back : 0u;
        up = reverse ? 0u : up | back;
        right |= after;
        left |= before;
        rows |= lines;
        cols |= w.lanes;
      }
    }
  }
  __syncwarp();
  if (rows == 0u && own) {  // nothing lowered
    finish(false, false, packed);
    return;
  }

  // changed rows (all of them the first time), in blocks of eight
#pragma unroll 1
  for (int c = 0; c < 32; c += 8) {
    if (own && ((rows >> c) & 0xFFu) == 0u) continue;
    const uint32_t* row = tile + (c + 1) * kPitch + 1 + lane;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const uint32_t v = row[k * kPitch];
      mine[(c + k) * 32] = v;
      if constexpr (kPriced) high = high || (v >= kPriceLimit && v < kTileInf);
    }
  }
  if (packed == goal_unit && lane == 0) {
    const uint32_t goal = tile[((goal_cell >> 5) + 1) * kPitch + 1 + (goal_cell & 31)];
    if (goal < kTileInf) {
      atomicMin(&st->goal, goal);
      // Priced, the search goes on to the end of the key level that holds the
      // goal, as the cell form does: a price that overflows there rejects
      // the net.
      uint32_t limit = goal;
      if constexpr (kPriced) {
        const unsigned long long width = peek(&st->level_width), first = peek(&st->start_key);
        limit = static_cast<uint32_t>(min(first + width * ((goal - first) / width + 1ull) - 1ull,
                                          static_cast<unsigned long long>(kNoLimit)));
      }
      atomicMin(&st->limit, limit);
    }
  }
  // the least key this unit lowers in each neighbour
  uint32_t out_key = kNoKey;
  const auto key_min = [&](bool lowers, uint32_t cost, int l, int x, int y) {
    if (!__any_sync(kFull, lowers)) return kNoKey;
    const uint32_t f = lowers ? cost + bound_to_goal(lat, win, l, x, y) : kNoKey;
    return __reduce_min_sync(kFull, f);
  };
  // a move's cost into a cell of a neighbour, with its price
  const auto priced = [&](uint32_t t, int l, int x, int y) {
    if constexpr (kPriced) {
      if (t < kTileInf) {
        const uint32_t price = price_of(p, win, ws, l, x, y);
        high = high || price >= kPriceLimit;
        t = min(t + min(price, kPriceLimit), kTileInf);
      }
      __syncwarp();
    }
    return t;
  };
  // rows above and below the unit, and its corners
#pragma unroll 1
  for (int k = 0; k < 2; ++k) {
    if (((k == 0 ? rows : rows >> 31) & 1u) == 0u) continue;
    const uint32_t* line = tile + (k == 0 ? 1 : 32) * kPitch + 1 + lane;
    const uint32_t* rim = tile + (k == 0 ? 0 : 33) * kPitch + 1 + lane;
    const uint32_t closed = ~(m.rim >> (2 * k));
    uint32_t t = unless(~(m.rim >> (8 + k)), 0, line[0]) + orth;
    if (lane > 0) t = __viaddmin_u32(unless(closed, 0, line[-1]), diag, t);
    if (lane < 31) t = __viaddmin_u32(unless(closed, 1, line[1]), diag, t);
    const int y = k == 0 ? u.by - 1 : u.by + 32;
    if (kCorr && confined && !in_corridor(corr, win, u.bx + lane, y)) t = kTileInf;
    t = priced(t, u.l, u.bx + lane, y);
    const uint32_t f = key_min(t < rim[0], t, u.l, u.bx + lane, y);
    if (lane == k) out_key = f;
    // corners: from the first and the last cell of the line
    uint32_t corner = lane == 0 || lane == 31 ? unless(closed, lane == 0 ? 0 : 1, line[0]) + diag : kTileInf;
    if (kCorr && confined && !in_corridor(corr, win, u.bx + (lane == 0 ? -1 : 32), y)) corner = kTileInf;
    corner = priced(corner, u.l, u.bx + (lane == 0 ? -1 : 32), y);
    const bool low = (lane == 0 && corner < rim[-1]) || (lane == 31 && corner < rim[1]);
    if (__any_sync(kFull, low)) {
      const uint32_t cf = low ? corner + bound_to_goal(lat, win, u.l, u.bx + (lane == 0 ? -1 : 32), y) : kNoKey;
      const uint32_t c0 = __shfl_sync(kFull, cf, 0), c1 = __shfl_sync(kFull, cf, 31);
      if (lane == 4 + 2 * k) out_key = c0;
      if (lane == 5 + 2 * k) out_key = c1;
    }
  }
  // columns left and right of the unit
#pragma unroll 1
  for (int k = 0; k < 2; ++k) {
    if (((k == 0 ? cols : cols >> 31) & 1u) == 0u) continue;
    const uint32_t* line = tile + (lane + 1) * kPitch + (k == 0 ? 1 : 32);
    const uint32_t* rim = tile + (lane + 1) * kPitch + (k == 0 ? 0 : 33);
    const uint32_t closed = ~(m.rim >> (4 + 2 * k));
    uint32_t t = unless(~(m.rim >> (10 + k)), 0, line[0]) + orth;
    if (lane > 0) t = __viaddmin_u32(unless(closed, 0, line[-kPitch]), diag, t);
    if (lane < 31) t = __viaddmin_u32(unless(closed, 1, line[kPitch]), diag, t);
    if (kCorr && confined && !in_corridor(corr, win, u.bx + (k == 0 ? -1 : 32), u.by + lane)) t = kTileInf;
    t = priced(t, u.l, u.bx + (k == 0 ? -1 : 32), u.by + lane);
    const uint32_t f = key_min(t < rim[0], t, u.l, u.bx + (k == 0 ? -1 : 32), u.by + lane);
    if (lane == 2 + k) out_key = f;
  }
  // the layers below and above, over the changed rows
#pragma unroll 1
  for (int k = 8; k < 10; ++k) {
    if (((exist >> k) & 1u) == 0u) continue;
    const int l = k == 8 ? u.l - 1 : u.l + 1;
    uint32_t unused;
    const uint32_t shut = ~(via_word(lat, win, min(l, u.l), u.bx + lane, u.by) & m.col_free &
                            column_word(lat, win, l, u.bx + lane, u.by, unused));
    const bool labelled = ((touched >> k) & 1u) != 0u;
    const uint32_t* other = k == 8 ? mine - plane : mine + plane;
    const uint32_t dx = static_cast<uint32_t>(abs(u.bx + lane - win.gx));
    uint32_t f = kNoKey;
#pragma unroll 1
    for (int c = 0; c < 32; c += 8) {
      if (((rows >> c) & 0xFFu) == 0u) continue;
      uint32_t o[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) o[i] = labelled ? __ldcg(other + (c + i) * 32) : kTileInf;
      const uint32_t closed = shut >> c;
      const uint32_t* row = tile + (c + 1) * kPitch + 1 + lane;
      bool lowers = false;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        uint32_t t = unless(closed, i, row[i * kPitch]) + via;
        // (an unchanged row of the block lowers nothing: no need of its prices)
        t = !kPriced || (rows & (1u << (c + i))) != 0u ? priced(t, l, u.bx + lane, u.by + c + i) : kTileInf;
        lowers = lowers || t < o[i];
        o[i] = t < o[i] ? t : kNoKey;
      }
      if (__any_sync(kFull, lowers)) {
        // the planar part of the bound, added where the label lowers
        const uint32_t step = diag >= orth ? min(diag, 2u * orth) - orth : 0u, far = diag >= orth ? orth : diag;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const uint32_t dy = static_cast<uint32_t>(abs(u.by + c + i - win.gy));
          const uint32_t h = min(dx, dy) * step + max(dx, dy) * far;
          if (o[i] != kNoKey) f = min(f, o[i] + h);
        }
      }
    }
    f = __reduce_min_sync(kFull, f);
    if (lane == k && f != kNoKey) out_key = f + static_cast<uint32_t>(abs(l - win.gl)) * via;
  }
  if constexpr (kCorr) {
    if (confined) {
      const uint32_t leaving = exit_key(lat, win, corr, u, tile, rows, lane);
      if (lane == 0 && leaving != kNoKey) atomicMin(&st->exit_key, leaving);
      __syncwarp();
    }
  }
  if constexpr (kPriced) {
    if (__any_sync(kFull, high) && lane == 0) atomicMax(&st->stop, 3u);
  }
  // What lands before what: the labels before the side bits and kTouched that
  // announce them, these before the neighbours' keys and before this unit's
  // own key is free again (in `finish`).  kTouched and the side bits may land
  // in either order, so a warp that takes a neighbour reads this unit's labels
  // on its side bit alone.
  __syncwarp();
  __threadfence();
  __syncwarp();
  const uint32_t limit = peek(&st->limit), thr = peek(&st->thr);
  const bool lowers = out_key <= limit;  // lanes 0..9 only: the others hold kNoKey
  const int nb = u.id + part.offset;
  if (!own && lane == 0) atomicOr(ws.flags + u.id, kTouched);
  if (lowers) atomicOr(ws.flags + nb, part.seen);
  if (!own || __any_sync(kFull, lowers)) {
    __syncwarp();
    __threadfence();
    __syncwarp();
  }
  bool near = false, far = false;
  if (lowers) {
    const uint32_t old = atomicMin(ws.pend + nb, out_key);
    if (old == kNoKey) {
      near = out_key < thr;
      far = !near;
      if (far) atomicOr(ws.flags + nb, kInFar);
    } else if (old != kBusyKey && out_key < thr && old >= thr) {
      near = (atomicAnd(ws.flags + nb, ~kInFar) & kInFar) != 0u;
    }
  }
  __syncwarp();
  finish(near, far, packed + part.packed);
}

// Canonical reverse path by one warp: the unit under the walk sits in shared
// memory, so a step costs a few shared-memory reads; a step onto another unit
// loads that one.  Vias are tried only when no planar predecessor matches
// (headings 0-7 come first).  Returns the path length, 0 when broken.
template <bool kPriced>
__device__ __forceinline__ uint32_t walk_path(const TileLaunch& p, const Win& win, const Space& ws,
                                              const LanePart& part, int sl, int sx, int sy, uint32_t goal, unsigned long long base,
                                              unsigned long long bound, uint32_t* tile, uint64_t* quads,
                                              uint32_t* prices, int lane) {
  const LatticeDeviceView& lat = p.lat;
  int l = win.gl, x = win.gx, y = win.gy;
  uint32_t here = goal, len = 0;
  uint32_t loaded = kNoKey;
  Unit u{};
  // heading of this lane: the step into the current cell
  const int dx = (lane == 0 || lane == 1 || lane == 7) ? 1 : (lane == 2 || lane == 6) ? 0 : -1;
  const int dy = (lane >= 1 && lane <= 3) ? 1 : (lane == 0 || lane == 4) ? 0 : -1;
  while (len < bound) {
    if (lane == 0) {
      p.path_arena[base + len] = static_cast<uint32_t>(
          (static_cast<size_t>(l) * lat.height + (win.y0 + y)) * lat.width + (win.x0 + x));
    }
    ++len;
    if (l == sl && x == sx && y == sy) return len;
    const uint32_t unit = pack_unit(l, y >> 5, x >> 5);
    if (unit != loaded) {
      u = unpack_unit(win, unit);
      __syncwarp();
      // 2 x 2 blocks over rows r - 1 and r (bit x: columns x - 1 and x)
      Masks m;
      Rims rims;
      unit_free(lat, win, u, lane, m, rims);
      const uint64_t line = line34(static_cast<uint32_t>(rims.left >> (lane + 1)), m.row_free,
                                   static_cast<uint32_t>(rims.right >> (lane + 1)));
      uint64_t above = __shfl_up_sync(kFull, line, 1);
      if (lane == 0) above = rims.top;
      quads[lane] = quads34(line, above);
      if (lane == 31) quads[32] = quads34(line, rims.bottom);
      load_unit(ws.labels, win, u, touched_neighbours(ws, part, u.id, neighbours(win, u, lat.layers), lane), true, tile, lane);
      if constexpr (kPriced) load_prices(p, win, ws, u, m.col_free, prices, lane);
      __syncwarp();
      loaded = unit;
    }
    const int r = y - u.by, c = x - u.bx;
    // the move into this cell paid its price
    const uint32_t paid = kPriced ? prices[r * kPricePitch + c] : 0u;
    bool ok = false;
    uint32_t label = kTileInf;
    if (lane < 8) {
      const int pr = r - dy, pc = c - dx;
      label = tile[(pr + 1) * kPitch + 1 + pc];
      const bool legal = (lane & 1) == 0 || ((quads[max(r, pr)] >> max(c, pc)) & 1ull) != 0ull;
      ok = legal && label < kTileInf && label + ((lane & 1) ? lat.diag : lat.orth) + paid == here;
    }
    unsigned hit = __ballot_sync(kFull, ok);
    int nl = l;
    if (hit == 0u) {
      if (lane == 8 || lane == 9) {
        nl = lane == 8 ? l - 1 : l + 1;
        if (free_at(lat, win, nl, x, y)) {
          const int other = u.id + (lane == 8 ? -1 : 1) * win.tx * win.ty;
          bool allowed = (*reinterpret_cast<volatile uint32_t*>(ws.flags + other) & kTouched) != 0u;
          if (allowed && lat.via_ok != nullptr) {
            const int X = win.x0 + x;
            const size_t row = static_cast<size_t>(min(l, nl)) * lat.height + (win.y0 + y);
            allowed = ((__ldg(lat.via_ok + row * lat.words + (X >> 5)) >> (X & 31)) & 1u) != 0u;
          }
          if (allowed) {
            label = __ldcg(ws.labels + static_cast<size_t>(other) * 1024u + r * 32 + c);
            ok = label < kTileInf && label + lat.via + paid == here;
          }
        }
      }
      hit = __ballot_sync(kFull, ok);
      if (hit == 0u) return 0u;
    }
    const int sel = __ffs(hit) - 1;
    here = __shfl_sync(kFull, label, sel);
    if (sel < 8) {
      x -= __shfl_sync(kFull, dx, sel);
      y -= __shfl_sync(kFull, dy, sel);
    } else {
      l = __shfl_sync(kFull, nl, sel);
    }
  }
  return 0u;
}

// A net as its searchers see it.
struct TileNet {
  Win win;
  Space ws;
  uint32_t units, start_unit, goal_unit;
  int start_cell, goal_cell;
  int sl, sx, sy;
  Corridor corr;
};

__device__ __forceinline__ TileNet net_at(const TileLaunch& p, uint32_t index, uint32_t slot) {
  const NetPlan plan = p.plans[index];
  const apgar_b200_lattice_net net = p.nets[plan.net];
  uint32_t* base = p.c[0].pool;
  if (p.per_net) {
    base += plan.dist_offset;
  } else {
    int k = 0;
    while (k < 4 && index >= p.c[k].end) ++k;
    base = p.c[k].pool + static_cast<uint64_t>(slot) * p.c[k].slot_words;
  }
  TileNet n;
  n.win.x0 = static_cast<int>(net.win_x0);
  n.win.y0 = static_cast<int>(net.win_y0);
  n.win.w = static_cast<int>(net.win_w);
  n.win.h = static_cast<int>(net.win_h);
  n.win.gl = static_cast<int>(net.goal_layer);
  n.win.gx = static_cast<int>(net.goal_x) - n.win.x0;
  n.win.gy = static_cast<int>(net.goal_y) - n.win.y0;
  n.win.tx = (n.win.w + 31) >> 5;
  n.win.ty = (n.win.h + 31) >> 5;
  n.sl = static_cast<int>(net.start_layer);
  n.sx = static_cast<int>(net.start_x) - n.win.x0;
  n.sy = static_cast<int>(net.start_y) - n.win.y0;
  n.units = static_cast<uint32_t>(p.lat.layers) * n.win.tx * n.win.ty;
  n.ws = space_at(base, n.units);
  n.corr.bits = p.corridor == nullptr ? nullptr : p.corridor + static_cast<size_t>(plan.net) * 128u;
  n.corr.shift = 2;  // at most 63 coarse cells a side
  while (((max(n.win.w, n.win.h) - 1) >> n.corr.shift) >= 63) ++n.corr.shift;
  if (p.cell_cost_own != nullptr) n.ws.own = p.own_bits + (base - p.c[0].pool) / 32;
  n.start_unit = pack_unit(n.sl, n.sy >> 5, n.sx >> 5);
  n.goal_unit = pack_unit(n.win.gl, n.win.gy >> 5, n.win.gx >> 5);
  n.start_cell = ((n.sy & 31) << 5) | (n.sx & 31);
  n.goal_cell = ((n.win.gy & 31) << 5) | (n.win.gx & 31);
  return n;
}

__device__ __forceinline__ LanePart lane_part(const Win& win, int lane) {
  return LanePart{neighbour_offset(win, lane), neighbour_packed(lane), lane < 10 ? seen_from(lane) : 0u};
}

// Units in a net's queue that its warps are not about to take themselves.
__device__ __forceinline__ uint32_t spare_units(const TileNetState* st) {
  if (peek(&st->phase) != 1u) return 0u;
  const uint32_t head = peek(&st->head), queued = peek(&st->tail) - head;
  if (static_cast<int32_t>(queued) <= 0 || peek(&st->guests) >= kGuestsPerNet) return 0u;
  return queued > 1u || peek(&st->active) > queued ? min(queued, 0xFFFFu) : 0u;
}

// What the idle warps of a CTA share.
struct Lookout {
  uint32_t probed;   // SM clock of the last search,
  uint32_t pause;    // and the clocks until the next
  uint32_t net;      // a net found with units to spare,
  uint32_t places;   // and how many more warps may visit it
  uint32_t over;     // every net is done
  uint32_t team;     // the net that the whole CTA searches
};

// A net to visit, or kNoKey.  One warp of the CTA searches at a time,
// kProbeClocks apart, the 32 unfinished nets from `low` on; the others look
// only at shared memory: their reads would slow the states' own warps.
__device__ __forceinline__ uint32_t find_net(const TileLaunch& p, uint32_t& low, uint32_t& skip, Lookout& look, int lane) {
  uint32_t found = kNoKey, mine = 0;
  if (lane == 0) {
    if (static_cast<int32_t>(peek(&look.places)) > 0 && static_cast<int32_t>(atomicSub(&look.places, 1u)) > 0) {
      found = peek(&look.net);
    } else {
      const uint32_t now = static_cast<uint32_t>(clock64()), then = peek(&look.probed);
      mine = now - then > peek(&look.pause) && atomicCAS(&look.probed, then, now) == then ? 1u : 0u;
    }
  }
  __syncwarp();
  found = __shfl_sync(kFull, found, 0);
  if (found != kNoKey || __shfl_sync(kFull, mine, 0) == 0u) return found;
  const uint32_t i = low + skip + lane;
  const uint32_t phase = i < p.total ? peek(&p.states[i].phase) : 0u;
  const uint32_t spare = phase == 1u ? spare_units(p.states + i) : 0u;
  const uint32_t best = __reduce_max_sync(kFull, spare << 8 | static_cast<uint32_t>(lane));
  const unsigned unfinished = __ballot_sync(kFull, phase != 2u);
  if (skip == 0u) low += unfinished == 0u ? 32u : static_cast<uint32_t>(__ffs(unfinished) - 1);
  if (low >= p.total) low = 0u;
  if (lane == 0) {
    if (peek(p.finished) >= p.total) *reinterpret_cast<volatile uint32_t*>(&look.over) = 1u;
    *reinterpret_cast<volatile uint32_t*>(&look.pause) =
        (best >> 8) != 0u ? kProbeClocks : min(2u * peek(&look.pause), kProbeClocksMost);
  }
  __syncwarp();
  if ((best >> 8) != 0u) {
    found = i - lane + (best & 31u);
    skip = 0u;
    if (lane == 0) {
      *reinterpret_cast<volatile uint32_t*>(&look.net) = found;
      __threadfence_block();
      *reinterpret_cast<volatile uint32_t*>(&look.places) = min(best >> 8, kTileThreads / 32u);
    }
    __syncwarp();
  } else {
    skip = low + skip + 32u < p.total ? skip + 32u : 0u;
  }
  return found;
}

// Whether the batch is cancelled (one lane).
__device__ __forceinline__ bool batch_cancelled(const TileLaunch& p) {
  if (p.cancel == nullptr) return false;
  if (peek(p.watch) != 0u) return true;
  uint32_t now;
  asm volatile("mov.u32 %0, %%globaltimer_lo;" : "=r"(now));
  const uint32_t then = peek(p.watch + 1);
  if (now - then < kCancelLookNs || atomicCAS(p.watch + 1, then, now) != then || *p.cancel == 0u) return false;
  *reinterpret_cast<volatile uint32_t*>(p.watch) = 1u;
  return true;
}

// Clears the net's workspace and queues its start.
__device__ __forceinline__ bool start_net(const TileLaunch& p, const TileNet& n, TileNetState* st, uint32_t level_width,
                                          uint32_t slot, uint32_t net, int lane) {
  const bool free_ends = free_at(p.lat, n.win, n.sl, n.sx, n.sy) &&
                         free_at(p.lat, n.win, n.win.gl, n.win.gx, n.win.gy);
  for (uint32_t i = lane; i < 2u * n.units; i += 32) __stcg(n.ws.pend + i, i < n.units ? kNoKey : 0u);
  for (uint32_t i = lane; i <= n.ws.ring_mask; i += 32) __stcg(n.ws.ring + i, kEmptySlot);
  if (n.ws.own != nullptr) {
    // the cells of the net's previous route (a packed reverse path of global
    // cells; a cell outside the window cannot be entered anyway)
    for (uint32_t i = lane; i < 32u * n.units; i += 32) __stcg(n.ws.own + i, 0u);
    __syncwarp();
    const apgar_b200_lattice_result prev = p.prev_results[net];
    if (prev.completion == APGAR_B200_COMPLETION_REACHED) {
      const uint32_t lw = static_cast<uint32_t>(p.lat.width), lh = static_cast<uint32_t>(p.lat.height);
      for (uint32_t j = lane; j < prev.path_len; j += 32) {
        const uint32_t c = p.prev_paths[prev.path_offset + j];
        const int x = static_cast<int>(c % lw) - n.win.x0, y = static_cast<int>((c / lw) % lh) - n.win.y0;
        const uint32_t l = c / lw / lh;
        if (l < static_cast<uint32_t>(p.lat.layers) && x >= 0 && x < n.win.w && y >= 0 && y < n.win.h) {
          const int id = (static_cast<int>(l) * n.win.ty + (y >> 5)) * n.win.tx + (x >> 5);
          atomicOr(n.ws.own + static_cast<size_t>(id) * 32u + (y & 31), 1u << (x & 31));
        }
      }
    }
  }
  uint32_t confined = 0, outcome = APGAR_B200_CORRIDOR_NONE;
  if (n.corr.bits != nullptr) {
    uint32_t any = 0;
    for (int i = lane; i < 128; i += 32) any |= __ldg(n.corr.bits + i);
    confined = in_corridor(n.corr, n.win, n.sx, n.sy) && in_corridor(n.corr, n.win, n.win.gx, n.win.gy) ? 1u : 0u;
    // an empty bitmap proposes no corridor
    const bool proposed = __any_sync(kFull, any != 0u);
    outcome = confined != 0u ? APGAR_B200_CORRIDOR_CERTIFIED
                             : (proposed ? APGAR_B200_CORRIDOR_FALLBACK_UNREACHED : APGAR_B200_CORRIDOR_NONE);
  }
  __syncwarp();
  if (lane == 0) {
    const uint32_t h0 = bound_to_goal(p.lat, n.win, n.sl, n.sx, n.sy);
    st->head = 0u;
    st->tail = st->active = free_ends ? 1u : 0u;
    st->level_width = level_width;
    st->thr = h0 + min(level_width, kNoKey - h0);
    st->far_par = st->far_count[0] = st->far_count[1] = 0u;
    st->goal = kTileInf;
    st->limit = kNoLimit;
    st->start_key = h0;
    st->confined = confined;
    st->exit_key = kNoKey;
    st->corridor = outcome;
    st->stop = batch_cancelled(p) ? 1u : 0u;
    st->steps = st->units = st->levels = 0u;
    st->slot = slot;
    st->guests = 0u;
    __stcg(n.ws.pend + unpack_unit(n.win, n.start_unit).id, h0);
    __stcg(n.ws.ring, n.start_unit);
  }
  __threadfence();
  __syncwarp();
  if (lane == 0) *reinterpret_cast<volatile uint32_t*>(&st->phase) = free_ends ? 1u : 2u;
  __syncwarp();
  return free_ends;
}

// A net that may not be searched: its slot may still be written to.
__device__ __forceinline__ void reject_net(TileNetState* st, int lane) {
  if (lane == 0) {
    st->goal = kTileInf;
    st->stop = 2u;
    __threadfence();
    *reinterpret_cast<volatile uint32_t*>(&st->phase) = 2u;
  }
  __syncwarp();
}

// The net's result, and its path by the canonical walk.
template <bool kPriced>
__device__ __forceinline__ void finish_net(const TileLaunch& p, const TileNet& n, const TileNetState* st, bool free_ends, bool team,
                                           uint32_t net, uint32_t* tile, uint64_t* quads, uint32_t* prices, int lane) {
  const LatticeDeviceView& lat = p.lat;
  __threadfence();
  const uint32_t goal = peek(&st->goal), stop = peek(&st->stop);
  if (kPriced && stop == 3u) {  // for the cell form
    if (lane == 0) {
      NetPlan plan{};
      plan.net = net;
      // (the team class's nets come first among the plans, so here too)
      const uint32_t first = team || p.c[0].team == 0u ? 0u : p.c[0].end;
      p.redo[first + atomicAdd(p.redo_count + (team ? 0 : 1), 1u)] = plan;
    }
    return;
  }
  apgar_b200_lattice_result res{};
  res.cost = APGAR_B200_UNREACHABLE;
  res.completion = APGAR_B200_COMPLETION_DISCONNECTED;
  res.sweeps = peek(&st->units);
  res.row_steps = peek(&st->steps);
  res.row_stores = peek(&st->levels);
  if (!free_ends) {
    // no search: disconnected
  } else if (stop != 0u) {
    res.completion = stop == 1u ? APGAR_B200_COMPLETION_CANCELLED : APGAR_B200_COMPLETION_REJECTED;
  } else if (goal < kTileInf) {
    const unsigned long long bound = goal / min(lat.orth, min(lat.diag, lat.via)) + 1ull;
    unsigned long long base = 0;
    if (lane == 0) base = atomicAdd(p.arena_cursor, bound);
    base = __shfl_sync(kFull, base, 0);
    uint32_t len = 0;
    if (base + bound <= p.path_arena_capacity) {
      len = walk_path<kPriced>(p, n.win, n.ws, lane_part(n.win, lane), n.sl, n.sx, n.sy, goal, base, bound, tile, quads,
                               prices, lane);
    }
    res.completion = len != 0u ? APGAR_B200_COMPLETION_REACHED : APGAR_B200_COMPLETION_REJECTED;
    if (len != 0u) {
      res.cost = goal;
      res.path_len = len;
      res.arena_offset = base;
    }
  }
  if (lane == 0) {
    p.results[net] = res;
    if (p.corridor_status != nullptr) p.corridor_status[net] = static_cast<uint8_t>(peek(&st->corridor));
  }
}

// A kept route (partial rip-up): the net's previous result and path go into
// this execution.
__device__ __forceinline__ void keep_net(const TileLaunch& p, uint32_t net, int lane) {
  apgar_b200_lattice_result res = p.prev_results[net];
  res.arena_offset = 0;
  if (res.completion == APGAR_B200_COMPLETION_REACHED && res.path_len > 0) {
    unsigned long long base = 0;
    if (lane == 0) base = atomicAdd(p.arena_cursor, static_cast<unsigned long long>(res.path_len));
    base = __shfl_sync(kFull, base, 0);
    if (base + res.path_len > p.path_arena_capacity) {
      res.completion = APGAR_B200_COMPLETION_REJECTED;
      res.cost = APGAR_B200_UNREACHABLE;
      res.path_len = 0;
    } else {
      for (uint32_t j = lane; j < res.path_len; j += 32) p.path_arena[base + j] = p.prev_paths[res.path_offset + j];
      res.arena_offset = base;
    }
  }
  if (lane == 0) p.results[net] = res;
}

// Every warp takes nets, largest first, and relaxes their units.  A warp that
// finds no net left is a guest of other warps' nets: it relaxes their units
// until they have none to spare.  A guest may leave at any time: a net's
// owner finishes it alone.
template <bool kCheapDiagonal, bool kPriced, bool kCorr>
__global__ void __launch_bounds__(kTileThreads, kTileBlocks) lattice_tiles_kernel(const __grid_constant__ TileLaunch p) {
  extern __shared__ __align__(16) uint32_t tile_smem[];
  __shared__ Lookout look;
  const int lane = threadIdx.x & 31;
  // numbered across the CTAs: where the workspace is in slots, the warps that
  // own nets are spread over the SMs
  const uint32_t warp = (threadIdx.x >> 5) * gridDim.x + blockIdx.x;
  uint32_t* const tile = tile_smem + (threadIdx.x >> 5) * (kWarpWords + (kPriced ? kPriceWords : 0));
  uint64_t* const quads = reinterpret_cast<uint64_t*>(tile + kTileWords);
  uint32_t* const prices = tile + kWarpWords;
  if (threadIdx.x == 0) {
    look.probed = static_cast<uint32_t>(clock64());
    look.net = kNoKey;
    look.pause = kProbeClocks;
    look.places = look.over = 0u;
  }
  __syncthreads();
  int k = 0;
  uint32_t index = 0, low = 0, skip = 0;
  bool busy = false, owner = false, member = false, free_ends = false, kept = false, given_up = false;
  TileNetState* st = nullptr;
  TileNet n;
  LanePart part{};
  uint32_t turns = 0, idle = 0, misses = 0, seen = kNoKey;
  for (;;) {
    if (!busy) {
      owner = member = false;
      // the next net of the widest class that has one left: a team class's
      // net is the whole CTA's, its first warp's to start and to finish
      for (; k < 5; ++k) {
        index = kNoKey;
        if (p.c[k].team != 0u) {
          __syncthreads();
          if (threadIdx.x == 0) {
            look.team = blockIdx.x < p.c[k].slots ? p.c[k].begin + atomicAdd(p.c[k].next_plan, 1u) : kNoKey;
          }
          __syncthreads();
          index = look.team;
          if (index < p.c[k].end) {
            owner = threadIdx.x < 32;
            member = !owner;
            break;
          }
        } else if (warp < p.c[k].slots) {
          if (lane == 0) index = p.c[k].begin + atomicAdd(p.c[k].next_plan, 1u);
          index = __shfl_sync(kFull, index, 0);
          if (index < p.c[k].end) {
            owner = true;
            break;
          }
        }
      }
      if (k == 5) {
        if (__shfl_sync(kFull, peek(&look.over), 0) != 0u || ++idle > kIdleLimit) return;
        index = find_net(p, low, skip, look, lane);
        if (index == kNoKey) {
          __nanosleep(kNapNs);
          continue;
        }
        __threadfence();  // the net's set-up before its queue
      }
      st = p.states + index;
      const uint32_t place = k < 5 && p.c[k].team != 0u ? blockIdx.x : warp;
      n = net_at(p, index, k < 5 ? place : peek(&st->slot));
      part = lane_part(n.win, lane);
      kept = p.skip != nullptr && k < 5 && p.skip[p.plans[index].net] != 0u;
      if (owner && kept) {
        keep_net(p, p.plans[index].net, lane);
        if (lane == 0) *reinterpret_cast<volatile uint32_t*>(&st->phase) = 2u;
        __syncwarp();
      } else if (owner) {
        if (p.per_net == 0u && __shfl_sync(kFull, peek(p.finished + 1), 0) != 0u) {
          reject_net(st, lane);
          free_ends = true;
        } else {
          free_ends = start_net(p, n, st, p.c[k].level_width, place, p.plans[index].net, lane);
        }
      }
      if (k < 5 && p.c[k].team != 0u) __syncthreads();  // the team waits for the net's set-up
      if (k == 5) {
        if (lane == 0) atomicAdd(&st->guests, 1u);
        __syncwarp();
      }
      busy = true;
      given_up = false;
      idle = misses = 0;
      seen = kNoKey;
    }
    if (owner && p.cancel != nullptr && (++turns % kCancelPollTurns) == 0u) {
      if (lane == 0 && batch_cancelled(p)) atomicMax(&st->stop, 1u);
      __syncwarp();
    }
    const uint32_t unit = pop_unit(st, n.ws, lane);
    if (unit != kEmptySlot) {
      relax_unit<kCheapDiagonal, kPriced, kCorr>(p, n.win, n.ws, unit, part, n.start_unit, n.start_cell, n.goal_unit,
                                                 n.goal_cell, st, n.corr, tile, prices, lane);
      __syncwarp();
      idle = misses = 0;
      continue;
    }
    const bool done = __shfl_sync(kFull, peek(&st->phase), 0) != 1u;
    if (member) {
      if (done || ++misses > kIdleLimit) {
        busy = false;
        continue;
      }
    } else if (!owner) {
      if (done || ++misses > kGuestMisses) {
        if (lane == 0) atomicSub(&st->guests, 1u);
        __syncwarp();
        busy = false;
        continue;
      }
    } else if (!done && idle > kIdleLimit && !given_up) {
      // Nothing finishes.  The net is rejected, once its units have drained
      // (each ends at once now): another warp may still be in one.
      if (lane == 0) atomicMax(&st->stop, 2u);
      __syncwarp();
      given_up = true;
      idle = 0u;
    } else if (done || idle > kIdleLimit) {
      if (!done && lane == 0) {
        // Given up for good: a warp that never left a unit may still write to
        // the net's workspace, so no later net takes a slot.
        *reinterpret_cast<volatile uint32_t*>(p.finished + 1) = 1u;
        *reinterpret_cast<volatile uint32_t*>(&st->phase) = 2u;
        __threadfence();
      }
      __syncwarp();
      if (!kept) finish_net<kPriced>(p, n, st, free_ends, p.c[k].team != 0u, p.plans[index].net, tile, quads, prices, lane);
      __syncwarp();
      if (lane == 0 && atomicAdd(p.finished, 1u) + 1u >= p.total) *reinterpret_cast<volatile uint32_t*>(&look.over) = 1u;
      __syncwarp();
      busy = false;
      continue;
    } else {
      const uint32_t progress = __shfl_sync(kFull, peek(&st->units), 0);
      idle = progress != seen ? 0u : idle + 1u;
      seen = progress;
    }
    __nanosleep(kNapNs);
  }
}

constexpr int tile_smem_bytes(bool priced) {
  return kTileThreads / 32 * (kWarpWords + (priced ? kPriceWords : 0)) * 4;
}

using TileKernel = void (*)(TileLaunch);

template <bool kCheapDiagonal>
TileKernel tile_kernel(bool priced, bool corridor) {
  if (corridor) return priced ? lattice_tiles_kernel<kCheapDiagonal, true, true> : lattice_tiles_kernel<kCheapDiagonal, false, true>;
  return priced ? lattice_tiles_kernel<kCheapDiagonal, true, false> : lattice_tiles_kernel<kCheapDiagonal, false, false>;
}

TileKernel tile_kernel(bool cheap_diagonal, bool priced, bool corridor) {
  return cheap_diagonal ? tile_kernel<true>(priced, corridor) : tile_kernel<false>(priced, corridor);
}

// CTAs per SM that every form of the kernel can keep resident.
std::atomic<int> g_tile_blocks[64];

cudaError_t tile_blocks_per_sm(int* out) {
  int device = 0;
  if (cudaError_t e = cudaGetDevice(&device); e != cudaSuccess) return e;
  const bool cacheable = device >= 0 && device < 64;
  if (cacheable) {
    const int cached = g_tile_blocks[device].load(std::memory_order_acquire);
    if (cached > 0) {
      *out = cached;
      return cudaSuccess;
    }
  }
  int least = kTileBlocks;
  for (int form = 0; form < 8; ++form) {
    const bool priced = (form & 2) != 0;
    const void* kernel = reinterpret_cast<const void*>(tile_kernel((form & 1) != 0, priced, (form & 4) != 0));
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, tile_smem_bytes(priced));
    int blocks = 0;
    if (e == cudaSuccess) {
      e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, kernel, kTileThreads, tile_smem_bytes(priced));
    }
    if (e != cudaSuccess) return e;
    least = std::min(least, blocks);
  }
  *out = std::max(1, least);
  if (cacheable) g_tile_blocks[device].store(*out, std::memory_order_release);
  return cudaSuccess;
}

}  // namespace

// Words of one net's workspace: labels, four words per unit and the ring.
uint64_t lattice_tile_words(int layers, uint32_t win_w, uint32_t win_h) {
  const uint64_t units = static_cast<uint64_t>(layers) * ((win_w + 31u) / 32u) * ((win_h + 31u) / 32u);
  return (units * 1028u + ring_slots(static_cast<uint32_t>(units)) + 31u) & ~31ull;
}

// Warps of a launch: every one that can be resident at once.
cudaError_t lattice_tile_warps(int sm_count, uint32_t* out) {
  int blocks = 0;
  if (cudaError_t e = tile_blocks_per_sm(&blocks); e != cudaSuccess) return e;
  *out = static_cast<uint32_t>(blocks) * static_cast<uint32_t>(std::max(1, sm_count)) * (kTileThreads / 32);
  return cudaSuccess;
}

cudaError_t launch_lattice_tiles(const TileLaunch& launch, int sm_count, cudaStream_t stream) {
  if (launch.total == 0) return cudaSuccess;
  uint32_t warps = 0;
  if (cudaError_t e = lattice_tile_warps(sm_count, &warps); e != cudaSuccess) return e;
  // A CTA for every eight units: more would only wait for the end (one net of
  // 4 x 4 cells: 52 us with all of them).
  const unsigned grid = static_cast<unsigned>(std::min<uint64_t>(warps, launch.units + 7u) / (kTileThreads / 32));
  const bool priced = launch.cell_cost != nullptr;
  const TileKernel kernel = tile_kernel(launch.lat.diag < launch.lat.orth, priced, launch.corridor != nullptr);
  kernel<<<grid, kTileThreads, tile_smem_bytes(priced), stream>>>(launch);
  return cudaGetLastError();
}

}  // namespace apgar_b200
