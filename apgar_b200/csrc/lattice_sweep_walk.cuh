// The end of both sweep kernels: the net's record and, from exact labels, its
// path, by the net's first warp.  Text, included where it is wanted: a function
// called at the end of the form with a warp a layer made the allocation-free
// call on 96 planar nets 0.6% longer (529 and 532 us).
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
