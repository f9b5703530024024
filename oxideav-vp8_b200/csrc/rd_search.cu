// rd_search.cu — the RD-effort inter search of decide_mb_rd
// (src/encoder/inter_search.rs:846-1060) for every MB of a frame.
//
// vp8a_rd_inter_search takes each MB's census neighbours as input, so all
// MBs are independent: one warp per MB, four warps per CTA. Per reference
// the warp runs whole_pixel_search (seeds, then the WIDE 8-point and NARROW
// 4-point descents on SAD + sqrt(lambda) * MV bits, :380-495), then for the
// leader (and, by effort, the runner-up) sub_pixel_refine (shared half-pel
// planes over the staged window plus four quarter-pel six-tap probes,
// :499-552) and the free ZERO / NEAREST / NEAR candidates; the cheapest
// candidate wins with the reference's strict '<'. MV rates are the
// reference's f32 table values (MvCostTable, :166-194): each component's
// f64 bit count rounded to f32, summed in f32, widened. The SAD early exits
// of whole_sad never change an outcome (an exiting candidate is rejected
// either way), so SADs are computed in full.
//
// What bounds it: each warp's chain of descent rounds (8160 warps at 1080p, about
// 55 an SM). A round's points do not depend on one another, and the reference's
// walk over them keeps the first smallest cost: so a round (or the seeds) takes
// all its SADs together from a staged window, two blocks a pass, lane q computes
// point q's cost, and one reduction finds the winner. (The same pairs read from
// the plane keep the L1 pipe 60 % busy, a line a lane: 292 us.) The quarter-pel
// probes share two six-tap planes as the half-pel ones do. Measured (1080p, three
// references, BALANCED effort): 657 us with byte loads and one point at a time,
// 149 us now.
#include "census.cuh"

namespace {
using namespace vp8a_dev;

struct Shape {
  uint32_t descent_rounds;
  int wide_pattern, half_diagonals, quarter, search_other_refs, refine_runner_up;
  unsigned long long split_gate;
};

// EncodeEffort::inter_shape (src/encoder/inter_search.rs:93-161), the
// fields this search reads.
Shape shape_for(uint32_t effort) {
  switch (effort) {
    case VP8A_EFFORT_FASTEST: return Shape{4, 0, 1, 0, 0, 0, ~0ull};
    case VP8A_EFFORT_FAST: return Shape{8, 1, 1, 1, 1, 0, ~0ull};
    case VP8A_EFFORT_BALANCED: return Shape{16, 1, 1, 1, 1, 1, 4ull};
    default: return Shape{32, 1, 1, 1, 1, 1, 0ull};
  }
}

constexpr int RD_WARPS = 4;
constexpr int MAX_REFS = 3;

struct RdArgs {
  const uint8_t* fy;
  uint64_t fys;
  int fw, fh;
  MePlane refs[MAX_REFS];
  uint8_t ref_ids[MAX_REFS];
  int n_refs;
  int mb_cols, mb_rows;
  vp8a_mv_contexts ctx;
  double lambda_sad;
  uint32_t good_enough;
  Shape shape;
  const double* bit_cost;
  const double* mvbits;  // mv_component_bits per context and value (2 x 2047)
  const MbInfoDev* nb;
  vp8a_rd_inter* out;
};

struct Found {
  vp8a_mv mv;
  uint32_t sad;
  double cost;
};

struct RdCensus {
  vp8a_mv best, nearest, near_;
  double mode_bits[5];
};

// MvCostTable::bits: f32 component costs summed in f32; false when the
// differential leaves [-1023, 1023].
__device__ __forceinline__ bool cost_bits(const double* mvb, vp8a_mv mv, vp8a_mv base, double* out) {
  const int dr = mv.row - base.row, dc = mv.col - base.col;
  if (dr < -1023 || dr > 1023 || dc < -1023 || dc > 1023) return false;
  const float s = (float)mv_bits_lookup(mvb, 0, dr) + (float)mv_bits_lookup(mvb, 1, dc);
  *out = (double)s;
  return true;
}

// Lane q's point (its vector, its SAD, whether it counts), for all lanes in order,
// each kept when its cost is below the best: the first smallest of them, if below.
// A point's cost is at least its rate, so the reference's early exit on the rate
// never decides. Costs are sums of non-negative terms: their order is that of
// their bits (a NaN, from a NaN lambda, is above all and never below the best).
__device__ __forceinline__ bool keep_first(const RdArgs& a, vp8a_mv base, double ls, Found& best, vp8a_mv mv,
                                           uint32_t sad, bool counts) {
  double bits, cost = __longlong_as_double(0x7ff0000000000000LL);
  if (counts && cost_bits(a.mvbits, mv, base, &bits)) cost = (double)sad + ls * bits;
  const uint32_t hi = (uint32_t)__double2hiint(cost), lo = (uint32_t)__double2loint(cost);
  const uint32_t mhi = __reduce_min_sync(FULL, hi), mlo = __reduce_min_sync(FULL, hi == mhi ? lo : ~0u);
  const int q = __ffs(__ballot_sync(FULL, hi == mhi && lo == mlo)) - 1;
  const double c = __hiloint2double((int)mhi, (int)mlo);
  if (!(c < best.cost)) return false;
  best.cost = c;
  best.sad = __shfl_sync(FULL, sad, q);
  best.mv.row = (int16_t)__shfl_sync(FULL, (int)mv.row, q);
  best.mv.col = (int16_t)__shfl_sync(FULL, (int)mv.col, q);
  return true;
}

__global__ void __launch_bounds__(RD_WARPS * 32) rd_search_kernel(RdArgs a) {
  __shared__ WarpScratch scratch[RD_WARPS];
  __shared__ __align__(16) uint8_t srcs[RD_WARPS][256];
  __shared__ double bit_cost[256];
  for (int i = threadIdx.x; i < 256; i += blockDim.x) bit_cost[i] = a.bit_cost[i];
  __syncthreads();
  const double* t = bit_cost;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int idx = blockIdx.x * RD_WARPS + warp;
  if (idx >= a.mb_cols * a.mb_rows) return;
  const int mb_row = idx / a.mb_cols, mb_col = idx - mb_row * a.mb_cols;
  WarpScratch& S = scratch[warp];
  uint8_t* src = srcs[warp];
  {
    // Eight source pixels a lane, edge-clamped.
    const int y = min(mb_row * 16 + (lane >> 1), a.fh - 1), x = mb_col * 16 + (lane & 1) * 8;
    const uint8_t* p = a.fy + (size_t)y * a.fys;
    uint32_t v[2] = {0, 0};
    if ((((uintptr_t)a.fy | a.fys) & 3) == 0 && x + 8 <= a.fw) {
      v[0] = __ldg((const uint32_t*)(p + x));
      v[1] = __ldg((const uint32_t*)(p + x) + 1);
    } else {
#pragma unroll
      for (int i = 0; i < 8; i++) v[i >> 2] |= (uint32_t)p[min(x + i, a.fw - 1)] << (8 * (i & 3));
    }
    *(uint2*)(src + lane * 8) = make_uint2(v[0], v[1]);
  }
  __syncwarp();
  const MbInfoDev above = a.nb[3 * idx], left = a.nb[3 * idx + 1], al = a.nb[3 * idx + 2];
  const int ox = mb_col * 16, oy = mb_row * 16;
  const int to_left = -((mb_col + 1) << 6), to_right = (a.mb_cols - mb_col) << 6;
  const int to_top = -((mb_row + 1) << 6), to_bottom = (a.mb_rows - mb_row) << 6;
  const int rx0 = max(to_left / 4, -255), rx1 = min(to_right / 4, 255);
  const int ry0 = max(to_top / 4, -255), ry1 = min(to_bottom / 4, 255);
  const uint32_t ge = a.good_enough;
  const double ls = a.lambda_sad;
  // The census does not depend on the reference (default sign bias).
  const Census cn = census(above, left, al, mb_col, mb_row, a.mb_cols, a.mb_rows);
  RdCensus cs;
  cs.best = cn.best_predictor;
  cs.nearest = cn.nearest;
  cs.near_ = cn.near_;
  for (int m = 0; m < 5; m++) {  // the `tree` closure (:905-914)
    double bits = 0.0;
    for (int q = 0; q < m; q++) bits += bb(t, cn.p[q], 1);
    if (m < 4) bits += bb(t, cn.p[m], 0);
    cs.mode_bits[m] = bits;
  }
  vp8a_rd_inter o;
  memset(&o, 0, sizeof o);
  for (int k = 0; k < 3; k++) {
    o.found[k].mv = vp8a_mv{0, 0};
    o.found[k].sad = 0xffffffffu;
  }
  Found found[MAX_REFS];
  double total[MAX_REFS];
  bool have[MAX_REFS] = {false, false, false};
  int leader = 0;
  double leader_cost = __longlong_as_double(0x7ff0000000000000LL);
  const double INF = __longlong_as_double(0x7ff0000000000000LL);

  int wx0 = -(1 << 28), wy0 = -(1 << 28), win_ref = -1;  // the window, and whose it is
  for (int n = 0; n < a.n_refs; n++) {
    const MePlane& P = a.refs[n];
    const uint8_t id = a.ref_ids[n];
    // whole_pixel_search (:380-495).
    Found best = {{0, 0}, 0xffffffffu, INF};
    // The SADs of points 0 .. m - 1 (m <= 8; lane q holds point q and whether it
    // counts), from the window where it covers them all.
    auto point_sads = [&](int px, int py, bool counts, int m) -> uint32_t {
      const int lx = ox + px - wx0, ly = oy + py - wy0;
      unsigned todo = __ballot_sync(FULL, counts && lane < m);
      uint32_t sad = 0;
      if (__all_sync(FULL, !(counts && lane < m) || (lx >= 0 && ly >= 0 && lx <= WS - 16 && ly <= WS - 16))) {
#pragma unroll 2
        for (int p = 0; p < m; p += 2) {
          // A point that does not count reads the window's corner.
          const int at = counts && lane < m ? ly << 16 | lx : 0;
          const int s0 = __shfl_sync(FULL, at, p), s1 = __shfl_sync(FULL, at, p + 1);
          const uint32_t both = sad_win16_pair(S.win, s0 & 0xffff, s0 >> 16, s1 & 0xffff, s1 >> 16, src, lane);
          if ((lane & ~1) == p) sad = (lane & 1) ? both >> 16 : both & 0xffffu;
        }
        return sad;
      }
#pragma unroll 1
      for (; todo; todo &= todo - 1) {
        const int q = __ffs(todo) - 1;
        const uint32_t s = sad_whole_at(P, S.win, wx0, wy0, ox + __shfl_sync(FULL, px, q),
                                        oy + __shfl_sync(FULL, py, q), src, lane);
        if (lane == q) sad = s;
      }
      return sad;
    };
    // Lane q's seed, snapped and clamped; a point tried before does not count.
    int len = 4;
    vp8a_mv seed = lane == 1 ? cs.nearest : (lane == 2 ? cs.near_ : (lane == 3 ? cs.best : vp8a_mv{0, 0}));
    if (left.ref_frame == id) {
      if (lane == len) seed = left.mv;
      len++;
    }
    if (above.ref_frame == id) {
      if (lane == len) seed = above.mv;
      len++;
    }
    // The seeds, then the rounds of the WIDE descent (offsets (-2,0) (2,0) (0,-2)
    // (0,2) (-1,-1) (1,-1) (-1,1) (1,1)) and of the NARROW one ((-1,0) (1,0) (0,-1)
    // (0,1)); one call site for the three keeps the kernel's code small.
    int px = clampi((seed.col + 2) >> 2, rx0, rx1), py = clampi((seed.row + 2) >> 2, ry0, ry1);
    const unsigned same = __match_any_sync(FULL, (py << 16) ^ (px & 0xffff));
    bool counts = (same & ((1u << lane) - 1u)) == 0;
    int m = len, phase = 0;
    uint32_t rounds = a.shape.descent_rounds;
    const int cx0 = __shfl_sync(FULL, px, 3), cy0 = __shfl_sync(FULL, py, 3);
    wx0 = ox + cx0 - WIN_LEAD;
    wy0 = oy + cy0 - WIN_LEAD;
    load_window(P, S.win, wx0, wy0, lane);
    __syncwarp();
    for (;;) {
      vp8a_mv mv;
      mv.row = (int16_t)(py * 4);
      mv.col = (int16_t)(px * 4);
      const bool improved = keep_first(a, cs.best, ls, best, mv, point_sads(px, py, counts, m), counts && lane < m);
      if (phase == 0) {
        if (!(n == 0 || a.shape.search_other_refs) || best.sad <= ge) break;
        phase = a.shape.wide_pattern && (unsigned long long)best.sad > 4ull * ge ? 1 : 2;
      } else if (phase == 1) {
        if (best.sad <= ge) break;
        if (--rounds == 0 || !improved) {
          phase = 2;
          rounds = a.shape.descent_rounds;
        }
      } else if (--rounds == 0 || !improved || best.sad <= ge) {
        break;
      }
      const int cx = best.mv.col / 4, cy = best.mv.row / 4;
      if (abs(ox + cx - WIN_LEAD - wx0) > WIN_LEAD - 2 || abs(oy + cy - WIN_LEAD - wy0) > WIN_LEAD - 2) {
        // The round would leave the window: another around its centre.
        wx0 = ox + cx - WIN_LEAD;
        wy0 = oy + cy - WIN_LEAD;
        __syncwarp();
        load_window(P, S.win, wx0, wy0, lane);
        __syncwarp();
      }
      if (phase == 1) {
        px = cx + (lane < 2 ? 4 * lane - 2 : (lane < 4 ? 0 : 2 * (lane & 1) - 1));
        py = cy + (lane < 2 ? 0 : (lane < 4 ? 4 * lane - 10 : (lane < 6 ? -1 : 1)));
        m = 8;
      } else {
        px = cx + (lane < 2 ? 2 * lane - 1 : 0);
        py = cy + (lane < 2 ? 0 : 2 * lane - 5);
        m = 4;
      }
      counts = px >= rx0 && px <= rx1 && py >= ry0 && py <= ry1;
    }
    win_ref = n;
    found[n] = best;
    // ref_frame_tree_bits(ref, 128, 128) (src/encoder.rs:9108).
    const double rbits = id == VP8A_REF_LAST ? bb(t, 128, 0)
                         : id == VP8A_REF_GOLDEN ? bb(t, 128, 1) + bb(t, 128, 0)
                                                 : bb(t, 128, 1) + bb(t, 128, 1);
    total[n] = best.cost + ls * rbits;
    if (total[n] < leader_cost) {
      leader_cost = total[n];
      leader = n;
    }
    have[n] = true;
    o.found[n].mv = best.mv;
    o.found[n].sad = best.sad;
    o.n_searched = (uint8_t)(n + 1);
    if (best.sad <= ge) break;
  }

  bool have_best = false;
  double best_cost = 0.0;
  for (int n = 0; n < a.n_refs; n++) {
    if (!have[n]) continue;
    const bool refine = n == leader || (a.shape.refine_runner_up &&
                                        (a.shape.split_gate == 0ull || total[n] < leader_cost * 1.125));
    if (!refine) continue;
    const MePlane& P = a.refs[n];
    const uint8_t id = a.ref_ids[n];
    const double ref_bits = id == VP8A_REF_LAST ? bb(t, 128, 0)
                            : id == VP8A_REF_GOLDEN ? bb(t, 128, 1) + bb(t, 128, 0)
                                                    : bb(t, 128, 1) + bb(t, 128, 1);
    Found f = found[n];
    if (f.sad > ge / 2) {
      // sub_pixel_refine (:499-552): window around the whole-pel start.
      const int fx = ox + f.mv.col / 4 - WIN_LEAD, fy = oy + f.mv.row / 4 - WIN_LEAD;
      if (win_ref != n || abs(fx - wx0) > WIN_LEAD - 4 || abs(fy - wy0) > WIN_LEAD - 4) {
        wx0 = fx;
        wy0 = fy;
        win_ref = n;
        __syncwarp();
        load_window(P, S.win, wx0, wy0, lane);
        __syncwarp();
      }
      uint32_t hs[8], sad = 0;
      half_plane_sads(S, wx0, wy0, ox, oy, f.mv, src, lane, hs);
#pragma unroll
      for (int k = 0; k < 8; k++)
        if (lane == k) sad = hs[k];
      // Lane k's half-pel candidate.
      vp8a_mv mv;
      const int dy = cand_dr(lane & 7), dx = cand_dc(lane & 7);
      mv.row = (int16_t)(f.mv.row + 2 * dy);
      mv.col = (int16_t)(f.mv.col + 2 * dx);
      keep_first(a, cs.best, ls, f, mv, sad,
                 lane < 8 && (a.shape.half_diagonals || dx == 0 || dy == 0) && abs((int)mv.row) <= 1020 &&
                     abs((int)mv.col) <= 1020);
      if (a.shape.quarter) {
        // Candidates (-1,0) (1,0) (0,-1) (0,1): 3 and 4, 1 and 6 of the eight
        // around the centre share planes where the window covers them.
        const vp8a_mv centre = f.mv;
        mv.row = (int16_t)(centre.row + (lane < 2 ? 0 : 2 * (lane & 1) - 1));
        mv.col = (int16_t)(centre.col + (lane < 2 ? 2 * lane - 1 : 0));
        if (quarter_inside(centre, ox, oy, wx0, wy0)) {
          int iy0, fr;
          quarter_pos(centre.row - 1, oy, wy0, iy0, fr);
          iy0 -= 2;
          auto taps = [](int x) { return taps_const(x); };
          quarter_planes_h(S.win, S.temp, taps, centre, ox, wx0, iy0, lane, 32);
          __syncwarp();
          const uint32_t h = quarter_pair_sads(S.temp, src, taps, centre, oy, wy0, iy0, lane < 16 ? 3 : 4, lane);
          const uint32_t v = quarter_pair_sads(S.temp, src, taps, centre, oy, wy0, iy0, lane < 16 ? 1 : 6, lane);
          const uint32_t both = lane < 2 ? h : v;
          sad = (lane & 1) ? both >> 16 : both & 0xffffu;
          __syncwarp();
        } else {
#pragma unroll 1
          for (int k = 0; k < 4; k++) {
            const uint32_t s = sad_at_mv(P, S, wx0, wy0, ox, oy, (int16_t)__shfl_sync(FULL, (int)mv.row, k),
                                         (int16_t)__shfl_sync(FULL, (int)mv.col, k), src, lane);
            if (lane == k) sad = s;
          }
        }
        keep_first(a, cs.best, ls, f, mv, sad, lane < 4 && abs((int)mv.row) <= 1022 && abs((int)mv.col) <= 1022);
      }
    }
    const vp8a_mv zero = {0, 0};
    int mode;
    double mode_bits;
    if (mv_eq(f.mv, zero)) {
      mode = VP8A_MODE_ZERO;
      mode_bits = cs.mode_bits[0];
    } else if (mv_eq(f.mv, cs.nearest)) {
      mode = VP8A_MODE_NEAREST;
      mode_bits = cs.mode_bits[1];
    } else if (mv_eq(f.mv, cs.near_)) {
      mode = VP8A_MODE_NEAR;
      mode_bits = cs.mode_bits[2];
    } else {
      double diff = 0.0;
      cost_bits(a.mvbits, f.mv, cs.best, &diff);
      mode = VP8A_MODE_NEW;
      mode_bits = cs.mode_bits[3] + diff;
    }
    auto consider = [&](int md, vp8a_mv mv, uint32_t sad, double bits) {
      const double cost = (double)sad + ls * bits;
      if (!have_best || cost < best_cost) {
        have_best = true;
        best_cost = cost;
        o.ref_frame = id;
        o.mode = (uint8_t)md;
        o.mv = mv;
        o.sad = sad;
        o.cost = cost;
        o.bits = bits;
      }
    };
    consider(mode, f.mv, f.sad, ref_bits + mode_bits);
    const vp8a_mv fm[3] = {zero, cs.nearest, cs.near_};
    // The window serves them when it is this reference's.
    const int vx0 = win_ref == n ? wx0 : -(1 << 28), vy0 = win_ref == n ? wy0 : -(1 << 28);
#pragma unroll 1
    for (int k = 0; k < 3; k++) {
      if (k == 1 && mv_eq(cs.nearest, zero)) continue;
      if (k == 2 && (mv_eq(cs.near_, zero) || mv_eq(cs.near_, cs.nearest))) continue;
      const vp8a_mv mv = fm[k];
      if (mv_eq(mv, f.mv)) continue;
      const uint32_t sad = ((mv.row & 3) == 0 && (mv.col & 3) == 0)
                               ? sad_whole_at(P, S.win, vx0, vy0, ox + mv.col / 4, oy + mv.row / 4, src, lane)
                               : sad_at_mv(P, S, vx0, vy0, ox, oy, mv.row, mv.col, src, lane);
      consider(k, mv, sad, ref_bits + cs.mode_bits[k]);
    }
  }
  o.leader = (uint8_t)leader;
  if (lane == 0) a.out[idx] = o;
}

}  // namespace

extern "C" vp8a_status vp8a_rd_inter_search(vp8a_ctx* ctx, const vp8a_i420* frame, const vp8a_planes* refs,
                                            const uint8_t* ref_ids, uint32_t n_refs,
                                            const vp8a_mv_contexts* mv_contexts, double lambda, uint32_t y1_ac,
                                            uint32_t effort, const vp8a_mb_info* neighbours, vp8a_rd_inter* out) {
  if (!ctx || !frame || !refs || !ref_ids || !neighbours || !out) {
    vp8a::set_error("null argument");
    return VP8A_E_INVALID_ARGUMENT;
  }
  if (frame->width == 0 || frame->height == 0 || frame->width > 0x3FFF || frame->height > 0x3FFF) {
    vp8a::set_error("invalid dimensions");
    return VP8A_E_INVALID_DIMENSIONS;
  }
  if (n_refs == 0 || n_refs > (uint32_t)MAX_REFS || effort > VP8A_EFFORT_THOROUGH) {
    vp8a::set_error("n_refs must be 1..3 and effort a VP8A_EFFORT_* value");
    return VP8A_E_INVALID_ARGUMENT;
  }
  const int mb_cols = (int)((frame->width + 15) / 16), mb_rows = (int)((frame->height + 15) / 16);
  VP8A_CUDA(cudaSetDevice(ctx->device));
  vp8a::Stager st(ctx);
  vp8a_status s;
  uint8_t ids[MAX_REFS];
  if ((s = st.read_to_host(ref_ids, n_refs, ids)) != VP8A_OK) return s;
  for (uint32_t k = 0; k < n_refs; k++) {
    if ((int)refs[k].mb_cols != mb_cols || (int)refs[k].mb_rows != mb_rows) {
      vp8a::set_error("reference planes do not match the frame's MB grid");
      return VP8A_E_REFERENCE_DIMENSIONS_MISMATCH;
    }
    if (ids[k] < VP8A_REF_LAST || ids[k] > VP8A_REF_ALTREF || !refs[k].y || refs[k].y_stride < (uint64_t)mb_cols * 16) {
      vp8a::set_error("bad reference id, plane or stride");
      return VP8A_E_INVALID_ARGUMENT;
    }
  }
  if (!frame->y || frame->y_stride < frame->width) {
    vp8a::set_error("bad source plane");
    return VP8A_E_INVALID_ARGUMENT;
  }
  RdArgs a{};
  const void* d;
  if ((s = st.in(frame->y, frame->y_stride * (size_t)(frame->height - 1) + frame->width, &d)) != VP8A_OK) return s;
  a.fy = (const uint8_t*)d;
  a.fys = frame->y_stride;
  a.fw = (int)frame->width;
  a.fh = (int)frame->height;
  for (uint32_t k = 0; k < n_refs; k++) {
    const size_t bytes = refs[k].y_stride * (size_t)(mb_rows * 16 - 1) + (size_t)mb_cols * 16;
    if ((s = st.in(refs[k].y, bytes, &d)) != VP8A_OK) return s;
    a.refs[k] = MePlane{(const uint8_t*)d, refs[k].y_stride, mb_cols * 16, mb_rows * 16};
    a.ref_ids[k] = ids[k];
  }
  a.n_refs = (int)n_refs;
  a.mb_cols = mb_cols;
  a.mb_rows = mb_rows;
  if (mv_contexts) {
    a.ctx = *mv_contexts;
  } else {
    static const uint8_t dflt[2][19] = {
        {162, 128, 225, 146, 172, 147, 214, 39, 156, 128, 129, 132, 75, 145, 178, 206, 239, 254, 254},
        {164, 128, 204, 170, 119, 235, 140, 230, 228, 128, 130, 130, 74, 148, 180, 203, 236, 254, 254}};
    memcpy(a.ctx.p, dflt, sizeof dflt);
  }
  // decide_mb_rd (:850-866): sqrt(lambda), good_enough from y1_ac.
  a.lambda_sad = std::sqrt(lambda);
  const uint32_t qpix = std::max(y1_ac / 8u, 1u);
  a.good_enough = 256u * qpix / 2u;
  a.shape = shape_for(effort);
  a.bit_cost = ctx->d_bit_cost;
  const size_t nmb = (size_t)mb_cols * mb_rows;
  if ((s = st.in(neighbours, sizeof(vp8a_mb_info) * nmb * 3, &d)) != VP8A_OK) return s;
  a.nb = (const MbInfoDev*)d;
  void *dout, *dmvb;
  if ((s = st.out(out, sizeof(vp8a_rd_inter) * nmb, &dout)) != VP8A_OK) return s;
  a.out = (vp8a_rd_inter*)dout;
  if ((s = st.scratch(sizeof(double) * 2 * MV_BITS_SPAN, &dmvb)) != VP8A_OK) return s;
  mv_bits_table_kernel<<<(2 * MV_BITS_SPAN + 255) / 256, 256, 0, ctx->stream>>>(ctx->d_bit_cost, a.ctx,
                                                                               (double*)dmvb);
  VP8A_CUDA(cudaGetLastError());
  ctx->launches++;
  a.mvbits = (const double*)dmvb;
  rd_search_kernel<<<vp8a::grid_for(nmb, RD_WARPS), RD_WARPS * 32, 0, ctx->stream>>>(a);
  VP8A_CUDA(cudaGetLastError());
  ctx->launches++;
  return st.finish();
}
