// lf.cu — §15 loop filter and the §9.4 (level, sharpness) search.
//
// Entry points:
//   vp8a_filter_frame                  filter_inter_frame_flags / filter_frame_flags
//                                      (src/loop_filter.rs:1364, :2506), in place
//   vp8a_reconstruction_ssd            (src/loop_filter.rs:1965)
//   vp8a_filter_sweep                  score_filter_candidate (:2062) for all 64 x 8
//   vp8a_select_filter_params          select_filter_params_threaded (:2133)
//   vp8a_select_filter_params_sampled  select_filter_params_sampled (:2288)
//
// Kernel design. A pass filters the picture for one (level, sharpness)
// candidate and adds its visible-window SSD against the source to the
// candidate's table entries. Luma and chroma never read each other, so a pass
// may take both or one of them. The §15 raster order makes MB (r, c) depend on
// (r, c-1) and (r-1, c+1) (the filter never writes right of or below the MB it
// processes): MBs run as a wavefront of steps, eight lanes an MB. A row keeps
// its last three MBs in a ring of shared-memory slots: an MB is read from the
// unfiltered reconstruction when its step comes, and is scored against the
// source (or written back) once no later MB writes it, when its slot is
// refilled. The picture therefore crosses HBM once per call, as a copy into MB
// tiles that all passes read from L2, and no filtered copy of the planes is
// ever materialised.
//
// Bound: the integer ALU (min/max, absolute difference, byte permute and
// logic run at 64 lanes a clock per SM; multiply-adds have a pipe of their
// own). Every lane therefore filters two pixels per instruction: taps are
// pairs of 16-bit fields (two rows for the vertical edges, two columns for
// the horizontal ones), clamps are single add-min-relu instructions, and the
// filters' (27 w + 63) >> 7 family is a multiply by a pre-scaled constant
// whose high byte a byte permute picks. The 64 x 8 grid over 1920x1080 (436
// passes) took 3.30 ms with one pixel per lane and instruction, 2.35 ms so
// paired, 1.27 ms with the rows read from tiles (ncu: 56 % of the issue slots
// and of the ALU's cycles, the rest mostly waiting at the step barriers for
// the MBs with inner edges).
//
// Parallelism. A grid of candidates fills the GPU with one CTA per pass. The
// selection walk's few candidates, and the single pass that filters a frame,
// would leave most SMs idle with the chain of steps exposed, so such a pass is
// split into bands of rows over a thread-block cluster whose CTAs hand each
// other the rows at their seams (filtering one 1280x720 frame: 0.88 ms in one
// CTA before, 0.14 ms; 3840x2160: 7.0 and 0.47 ms).
//
// The sampled search's two-row bands are rows whose steps restart at 0 and
// whose first row has no top edge.
#include <cooperative_groups.h>

#include <algorithm>
#include <mutex>

#include "vp8a_internal.cuh"

namespace {
using namespace vp8a_dev;
namespace cg = cooperative_groups;
constexpr unsigned FULL = 0xffffffffu;

// Wavefront. A whole pass runs MB (r, c)'s vertical and then its horizontal
// edges at step 2 r + c, one barrier a step: MB (r - 1, c + 1) ran the step
// before. A split pass, which is bound by the length of its chain of steps,
// runs at step r + c, all vertical edges before all horizontal ones: the
// horizontal edges of (r, c) need only the vertical ones of (r - 1, c + 1).
__host__ __device__ constexpr int skew_of(int split) { return split > 1 ? 1 : 2; }

// Slots per MB row: MB (r, c) takes slot c % 3 once MB (r, c - 3) is final and
// scored. In a whole pass MB (r, c - 3)'s last writer, MB (r + 1, c - 3), ran
// the step before; while MB (r, c) runs, row r - 1 runs (r - 1, c + 2) and row
// r + 1 runs (r + 1, c - 2): the slots they touch are never the one being
// refilled. In a split pass the last writer ran two steps before.
constexpr int RING = 3;

// Lanes per MB, MBs per warp.
constexpr int LPM = 8, MPW = 32 / LPM;
// CTAs of a split pass: 8 is the portable cluster size; 16 only where a CTA
// could not hold its rows otherwise (pictures over 8192 rows).
constexpr int MAX_CLUSTER = 8, MAX_CLUSTER_FIT = 16;

// MB slots of one plane kind. Luma: 16 rows of 16 bytes; chroma: 8 rows of 8
// bytes of U, then of V. Lane q of an MB owns two rows for the vertical
// edges (luma q and q + 8; chroma q & 3 and (q & 3) + 4 of plane q >> 2) and
// two adjacent columns for the horizontal ones. A set's stride offsets
// neighbouring sets by 16 bytes (luma; 8 chroma), so that the MBs of
// consecutive rows read their columns from distinct banks.
template <bool LUMA>
struct Geo {
  static constexpr int NW = LUMA ? 4 : 2;  // words per row
  static constexpr int ROWB = NW * 4;
  static constexpr int SLOT = LUMA ? 256 : 128;
  static constexpr int SET = RING * SLOT + (LUMA ? 16 : 8);
  // The MB's last four rows: lane q's eight bytes of them in a slot, and its
  // two columns in a 64-byte message of them.
  static __device__ __forceinline__ int tail_off(int q) { return LUMA ? 192 + q * 8 : (q >> 2) * 64 + 32 + (q & 3) * 8; }
  static __device__ __forceinline__ int msg_col(int q) { return LUMA ? q * 2 : (q >> 2) * 32 + (q & 3) * 2; }
  static constexpr int HALF = LUMA ? 8 : 4;  // distance of the lane's rows
  static __device__ __forceinline__ int row(int q) { return LUMA ? q : q & 3; }
  static __device__ __forceinline__ int row_off(int q) { return LUMA ? q * 16 : (q >> 2) * 64 + (q & 3) * 8; }
  static __device__ __forceinline__ int col_off(int q) { return LUMA ? q * 2 : (q >> 2) * 64 + (q & 3) * 2; }
};

struct LfArgs {
  const uint8_t* y;
  const uint8_t* u;
  const uint8_t* v;
  uint64_t ys, cs;
  int mb_cols, mb_rows;
  const vp8a_mb_lf_info* mbs;
  vp8a_filter_config base;
  const uint8_t* sy;
  const uint8_t* su;
  const uint8_t* sv;
  uint64_t sys, scs;
  int width, height;
  const uint8_t* cands;  // [n][2] (level, sharpness)
  // [n] or null: the sharpness values whose table entries candidate i's
  // SSD fills (bit s = level * 8 + s), null = its own sharpness only.
  const uint8_t* cand_mask;
  int n_cands;
  // Row schedule (lf_schedule_kernel). Scored rows are numbered s = 0 ..
  // n_scored - 1: every MB row, or (band_step > 0) the two rows at the start
  // of each band_step rows. `split` ranks (CTAs of a cluster) take
  // consecutive bands of them. In a whole pass meta[t] = (first entry, entries
  // with inner edges, entries to filter, entries) of step t, and an entry is
  // s << 6 | filter class.
  int n_scored, band_step, max_t0, steps, split;
  uint4* meta;
  uint16_t* list;
  // Row s of a whole pass keeps its slots in ring set s & set_mask; a rank's
  // rows have a set each.
  int n_sets, set_mask;
  int recon_align, source_align;  // 2: whole-row vector loads, 1: word loads, 0: bytes
  // The scored rows' reconstruction and source as MB tiles (tile_mb), or null:
  // MB (s, c)'s 384 bytes (Y rows, U rows, V rows) at (s * mb_cols + c) * 384.
  uint8_t* recon_tiles;
  uint8_t* source_tiles;
  uint8_t* info;  // split passes: MB (s, c)'s filter class, bit 7 = has inner edges
  uint64_t* ssd_out;              // [64 * 8], indexed level * 8 + sharpness; added to
  uint8_t* oy;                    // write-back planes (apply mode) or null
  uint8_t* ou;
  uint8_t* ov;
  // Sweep mode: a level-0 candidate scores the unfiltered planes
  // (score_filter_candidate's short cut, src/loop_filter.rs:2071). Apply
  // mode runs the pass with the base level as given, since per-MB
  // segment overrides and deltas can still filter MBs at base level 0.
  int level0_unfiltered;
  unsigned spin_limit;  // polls of the waits between a split pass's CTAs (microseconds each message)
  unsigned* status;     // set to DEV_TIMEOUT when they run out
};

__host__ __device__ __forceinline__ int clamp63(int v) { return v < 0 ? 0 : (v > 63 ? 63 : v); }

// calculate_mb_filter_level_inter (src/loop_filter.rs:1280-1331).
__host__ __device__ __forceinline__ int mb_level(const vp8a_filter_config& c, int level0, const vp8a_mb_lf_info& m) {
  int level = level0;
  if (c.segmentation_enabled) {
    int seg = m.segment_id < 0 ? 0 : (m.segment_id > 3 ? 3 : (int)m.segment_id);
    if (c.segment_abs) level = c.segment_lf_level[seg];
    else level += c.segment_lf_level[seg];
  }
  level = clamp63(level);
  if (c.delta_enabled) {
    int rd = m.ref_frame == VP8A_REF_LAST     ? c.ref_delta_last
             : m.ref_frame == VP8A_REF_GOLDEN ? c.ref_delta_golden
             : m.ref_frame == VP8A_REF_ALTREF ? c.ref_delta_altref
                                              : c.ref_delta_current;
    level += rd;
    if (m.ref_frame == VP8A_REF_INTRA) {
      if (m.y_mode_is_bpred) level += c.bpred_mode_delta;
    } else if (m.inter_mode == VP8A_MODE_ZERO) {
      level += c.zero_mv_mode_delta;
    } else if (m.inter_mode == VP8A_MODE_SPLIT) {
      level += c.split_mv_mode_delta;
    } else {
      level += c.other_mv_mode_delta;
    }
  }
  return clamp63(level);
}

// LoopFilterParams::derive's interior limit (src/loop_filter.rs:99-148):
// with the level, it fixes every parameter of the §15 filters.
__host__ __device__ __forceinline__ int interior_limit(int level, int sharp) {
  int interior = level;
  if (sharp != 0) {
    interior >>= (sharp > 4) ? 2 : 1;
    const int cap = 9 - sharp > 0 ? 9 - sharp : 0;
    if (interior > cap) interior = cap;
  }
  return interior == 0 ? 1 : interior;
}

// An MB's filter class: everything of its record that mb_level reads. 14
// kinds (intra without and with B_PRED; four reference cases x ZERO, SPLIT,
// other) x 4 segments, so an entry's 6 bits hold it and a pass derives the
// parameters of each class once.
constexpr int KINDS = 14, CLASSES = 4 * KINDS;
static_assert(CLASSES <= 64, "a class fits in a schedule entry");

__device__ __forceinline__ int mb_class(const vp8a_mb_lf_info& m) {
  int kind;
  if (m.ref_frame == VP8A_REF_INTRA) {
    kind = m.y_mode_is_bpred ? 1 : 0;
  } else {
    const int ri = m.ref_frame == VP8A_REF_LAST ? 0 : (m.ref_frame == VP8A_REF_GOLDEN ? 1
                                                       : m.ref_frame == VP8A_REF_ALTREF ? 2 : 3);
    kind = 2 + 3 * ri + (m.inter_mode == VP8A_MODE_ZERO ? 0 : (m.inter_mode == VP8A_MODE_SPLIT ? 1 : 2));
  }
  const int seg = m.segment_id < 0 ? 0 : (m.segment_id > 3 ? 3 : (int)m.segment_id);
  return seg * KINDS + kind;
}

__device__ __forceinline__ vp8a_mb_lf_info class_record(int cls) {
  const int seg = cls / KINDS, kind = cls - seg * KINDS;
  vp8a_mb_lf_info m{};
  m.segment_id = (int8_t)seg;
  m.inter_mode = VP8A_MODE_NONE;
  if (kind < 2) {
    m.ref_frame = VP8A_REF_INTRA;
    m.y_mode_is_bpred = (uint8_t)kind;
  } else {
    const int ri = (kind - 2) / 3, mi = (kind - 2) - 3 * ri;
    m.ref_frame = ri == 0 ? VP8A_REF_LAST : (ri == 1 ? VP8A_REF_GOLDEN : (ri == 2 ? VP8A_REF_ALTREF : 0xff));
    m.inter_mode = mi == 0 ? VP8A_MODE_ZERO : (mi == 1 ? VP8A_MODE_SPLIT : VP8A_MODE_NEW);
  }
  return m;
}

// ------------------------------------------------------------ row schedule

struct Rows {
  int band, skew;
  __device__ __forceinline__ Rows(const LfArgs& a, int split) : band(a.band_step), skew(skew_of(split)) {}
  __device__ __forceinline__ int t0(int s) const { return skew * (band ? s & 1 : s); }
  __device__ __forceinline__ bool top(int s) const { return band ? (s & 1) != 0 : s > 0; }
  __device__ __forceinline__ int mb_row(int s) const { return band ? (s >> 1) * band + (s & 1) : s; }
};

// Rank k's first row: equal bands, so that only the last ranks of a picture
// with few rows have none.
__host__ __device__ __forceinline__ int rank_row(int n_scored, int split, int k) {
  const int each = (n_scored + split - 1) / split;
  return k * each < n_scored ? k * each : n_scored;
}

// One warp lists the MBs of one step: those with inner edges first (they run
// the long path, so they share warps), then those without, then the rows'
// trailing columns, which only score.
__device__ __forceinline__ void schedule_step(const LfArgs& a, int t, int lane) {
  const Rows R(a, 1);
  const int n = a.n_scored, span = a.mb_cols + RING;
  unsigned before = 0;
  for (int s = lane; s < n; s += 32) before += (unsigned)min(max(t - R.t0(s), 0), span);
  const unsigned first = __reduce_add_sync(FULL, before);
  unsigned n_sub = 0, n_main = 0, n_all = 0;
  for (int pass = 0; pass < 2; pass++) {
    unsigned b_sub = first, b_edge = first + n_sub, b_tail = first + n_main;
    for (int b = 0; b < n; b += 32) {
      const int s = b + lane, c = s < n ? t - R.t0(s) : -1;
      const bool tail = c >= a.mb_cols && c < span;
      bool main = c >= 0 && c < a.mb_cols, sub = false;
      int cls = 0;
      if (main) {
        const vp8a_mb_lf_info m = a.mbs[(size_t)R.mb_row(s) * a.mb_cols + c];
        sub = m.y_mode_is_bpred || m.has_coeffs;
        cls = mb_class(m);
      }
      const unsigned v_sub = __ballot_sync(FULL, main && sub), v_edge = __ballot_sync(FULL, main && !sub),
                     v_tail = __ballot_sync(FULL, tail);
      if (pass == 0) {
        n_sub += __popc(v_sub);
        n_main += __popc(v_sub | v_edge);
        n_all += __popc(v_sub | v_edge | v_tail);
      } else {
        const unsigned lt = (1u << lane) - 1u;
        if (main || tail) {
          const unsigned at = tail ? b_tail + __popc(v_tail & lt)
                                   : (sub ? b_sub + __popc(v_sub & lt) : b_edge + __popc(v_edge & lt));
          a.list[at] = (uint16_t)(s << 6 | cls);
        }
        b_sub += __popc(v_sub);
        b_edge += __popc(v_edge);
        b_tail += __popc(v_tail);
      }
    }
  }
  if (lane == 0) a.meta[t] = make_uint4(first, n_sub, n_main, n_all);
}

// The table entries candidate `q` fills.
__device__ __forceinline__ int entry_mask(const LfArgs& a, int q, int lv, int sh) {
  return (lv == 0 && a.level0_unfiltered) ? 0xff : (a.cand_mask ? a.cand_mask[q] : 1 << sh);
}

__device__ __forceinline__ void clear_entries(const LfArgs& a, int i, int n) {
  if (!a.ssd_out) return;
  for (; i < a.n_cands; i += n) {
    const int lv = a.cands[2 * i], mk = entry_mask(a, i, lv, a.cands[2 * i + 1]);
    for (int s = 0; s < 8; s++)
      if ((mk >> s) & 1) a.ssd_out[lv * 8 + s] = 0;
  }
}

// The passes read an MB's rows eight lanes at a time; in the planes every row
// is a cache line of its own (32 lines per load instruction, half of each
// sector unused), so the planes are copied once per call into MB tiles, where
// the eight lanes' rows are 128 consecutive bytes. One warp copies two
// neighbouring MBs: lane (row, MB).
constexpr int TILE = 384;

__device__ __forceinline__ uint32_t load_word(const uint8_t* p, int align, int n) {
  // The first n of four bytes, the rest 0.
  if (align && n >= 4) return *(const uint32_t*)p;
  uint32_t w = 0;
#pragma unroll
  for (int k = 0; k < 4; k++)
    if (k < n) w |= (uint32_t)p[k] << (8 * k);
  return w;
}

// `w` x `h`: the picture the planes hold (the MB-padded planes or the visible
// source); bytes outside it become 0.
__device__ __forceinline__ void tile_mb(const uint8_t* y, const uint8_t* u, const uint8_t* v, uint64_t ys, uint64_t cs,
                                        int align, int w, int h, int r, int c, uint8_t* tile, int l) {
  const int yr = r * 16 + l, n = yr < h ? w - c * 16 : 0;
  const uint8_t* p = y + (uint64_t)(unsigned)yr * ys + (unsigned)(c * 16);
  uint4 o;
  if (align == 2 && n >= 16) o = *(const uint4*)p;
  else o = make_uint4(load_word(p, align, n), load_word(p + 4, align, n - 4), load_word(p + 8, align, n - 8),
                      load_word(p + 12, align, n - 12));
  *(uint4*)(tile + l * 16) = o;
  const int cr = r * 8 + (l & 7), m = cr < (h + 1) / 2 ? (w + 1) / 2 - c * 8 : 0;
  const uint8_t* q = (l < 8 ? u : v) + (uint64_t)(unsigned)cr * cs + (unsigned)(c * 8);
  uint2 e;
  if (align == 2 && m >= 8) e = *(const uint2*)q;
  else e = make_uint2(load_word(q, align, m), load_word(q + 4, align, m - 4));
  *(uint2*)(tile + 256 + l * 8) = e;
}

__device__ __forceinline__ int tile_warps(const LfArgs& a) {
  return a.recon_tiles ? a.n_scored * ((a.mb_cols + 1) / 2) : 0;
}

__device__ __forceinline__ void tile_pair(const LfArgs& a, int idx, int lane) {
  const int pairs = (a.mb_cols + 1) / 2, s = idx / pairs, c = 2 * (idx - s * pairs) + (lane >> 4), l = lane & 15;
  if (c >= a.mb_cols) return;
  const int r = Rows(a, a.split).mb_row(s);
  const size_t mb = (size_t)s * a.mb_cols + c, at = mb * TILE;
  if (l == 0 && a.split > 1) {
    const vp8a_mb_lf_info m = a.mbs[(size_t)r * a.mb_cols + c];
    a.info[mb] = (uint8_t)(mb_class(m) | (m.y_mode_is_bpred || m.has_coeffs ? 0x80 : 0));
  }
  tile_mb(a.y, a.u, a.v, a.ys, a.cs, a.recon_align, a.mb_cols * 16, a.mb_rows * 16, r, c, a.recon_tiles + at, l);
  if (a.sy)
    tile_mb(a.sy, a.su, a.sv, a.sys, a.scs, a.source_align, a.width, a.height, r, c, a.source_tiles + at, l);
}

constexpr int SCHED_WARPS = 8;

// Work item `idx` of a picture's preparation: the schedule's steps, then the
// tiles.
__device__ __forceinline__ void prepare_item(const LfArgs& a, int idx, int lane) {
  const int n = a.split > 1 ? 0 : a.steps;
  if (idx < n) schedule_step(a, idx, lane);
  else if (idx - n < tile_warps(a)) tile_pair(a, idx - n, lane);
}

__global__ void __launch_bounds__(SCHED_WARPS * 32) lf_schedule_kernel(const __grid_constant__ LfArgs a) {
  if (blockIdx.x == 0) clear_entries(a, threadIdx.x, blockDim.x);
  prepare_item(a, blockIdx.x * SCHED_WARPS + (threadIdx.x >> 5), threadIdx.x & 31);
}

__global__ void __launch_bounds__(SCHED_WARPS * 32)
    lf_schedule_batch_kernel(const LfArgs* __restrict__ jobs, const uint32_t* __restrict__ cta_start, int n_jobs) {
  __shared__ LfArgs sa;
  __shared__ uint32_t first[2];
  find_job(jobs, cta_start, n_jobs, &sa, first);
  if (blockIdx.x == first[0]) clear_entries(sa, threadIdx.x, blockDim.x);
  prepare_item(sa, (int)(blockIdx.x - first[0]) * SCHED_WARPS + (threadIdx.x >> 5), threadIdx.x & 31);
}

// ---------------------------------------------------------------- filters
//
// Taps are pairs of pixels in the 16-bit fields of a word. Sums below keep
// every field non-negative before a field-wise instruction reads it, so
// plain 32-bit adds and multiplies act on both fields at once.

__device__ __forceinline__ uint32_t pk(int v) { return (uint32_t)(uint16_t)(int16_t)v * 0x00010001u; }
constexpr uint32_t DISABLED = 0x80008000u;  // a limit that no pixel passes

// Bytes 1 and 3 as fields: each field >> 8.
__device__ __forceinline__ uint32_t high_bytes(uint32_t x) { return __byte_perm(x, 0u, 0x4341); }
// 0xffff where the field's sign bit is set.
__device__ __forceinline__ uint32_t sign_mask(uint32_t x) {
  uint32_t r;
  asm("prmt.b32 %0, %1, 0, 0xbb99;" : "=r"(r) : "r"(x));
  return r;
}
// clamp(x + k, 0, 255) per field.
__device__ __forceinline__ uint32_t clamp_add(uint32_t x, int k) { return __viaddmin_s16x2_relu(x, pk(k), pk(255)); }
// m ? x : y, bitwise.
__device__ __forceinline__ uint32_t sel(uint32_t m, uint32_t x, uint32_t y) { return (x & m) | (y & ~m); }

// Limits of one MB as packed biases: a field's sign bit is set when the
// measure exceeds its limit. flat: 0x7fff - interior; edge: 0x7fff - (2 E +
// 1), since 2 |p0 - q0| + (|p1 - q1| >> 1) <= E is 4 |p0 - q0| + |p1 - q1| <=
// 2 E + 1; hev: 0x7fff - threshold.
struct Limits {
  uint32_t flat, hev, mb, sub;
};

// The tests of §15.3 on eight taps: `no` = the edge is left alone, `hv` =
// high edge variance.
__device__ __forceinline__ void edge_masks(const uint32_t* p, uint32_t kflat, uint32_t kedge, uint32_t khev,
                                           uint32_t& no, uint32_t& hv) {
  const uint32_t inner = __vmaxs2(__vabsdiffu4(p[2], p[3]), __vabsdiffu4(p[5], p[4]));
  uint32_t flat = __vimax3_s16x2(__vabsdiffu4(p[0], p[1]), __vabsdiffu4(p[1], p[2]), inner);
  flat = __vimax3_s16x2(flat, __vabsdiffu4(p[7], p[6]), __vabsdiffu4(p[6], p[5]));
  const uint32_t e = __vabsdiffu4(p[3], p[4]) * 4u + (__vabsdiffu4(p[2], p[5]) + kedge);
  no = sign_mask((flat + kflat) | e);
  hv = sign_mask(inner + khev);
}

// c8(p1 - q1) + 128.
__device__ __forceinline__ uint32_t outer_tap(const uint32_t* p) { return clamp_add(p[2] - p[5] + pk(256), -128); }
// c8(s + 3 (q0 - p0)) + 128 of S = s + 128.
__device__ __forceinline__ uint32_t common_adjust(const uint32_t* p, uint32_t S) {
  return clamp_add((p[4] - p[3] + pk(256)) * 3u + S, -768);
}

// §15.3 MBfilter (src/loop_filter.rs:331-371) on taps p3..q3 = p[0..8).
// W = w + 128; each a = (k w + 63) >> 7 comes out as (2 k W + 126) >> 8 = a +
// k. A field that is left alone gets w = 0, which changes nothing.
__device__ __forceinline__ void mb_filter(uint32_t* p, const Limits& L, uint32_t kflat) {
  uint32_t no, hv;
  edge_masks(p, kflat, L.mb, L.hev, no, hv);
  const uint32_t W = sel(no, pk(128), common_adjust(p, outer_tap(p)));
  const uint32_t Ww = sel(hv, pk(128), W), Wn = sel(hv, W, pk(128));
  const uint32_t a27 = high_bytes(Ww * 54u + pk(126)), a18 = high_bytes(Ww * 36u + pk(126)),
                 a9 = high_bytes(Ww * 18u + pk(126));
  // c8(w + 4) >> 3 and c8(w + 3) >> 3, each + 16.
  const uint32_t nq = high_bytes(__viaddmin_s16x2(Wn, pk(4), pk(255)) * 32u);
  const uint32_t np = high_bytes(__viaddmin_s16x2(Wn, pk(3), pk(255)) * 32u);
  const uint32_t q0 = p[4], p0 = p[3], q1 = p[5], p1 = p[2], q2 = p[6], p2 = p[1];
  p[4] = clamp_add(q0 - (a27 + nq) + pk(43 + 256), -256);
  p[3] = clamp_add(p0 + (a27 + np), -43);
  p[5] = clamp_add(q1 - a18 + pk(18 + 256), -256);
  p[2] = clamp_add(p1 + a18, -18);
  p[6] = clamp_add(q2 - a9 + pk(9 + 256), -256);
  p[1] = clamp_add(p2 + a9, -9);
}

// §15.3 subblock_filter (src/loop_filter.rs:292-318). With a = c8(w + 4) >>
// 3, (a + 1) >> 1 is (c8(w + 4) + 8) >> 4. The §15.2 simple_segment (:235-247)
// is this filter with every pixel flat and of high edge variance.
__device__ __forceinline__ void sb_filter(uint32_t* p, uint32_t kedge, uint32_t khev, uint32_t kflat) {
  uint32_t no, hv;
  edge_masks(p, kflat, kedge, khev, no, hv);
  const uint32_t W = sel(no, pk(128), common_adjust(p, sel(hv, outer_tap(p), pk(128))));
  const uint32_t C = __viaddmin_s16x2(W, pk(4), pk(255));
  const uint32_t aq = high_bytes(C * 32u), ap = high_bytes(__viaddmin_s16x2(W, pk(3), pk(255)) * 32u);
  const uint32_t a2 = sel(hv, pk(8), high_bytes(C * 16u + pk(128)));
  const uint32_t q0 = p[4], p0 = p[3], q1 = p[5], p1 = p[2];
  p[4] = clamp_add(q0 - aq + pk(16 + 256), -256);
  p[3] = clamp_add(p0 + ap, -16);
  p[5] = clamp_add(q1 - a2 + pk(8 + 256), -256);
  p[2] = clamp_add(p1 + a2, -8);
}

// The MB edge: the normal or (a frame-wide choice) the simple filter.
template <bool SIMPLE>
__device__ __forceinline__ void mb_edge(uint32_t* p, const Limits& L, uint32_t kflat) {
  if constexpr (SIMPLE) sb_filter(p, L.mb, L.hev, kflat);
  else mb_filter(p, L, kflat);
}

// Words of two rows to taps (one row per field) and back.
__device__ __forceinline__ void rows_to_taps(uint32_t a, uint32_t b, uint32_t* t) {
  const uint32_t lo = __byte_perm(a, b, 0x5410), hi = __byte_perm(a, b, 0x7632);
  t[0] = lo & 0x00ff00ffu;
  t[1] = high_bytes(lo);
  t[2] = hi & 0x00ff00ffu;
  t[3] = high_bytes(hi);
}
__device__ __forceinline__ void taps_to_rows(const uint32_t* t, uint32_t& a, uint32_t& b) {
  const uint32_t lo = t[1] * 256u + t[0], hi = t[3] * 256u + t[2];
  a = __byte_perm(lo, hi, 0x5410);
  b = __byte_perm(lo, hi, 0x7632);
}

// -------------------------------------------------------------- MB access

// One lane's two rows of an MB.
template <bool LUMA>
struct LaneRows {
  uint32_t w[2][Geo<LUMA>::NW];
};

// The lane's two rows at `p` and `p + half`: whole-row vector loads where
// the plane allows them (align 2), else words or bytes.
template <bool LUMA>
__device__ __noinline__ LaneRows<LUMA> load_rows_unaligned(const uint8_t* p, uint64_t half, int align) {
  LaneRows<LUMA> o;
  for (int i = 0; i < 2; i++, p += half)
#pragma unroll
    for (int k = 0; k < Geo<LUMA>::NW; k++) {
      const uint8_t* b = p + 4 * k;
      const uint32_t w = align == 1 ? *(const uint32_t*)b
                                    : (uint32_t)b[0] | (uint32_t)b[1] << 8 | (uint32_t)b[2] << 16 | (uint32_t)b[3] << 24;
      if (i == 0) o.w[0][k] = w;
      else o.w[1][k] = w;
    }
  return o;
}

template <bool LUMA>
__device__ __forceinline__ void load_rows(const uint8_t* p, uint64_t half, int align, LaneRows<LUMA>& o) {
  if (align == 2) {
    // Plain loads: apply mode writes final MBs back into the planes.
    if constexpr (LUMA) {
      const uint4 v = *(const uint4*)p, w = *(const uint4*)(p + half);
      o.w[0][0] = v.x;
      o.w[0][1] = v.y;
      o.w[0][2] = v.z;
      o.w[0][3] = v.w;
      o.w[1][0] = w.x;
      o.w[1][1] = w.y;
      o.w[1][2] = w.z;
      o.w[1][3] = w.w;
    } else {
      const uint2 v = *(const uint2*)p, w = *(const uint2*)(p + half);
      o.w[0][0] = v.x;
      o.w[0][1] = v.y;
      o.w[1][0] = w.x;
      o.w[1][1] = w.y;
    }
  } else {
    o = load_rows_unaligned<LUMA>(p, half, align);
  }
}

// A plane set (or its MB tiles) seen by one lane: its first row of MB 0.
template <bool LUMA, bool TILED>
struct LanePlane {
  const uint8_t* p;
  uint64_t mb_row, half;  // planes: bytes per MB row; bytes between the lane's rows
  int cols;
  __device__ __forceinline__ LanePlane(const uint8_t* tiles, int mb_cols, const uint8_t* y, const uint8_t* u,
                                       const uint8_t* v, uint64_t ys, uint64_t cs, int q) {
    cols = mb_cols;
    if constexpr (TILED) {
      p = tiles + (LUMA ? 0 : 256) + Geo<LUMA>::row_off(q);
      mb_row = 0;
      half = Geo<LUMA>::HALF * Geo<LUMA>::ROWB;
    } else {
      const uint64_t st = LUMA ? ys : cs;
      p = (LUMA ? y : (q < 4 ? u : v)) + (uint64_t)(unsigned)Geo<LUMA>::row(q) * st;
      half = Geo<LUMA>::HALF * st;
      mb_row = 2 * half;
    }
  }
  // MB (r, c), the scored row s.
  __device__ __forceinline__ const uint8_t* mb(int s, int r, int c) const {
    if constexpr (TILED) return p + (size_t)(unsigned)(s * cols + c) * TILE;
    else return p + (uint64_t)(unsigned)r * mb_row + (unsigned)(c * Geo<LUMA>::ROWB);
  }
};

// Sum of squared differences of four byte pairs.
__device__ __forceinline__ uint32_t ssd4(uint32_t x, uint32_t y, uint32_t acc) {
  const uint32_t d = __vabsdiffu4(x, y);
  return (uint32_t)__dp4a(d, d, acc);
}

template <int NW>
__device__ __forceinline__ void slot_row(const uint8_t* s, uint32_t (&w)[NW]) {
  if constexpr (NW == 4) {
    const uint4 v = *(const uint4*)s;
    w[0] = v.x;
    w[1] = v.y;
    w[2] = v.z;
    w[3] = v.w;
  } else {
    const uint2 v = *(const uint2*)s;
    w[0] = v.x;
    w[1] = v.y;
  }
}
template <int NW>
__device__ __forceinline__ void set_slot_row(uint8_t* s, const uint32_t (&w)[NW]) {
  if constexpr (NW == 4) *(uint4*)s = make_uint4(w[0], w[1], w[2], w[3]);
  else *(uint2*)s = make_uint2(w[0], w[1]);
}

// Final MB (r, c) in its slot: this lane's share of its SSD against `src`
// (an MB inside the window).
template <bool LUMA>
__device__ __forceinline__ uint32_t score_mb(const uint8_t* slot, int q, const LaneRows<LUMA>& src) {
  constexpr int NW = Geo<LUMA>::NW;
  uint32_t acc = 0;
#pragma unroll
  for (int i = 0; i < 2; i++) {
    uint32_t w[NW];
    slot_row(slot + Geo<LUMA>::row_off(q) + i * Geo<LUMA>::HALF * Geo<LUMA>::ROWB, w);
#pragma unroll
    for (int k = 0; k < NW; k++) acc = ssd4(w[k], src.w[i][k], acc);
  }
  return acc;
}

// The same for an MB across the window's edge: source bytes outside are not
// read and do not count.
template <bool LUMA>
__device__ __noinline__ uint32_t score_edge_mb(const uint8_t* slot, const uint8_t* g, uint64_t half, int cols,
                                               int rows, int q) {
  const int n = min(cols, Geo<LUMA>::ROWB);
  uint32_t acc = 0;
  for (int i = 0; i < 2; i++) {
    if (Geo<LUMA>::row(q) + i * Geo<LUMA>::HALF >= rows) break;
    const uint8_t* s = slot + Geo<LUMA>::row_off(q) + i * Geo<LUMA>::HALF * Geo<LUMA>::ROWB;
    for (int x = 0; x < n; x++) {
      const int d = (int)s[x] - (int)g[x];
      acc += (uint32_t)(d * d);
    }
    g += half;
  }
  return acc;
}

// Write the lane's rows of a final MB back (apply mode).
template <bool LUMA>
__device__ __forceinline__ void store_rows(uint8_t* g, uint64_t half, int align, const LaneRows<LUMA>& o) {
#pragma unroll
  for (int i = 0; i < 2; i++, g += half) {
    if (align == 2) set_slot_row(g, o.w[i]);
    else
#pragma unroll
      for (int k = 0; k < Geo<LUMA>::NW; k++) {
        if (align == 1) {
          ((uint32_t*)g)[k] = o.w[i][k];
        } else {
          g[4 * k] = (uint8_t)o.w[i][k];
          g[4 * k + 1] = (uint8_t)(o.w[i][k] >> 8);
          g[4 * k + 2] = (uint8_t)(o.w[i][k] >> 16);
          g[4 * k + 3] = (uint8_t)(o.w[i][k] >> 24);
        }
      }
  }
}

// ------------------------------------------------------------ MB filtering

// Two adjacent pixels as fields, and back.
__device__ __forceinline__ uint32_t spread2(uint32_t w) { return __byte_perm(w, 0u, 0x4140); }
__device__ __forceinline__ uint32_t join2(uint32_t t) { return __byte_perm(t, 0u, 0x4420); }

// Vertical edges of one MB (its left MB edge and, with FULL_MB, its inner
// edges) on the lane's two rows, from the unfiltered rows `rec` into the slot
// `me`; the left neighbour's last word is filtered in place.
template <bool LUMA, bool SIMPLE, bool FULL_MB>
__device__ __forceinline__ void vertical_edges(LaneRows<LUMA>& rec, uint8_t* me, uint8_t* left, int q, bool has_left,
                                               const Limits& L, uint32_t kleft, uint32_t kinner) {
  constexpr int NW = Geo<LUMA>::NW, NT = FULL_MB ? NW : 1, B = Geo<LUMA>::HALF * Geo<LUMA>::ROWB;
  uint8_t* l = left + Geo<LUMA>::row_off(q) + 4 * (NW - 1);
  uint32_t t[4 + 4 * NT];
  rows_to_taps(*(const uint32_t*)l, *(const uint32_t*)(l + B), t);
#pragma unroll
  for (int k = 0; k < NT; k++) rows_to_taps(rec.w[0][k], rec.w[1][k], t + 4 + 4 * k);
  mb_edge<SIMPLE>(t, L, kleft);
  if constexpr (FULL_MB) {
#pragma unroll
    for (int k = 0; k + 1 < NW; k++) sb_filter(t + 4 + 4 * k, L.sub, L.hev, kinner);
  }
  uint32_t wa, wb;
  taps_to_rows(t, wa, wb);
  if (has_left) {
    *(uint32_t*)l = wa;
    *(uint32_t*)(l + B) = wb;
  }
#pragma unroll
  for (int k = 0; k < NT; k++) taps_to_rows(t + 4 + 4 * k, rec.w[0][k], rec.w[1][k]);
  uint8_t* m = me + Geo<LUMA>::row_off(q);
  set_slot_row(m, rec.w[0]);
  set_slot_row(m + B, rec.w[1]);
}

// Horizontal edges of one MB on the lane's two columns: the top MB edge (the
// last four rows of the MB above, at `up`) and, with FULL_MB, the inner edges.
template <bool LUMA, bool SIMPLE, bool FULL_MB>
__device__ __forceinline__ void horizontal_edges(uint8_t* me, uint8_t* up, int q, bool has_top, const Limits& L,
                                                 uint32_t ktop, uint32_t kinner) {
  constexpr int NW = Geo<LUMA>::NW, ROWB = Geo<LUMA>::ROWB, NT = FULL_MB ? NW : 1;
  uint32_t t[4 + 4 * NT];
  uint8_t* col = me + Geo<LUMA>::col_off(q);
#pragma unroll
  for (int k = 0; k < 4; k++) t[k] = spread2(*(const uint16_t*)(up + k * ROWB));
#pragma unroll
  for (int k = 0; k < 4 * NT; k++) t[4 + k] = spread2(*(const uint16_t*)(col + k * ROWB));
  mb_edge<SIMPLE>(t, L, ktop);
  if (has_top)
#pragma unroll
    for (int k = 1; k < 4; k++) *(uint16_t*)(up + k * ROWB) = (uint16_t)join2(t[k]);
  if constexpr (FULL_MB) {
#pragma unroll
    for (int k = 0; k + 1 < NW; k++) sb_filter(t + 4 + 4 * k, L.sub, L.hev, kinner);
  }
  // The MB edge changes the first three rows, an inner edge two on each side.
#pragma unroll
  for (int k = 0; k < (FULL_MB ? 4 * NW - 2 : 3); k++) *(uint16_t*)(col + k * ROWB) = (uint16_t)join2(t[4 + k]);
}

// ------------------------------------------------------------------ a pass

// The MB a lane works on.
struct Item {
  int s, r, c, slot, set;      // scored row, MB row and column, slot (column % RING), ring set
  bool live, main, sub, full;  // scores; filters; has inner edges; an MB of the warp's group has
  bool top;
};

// One plane kind of a pass, as one lane sees it.
template <bool LUMA, bool SIMPLE, bool TILED>
struct PlanePass {
  static constexpr int SLOT = Geo<LUMA>::SLOT, SET = Geo<LUMA>::SET;
  LanePlane<LUMA, TILED> recon, source;
  int whole_cols, whole_rows;  // MBs inside the visible window whole
  uint8_t* rings;
  LaneRows<LUMA> rec, src;

  __device__ __forceinline__ PlanePass(const LfArgs& a, uint8_t* ring, int q)
      : recon(a.recon_tiles, a.mb_cols, a.y, a.u, a.v, a.ys, a.cs, q),
        source(a.source_tiles, a.mb_cols, a.sy, a.su, a.sv, a.sys, a.scs, q),
        rings(ring) {
    const int w = LUMA ? a.width : (a.width + 1) >> 1, h = LUMA ? a.height : (a.height + 1) >> 1;
    whole_cols = w / Geo<LUMA>::ROWB;
    whole_rows = h / (2 * Geo<LUMA>::HALF);
  }
  __device__ __forceinline__ bool whole(int r, int c) const { return c < whole_cols && r < whole_rows; }
  // The rows item (s, r, c) needs: its own and the source under the MB that
  // leaves its slot.
  __device__ __forceinline__ void fetch(const LfArgs& a, int s, int r, int c, bool main, bool live) {
    if (main) load_rows<LUMA>(recon.mb(s, r, c), recon.half, TILED ? 2 : a.recon_align, rec);
    if (live && a.ssd_out && c >= RING && whole(r, c - RING))
      load_rows<LUMA>(source.mb(s, r, c - RING), source.half, TILED ? 2 : a.source_align, src);
  }
  // MB (r, c - RING) is final: score it (or write it back).
  __device__ __forceinline__ uint32_t finish(const LfArgs& a, const Item& m, int q) {
    if (!m.live || m.c < RING) return 0;
    const uint8_t* slot = rings + m.set * SET + m.slot * SLOT;
    const int c = m.c - RING;
    if (a.oy) {
      const LanePlane<LUMA, false> out(nullptr, 0, a.oy, a.ou, a.ov, a.ys, a.cs, q);
      LaneRows<LUMA> fin;
      slot_row(slot + Geo<LUMA>::row_off(q), fin.w[0]);
      slot_row(slot + Geo<LUMA>::row_off(q) + Geo<LUMA>::HALF * Geo<LUMA>::ROWB, fin.w[1]);
      store_rows<LUMA>(const_cast<uint8_t*>(out.mb(m.s, m.r, c)), out.half, a.recon_align, fin);
    }
    if (!a.ssd_out) return 0;
    if (whole(m.r, c)) return score_mb<LUMA>(slot, q, src);
    const int w = LUMA ? a.width : (a.width + 1) >> 1, h = LUMA ? a.height : (a.height + 1) >> 1;
    return score_edge_mb<LUMA>(slot, source.mb(m.s, m.r, c), source.half, w - c * Geo<LUMA>::ROWB,
                               h - m.r * 2 * Geo<LUMA>::HALF, q);
  }
  __device__ __forceinline__ void vertical(const Item& m, const Limits& L, int q) {
    uint8_t* set = rings + m.set * SET;
    uint8_t *me = set + m.slot * SLOT, *left = set + (m.slot ? m.slot - 1 : RING - 1) * SLOT;
    const uint32_t kleft = m.c > 0 ? L.flat : DISABLED, kinner = m.sub ? L.flat : DISABLED;
    if (m.full) vertical_edges<LUMA, SIMPLE, true>(rec, me, left, q, m.c > 0, L, kleft, kinner);
    else vertical_edges<LUMA, SIMPLE, false>(rec, me, left, q, m.c > 0, L, kleft, kinner);
  }
  // `up_set`: the ring set of the row above; without a top edge the row's own
  // slot stands in, and is only read.
  __device__ __forceinline__ void horizontal(const Item& m, const Limits& L, int q, int up_set) {
    constexpr int LAST = (Geo<LUMA>::NW - 1) * 4 * Geo<LUMA>::ROWB;  // offset of the MB's last four rows
    uint8_t* me = rings + m.set * SET + m.slot * SLOT;
    uint8_t* up = rings + up_set * SET + m.slot * SLOT + LAST + Geo<LUMA>::col_off(q);
    const uint32_t ktop = m.top ? L.flat : DISABLED, kinner = m.sub ? L.flat : DISABLED;
    if (m.full) horizontal_edges<LUMA, SIMPLE, true>(me, up, q, m.top, L, ktop, kinner);
    else horizontal_edges<LUMA, SIMPLE, false>(me, up, q, m.top, L, ktop, kinner);
  }
};

struct NoPlane {
  __device__ __forceinline__ void fetch(const LfArgs&, int, int, int, bool, bool) {}
  __device__ __forceinline__ uint32_t finish(const LfArgs&, const Item&, int) { return 0; }
  __device__ __forceinline__ void vertical(const Item&, const Limits&, int) {}
  __device__ __forceinline__ void horizontal(const Item&, const Limits&, int, int) {}
};

// One whole pass's steps over plane kind A (and B). `lim`, `lim_b`: the
// candidate's limits per filter class; `turn` spreads the warps' first groups
// over the SM's quarters. Returns this thread's share of the SSD.
template <bool PRE, class A, class B>
__device__ __forceinline__ uint64_t run_pass(const LfArgs& a, const Limits* lim, const Limits* lim_b, unsigned* taken,
                                             int turn, A& pa, B& pb) {
  const Rows R(a, 1);
  const int lane = threadIdx.x & 31, q = lane & (LPM - 1), sub_lane = lane / LPM;
  const unsigned nwarps = blockDim.x >> 5;
  uint64_t total = 0;
  // The step's MBs are taken in groups of MPW. The groups with inner edges
  // come first in the list and take about twice as long: each warp starts on
  // a group of its own (turned every step, so that the long groups move over
  // the SM's quarters) and then takes the next free group.
  unsigned turned = ((threadIdx.x >> 5) + (unsigned)turn) % nwarps;
  uint4 mt = a.meta[0];
  int base0 = turned * MPW;
  int entry = base0 + sub_lane < (int)mt.w ? a.list[mt.x + base0 + sub_lane] : 0;
  auto fetch = [&](const uint4& m, int i, int e, int t) {
    const int s = e >> 6, r = R.mb_row(s), c = t - R.t0(s);
    pa.fetch(a, s, r, c, i < (int)m.z, i < (int)m.w);
    pb.fetch(a, s, r, c, i < (int)m.z, i < (int)m.w);
  };
  if constexpr (PRE) fetch(mt, base0 + sub_lane, entry, 0);
  for (int t = 0; t < a.steps; t++) {
    const uint4 next = t + 1 < a.steps ? a.meta[t + 1] : make_uint4(0, 0, 0, 0);
    turned = turned + 1 == nwarps ? 0 : turned + 1;
    const int next0 = turned * MPW;
    const int next_entry = next0 + sub_lane < (int)next.w ? a.list[next.x + next0 + sub_lane] : 0;
    if (threadIdx.x == 0) taken[(t + 1) & 1] = nwarps;
    int base = base0, e = entry;
    bool fetched = PRE;
    while (base < (int)mt.w) {
      const int i = base + sub_lane;
      Item m;
      m.s = e >> 6;
      m.r = R.mb_row(m.s);
      m.c = t - R.t0(m.s);
      m.slot = (unsigned)m.c % RING;
      m.set = m.s & a.set_mask;
      m.live = i < (int)mt.w;
      m.main = i < (int)mt.z;
      m.sub = i < (int)mt.y;
      m.full = base < (int)mt.y;
      m.top = R.top(m.s);
      if (!fetched) {
        pa.fetch(a, m.s, m.r, m.c, m.main, m.live);
        pb.fetch(a, m.s, m.r, m.c, m.main, m.live);
      }
      // MB (r, c - RING) leaves the slot that MB (r, c) takes.
      total += pa.finish(a, m, q) + pb.finish(a, m, q);
      const Limits La = lim[e & 63];
      if (m.main) {
        pa.vertical(m, La, q);
        pb.vertical(m, lim_b[e & 63], q);
      }
      // The warp's next group; after its last one the row registers are free
      // for the next step's rows.
      int nb = (int)mt.w;
      if (nwarps * MPW < mt.w) {
        unsigned g = 0;
        if (lane == 0) g = atomicAdd(&taken[t & 1], 1u);
        nb = (int)__shfl_sync(FULL, g, 0) * MPW;
      }
      if (PRE && nb >= (int)mt.w) fetch(next, next0 + sub_lane, next_entry, t + 1);
      __syncwarp();
      if (m.main) {
        const int up_set = (m.s - (m.top ? 1 : 0)) & a.set_mask;
        pa.horizontal(m, La, q, up_set);
        pb.horizontal(m, lim_b[e & 63], q, up_set);
      }
      __syncwarp();
      base = nb;
      fetched = false;
      if (base + sub_lane < (int)mt.w) e = a.list[mt.x + base + sub_lane];
    }
    if (PRE && base0 >= (int)mt.w) fetch(next, next0 + sub_lane, next_entry, t + 1);
    mt = next;
    base0 = next0;
    entry = next_entry;
    __syncthreads();
  }
  return total;
}

// ------------------------------------------------- between a split's CTAs
//
// The CTA of rows [s0, s1) hands each MB's last four rows of row s1 - 1 to the
// next CTA once the vertical edges have passed them (64 bytes), and gets them
// back filtered, straight into its ring, for scoring. Both are asynchronous
// stores into the neighbour's shared memory that complete a transaction on its
// mbarrier, so the CTAs are ordered pairwise, message by message, and no CTA
// waits for one that it does not depend on (a cluster barrier a step cost
// about 2,000 of a step's 4,400 cycles: its release alone is a fence of 700 to
// 900, and reads of a neighbour's memory are slow). Two messages are in flight
// at most: message c is sent at column c + 1, after column c - 2's return has
// been waited for.
//
// A lane whose wait runs out closes its end of the link: it sends and waits no more,
// so its shares sent are the first so many messages'. Before the CTAs leave
// (leave_split), each tells its neighbours how many that was and waits for what was
// sent to it and not taken in.

struct Link {
  alignas(16) uint8_t inbox[2][64];  // message c in entry c & 1
  uint64_t in_bar[2], ret_bar[2];
  // By lane: messages sent down, returns taken in, messages taken in and returned;
  // what the neighbours have sent, told at the end.
  unsigned n_down[LPM], n_back[LPM], n_up[LPM], sent_in[LPM], sent_ret[LPM];
  int turns;  // polls left for this CTA's waits, in thousands (POLL_TURN)
  int dead;   // they have run out: a wait's first poll that fails ends it
};
constexpr int POLL_TURN = 1024;

__device__ __forceinline__ uint32_t smem_at(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ uint32_t cluster_at(uint32_t at, int rank) {
  uint32_t r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(at), "r"(rank));
  return r;
}
__device__ __forceinline__ void expect_message(uint64_t* bar) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], 64;" ::"r"(smem_at(bar)) : "memory");
}
__device__ __forceinline__ void send8(uint32_t at, uint2 v, uint32_t bar) {
  asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v2.b32 [%0], {%1, %2}, [%3];" ::"r"(at),
               "r"(v.x), "r"(v.y), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void store_cluster(uint32_t at, unsigned v) {
  asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(at), "r"(v) : "memory");
}
__device__ __forceinline__ bool message_in(uint32_t bar, unsigned parity) {
  uint32_t done;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.test_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n"
      " selp.u32 %0, 1, 0, p;\n}"
      : "=r"(done)
      : "r"(bar), "r"(parity)
      : "memory");
  return done != 0;
}
// Message (or return) m; false when the wait ran out (the pass then runs on without
// that neighbour). The limit is counted outside the polls' way, in turns: a load of it
// and a comparison a poll made a 1280x720 pass 162 us instead of 155.
__device__ __forceinline__ bool wait_message(const LfArgs& a, Link* k, uint64_t* bars, int m) {
  const uint32_t at = smem_at(bars + (m & 1));
  const unsigned parity = (unsigned)(m >> 1) & 1u;
#pragma unroll 1
  for (int polls = 0;;) {
    if (message_in(at, parity)) return true;
    if (*(volatile int*)&k->dead) break;
    if (++polls > POLL_TURN) {
      polls = 0;
      if (atomicSub(&k->turns, 1) <= 1) *(volatile int*)&k->dead = 1;
    }
  }
  atomicCAS(a.status, 0u, (unsigned)vp8a::DEV_TIMEOUT);
  return false;
}
// On the way out: the messages from `got` on of which a lane sent its share (lane q
// those of the first sent[q]). They arrive within microseconds.
__device__ __forceinline__ void await_messages(uint64_t* bars, unsigned got, const unsigned* sent) {
  unsigned most = 0;
  for (int q = 0; q < LPM; q++) most = max(most, sent[q]);
  for (; got < most; got++) {
    const uint32_t at = smem_at(bars + (got & 1));
    unsigned missing = 0;
    for (int q = 0; q < LPM; q++) missing += sent[q] <= got ? 8u : 0u;
    if (missing)
      asm volatile("mbarrier.complete_tx.relaxed.cta.shared::cta.b64 [%0], %1;" ::"r"(at), "r"(missing) : "memory");
    for (int polls = 0; polls < 1 << 20 && !message_in(at, got >> 1 & 1u); polls++) {
    }
  }
}

__device__ __forceinline__ void init_link(Link* k, unsigned limit) {
  k->turns = (int)(limit / POLL_TURN) + 1;
  k->dead = limit == 0;
  for (int q = 0; q < LPM; q++) k->sent_in[q] = k->sent_ret[q] = 0;
  for (int i = 0; i < 2; i++) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_at(&k->in_bar[i])) : "memory");
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_at(&k->ret_bar[i])) : "memory");
  }
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  for (int i = 0; i < 2; i++) {
    expect_message(&k->in_bar[i]);
    expect_message(&k->ret_bar[i]);
  }
}

// One CTA's rows of a split pass: every eight lanes own one row for the whole
// pass, so that a step has no list to read and no address to build. The warp
// takes the long path when one of its four MBs has inner edges.
template <bool LUMA, bool SIMPLE>
__device__ __forceinline__ uint64_t run_split(const LfArgs& a, const Limits* lim, uint8_t* rings, Link* link,
                                              int rank) {
  constexpr int SLOT = Geo<LUMA>::SLOT, SET = Geo<LUMA>::SET, ROWB = Geo<LUMA>::ROWB;
  constexpr int LAST = (Geo<LUMA>::NW - 1) * 4 * ROWB, HALF_OFF = Geo<LUMA>::HALF * ROWB;
  const Rows R(a, 2);
  const int g = threadIdx.x / LPM, q = threadIdx.x & (LPM - 1), cols = a.mb_cols;
  const int s0 = rank_row(a.n_scored, a.split, rank), s1 = rank_row(a.n_scored, a.split, rank + 1);
  const bool have = s0 + g < s1;
  const int s = have ? s0 + g : s0, t0 = have ? R.t0(s) : 1 << 30, r = R.mb_row(s);
  const bool top = R.top(s), handed = top && g == 0, hand_down = have && s == s1 - 1 && s1 < a.n_scored && R.top(s1);
  const int w = LUMA ? a.width : (a.width + 1) >> 1, h = LUMA ? a.height : (a.height + 1) >> 1;
  const int rows_left = h - r * 2 * Geo<LUMA>::HALF;
  const int whole_cols = rows_left >= 2 * Geo<LUMA>::HALF ? w / ROWB : 0;
  const bool score = a.ssd_out != nullptr;
  uint8_t* set = rings + g * SET;
  uint8_t* up_set = top && !handed ? set - SET : set;
  const size_t row_tiles = (size_t)s * cols;
  const int off = (LUMA ? 0 : 256) + Geo<LUMA>::row_off(q);
  const uint8_t *rp = a.recon_tiles + row_tiles * TILE + off, *sp = a.source_tiles + row_tiles * TILE + off;
  const uint8_t* ip = a.info + row_tiles;
  const LanePlane<LUMA, false> out(nullptr, 0, a.oy, a.ou, a.ov, a.ys, a.cs, q);
  uint8_t* op = a.oy ? const_cast<uint8_t*>(out.mb(0, r, 0)) : nullptr;
  uint32_t down_inbox, down_bar, up_rings, up_bar;
  {
    const int d = min(rank + 1, a.split - 1), u = max(rank - 1, 0);
    down_inbox = cluster_at(smem_at(link->inbox), d) + q * 8;
    down_bar = cluster_at(smem_at(link->in_bar), d);
    // The previous rank's last row (its rows are as many as any full rank's).
    up_rings = cluster_at(smem_at(rings), u) + (s0 - 1 - rank_row(a.n_scored, a.split, u)) * SET + Geo<LUMA>::tail_off(q);
    up_bar = cluster_at(smem_at(link->ret_bar), u);
  }
  uint64_t total = 0;
  LaneRows<LUMA> rec, src, fin;
  bool down = hand_down, up = handed;  // this lane's ends of the links are open
  if (down) link->n_down[q] = link->n_back[q] = cols;
  if (up) link->n_up[q] = cols;
  unsigned info = 0;
  int slot = 0;  // c % RING
  auto fetch = [&](int c) {
    if (c >= 0 && c < cols) {
      info = ip[c];
      load_rows<LUMA>(rp + (size_t)(unsigned)c * TILE, HALF_OFF, 2, rec);
    }
    if (score && c >= RING && c - RING < whole_cols)
      load_rows<LUMA>(sp + (size_t)(unsigned)(c - RING) * TILE, HALF_OFF, 2, src);
  };
  fetch(0 - t0);
  for (int t = 0; t < a.steps; t++) {
    const int c = t - t0;
    const bool live = c >= 0 && c < cols + RING, main = c >= 0 && c < cols;
    const bool sub = main && (info & 0x80) != 0, full = __any_sync(FULL, sub);
    uint8_t* me = set + slot * SLOT;
    const int left_at = (slot ? slot - 1 : RING - 1) * SLOT;
    const Limits L = lim[info & 63];
    const uint32_t kinner = sub ? L.flat : DISABLED;
    bool written = false;
    if (live && c >= RING) {
      // MB (r, c - RING) is final (its last rows back from the next CTA).
      const int f = c - RING;
      if (down) {
        if (!wait_message(a, link, link->ret_bar, f)) {
          down = false;
          link->n_down[q] = min(c - 1, cols);
          link->n_back[q] = f;
        } else if (q == 0) {
          expect_message(&link->ret_bar[f & 1]);
        }
      }
      if (score) {
        total += f < whole_cols ? score_mb<LUMA>(me, q, src)
                                : score_edge_mb<LUMA>(me, sp + (size_t)(unsigned)f * TILE, HALF_OFF, w - f * ROWB,
                                                      rows_left, q);
      }
      if (op) {
        slot_row(me + Geo<LUMA>::row_off(q), fin.w[0]);
        slot_row(me + Geo<LUMA>::row_off(q) + HALF_OFF, fin.w[1]);
        written = true;
      }
    }
    if (main) {
      const uint32_t kleft = c > 0 ? L.flat : DISABLED;
      if (full) vertical_edges<LUMA, SIMPLE, true>(rec, me, set + left_at, q, c > 0, L, kleft, kinner);
      else vertical_edges<LUMA, SIMPLE, false>(rec, me, set + left_at, q, c > 0, L, kleft, kinner);
    }
    __syncwarp();
    if (down && c >= 1 && c <= cols)
      send8(down_inbox + ((c - 1) & 1) * 64, *(const uint2*)(set + left_at + Geo<LUMA>::tail_off(q)),
            down_bar + ((c - 1) & 1) * 8);
    fetch(c + 1);
    if (written) store_rows<LUMA>(op + (c - RING) * ROWB, out.half, a.recon_align, fin);
    __syncthreads();
    if (main) {
      uint8_t* msg = link->inbox[c & 1];
      if (up && !wait_message(a, link, link->in_bar, c)) {
        up = false;
        link->n_up[q] = c;
      }
      uint8_t* above = handed ? msg + Geo<LUMA>::msg_col(q) : up_set + slot * SLOT + LAST + Geo<LUMA>::col_off(q);
      const uint32_t ktop = top ? L.flat : DISABLED;
      if (full) horizontal_edges<LUMA, SIMPLE, true>(me, above, q, top, L, ktop, kinner);
      else horizontal_edges<LUMA, SIMPLE, false>(me, above, q, top, L, ktop, kinner);
      if (handed) __syncwarp((1u << LPM) - 1u);
      if (up) {
        const uint2 v = *(const uint2*)(msg + q * 8);
        if (q == 0) expect_message(&link->in_bar[c & 1]);
        send8(up_rings + slot * SLOT, v, up_bar + (c & 1) * 8);
      }
    }
    slot = c < 0 ? 0 : (slot == RING - 1 ? 0 : slot + 1);
    __syncthreads();
  }
  return total;
}

// The end of a split pass. A CTA's shared memory must not go away under a message on
// its way to it, and a cluster barrier does not order asynchronous stores: it orders
// the plain ones that tell each neighbour how many messages it was sent. Nothing is
// left to wait for unless a wait ran out (tests/test_cluster_leave.py runs this under
// random interleavings). Written with the instructions themselves and apart from
// run_split: through cooperative groups' remote pointer and barrier a 1280x720 pass
// took 170 us instead of 158, every step of it slower.
__device__ __forceinline__ void leave_split(const LfArgs& a, Link* link, int rank) {
  const Rows R(a, 2);
  const int g = threadIdx.x / LPM, q = threadIdx.x & (LPM - 1);
  const int s0 = rank_row(a.n_scored, a.split, rank), s1 = rank_row(a.n_scored, a.split, rank + 1);
  const bool handed = g == 0 && s0 < s1 && R.top(s0);
  const bool hand_down = s0 + g == s1 - 1 && s1 < a.n_scored && R.top(s1);
  if (hand_down) store_cluster(cluster_at(smem_at(&link->sent_in[q]), rank + 1), link->n_down[q]);
  if (handed) store_cluster(cluster_at(smem_at(&link->sent_ret[q]), rank - 1), link->n_up[q]);
  __syncwarp();
  asm volatile("barrier.cluster.arrive.release.aligned;\n barrier.cluster.wait.acquire.aligned;" ::: "memory");
  if (handed && q == 0) await_messages(link->in_bar, link->n_up[0], link->sent_in);
  if (hand_down && q == 0) await_messages(link->ret_bar, link->n_back[0], link->sent_ret);
}

// LoopFilterParams::derive (src/loop_filter.rs:99-148) for every filter
// class of candidate (lv, sh).
template <bool SIMPLE>
__device__ __forceinline__ void class_limits(const LfArgs& a, int lv, int sh, bool luma, Limits* lim) {
  for (int i = threadIdx.x; i < CLASSES; i += blockDim.x) {
    const int level = (lv == 0 && a.level0_unfiltered) ? 0 : mb_level(a.base, lv, class_record(i));
    const int interior = interior_limit(level, sh);
    const int hev = a.base.key_frame ? (level >= 40 ? 2 : (level >= 15 ? 1 : 0))
                                     : (level >= 40 ? 3 : (level >= 20 ? 2 : (level >= 15 ? 1 : 0)));
    const int mbedge = min((level + 2) * 2 + interior, 255), subedge = min(level * 2 + interior, 255);
    // The simple filter leaves chroma alone and has no flatness or variance
    // test.
    const bool off = level == 0 || (SIMPLE && !luma);
    Limits L;
    L.flat = off ? DISABLED : (SIMPLE ? pk(0x7fff - 255) : pk(0x7fff - interior));
    L.hev = SIMPLE ? DISABLED : pk(0x7fff - hev);
    L.mb = pk(0x7fff - (2 * mbedge + 1));
    L.sub = pk(0x7fff - (2 * subedge + 1));
    lim[i] = L;
  }
}

// CTA `cta` of a picture's passes: `split` CTAs per pass; one pass per
// candidate (BOTH), or the luma passes of every candidate and then the chroma
// passes; `np` candidates one after another.
template <bool SIMPLE, bool CL, bool BOTH, bool PRE, bool TILED>
__device__ __forceinline__ void sweep_body(const LfArgs& a, int cta, int np) {
  extern __shared__ __align__(16) uint8_t rings[];
  __shared__ Limits lim[CLASSES];
  __shared__ Limits lim_c[BOTH && SIMPLE ? CLASSES : 1];  // the simple filter's chroma limits differ
  __shared__ unsigned long long red[32];
  __shared__ unsigned taken[2];  // groups taken at even and odd steps
  __shared__ Link link;
  const int rank = CL ? cta % a.split : 0, item = CL ? cta / a.split : cta;
  const int per_plane = (a.n_cands + np - 1) / np;
  const bool luma = BOTH || item < per_plane;
  const int first = (luma ? item : item - per_plane) * np, last = min(first + np, a.n_cands);
  const int q = threadIdx.x & (LPM - 1);
  for (int k = first; k < last; k++) {
    const int lv = a.cands[2 * k], sh = a.cands[2 * k + 1], mk = entry_mask(a, k, lv, sh);
    class_limits<SIMPLE>(a, lv, sh, luma, lim);
    if constexpr (BOTH && SIMPLE) class_limits<SIMPLE>(a, lv, sh, false, lim_c);
    if (threadIdx.x == 0) {
      taken[0] = blockDim.x >> 5;
      if constexpr (CL) init_link(&link, a.spin_limit);
    }
    if constexpr (CL) cg::this_cluster().sync();
    else __syncthreads();
    uint64_t v;
    NoPlane none;
    if constexpr (CL) {
      v = luma ? run_split<true, SIMPLE>(a, lim, rings, &link, rank)
               : run_split<false, SIMPLE>(a, lim, rings, &link, rank);
      leave_split(a, &link, rank);
    } else if constexpr (BOTH) {
      PlanePass<true, SIMPLE, TILED> y(a, rings, q);
      PlanePass<false, SIMPLE, TILED> c(a, rings + a.n_sets * Geo<true>::SET, q);
      v = run_pass<PRE>(a, lim, SIMPLE ? lim_c : lim, taken, (int)blockIdx.x, y, c);
    } else if (luma) {
      PlanePass<true, SIMPLE, TILED> y(a, rings, q);
      v = run_pass<PRE>(a, lim, lim, taken, (int)blockIdx.x, y, none);
    } else {
      PlanePass<false, SIMPLE, TILED> c(a, rings, q);
      v = run_pass<PRE>(a, lim, lim, taken, (int)blockIdx.x, c, none);
    }
    if (!a.ssd_out) continue;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(FULL, v, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    if (threadIdx.x < 32) {
      unsigned long long x = threadIdx.x < (blockDim.x >> 5) ? red[threadIdx.x] : 0ull;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(FULL, x, o);
      if (threadIdx.x < 8 && ((mk >> threadIdx.x) & 1))
        atomicAdd((unsigned long long*)&a.ssd_out[lv * 8 + threadIdx.x], x);
    }
    __syncthreads();
  }
}

// Threads a CTA may have: the register budget of the three shapes.
constexpr int max_threads(bool cl, bool both) { return cl ? 512 : (both ? 768 : 1024); }

template <bool SIMPLE, bool CL, bool BOTH, bool PRE, bool TILED>
__global__ void __launch_bounds__(max_threads(CL, BOTH), 1) lf_sweep_kernel(const __grid_constant__ LfArgs a, int np) {
  sweep_body<SIMPLE, CL, BOTH, PRE, TILED>(a, blockIdx.x, np);
}

// Many pictures' sweeps in one launch: CTA offsets per job as in find_job.
template <bool SIMPLE, bool CL, bool BOTH, bool PRE, bool TILED>
__global__ void __launch_bounds__(max_threads(CL, BOTH), 1)
    lf_sweep_batch_kernel(const LfArgs* __restrict__ jobs, const uint32_t* __restrict__ cta_start, int n_jobs,
                          int np) {
  __shared__ LfArgs sa;
  __shared__ uint32_t first[2];
  find_job(jobs, cta_start, n_jobs, &sa, first);
  sweep_body<SIMPLE, CL, BOTH, PRE, TILED>(sa, (int)(blockIdx.x - first[0]), np);
}

// Plain visible-window SSD of a reconstruction (reconstruction_ssd).
__global__ void __launch_bounds__(256) ssd_kernel(const uint8_t* rec, uint64_t rs, const uint8_t* src, uint64_t ss,
                                                  int w, int h, unsigned long long* out) {
  uint64_t acc = 0;
  const size_t n = (size_t)w * h;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    int y = (int)(i / w), x = (int)(i % w);
    int d = (int)rec[(size_t)y * rs + x] - (int)src[(size_t)y * ss + x];
    acc += (uint64_t)(d * d);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(FULL, acc, o);
  if ((threadIdx.x & 31) == 0) atomicAdd(out, (unsigned long long)acc);
}

// ------------------------------------------------------------------- host

vp8a_status validate_config(const vp8a_filter_config* c) {
  if (c->loop_filter_level > 63) {
    vp8a::set_error("loop_filter_level > 63");
    return VP8A_E_LOOP_FILTER_LEVEL_OUT_OF_RANGE;
  }
  if (c->sharpness_level > 7) {
    vp8a::set_error("sharpness_level > 7");
    return VP8A_E_SHARPNESS_LEVEL_OUT_OF_RANGE;
  }
  return VP8A_OK;
}

// The scored rows of whole frames (every_rows = 0) or two-row bands, and
// the wavefront's steps.
void set_rows(LfArgs& a, uint32_t every_rows) {
  if (every_rows == 0) {
    a.band_step = 0;
    a.n_scored = a.mb_rows;
    a.max_t0 = a.n_scored - 1;
  } else {
    const int step = every_rows < 2 ? 2 : (int)std::min<uint32_t>(every_rows, 1u << 20);
    const int bands = (a.mb_rows + step - 1) / step;
    a.band_step = step;
    // The last band holds one row when the picture ends after it.
    a.n_scored = 2 * bands - ((bands - 1) * step + 1 >= a.mb_rows ? 1 : 0);
    a.max_t0 = a.n_scored > 1 ? 1 : 0;
  }
}

// The widest loads the planes' bases and strides allow.
void set_alignment(LfArgs& a) {
  auto al = [](const void* p, uint64_t stride, unsigned k) { return (uintptr_t)p % k == 0 && stride % k == 0; };
  auto of = [&](const uint8_t* y, const uint8_t* u, const uint8_t* v, uint64_t ys, uint64_t cs) {
    if (al(y, ys, 16) && al(u, cs, 8) && al(v, cs, 8)) return 2;
    return al(y, ys, 4) && al(u, cs, 4) && al(v, cs, 4) ? 1 : 0;
  };
  a.recon_align = of(a.y, a.u, a.v, a.ys, a.cs);
  a.source_align = a.sy ? of(a.sy, a.su, a.sv, a.sys, a.scs) : 0;
}

// Stages planes, per-MB info and (optionally) the source; sets the scored
// rows: whole frames (every_rows = 0) or sampled bands.
vp8a_status stage_lf(vp8a_ctx* ctx, vp8a::Stager& st, const vp8a_planes* planes, const vp8a_mb_lf_info* mbs,
                     const vp8a_filter_config* base, const vp8a_source* src, uint32_t every_rows, bool write_back,
                     LfArgs* out) {
  if (!planes || !mbs || !base) {
    vp8a::set_error("null argument");
    return VP8A_E_INVALID_ARGUMENT;
  }
  if (planes->mb_cols == 0 || planes->mb_rows == 0 || planes->mb_cols > 1024 || planes->mb_rows > 1024) {
    vp8a::set_error("plane MB grid out of range");
    return VP8A_E_INVALID_DIMENSIONS;
  }
  if (planes->y_stride < (uint64_t)planes->mb_cols * 16 || planes->uv_stride < (uint64_t)planes->mb_cols * 8) {
    vp8a::set_error("plane stride below the MB-padded width");
    return VP8A_E_INVALID_ARGUMENT;
  }
  vp8a_status s = validate_config(base);
  if (s != VP8A_OK) return s;
  LfArgs& a = *out;
  const int cols = (int)planes->mb_cols, rows = (int)planes->mb_rows;
  const size_t yb = planes->y_stride * (size_t)rows * 16, cb = planes->uv_stride * (size_t)rows * 8;
  const void* d;
  void* dm;
  if (write_back) {
    if ((s = st.inout(planes->y, yb, &dm)) != VP8A_OK) return s;
    a.y = (const uint8_t*)dm;
    a.oy = (uint8_t*)dm;
    if ((s = st.inout(planes->u, cb, &dm)) != VP8A_OK) return s;
    a.u = (const uint8_t*)dm;
    a.ou = (uint8_t*)dm;
    if ((s = st.inout(planes->v, cb, &dm)) != VP8A_OK) return s;
    a.v = (const uint8_t*)dm;
    a.ov = (uint8_t*)dm;
  } else {
    if ((s = st.in(planes->y, yb, &d)) != VP8A_OK) return s;
    a.y = (const uint8_t*)d;
    if ((s = st.in(planes->u, cb, &d)) != VP8A_OK) return s;
    a.u = (const uint8_t*)d;
    if ((s = st.in(planes->v, cb, &d)) != VP8A_OK) return s;
    a.v = (const uint8_t*)d;
  }
  a.ys = planes->y_stride;
  a.cs = planes->uv_stride;
  a.mb_cols = cols;
  a.mb_rows = rows;
  if ((s = st.in(mbs, sizeof(vp8a_mb_lf_info) * (size_t)cols * rows, &d)) != VP8A_OK) return s;
  a.mbs = (const vp8a_mb_lf_info*)d;
  a.base = *base;
  a.status = ctx->d_status;
  a.spin_limit = (unsigned)std::min<uint64_t>(ctx->wait_limit, 0xffffffffu);
  if (src) {
    if (src->width == 0 || src->height == 0 || src->width > (uint32_t)cols * 16 ||
        src->height > (uint32_t)rows * 16) {
      vp8a::set_error("source size does not fit the MB grid");
      return VP8A_E_REFERENCE_DIMENSIONS_MISMATCH;
    }
    const uint32_t w = src->width, h = src->height, cw = (w + 1) / 2, ch = (h + 1) / 2;
    if (src->y_stride < w || src->uv_stride < cw) {
      vp8a::set_error("source stride below width");
      return VP8A_E_INVALID_ARGUMENT;
    }
    if ((s = st.in(src->y, src->y_stride * (size_t)(h - 1) + w, &d)) != VP8A_OK) return s;
    a.sy = (const uint8_t*)d;
    if ((s = st.in(src->u, src->uv_stride * (size_t)(ch - 1) + cw, &d)) != VP8A_OK) return s;
    a.su = (const uint8_t*)d;
    if ((s = st.in(src->v, src->uv_stride * (size_t)(ch - 1) + cw, &d)) != VP8A_OK) return s;
    a.sv = (const uint8_t*)d;
    a.sys = src->y_stride;
    a.scs = src->uv_stride;
    a.width = (int)w;
    a.height = (int)h;
  }
  set_rows(a, every_rows);
  set_alignment(a);
  return VP8A_OK;
}

// ------------------------------------------------------------ launch shape

// Rows one rank carries at once, at most: all of its rows, or those of the
// wavefront (a row is busy for mb_cols + RING steps, and the next starts
// `skew` steps later).
int active_rows(const LfArgs& a, int split) {
  const int mine = (a.n_scored + split - 1) / split;
  return a.band_step ? mine : std::min(mine, (a.mb_cols + RING + skew_of(split) - 1) / skew_of(split));
}

// The split's steps and ring sets: a row takes set (s - s0) & mask, free again
// once the row using it has scored its last MB.
void set_split(LfArgs& a, int split) {
  const int mine = (a.n_scored + split - 1) / split;
  int pow2 = 1;
  while (pow2 < active_rows(a, split)) pow2 *= 2;
  a.split = split;
  a.steps = skew_of(split) * a.max_t0 + a.mb_cols + RING;
  const bool wrap = split == 1 && !a.band_step && pow2 < mine;
  a.n_sets = wrap ? pow2 : mine;
  a.set_mask = wrap ? pow2 - 1 : 0x7fffffff;
}

size_t ring_bytes(const LfArgs& a, bool both) {
  return (size_t)a.n_sets * (Geo<true>::SET + (both ? Geo<false>::SET : 0));
}

// The shared memory a CTA's rings may take, and what a CTA takes besides them
// (its static part and the 1 KB the system reserves).
constexpr size_t MAX_RING_BYTES = 220 << 10, CTA_SMEM = 2304;

// What a launch of `candidates` per picture takes, in seconds, whole or split
// (fits of measured launches, 176x144 to 3840x2160 and 32x4096 to 4096x128). Whole
// passes: 0.36 ns per MB and candidate, but no less than one pass's chain of steps,
// whose step grows with the rows that are busy at once and so with the MBs that the
// CTA's warps take one after another (one pass alone, 1080p: 0.76 ms for 257 steps).
// Split passes: a step of 1.1 us whatever the picture (0.22 ms), 2.7 times the work
// (half of the lanes wait for inner edges that their own MB does not have), and
// every CTA stays for all the steps, 16 threads a row of the 512 that an SM holds,
// though in a tall and narrow picture few steps have work for it (128x4096, the whole
// grid: 6.6 ms split, 0.8 ms whole; one frame's filter 0.3 and 0.8).
double whole_time(const std::vector<LfArgs*>& jobs, double candidates) {
  double chain = 0, mbs = 0;
  for (const LfArgs* a : jobs) {
    chain = std::max(chain, (skew_of(1) * a->max_t0 + a->mb_cols) * (0.9e-6 + 0.0296e-6 * active_rows(*a, 1)));
    mbs += (double)a->n_scored * a->mb_cols;
  }
  return std::max(chain, 0.36e-9 * candidates * mbs);
}
double split_time(const std::vector<LfArgs*>& jobs, double candidates) {
  constexpr double THREADS = 148 * max_threads(true, false);
  double chain = 0, mbs = 0, stay = 0;
  for (const LfArgs* a : jobs) {
    const double c = (skew_of(2) * a->max_t0 + a->mb_cols) * 1.1e-6;
    chain = std::max(chain, c);
    mbs += (double)a->n_scored * a->mb_cols;
    stay += c * 2 * LPM * a->n_scored;
  }
  return std::max({chain, 0.97e-9 * candidates * mbs, candidates * stay / THREADS});
}

// CTAs per pass for a call whose largest launch has `candidates` per picture:
// where splitting pays, bands of about 12 rows (one pass, ms: 3840x2160 in 8
// bands 0.49, in 4 0.60; 1920x1080 8: 0.22, 4: 0.27; 1280x720 8: 0.16, 4: 0.15,
// 2: 0.16; 640x360 4: 0.08, 2: 0.08), of 17 when there are many candidates; and
// always as many as make the rings and rows fit.
int pick_split(const vp8a_ctx* ctx, double candidates, const std::vector<LfArgs*>& jobs) {
  int split = 1, rows = 1;
  auto feasible = [&](int k) {
    for (const LfArgs* a : jobs) {
      LfArgs b = *a;
      set_split(b, k);
      if (ring_bytes(b, false) > MAX_RING_BYTES || (k > 1 && LPM * b.n_sets > max_threads(true, false))) return false;
    }
    return true;
  };
  for (const LfArgs* a : jobs) rows = std::max(rows, a->n_scored);
  if (!ctx->force_layout[0] && split_time(jobs, candidates) < whole_time(jobs, candidates)) {
    const int band = candidates < 32 ? 12 : 17;
    while (split < MAX_CLUSTER && rows > band * split) split *= 2;
  }
  while (split < MAX_CLUSTER_FIT && !feasible(split)) split *= 2;
  return split;
}

// The schedule's buffers.
size_t meta_bytes(const LfArgs& a) { return sizeof(uint4) * (size_t)a.steps; }
size_t list_bytes(const LfArgs& a) {  // or the split passes' info bytes
  return (sizeof(uint16_t) * (size_t)a.n_scored * (a.mb_cols + RING) + 15) & ~(size_t)15;
}
size_t tile_bytes(const LfArgs& a) { return (size_t)TILE * a.n_scored * a.mb_cols; }
size_t prepared_bytes(const LfArgs& a) { return meta_bytes(a) + list_bytes(a) + tile_bytes(a) * (a.sy ? 2 : 1); }
void place_prepared(LfArgs& a, uint8_t* at) {
  a.meta = (uint4*)at;
  a.list = (uint16_t*)(at + meta_bytes(a));
  a.info = at + meta_bytes(a);
  a.recon_tiles = at + meta_bytes(a) + list_bytes(a);
  a.source_tiles = a.recon_tiles + tile_bytes(a);
}
// CTAs of lf_schedule_kernel.
unsigned prepare_ctas(const LfArgs& a) {
  const long warps = (long)(a.split > 1 ? 0 : a.steps) + (long)a.n_scored * ((a.mb_cols + 1) / 2);
  return (unsigned)((warps + SCHED_WARPS - 1) / SCHED_WARPS);
}

// A launch's shape: threads per CTA, next-row prefetch, luma and chroma in
// one pass, candidates per CTA.
struct Shape {
  int threads, pre, both, np;
};

template <bool SIMPLE, bool CL, bool BOTH, bool PRE, bool TILED>
vp8a_status launch_variant(vp8a_ctx* ctx, const Shape& S, unsigned grid, size_t smem, int split, const LfArgs& a,
                           const LfArgs* dj, const uint32_t* ds, int n_jobs) {
  const auto one = lf_sweep_kernel<SIMPLE, CL, BOTH, PRE, TILED>;
  const auto many = lf_sweep_batch_kernel<SIMPLE, CL, BOTH, PRE, true>;
  const void* k = dj ? (const void*)many : (const void*)one;
  // The kernel's limit, shared by every context's launches on the device: always the
  // most that any takes, so that no thread lowers it between another's two calls.
  VP8A_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)MAX_RING_BYTES));
  if (split > MAX_CLUSTER) VP8A_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = (unsigned)split;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3((unsigned)S.threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = ctx->stream;
  cfg.attrs = at;
  cfg.numAttrs = CL ? 1 : 0;
  int per_sm = 0;
  VP8A_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, S.threads, smem));
  ctx->last_layout[0] = S.np;
  ctx->last_layout[1] = S.threads;
  ctx->last_layout[2] = S.pre;
  ctx->last_layout[3] = std::max(per_sm, 1);
  if (dj) VP8A_CUDA(cudaLaunchKernelEx(&cfg, many, dj, ds, n_jobs, S.np));
  else VP8A_CUDA(cudaLaunchKernelEx(&cfg, one, a, S.np));
  VP8A_CUDA(cudaGetLastError());
  ctx->launches++;
  return VP8A_OK;
}

template <bool SIMPLE>
vp8a_status launch(vp8a_ctx* ctx, const Shape& S, unsigned grid, size_t smem, int split, const LfArgs& a,
                   const LfArgs* dj, const uint32_t* ds, int n_jobs) {
  if (split > 1) return launch_variant<SIMPLE, true, false, true, true>(ctx, S, grid, smem, split, a, dj, ds, n_jobs);
  if (!a.recon_tiles)
    return launch_variant<SIMPLE, false, false, false, false>(ctx, S, grid, smem, split, a, dj, ds, n_jobs);
  if (S.both)
    return S.pre ? launch_variant<SIMPLE, false, true, true, true>(ctx, S, grid, smem, split, a, dj, ds, n_jobs)
                 : launch_variant<SIMPLE, false, true, false, true>(ctx, S, grid, smem, split, a, dj, ds, n_jobs);
  return S.pre ? launch_variant<SIMPLE, false, false, true, true>(ctx, S, grid, smem, split, a, dj, ds, n_jobs)
               : launch_variant<SIMPLE, false, false, false, true>(ctx, S, grid, smem, split, a, dj, ds, n_jobs);
}

unsigned cta_count(const LfArgs& a, const Shape& S) {
  return (S.both ? 1u : 2u) * (unsigned)((a.n_cands + S.np - 1) / S.np) * (unsigned)a.split;
}

// The shape for a picture's passes. Measured over the grid's 436 candidates
// (ms; one pass per candidate with t threads | luma and chroma apart):
// 3840x2160 (rings 146 KB, one CTA an SM) t 768 5.12, 512 5.37, 256 6.69 |
// 5.14; 1920x1080 (73 KB, three) 256 1.27, 384 1.66, 192 1.30 | 1.50;
// 1280x720 0.60 | 0.63; 640x360 (23 rows) 0.28 | 0.24. So: the SM's 768
// threads shared by the CTAs whose rings fit, but no fewer than 256 (more
// than three CTAs an SM never run); where a step has few MBs the passes are
// bound by their step latency and twice as many, half as long, run better.
vp8a_status pick_shape(vp8a_ctx* ctx, const LfArgs& a, Shape* S) {
  const int rows = active_rows(a, a.split), full = std::max(32, (LPM * rows + 31) / 32 * 32);
  const bool fits = a.recon_tiles && a.split == 1 && ring_bytes(a, true) <= MAX_RING_BYTES;
  if (a.split > 1) {
    *S = Shape{(LPM * a.n_sets + 31) / 32 * 32, 1, 0, 1};
  } else if (fits && rows > 32) {
    const int per_sm = std::max(1, std::min(3, (int)((228 << 10) / (ring_bytes(a, true) + CTA_SMEM))));
    *S = Shape{std::min(full, max_threads(false, true) / per_sm), 0, 1, 1};
  } else {
    *S = Shape{std::min(full, rows > 32 ? 512 : 128), 0, 0, 1};
  }
  if (ctx->force_layout[0]) {
    if (ctx->force_layout[1] > max_threads(false, false) || a.split > 1) {
      vp8a::set_error("the forced sweep layout does not fit this picture");
      return VP8A_E_INVALID_ARGUMENT;
    }
    *S = Shape{ctx->force_layout[1], ctx->force_layout[2],
               fits && ctx->force_layout[1] <= max_threads(false, true), ctx->force_layout[0]};
  }
  return VP8A_OK;
}

// Splits and schedules one picture's passes; the schedule serves every launch
// of the call, whose largest has `candidates`. The first launch's candidates
// must be in place (their table entries are cleared).
vp8a_status schedule(vp8a_ctx* ctx, vp8a::Stager& st, LfArgs* a, int candidates) {
  set_split(*a, pick_split(ctx, candidates, {a}));
  void* d;
  vp8a_status s;
  if ((s = st.scratch(prepared_bytes(*a), &d)) != VP8A_OK) return s;
  place_prepared(*a, (uint8_t*)d);
  lf_schedule_kernel<<<prepare_ctas(*a), SCHED_WARPS * 32, 0, ctx->stream>>>(*a);
  VP8A_CUDA(cudaGetLastError());
  ctx->launches++;
  return VP8A_OK;
}

// Runs the scheduled passes of a.n_cands candidates already in device memory.
vp8a_status run_sweep(vp8a_ctx* ctx, const LfArgs& a) {
  if (a.n_cands == 0) return VP8A_OK;
  Shape S;
  vp8a_status s = pick_shape(ctx, a, &S);
  if (s != VP8A_OK) return s;
  const size_t smem = ring_bytes(a, S.both);
  return a.base.simple ? launch<true>(ctx, S, cta_count(a, S), smem, a.split, a, nullptr, nullptr, 0)
                       : launch<false>(ctx, S, cta_count(a, S), smem, a.split, a, nullptr, nullptr, 0);
}

// The whole 64 x 8 grid as distinct filter passes. Two sharpness values
// of one level filter identically when every MB level the configuration can
// produce from that level (each segment, reference and mode class of
// calculate_mb_filter_level_inter) has the same interior limit under both:
// the interior limit and the level fix every parameter of the §15 filters
// (LoopFilterParams::derive, src/loop_filter.rs:99-148). Each pass fills the
// table entries of its sharpness group (`masks`); level 0 is one pass for
// all eight (score_filter_candidate's unfiltered short cut).
// Writes the passes into `pairs` (2 per pass) and `masks` (1 per pass;
// room for 1 + 63 * 8 passes) and returns their number. No heap memory.
int grid_passes(const vp8a_filter_config& base, uint8_t* pairs, uint8_t* masks) {
  int n = 0;
  pairs[0] = pairs[1] = 0;
  masks[n++] = 0xff;
  vp8a_mb_lf_info classes[4 * 11];
  int nc = 0;
  const int nseg = base.segmentation_enabled ? 4 : 1;
  for (int seg = 0; seg < nseg; seg++) {
    vp8a_mb_lf_info m{};
    m.segment_id = (int8_t)seg;
    m.ref_frame = VP8A_REF_INTRA;
    m.inter_mode = VP8A_MODE_NONE;
    for (int bp = 0; bp < 2; bp++) {
      m.y_mode_is_bpred = (uint8_t)bp;
      classes[nc++] = m;
    }
    m.y_mode_is_bpred = 0;
    for (int ref = VP8A_REF_LAST; ref <= VP8A_REF_ALTREF; ref++)
      for (int mode : {VP8A_MODE_ZERO, VP8A_MODE_SPLIT, VP8A_MODE_NEAREST}) {
        m.ref_frame = (uint8_t)ref;
        m.inter_mode = (uint8_t)mode;
        classes[nc++] = m;
      }
  }
  for (int level = 1; level < 64; level++) {
    uint8_t done = 0;
    for (int s0 = 0; s0 < 8; s0++) {
      if (done >> s0 & 1) continue;
      uint8_t mask = 0;
      for (int s1 = s0; s1 < 8; s1++) {
        bool same = true;
        for (int c = 0; c < nc; c++) {
          const int l = mb_level(base, level, classes[c]);
          if (l != 0 && interior_limit(l, s0) != interior_limit(l, s1)) same = false;
        }
        if (same) mask |= (uint8_t)(1u << s1);
      }
      done |= mask;
      pairs[2 * n] = (uint8_t)level;
      pairs[2 * n + 1] = (uint8_t)s0;
      masks[n++] = mask;
    }
  }
  return n;
}

void grid_candidates(const vp8a_filter_config& base, std::vector<uint8_t>& pairs, std::vector<uint8_t>& masks) {
  pairs.resize(2 * (1 + 63 * 8));
  masks.resize(1 + 63 * 8);
  const int n = grid_passes(base, pairs.data(), masks.data());
  pairs.resize(2 * n);
  masks.resize(n);
}

// Upload a grid's candidate pairs and masks into `a` (level 0 and the
// levels lo..hi).
vp8a_status upload_grid(vp8a_ctx* ctx, vp8a::Stager& st, const vp8a_filter_config& base, LfArgs* a, int lo = 1,
                        int hi = 63) {
  std::vector<uint8_t> all_pairs, all_masks, pairs, masks;
  grid_candidates(base, all_pairs, all_masks);
  for (size_t i = 0; i < all_masks.size(); i++) {
    const int level = all_pairs[2 * i];
    if (level != 0 && (level < lo || level > hi)) continue;
    pairs.push_back(all_pairs[2 * i]);
    pairs.push_back(all_pairs[2 * i + 1]);
    masks.push_back(all_masks[i]);
  }
  const size_t n = masks.size();
  std::vector<uint8_t> blob(3 * n);
  memcpy(blob.data(), pairs.data(), 2 * n);
  memcpy(blob.data() + 2 * n, masks.data(), n);
  void* d;
  vp8a_status s;
  if ((s = st.upload(blob.data(), blob.size(), &d)) != VP8A_OK) return s;
  a->cands = (const uint8_t*)d;
  a->cand_mask = (const uint8_t*)d + 2 * n;
  a->n_cands = (int)n;
  return VP8A_OK;
}

vp8a_status upload_candidates(vp8a::Stager& st, LfArgs* a, const uint8_t* cands, int n) {
  void* d;
  vp8a_status s;
  if ((s = st.upload(cands, (size_t)n * 2, &d)) != VP8A_OK) return s;
  a->cands = (const uint8_t*)d;
  a->cand_mask = nullptr;
  a->n_cands = n;
  return VP8A_OK;
}

// Whether a walk scores every level of the base sharpness in one launch
// instead of its `first` candidates and then the refinements (`stages`
// launches of up to 6 candidates, each with about 25 us of copies and waiting
// around it): the 64 levels cost more work but one chain of steps.
bool score_all_levels(const std::vector<LfArgs*>& jobs, int first, int stages) {
  auto time = [&](int n) { return std::min(split_time(jobs, n), whole_time(jobs, n)); };
  return time(64) < time(first) + stages * (time(6) + 25e-6);
}

std::vector<uint8_t> all_levels(uint8_t sharp) {
  std::vector<uint8_t> c;
  for (int l = 0; l < 64; l++) c.insert(c.end(), {(uint8_t)l, sharp});
  return c;
}

vp8a_status timed_out() {
  vp8a::set_error("device wavefront wait exceeded its iteration budget");
  return VP8A_E_DEVICE_TIMEOUT;
}

// Ends a call whose launch may be split: with host buffers the call has
// waited for it, so a wait that ran out is reported now; with device buffers
// the next vp8a_ctx_synchronize reports it.
vp8a_status finish_sweep(vp8a_ctx* ctx, vp8a::Stager& st, bool split) {
  vp8a_status s = st.finish();
  return s == VP8A_OK && split && st.touched_host() ? vp8a::check_device_status(ctx) : s;
}

// Score `cands` into `table` (host, 513 entries, level * 8 + sharp).
// The first call of a walk schedules the picture.
vp8a_status score_candidates(vp8a_ctx* ctx, vp8a::Stager& st, LfArgs& a, const std::vector<uint8_t>& cands,
                             uint64_t* table) {
  const int n = (int)(cands.size() / 2);
  vp8a_status s = upload_candidates(st, &a, cands.data(), n);
  if (s != VP8A_OK) return s;
  // The launch's status word is the table's entry 512.
  VP8A_CUDA(cudaMemsetAsync(a.ssd_out, 0, 513 * sizeof(uint64_t), ctx->stream));
  a.status = (unsigned*)(a.ssd_out + 512);
  if (!a.meta && (s = schedule(ctx, st, &a, n)) != VP8A_OK) return s;
  if ((s = run_sweep(ctx, a)) != VP8A_OK) return s;
  VP8A_CUDA(cudaMemcpyAsync(table, a.ssd_out, 513 * sizeof(uint64_t), cudaMemcpyDeviceToHost, ctx->stream));
  VP8A_CUDA(cudaStreamSynchronize(ctx->stream));
  return table[512] ? timed_out() : VP8A_OK;
}

// ----------------------------------------------- sweep without allocation
//
// vp8a_filter_sweep_noalloc runs the same sweep kernel as vp8a_filter_sweep
// for callers that cannot allocate device memory while they run. Its scratch
// (the candidate list and the step schedule) lives in one fixed array of
// device memory owned by the library; every buffer the caller names must
// already be on the device.
constexpr int NA_MAX_MB_COLS = 256;  // 4096 pixels
constexpr int NA_MAX_MB_ROWS = 136;  // 2176 pixels
constexpr int NA_MAX_STEPS = 2 * (NA_MAX_MB_ROWS - 1) + NA_MAX_MB_COLS + RING;
constexpr int NA_CANDIDATES = 1 + 63 * 8;
// Scratch layout (bytes).
constexpr size_t NA_CANDS = 0;                                        // (level, sharpness) pairs
constexpr size_t NA_MASK = (2 * NA_CANDIDATES + 15) & ~(size_t)15;    // u8 sharpness mask per pass
constexpr size_t NA_META = (NA_MASK + NA_CANDIDATES + 15) & ~(size_t)15;
constexpr size_t NA_LIST = NA_META + sizeof(uint4) * NA_MAX_STEPS;
constexpr size_t NA_BYTES = NA_LIST + sizeof(uint16_t) * (size_t)NA_MAX_MB_ROWS * (NA_MAX_MB_COLS + RING);
static_assert((size_t)NA_MAX_MB_ROWS * Geo<true>::SET <= MAX_RING_BYTES, "every row's slot ring fits in one CTA");

// The grid's filter passes (grid_candidates: level 0, then one pass per
// group of sharpness values that filter identically), passed to the
// schedule kernel by value (1.5 KB of kernel parameters) so that no host
// buffer has to be staged.
struct NaGrid {
  int n;
  uint8_t pairs[2 * NA_CANDIDATES];
  uint8_t masks[NA_CANDIDATES];
};

// The library's only copy; every call on a device shares it (about 80 KiB,
// held by each device that loads the library until the process exits).
static __device__ __align__(256) uint8_t g_sweep_scratch[NA_BYTES];

// Candidates, cleared table (the grid fills every entry) and step schedule.
__global__ void __launch_bounds__(SCHED_WARPS * 32)
    sweep_schedule_kernel(const __grid_constant__ LfArgs a, uint8_t* scr, const __grid_constant__ NaGrid grid) {
  if (blockIdx.x == 0) {
    for (int i = threadIdx.x; i < grid.n; i += blockDim.x) {
      scr[NA_CANDS + 2 * i] = grid.pairs[2 * i];
      scr[NA_CANDS + 2 * i + 1] = grid.pairs[2 * i + 1];
      scr[NA_MASK + i] = grid.masks[i];
    }
    for (int i = threadIdx.x; i < 512; i += blockDim.x) a.ssd_out[i] = 0;
  }
  const int idx = blockIdx.x * SCHED_WARPS + (threadIdx.x >> 5);
  if (idx < a.steps) schedule_step(a, idx, threadIdx.x & 31);
}

// Device address of g_sweep_scratch on `dev` (current), looked up once per
// device. In host code the array's name only stands in for the symbol.
vp8a_status sweep_scratch(int dev, uint8_t** out) {
  static std::mutex mu;
  static void* ptr[64] = {};
  std::lock_guard<std::mutex> lock(mu);
  if (dev < 0 || dev >= 64) {
    vp8a::set_error("device index out of range");
    return VP8A_E_INVALID_ARGUMENT;
  }
  if (!ptr[dev]) {
    void* p = nullptr;
    const cudaError_t e = cudaGetSymbolAddress(&p, g_sweep_scratch);
    if (e != cudaSuccess) return vp8a::cuda_fail(e, "cudaGetSymbolAddress(g_sweep_scratch)");
    ptr[dev] = p;
  }
  *out = (uint8_t*)ptr[dev];
  return VP8A_OK;
}

// True when `p` is device (or managed) memory usable on `dev`.
bool device_resident(const void* p, int dev) {
  if (!p) return false;
  cudaPointerAttributes at;
  if (cudaPointerGetAttributes(&at, p) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return (at.type == cudaMemoryTypeDevice && at.device == dev) || at.type == cudaMemoryTypeManaged;
}

}  // namespace

extern "C" {

vp8a_status vp8a_filter_frame(vp8a_ctx* ctx, vp8a_planes* planes, const vp8a_mb_lf_info* mbs,
                              const vp8a_filter_config* config) {
  if (!ctx) return VP8A_E_INVALID_ARGUMENT;
  VP8A_CUDA(cudaSetDevice(ctx->device));
  vp8a::Stager st(ctx);
  LfArgs a{};
  vp8a_status s = stage_lf(ctx, st, planes, mbs, config, nullptr, 0, true, &a);
  if (s != VP8A_OK) return s;
  const uint8_t cand[2] = {config->loop_filter_level, config->sharpness_level};
  if ((s = upload_candidates(st, &a, cand, 1)) != VP8A_OK) return s;
  if ((s = schedule(ctx, st, &a, 1)) != VP8A_OK) return s;
  if ((s = run_sweep(ctx, a)) != VP8A_OK) return s;
  return finish_sweep(ctx, st, a.split > 1);
}

vp8a_status vp8a_reconstruction_ssd(vp8a_ctx* ctx, const vp8a_planes* planes, const vp8a_source* src,
                                    uint64_t* ssd_out) {
  if (!ctx || !planes || !src || !ssd_out) return VP8A_E_INVALID_ARGUMENT;
  VP8A_CUDA(cudaSetDevice(ctx->device));
  vp8a::Stager st(ctx);
  const uint32_t w = src->width, h = src->height, cw = (w + 1) / 2, ch = (h + 1) / 2;
  if (w == 0 || h == 0 || w > planes->mb_cols * 16 || h > planes->mb_rows * 16) {
    vp8a::set_error("source size does not fit the MB grid");
    return VP8A_E_REFERENCE_DIMENSIONS_MISMATCH;
  }
  vp8a_status s;
  const void *ry, *ru, *rv, *sy, *su, *sv;
  if ((s = st.in(planes->y, planes->y_stride * (size_t)(h - 1) + w, &ry)) != VP8A_OK) return s;
  if ((s = st.in(planes->u, planes->uv_stride * (size_t)(ch - 1) + cw, &ru)) != VP8A_OK) return s;
  if ((s = st.in(planes->v, planes->uv_stride * (size_t)(ch - 1) + cw, &rv)) != VP8A_OK) return s;
  if ((s = st.in(src->y, src->y_stride * (size_t)(h - 1) + w, &sy)) != VP8A_OK) return s;
  if ((s = st.in(src->u, src->uv_stride * (size_t)(ch - 1) + cw, &su)) != VP8A_OK) return s;
  if ((s = st.in(src->v, src->uv_stride * (size_t)(ch - 1) + cw, &sv)) != VP8A_OK) return s;
  void* acc;
  if ((s = st.out(ssd_out, sizeof(uint64_t), &acc)) != VP8A_OK) return s;
  VP8A_CUDA(cudaMemsetAsync(acc, 0, sizeof(uint64_t), ctx->stream));
  unsigned grid = (unsigned)std::max(1, ctx->sm_count * 4);
  ssd_kernel<<<grid, 256, 0, ctx->stream>>>((const uint8_t*)ry, planes->y_stride, (const uint8_t*)sy, src->y_stride,
                                            (int)w, (int)h, (unsigned long long*)acc);
  ssd_kernel<<<grid, 256, 0, ctx->stream>>>((const uint8_t*)ru, planes->uv_stride, (const uint8_t*)su,
                                            src->uv_stride, (int)cw, (int)ch, (unsigned long long*)acc);
  ssd_kernel<<<grid, 256, 0, ctx->stream>>>((const uint8_t*)rv, planes->uv_stride, (const uint8_t*)sv,
                                            src->uv_stride, (int)cw, (int)ch, (unsigned long long*)acc);
  VP8A_CUDA(cudaGetLastError());
  ctx->launches += 3;
  return st.finish();
}

vp8a_status vp8a_filter_sweep(vp8a_ctx* ctx, const vp8a_planes* planes, const vp8a_mb_lf_info* mbs,
                              const vp8a_filter_config* base, const vp8a_source* src, uint32_t every_rows,
                              uint64_t* ssd_out) {
  if (!ctx || !src || !ssd_out) return VP8A_E_INVALID_ARGUMENT;
  VP8A_CUDA(cudaSetDevice(ctx->device));
  vp8a::Stager st(ctx);
  LfArgs a{};
  vp8a_status s = stage_lf(ctx, st, planes, mbs, base, src, every_rows, false, &a);
  if (s != VP8A_OK) return s;
  void* dt;
  if ((s = st.out(ssd_out, 512 * sizeof(uint64_t), &dt)) != VP8A_OK) return s;
  a.ssd_out = (uint64_t*)dt;
  a.level0_unfiltered = 1;
  if ((s = upload_grid(ctx, st, *base, &a)) != VP8A_OK) return s;
  if ((s = schedule(ctx, st, &a, a.n_cands)) != VP8A_OK) return s;
  if ((s = run_sweep(ctx, a)) != VP8A_OK) return s;
  return finish_sweep(ctx, st, a.split > 1);
}

vp8a_status vp8a_filter_sweep_window(vp8a_ctx* ctx, const vp8a_planes* planes, const vp8a_mb_lf_info* mbs,
                                     const vp8a_filter_config* base, const vp8a_source* src, uint32_t lo_level,
                                     uint32_t hi_level, uint64_t* ssd_out) {
  if (!ctx || !src || !ssd_out || !base) return VP8A_E_INVALID_ARGUMENT;
  if (lo_level > hi_level || hi_level > 63) {
    vp8a::set_error("window levels must satisfy lo <= hi <= 63");
    return VP8A_E_LOOP_FILTER_LEVEL_OUT_OF_RANGE;
  }
  VP8A_CUDA(cudaSetDevice(ctx->device));
  vp8a::Stager st(ctx);
  LfArgs a{};
  vp8a_status s = stage_lf(ctx, st, planes, mbs, base, src, 0, false, &a);
  if (s != VP8A_OK) return s;
  void* dt;
  if ((s = st.out(ssd_out, 512 * sizeof(uint64_t), &dt)) != VP8A_OK) return s;
  VP8A_CUDA(cudaMemsetAsync(dt, 0xff, 512 * sizeof(uint64_t), ctx->stream));
  a.ssd_out = (uint64_t*)dt;
  a.level0_unfiltered = 1;
  if ((s = upload_grid(ctx, st, *base, &a, (int)std::max(1u, lo_level), (int)hi_level)) != VP8A_OK) return s;
  if ((s = schedule(ctx, st, &a, a.n_cands)) != VP8A_OK) return s;
  if ((s = run_sweep(ctx, a)) != VP8A_OK) return s;
  return finish_sweep(ctx, st, a.split > 1);
}

// Splits and schedules a batch's pictures (one split for all; the schedule
// serves every launch of the call, whose largest has `candidates` per picture).
static vp8a_status schedule_batch(vp8a_ctx* ctx, vp8a::Stager& st, std::vector<LfArgs>& args, double candidates) {
  std::vector<LfArgs*> ptrs;
  for (LfArgs& a : args) ptrs.push_back(&a);
  const int split = pick_split(ctx, candidates, ptrs);
  std::vector<uint32_t> start{0};
  size_t bytes = 0;
  for (LfArgs& a : args) {
    set_split(a, split);
    bytes += prepared_bytes(a);
    start.push_back(start.back() + prepare_ctas(a));
  }
  void* d;
  vp8a_status s;
  if ((s = st.scratch(bytes, &d)) != VP8A_OK) return s;
  uint8_t* at = (uint8_t*)d;
  for (LfArgs& a : args) {
    place_prepared(a, at);
    at += prepared_bytes(a);
  }
  const size_t o_start = sizeof(LfArgs) * args.size();
  std::vector<uint8_t> blob(o_start + sizeof(uint32_t) * start.size());
  memcpy(blob.data(), args.data(), o_start);
  memcpy(blob.data() + o_start, start.data(), sizeof(uint32_t) * start.size());
  if ((s = st.upload(blob.data(), blob.size(), &d)) != VP8A_OK) return s;
  lf_schedule_batch_kernel<<<start.back(), SCHED_WARPS * 32, 0, ctx->stream>>>(
      (const LfArgs*)d, (const uint32_t*)((const uint8_t*)d + o_start), (int)args.size());
  VP8A_CUDA(cudaGetLastError());
  ctx->launches++;
  return VP8A_OK;
}

// Every scheduled job's candidates: one launch for the jobs of one shape and
// ring size class (a launch's shared memory is its largest job's, and would
// keep the others' CTAs off the SMs), largest pictures first: their CTAs run
// longest, so they start first and the short ones fill in behind them. A
// split batch (few candidates) is one launch: its CTAs are all resident.
static vp8a_status run_batch(vp8a_ctx* ctx, vp8a::Stager& st, const std::vector<const LfArgs*>& jobs) {
  struct Group {
    std::array<int, 5> key;
    Shape S;
    std::vector<const LfArgs*> jobs;
  };
  std::vector<const LfArgs*> order(jobs);
  std::stable_sort(order.begin(), order.end(), [](const LfArgs* x, const LfArgs* y) {
    return (long)x->mb_cols * x->mb_rows > (long)y->mb_cols * y->mb_rows;
  });
  std::vector<Group> groups;
  vp8a_status s;
  for (const LfArgs* a : order) {
    Shape S;
    if ((s = pick_shape(ctx, *a, &S)) != VP8A_OK) return s;
    const int per_sm = a->split > 1 ? 0 : std::min(8, (int)((228 << 10) / (ring_bytes(*a, S.both) + CTA_SMEM)));
    const std::array<int, 5> key{a->base.simple != 0, S.both, per_sm, a->split > 1 ? 0 : S.threads, S.pre};
    Group* g = nullptr;
    for (Group& x : groups)
      if (x.key == key) g = &x;
    if (!g) {
      groups.push_back(Group{key, S, {}});
      g = &groups.back();
    }
    g->S.threads = std::max(g->S.threads, S.threads);
    g->jobs.push_back(a);
  }
  for (const Group& g : groups) {
    std::vector<LfArgs> table;
    std::vector<uint32_t> start{0};
    size_t smem = 0;
    for (const LfArgs* a : g.jobs) {
      table.push_back(*a);
      start.push_back(start.back() + cta_count(*a, g.S));
      smem = std::max(smem, ring_bytes(*a, g.S.both));
    }
    const size_t o_start = sizeof(LfArgs) * table.size();
    std::vector<uint8_t> blob(o_start + sizeof(uint32_t) * start.size());
    memcpy(blob.data(), table.data(), o_start);
    memcpy(blob.data() + o_start, start.data(), sizeof(uint32_t) * start.size());
    void* d;
    if ((s = st.upload(blob.data(), blob.size(), &d)) != VP8A_OK) return s;
    const uint32_t* ds = (const uint32_t*)((const uint8_t*)d + o_start);
    const int split = table[0].split, n = (int)table.size();
    s = g.key[0] ? launch<true>(ctx, g.S, start.back(), smem, split, table[0], (const LfArgs*)d, ds, n)
                 : launch<false>(ctx, g.S, start.back(), smem, split, table[0], (const LfArgs*)d, ds, n);
    if (s != VP8A_OK) return s;
  }
  return VP8A_OK;
}

vp8a_status vp8a_filter_sweeps(vp8a_ctx* ctx, const vp8a_sweep_job* jobs, uint32_t n_jobs) {
  if (!ctx || (!jobs && n_jobs)) {
    vp8a::set_error("null argument");
    return VP8A_E_INVALID_ARGUMENT;
  }
  if (n_jobs > VP8A_MAX_BATCH_JOBS) {
    vp8a::set_error("more jobs than VP8A_MAX_BATCH_JOBS");
    return VP8A_E_INVALID_ARGUMENT;
  }
  if (n_jobs == 0) return VP8A_OK;
  VP8A_CUDA(cudaSetDevice(ctx->device));
  vp8a::Stager st(ctx);
  vp8a_status s;
  std::vector<LfArgs> args(n_jobs);
  long candidates = 0;
  for (uint32_t j = 0; j < n_jobs; j++) {
    const vp8a_sweep_job& J = jobs[j];
    if (!J.ssd_out) {
      vp8a::set_error("null ssd_out");
      return VP8A_E_INVALID_ARGUMENT;
    }
    LfArgs& a = args[j];
    if ((s = stage_lf(ctx, st, &J.planes, J.mbs, &J.base, &J.src, J.every_rows, false, &a)) != VP8A_OK) return s;
    void* dt;
    if ((s = st.out(J.ssd_out, 512 * sizeof(uint64_t), &dt)) != VP8A_OK) return s;
    a.ssd_out = (uint64_t*)dt;
    a.level0_unfiltered = 1;
    if ((s = upload_grid(ctx, st, J.base, &a)) != VP8A_OK) return s;
    candidates += a.n_cands;
  }
  if ((s = schedule_batch(ctx, st, args, (double)candidates / n_jobs)) != VP8A_OK) return s;
  std::vector<const LfArgs*> all;
  for (const LfArgs& a : args) all.push_back(&a);
  if ((s = run_batch(ctx, st, all)) != VP8A_OK) return s;
  return finish_sweep(ctx, st, args[0].split > 1);
}

vp8a_status vp8a_select_filter_params_batch(vp8a_ctx* ctx, const vp8a_sweep_job* jobs, uint32_t n_jobs,
                                            uint8_t* level_out, uint8_t* sharpness_out) {
  if (!ctx || (!jobs && n_jobs) || (n_jobs && (!level_out || !sharpness_out))) {
    vp8a::set_error("null argument");
    return VP8A_E_INVALID_ARGUMENT;
  }
  if (n_jobs > VP8A_MAX_BATCH_JOBS) {
    vp8a::set_error("more jobs than VP8A_MAX_BATCH_JOBS");
    return VP8A_E_INVALID_ARGUMENT;
  }
  if (n_jobs == 0) return VP8A_OK;
  VP8A_CUDA(cudaSetDevice(ctx->device));
  vp8a::Stager st(ctx);
  vp8a_status s;
  std::vector<LfArgs> base_args(n_jobs);
  void* dt;
  if ((s = st.scratch(sizeof(uint64_t) * ((size_t)512 * n_jobs + 1), &dt)) != VP8A_OK) return s;
  std::vector<uint8_t> bs(n_jobs), best_level(n_jobs, 0), best_sharp(n_jobs);
  std::vector<uint64_t> best(n_jobs), t((size_t)512 * n_jobs + 1, 0);
  for (uint32_t j = 0; j < n_jobs; j++) {
    const vp8a_sweep_job& J = jobs[j];
    if (J.every_rows != 0) {
      vp8a::set_error("vp8a_select_filter_params_batch scores whole frames (every_rows must be 0)");
      return VP8A_E_INVALID_ARGUMENT;
    }
    LfArgs& a = base_args[j];
    if ((s = stage_lf(ctx, st, &J.planes, J.mbs, &J.base, &J.src, 0, false, &a)) != VP8A_OK) return s;
    a.ssd_out = (uint64_t*)dt + (size_t)512 * j;
    a.status = (unsigned*)((uint64_t*)dt + (size_t)512 * n_jobs);  // one word for the stage
    a.level0_unfiltered = 1;
    bs[j] = J.base.sharpness_level > 7 ? 7 : J.base.sharpness_level;
    best_sharp[j] = bs[j];
  }
  // One stage of the walk: job j scores the (level, sharpness) pairs in
  // cands[j] (none: the job sits the stage out); the tables come back.
  auto stage = [&](const std::vector<std::vector<uint8_t>>& cands) -> vp8a_status {
    std::vector<const LfArgs*> run;
    std::vector<uint8_t> pairs;
    for (uint32_t j = 0; j < n_jobs; j++) pairs.insert(pairs.end(), cands[j].begin(), cands[j].end());
    if (pairs.empty()) return VP8A_OK;
    void* dc;
    vp8a_status e = st.upload(pairs.data(), pairs.size(), &dc);
    if (e != VP8A_OK) return e;
    const uint8_t* at = (const uint8_t*)dc;
    for (uint32_t j = 0; j < n_jobs; j++) {
      base_args[j].cands = at;
      base_args[j].n_cands = (int)(cands[j].size() / 2);
      at += cands[j].size();
      if (!cands[j].empty()) run.push_back(&base_args[j]);
    }
    VP8A_CUDA(cudaMemsetAsync(dt, 0, t.size() * sizeof(uint64_t), ctx->stream));
    // The first stage schedules the pictures.
    if (!base_args[0].meta && (e = schedule_batch(ctx, st, base_args, pairs.size() / 2.0 / n_jobs)) != VP8A_OK) return e;
    if ((e = run_batch(ctx, st, run)) != VP8A_OK) return e;
    VP8A_CUDA(cudaMemcpyAsync(t.data(), dt, t.size() * sizeof(uint64_t), cudaMemcpyDeviceToHost, ctx->stream));
    VP8A_CUDA(cudaStreamSynchronize(ctx->stream));
    return t.back() ? timed_out() : VP8A_OK;
  };
  std::vector<std::vector<uint8_t>> c(n_jobs);
  std::vector<LfArgs*> all_jobs;
  for (LfArgs& a : base_args) all_jobs.push_back(&a);
  const bool all = score_all_levels(all_jobs, 17, 1);
  if (all) {
    for (uint32_t j = 0; j < n_jobs; j++) c[j] = all_levels(bs[j]);
    if ((s = stage(c)) != VP8A_OK) return s;
    for (auto& v : c) v.clear();
  }
  // Stage 1: grid 0, 4, ..., 60, 63 at the base sharpness.
  for (uint32_t j = 0; j < n_jobs; j++) {
    for (int l = 0; l <= 60; l += 4) c[j].insert(c[j].end(), {(uint8_t)l, bs[j]});
    c[j].insert(c[j].end(), {63, bs[j]});
  }
  if (!all && (s = stage(c)) != VP8A_OK) return s;
  for (uint32_t j = 0; j < n_jobs; j++) {
    const uint64_t* tj = t.data() + (size_t)512 * j;
    best[j] = tj[0 * 8 + bs[j]];
    for (size_t i = 2; i < c[j].size(); i += 2)
      if (tj[c[j][i] * 8 + bs[j]] < best[j]) {
        best[j] = tj[c[j][i] * 8 + bs[j]];
        best_level[j] = c[j][i];
      }
  }
  // Refine +/-3 around each grid winner, excluding it.
  for (uint32_t j = 0; j < n_jobs; j++) {
    c[j].clear();
    const int lo = best_level[j] >= 3 ? best_level[j] - 3 : 0, hi = std::min(63, best_level[j] + 3);
    for (int l = lo; l <= hi; l++)
      if (l != best_level[j]) c[j].insert(c[j].end(), {(uint8_t)l, bs[j]});
  }
  if (!all && (s = stage(c)) != VP8A_OK) return s;
  for (uint32_t j = 0; j < n_jobs; j++) {
    const uint64_t* tj = t.data() + (size_t)512 * j;
    for (size_t i = 0; i < c[j].size(); i += 2)
      if (tj[c[j][i] * 8 + bs[j]] < best[j]) {
        best[j] = tj[c[j][i] * 8 + bs[j]];
        best_level[j] = c[j][i];
      }
  }
  // Stage 2: the other sharpness values at each chosen non-zero level.
  for (uint32_t j = 0; j < n_jobs; j++) {
    c[j].clear();
    if (best_level[j] == 0) continue;
    for (int sh = 0; sh < 8; sh++)
      if (sh != bs[j]) c[j].insert(c[j].end(), {best_level[j], (uint8_t)sh});
  }
  if ((s = stage(c)) != VP8A_OK) return s;
  for (uint32_t j = 0; j < n_jobs; j++) {
    const uint64_t* tj = t.data() + (size_t)512 * j;
    for (size_t i = 0; i < c[j].size(); i += 2)
      if (tj[best_level[j] * 8 + c[j][i + 1]] < best[j]) {
        best[j] = tj[best_level[j] * 8 + c[j][i + 1]];
        best_sharp[j] = c[j][i + 1];
      }
    level_out[j] = best_level[j];
    sharpness_out[j] = best_sharp[j];
  }
  return st.finish();
}

vp8a_status vp8a_select_filter_params(vp8a_ctx* ctx, const vp8a_planes* planes, const vp8a_mb_lf_info* mbs,
                                      const vp8a_filter_config* base, const vp8a_source* src, uint8_t* level_out,
                                      uint8_t* sharpness_out) {
  if (!ctx || !src || !level_out || !sharpness_out) return VP8A_E_INVALID_ARGUMENT;
  VP8A_CUDA(cudaSetDevice(ctx->device));
  vp8a::Stager st(ctx);
  LfArgs a{};
  vp8a_status s = stage_lf(ctx, st, planes, mbs, base, src, 0, false, &a);
  if (s != VP8A_OK) return s;
  void* dt;
  if ((s = st.scratch(513 * sizeof(uint64_t), &dt)) != VP8A_OK) return s;
  a.ssd_out = (uint64_t*)dt;
  a.level0_unfiltered = 1;
  std::vector<uint64_t> t(513, 0);
  const uint8_t bs = base->sharpness_level > 7 ? 7 : base->sharpness_level;
  // Stage 1: grid 0, 4, ..., 60, 63 at the base sharpness.
  std::vector<uint8_t> c;
  for (int l = 0; l <= 60; l += 4) {
    c.push_back((uint8_t)l);
    c.push_back(bs);
  }
  c.push_back(63);
  c.push_back(bs);
  const bool all = score_all_levels({&a}, 17, 1);
  if ((s = score_candidates(ctx, st, a, all ? all_levels(bs) : c, t.data())) != VP8A_OK) return s;
  uint8_t best_level = 0;
  uint64_t best = t[0 * 8 + bs];
  for (size_t i = 2; i < c.size(); i += 2)
    if (t[c[i] * 8 + bs] < best) {
      best = t[c[i] * 8 + bs];
      best_level = c[i];
    }
  // Refine +/-3 around the grid winner, excluding it.
  const int lo = best_level >= 3 ? best_level - 3 : 0, hi = std::min(63, best_level + 3);
  c.clear();
  for (int l = lo; l <= hi; l++)
    if (l != best_level) {
      c.push_back((uint8_t)l);
      c.push_back(bs);
    }
  if (!all && (s = score_candidates(ctx, st, a, c, t.data())) != VP8A_OK) return s;
  for (size_t i = 0; i < c.size(); i += 2)
    if (t[c[i] * 8 + bs] < best) {
      best = t[c[i] * 8 + bs];
      best_level = c[i];
    }
  if (best_level == 0) {
    const uint8_t zero = 0;
    if ((s = st.write_from_host(level_out, &zero, 1)) != VP8A_OK) return s;
    if ((s = st.write_from_host(sharpness_out, &bs, 1)) != VP8A_OK) return s;
      return st.finish();
  }
  // Stage 2: the other sharpness values at the chosen level.
  c.clear();
  for (int sh = 0; sh < 8; sh++)
    if (sh != bs) {
      c.push_back(best_level);
      c.push_back((uint8_t)sh);
    }
  if ((s = score_candidates(ctx, st, a, c, t.data())) != VP8A_OK) return s;
  uint8_t best_sharp = bs;
  for (size_t i = 0; i < c.size(); i += 2)
    if (t[best_level * 8 + c[i + 1]] < best) {
      best = t[best_level * 8 + c[i + 1]];
      best_sharp = c[i + 1];
    }
  if ((s = st.write_from_host(level_out, &best_level, 1)) != VP8A_OK) return s;
  if ((s = st.write_from_host(sharpness_out, &best_sharp, 1)) != VP8A_OK) return s;
  return st.finish();
}

void vp8a_key_frame_sampling(uint32_t mb_rows, uint32_t* every_rows, uint32_t* sweep_sharpness) {
  // bands = clamp(mb_rows / 32, 3, 6); every_rows = max(mb_rows / bands, 2).
  const uint32_t bands = std::min<uint32_t>(std::max<uint32_t>(mb_rows / 32, 3), 6);
  if (every_rows) *every_rows = std::max<uint32_t>(mb_rows / bands, 2);
  if (sweep_sharpness) *sweep_sharpness = 1;
}

vp8a_status vp8a_select_filter_params_sampled(vp8a_ctx* ctx, const vp8a_planes* planes, const vp8a_mb_lf_info* mbs,
                                              const vp8a_filter_config* base, const vp8a_source* src,
                                              uint32_t every_rows, uint32_t sweep_sharpness, uint8_t* level_out,
                                              uint8_t* sharpness_out) {
  if (!ctx || !src || !level_out || !sharpness_out) return VP8A_E_INVALID_ARGUMENT;
  VP8A_CUDA(cudaSetDevice(ctx->device));
  vp8a::Stager st(ctx);
  LfArgs a{};
  const uint32_t er = every_rows < 2 ? 2 : every_rows;
  vp8a_status s = stage_lf(ctx, st, planes, mbs, base, src, er, false, &a);
  if (s != VP8A_OK) return s;
  void* dt;
  if ((s = st.scratch(513 * sizeof(uint64_t), &dt)) != VP8A_OK) return s;
  a.ssd_out = (uint64_t*)dt;
  a.level0_unfiltered = 1;
  std::vector<uint64_t> t(513, 0);
  const uint8_t bs = base->sharpness_level > 7 ? 7 : base->sharpness_level;
  static const uint8_t coarse[9] = {0, 8, 16, 24, 32, 40, 48, 56, 63};
  std::vector<uint8_t> c;
  for (uint8_t l : coarse) {
    c.push_back(l);
    c.push_back(bs);
  }
  const bool all = score_all_levels({&a}, 9, 3);
  if ((s = score_candidates(ctx, st, a, all ? all_levels(bs) : c, t.data())) != VP8A_OK) return s;
  uint8_t best_level = 0;
  uint64_t best = t[0 * 8 + bs];
  for (int i = 1; i < 9; i++)
    if (t[coarse[i] * 8 + bs] < best) {
      best = t[coarse[i] * 8 + bs];
      best_level = coarse[i];
    }
  for (uint8_t stp : {4, 2, 1}) {
    c.clear();
    if (best_level >= stp) {
      c.push_back((uint8_t)(best_level - stp));
      c.push_back(bs);
    }
    if (best_level + stp <= 63) {
      c.push_back((uint8_t)(best_level + stp));
      c.push_back(bs);
    }
    if (!all && (s = score_candidates(ctx, st, a, c, t.data())) != VP8A_OK) return s;
    uint8_t bl = best_level;
    for (size_t i = 0; i < c.size(); i += 2)
      if (t[c[i] * 8 + bs] < best) {
        best = t[c[i] * 8 + bs];
        bl = c[i];
      }
    best_level = bl;
  }
  uint8_t best_sharp = bs;
  if (sweep_sharpness && best_level != 0) {
    c.clear();
    for (int sh = 0; sh < 8; sh++)
      if (sh != bs) {
        c.push_back(best_level);
        c.push_back((uint8_t)sh);
      }
    if ((s = score_candidates(ctx, st, a, c, t.data())) != VP8A_OK) return s;
    for (size_t i = 0; i < c.size(); i += 2)
      if (t[best_level * 8 + c[i + 1]] < best) {
        best = t[best_level * 8 + c[i + 1]];
        best_sharp = c[i + 1];
      }
  }
  if ((s = st.write_from_host(level_out, &best_level, 1)) != VP8A_OK) return s;
  if ((s = st.write_from_host(sharpness_out, &best_sharp, 1)) != VP8A_OK) return s;
  return st.finish();
}

// The sweep of vp8a_filter_sweep without any allocation: see the header.
vp8a_status vp8a_filter_sweep_noalloc(vp8a_ctx* ctx, const vp8a_planes* planes, const vp8a_mb_lf_info* mbs,
                                      const vp8a_filter_config* base, const vp8a_source* src, uint32_t every_rows,
                                      uint64_t* ssd_out) {
  if (!ctx || !planes || !mbs || !base || !src || !ssd_out) {
    vp8a::set_error("null argument");
    return VP8A_E_INVALID_ARGUMENT;
  }
  const int cols = (int)planes->mb_cols, rows = (int)planes->mb_rows;
  if (cols < 1 || rows < 1 || cols > NA_MAX_MB_COLS || rows > NA_MAX_MB_ROWS) {
    vp8a::set_error("vp8a_filter_sweep_noalloc: the MB grid must be 1..256 columns by 1..136 rows "
                    "(its fixed scratch holds the schedule of at most 4096x2176 pixels)");
    return VP8A_E_INVALID_DIMENSIONS;
  }
  if (planes->y_stride < (uint64_t)cols * 16 || planes->uv_stride < (uint64_t)cols * 8) {
    vp8a::set_error("plane stride below the MB-padded width");
    return VP8A_E_INVALID_ARGUMENT;
  }
  vp8a_status s = validate_config(base);
  if (s != VP8A_OK) return s;
  if (src->width == 0 || src->height == 0 || src->width > (uint32_t)cols * 16 || src->height > (uint32_t)rows * 16) {
    vp8a::set_error("source size does not fit the MB grid");
    return VP8A_E_REFERENCE_DIMENSIONS_MISMATCH;
  }
  const uint32_t cw = (src->width + 1) / 2;
  if (src->y_stride < src->width || src->uv_stride < cw) {
    vp8a::set_error("source stride below width");
    return VP8A_E_INVALID_ARGUMENT;
  }
  VP8A_CUDA(cudaSetDevice(ctx->device));
  const void* bufs[8] = {planes->y, planes->u, planes->v, mbs, src->y, src->u, src->v, ssd_out};
  for (const void* b : bufs)
    if (!device_resident(b, ctx->device)) {
      vp8a::set_error("vp8a_filter_sweep_noalloc: every buffer must be device memory of the context's GPU "
                      "(this entry point stages nothing)");
      return VP8A_E_INVALID_ARGUMENT;
    }
  uint8_t* scr = nullptr;
  if ((s = sweep_scratch(ctx->device, &scr)) != VP8A_OK) return s;
  LfArgs a{};
  a.y = (const uint8_t*)planes->y;
  a.u = (const uint8_t*)planes->u;
  a.v = (const uint8_t*)planes->v;
  a.ys = planes->y_stride;
  a.cs = planes->uv_stride;
  a.mb_cols = cols;
  a.mb_rows = rows;
  a.mbs = mbs;
  a.base = *base;
  a.sy = (const uint8_t*)src->y;
  a.su = (const uint8_t*)src->u;
  a.sv = (const uint8_t*)src->v;
  a.sys = src->y_stride;
  a.scs = src->uv_stride;
  a.width = (int)src->width;
  a.height = (int)src->height;
  a.ssd_out = ssd_out;
  a.level0_unfiltered = 1;
  set_rows(a, every_rows);
  set_alignment(a);
  set_split(a, 1);
  a.cands = scr + NA_CANDS;
  a.cand_mask = scr + NA_MASK;
  a.meta = (uint4*)(scr + NA_META);
  a.list = (uint16_t*)(scr + NA_LIST);
  NaGrid grid{};
  grid.n = a.n_cands = grid_passes(*base, grid.pairs, grid.masks);  // <= NA_CANDIDATES
  sweep_schedule_kernel<<<(unsigned)((a.steps + SCHED_WARPS - 1) / SCHED_WARPS), SCHED_WARPS * 32, 0, ctx->stream>>>(
      a, scr, grid);
  VP8A_CUDA(cudaGetLastError());
  ctx->launches++;
  return run_sweep(ctx, a);
}

}  // extern "C"
