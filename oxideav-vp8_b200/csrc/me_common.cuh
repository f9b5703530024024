// me_common.cuh — warp-level motion-search building blocks shared by the
// batched search kernels (me.cu) and the wavefront analysis (analysis.cu).
//
// A warp owns one (MB, reference) item. The reference luma around the
// search centre is staged once in shared memory as an edge-clamped window
// (the §20.14 edge replication of fetch_luma_mb_whole_pixel /
// fetch_luma_mb_halo, src/motion_comp.rs:837,1513, is applied while the
// window is filled), so every later SAD or six-tap read is an unchecked
// shared-memory access. Candidates that leave the window fall back to
// clamped global loads with identical results.
#pragma once

#include "vp8a_internal.cuh"

namespace vp8a_dev {

constexpr unsigned FULL = 0xffffffffu;
constexpr int WS = 40;              // window extent and stride (bytes)
constexpr int WIN_BYTES = WS * WS + 16;
constexpr int WIN_R = 8;            // diamond radius the window is sized for
constexpr int WIN_LEAD = WIN_R + 3; // window origin = centre - WIN_LEAD

struct MePlane {
  const uint8_t* plane;
  uint64_t stride;
  int width;
  int height;
};

// Every member is a multiple of 16 bytes and the struct is 16-byte aligned,
// so arrays of it (and structs embedding it) keep word access aligned.
struct __align__(16) WarpScratch {
  uint8_t win[WIN_BYTES];        // 1616
  uint8_t temp[21 * 16 + 16];    // 352
  uint8_t halo[21 * 24 + 24];    // 528
  uint8_t more[192];             // with temp and halo: the shared sub-pel planes
};
static_assert(sizeof(WarpScratch) % 16 == 0, "WarpScratch must keep 16-byte multiples");

__device__ __forceinline__ int16_t clamp_component(int v) { return (int16_t)clampi(v, -1023, 1023); }
__device__ __forceinline__ int16_t snap_whole(int v) { return (int16_t)((v / 4) * 4); }
// stored_luma_mv (src/motion_comp.rs:187): wrapping doubling.
__device__ __forceinline__ int eighth(int16_t v) { return (int)(int16_t)(uint16_t)((uint16_t)v * 2u); }

// 8 unaligned bytes from shared memory as two little-endian words.
__device__ __forceinline__ void load8u(const uint8_t* p, uint32_t& o0, uint32_t& o1) {
  uintptr_t a = (uintptr_t)p;
  const uint32_t* w = (const uint32_t*)(a & ~(uintptr_t)3);
  unsigned sh = (unsigned)(a & 3) * 8u;
  uint32_t w0 = w[0], w1 = w[1], w2 = w[2];
  o0 = __funnelshift_r(w0, w1, sh);
  o1 = __funnelshift_r(w1, w2, sh);
}

// ------------------------------------------------------- packed six-tap
//
// The §18.3 filters run four pixels a thread, two to a register (16-bit
// fields), with the pixels read four to a word: a fifth of the loads and a
// third of the arithmetic of one pixel a thread.
__device__ __forceinline__ uint32_t pk16(int v) { return (uint32_t)(uint16_t)(int16_t)v * 0x00010001u; }
// Bytes 1 and 3 as fields.
__device__ __forceinline__ uint32_t odd_bytes(uint32_t x) { return __byte_perm(x, 0u, 0x4341); }
// (t >> 7) - 64 clamped to 0..255, per field: t is the filter's sum plus 64 + 64 *
// 128. The taps' negative sums reach -32 * 255 and the positive ones 160 * 255 (the
// half-pel taps both), so every field lies in 96 .. 49056 and takes nothing from its
// neighbour.
constexpr int TAP_BIAS = 64 + 64 * 128;
static_assert(TAP_BIAS - 32 * 255 >= 0 && TAP_BIAS + 160 * 255 <= 0xffff, "sums stay in their fields");
__device__ __forceinline__ uint32_t tap_result(uint32_t t) {
  return __viaddmin_s16x2_relu((t >> 7) & 0x01ff01ffu, pk16(-64), pk16(255));
}
// The half-pel taps 3, -16, 77, 77, -16, 3.
__device__ __forceinline__ uint32_t half6(uint32_t a, uint32_t b, uint32_t c, uint32_t d, uint32_t e, uint32_t f) {
  return tap_result((c + d) * 77u + pk16(TAP_BIAS) + (a + f) * 3u - (b + e) * 16u);
}
struct Taps {
  int f[6];
};
__device__ __forceinline__ uint32_t six(const Taps& k, uint32_t a, uint32_t b, uint32_t c, uint32_t d, uint32_t e,
                                        uint32_t f) {
  return tap_result(pk16(TAP_BIAS) + a * (uint32_t)k.f[0] + b * (uint32_t)k.f[1] + c * (uint32_t)k.f[2] +
                    d * (uint32_t)k.f[3] + e * (uint32_t)k.f[4] + f * (uint32_t)k.f[5]);
}
__device__ __forceinline__ Taps taps_const(int f) {
  const int* t = c_sixtap[f];
  return Taps{{t[0], t[1], t[2], t[3], t[4], t[5]}};
}
// Twelve bytes of a shared-memory row from byte offset `o` on, as words.
__device__ __forceinline__ void row_words(const uint8_t* row, int o, uint32_t& u0, uint32_t& u1, uint32_t& u2) {
  const uint32_t* w = (const uint32_t*)(row + (o & ~3));
  const unsigned sh = (unsigned)(o & 3) * 8u;
  const uint32_t w1 = w[1], w2 = w[2];
  u0 = __funnelshift_r(w[0], w1, sh);
  u1 = __funnelshift_r(w1, w2, sh);
  u2 = __funnelshift_r(w2, w[3], sh);
}
__device__ __forceinline__ uint32_t row_word(const uint8_t* row, int o) {
  const uint32_t* w = (const uint32_t*)(row + (o & ~3));
  return __funnelshift_r(w[0], w[1], (unsigned)(o & 3) * 8u);
}
// Four outputs of a horizontal filter over the bytes of u0, u1, u2: output i
// takes bytes i .. i + 5.
template <class F>
__device__ __forceinline__ uint32_t filter_row(uint32_t u0, uint32_t u1, uint32_t u2, F&& tap6) {
  constexpr uint32_t M = 0x00ff00ffu;
  const uint32_t s2 = __byte_perm(u0, u1, 0x5432), s6 = __byte_perm(u1, u2, 0x5432);
  const uint32_t p1 = odd_bytes(u0), p2 = s2 & M, p3 = odd_bytes(s2), p4 = u1 & M, p5 = odd_bytes(u1);
  return tap6(p1, p2, p3, p4, p5, s6 & M) * 256u + tap6(u0 & M, p1, p2, p3, p4, p5);
}

// Whether the plane can be read as aligned words.
__device__ __forceinline__ bool word_plane(const MePlane& P) {
  return (((uintptr_t)P.plane | (uintptr_t)P.stride) & 3) == 0;
}

// Fill a WS x WS window whose top-left is plane pixel (x0, y0), clamping
// every coordinate into the plane: words where they lie inside it, at the edges
// too. (Byte loads for a whole window at an edge, a row at a time, made a
// three-reference search of a 16x16 frame at the fastest effort 62 us instead of 54,
// and of a 1920x1080 frame at the middle effort 161 instead of 149.)
__device__ __forceinline__ void load_window(const MePlane& P, uint8_t* win, int x0, int y0, int lane) {
  if (word_plane(P) && x0 >= 0 && (x0 & ~3) + WS + 4 <= P.width) {
    const int sh = x0 & 3, xa = x0 - sh;
    for (int t = lane; t < WS * (WS / 4); t += 32) {
      const int r = t / (WS / 4), w = t - r * (WS / 4);
      const uint32_t* p = (const uint32_t*)(P.plane + (size_t)clampi(y0 + r, 0, P.height - 1) * P.stride + xa) + w;
      *(uint32_t*)(win + r * WS + 4 * w) = __funnelshift_r(__ldg(p), __ldg(p + 1), 8u * (unsigned)sh);
    }
    __syncwarp();
    return;
  }
  // Four words a lane in flight.
  const bool words = word_plane(P);
#pragma unroll 4
  for (int t = lane; t < WS * (WS / 4); t += 32) {
    const int r = t / (WS / 4), w = t - r * (WS / 4), x = x0 + 4 * w, sh = x & 3;
    const uint8_t* row = P.plane + (size_t)clampi(y0 + r, 0, P.height - 1) * P.stride;
    uint32_t v = 0;
    if (words && x >= 0 && x - sh + 8 <= P.width) {
      const uint32_t* p = (const uint32_t*)(row + (x - sh));
      v = __funnelshift_r(__ldg(p), __ldg(p + 1), 8u * (unsigned)sh);
    } else {
#pragma unroll
      for (int k = 0; k < 4; k++) v |= (uint32_t)row[clampi(x + k, 0, P.width - 1)] << (8 * k);
    }
    *(uint32_t*)(win + r * WS + 4 * w) = v;
  }
  __syncwarp();
}

// Source MB in shared memory (16x16, stride 16); each lane's 8-byte slice
// is lane>>1 = row, (lane&1)*8 = column.
__device__ __forceinline__ uint32_t sad_win16(const uint8_t* win, int lx, int ly, const uint8_t* src, int lane) {
  int row = lane >> 1, c0 = (lane & 1) * 8;
  uint32_t r0, r1;
  load8u(win + (ly + row) * WS + lx + c0, r0, r1);
  const uint32_t* sp = (const uint32_t*)(src + row * 16 + c0);
  uint32_t s = __vsadu4(r0, sp[0]) + __vsadu4(r1, sp[1]);
  return __reduce_add_sync(FULL, s);
}

// Whole-pel SAD of the 16x16 block at plane pixel (x0, y0), clamped loads.
__device__ __forceinline__ uint32_t sad_global16(const MePlane& P, int x0, int y0, const uint8_t* src, int lane) {
  int row = lane >> 1, c0 = (lane & 1) * 8;
  int y = clampi(y0 + row, 0, P.height - 1);
  const uint8_t* pr = P.plane + (size_t)y * P.stride;
  uint32_t s = 0;
  if (word_plane(P) && x0 >= 0 && (x0 & ~3) + 20 <= P.width) {
    const int x = x0 + c0;
    const uint32_t* w = (const uint32_t*)(pr + (x & ~3));
    const unsigned sh = (unsigned)(x & 3) * 8u;
    const uint32_t w1 = __ldg(w + 1);
    const uint2 sv = *(const uint2*)(src + row * 16 + c0);
    s = __vsadu4(__funnelshift_r(__ldg(w), w1, sh), sv.x) + __vsadu4(__funnelshift_r(w1, __ldg(w + 2), sh), sv.y);
    return __reduce_add_sync(FULL, s);
  }
#pragma unroll
  for (int k = 0; k < 8; k++) {
    int d = (int)pr[clampi(x0 + c0 + k, 0, P.width - 1)] - (int)src[row * 16 + c0 + k];
    s += (uint32_t)(d < 0 ? -d : d);
  }
  return __reduce_add_sync(FULL, s);
}

// Whole-pel SAD at plane pixel (x0, y0): window when it covers the block.
__device__ __forceinline__ uint32_t sad_whole_at(const MePlane& P, const uint8_t* win, int wx0, int wy0,
                                                 int x0, int y0, const uint8_t* src, int lane) {
  int lx = x0 - wx0, ly = y0 - wy0;
  if (lx >= 0 && ly >= 0 && lx <= WS - 16 && ly <= WS - 16) return sad_win16(win, lx, ly, src, lane);
  return sad_global16(P, x0, y0, src, lane);
}

// Whole-pel SADs of two blocks of the window, at its pixels (xa, ya) and (xb, yb):
// block a's in the low half of the result. A half-warp takes a block, a lane a row
// (the window's 40-byte rows fall on distinct banks).
__device__ __forceinline__ uint32_t sad_win16_pair(const uint8_t* win, int xa, int ya, int xb, int yb,
                                                   const uint8_t* src, int lane) {
  const int x = lane < 16 ? xa : xb, row = lane & 15;
  const uint32_t* w = (const uint32_t*)(win + ((lane < 16 ? ya : yb) + row) * WS + (x & ~3));
  const uint4 sv = *(const uint4*)(src + row * 16);
  const unsigned sh = (unsigned)(x & 3) * 8u;
  const uint32_t w1 = w[1], w2 = w[2], w3 = w[3];
  const uint32_t s = __vsadu4(__funnelshift_r(w[0], w1, sh), sv.x) + __vsadu4(__funnelshift_r(w1, w2, sh), sv.y) +
                     __vsadu4(__funnelshift_r(w2, w3, sh), sv.z) + __vsadu4(__funnelshift_r(w3, w[4], sh), sv.w);
  return __reduce_add_sync(FULL, lane < 16 ? s : s << 16);
}

// §18.3 two-pass six-tap prediction SAD (sixtap_mb_luma,
// src/motion_comp.rs:902-1057) from a 21x21 halo at `h` (stride hs, a multiple
// of 4; block origin at (2, 2); reads up to 27 bytes of a row from h on). The
// horizontal pass keeps its 8-bit clamp; a pass whose fraction is 0 is the
// identity (the reference's own identity elision, src/motion_comp.rs:960-1007),
// which the taps 0, 0, 128, 0, 0, 0 reproduce.
__device__ __forceinline__ uint32_t subpel_sad(const uint8_t* h, int hs, int mx, int my, const uint8_t* src,
                                               uint8_t* temp, int lane) {
  const int o = (int)((uintptr_t)h & 3);
  const Taps fh = taps_const(mx), fv = taps_const(my);
#pragma unroll 1
  for (int t = lane; t < 21 * 4; t += 32) {
    const int r = t >> 2, j = t & 3;
    uint32_t u0, u1, u2;
    row_words(h - o + r * hs, o + 4 * j, u0, u1, u2);
    *(uint32_t*)(temp + t * 4) = filter_row(u0, u1, u2, [&](uint32_t a, uint32_t b, uint32_t c, uint32_t d, uint32_t e,
                                                            uint32_t f) { return six(fh, a, b, c, d, e, f); });
  }
  __syncwarp();
  // Word column j, rows 2 strip and 2 strip + 1.
  const int j = lane & 3, r0 = (lane >> 2) * 2;
  uint32_t e[7], d[7];
#pragma unroll
  for (int k = 0; k < 7; k++) {
    const uint32_t w = *(const uint32_t*)(temp + (r0 + k) * 16 + j * 4);
    e[k] = w & 0x00ff00ffu;
    d[k] = odd_bytes(w);
  }
  uint32_t s = 0;
#pragma unroll
  for (int r = 0; r < 2; r++)
    s += __vsadu4(six(fv, d[r], d[r + 1], d[r + 2], d[r + 3], d[r + 4], d[r + 5]) * 256u +
                      six(fv, e[r], e[r + 1], e[r + 2], e[r + 3], e[r + 4], e[r + 5]),
                  *(const uint32_t*)(src + (r0 + r) * 16 + j * 4));
  __syncwarp();
  return __reduce_add_sync(FULL, s);
}

// mb_luma_sad_at_mv (src/motion_search.rs:470-529) for the MB at plane
// pixel (mbx, mby), served from the window when it covers the candidate.
// `temp` (21 x 16 bytes) and `halo` (21 x 24) are the warp's own scratch.
__device__ __forceinline__ uint32_t sad_at_mv(const MePlane& P, const uint8_t* win, uint8_t* temp, uint8_t* halo,
                                              int wx0, int wy0, int mbx, int mby, int16_t mv_row, int16_t mv_col,
                                              const uint8_t* src, int lane) {
  int er = eighth(mv_row), ec = eighth(mv_col);
  int mx = ec & 7, my = er & 7;
  int bx = mbx + (ec >> 3), by = mby + (er >> 3);
  if (mx == 0 && my == 0) return sad_whole_at(P, win, wx0, wy0, bx, by, src, lane);
  int hx = bx - 2, hy = by - 2;
  int lx = hx - wx0, ly = hy - wy0;
  if (lx >= 0 && ly >= 0 && lx <= WS - 21 && ly <= WS - 21)
    return subpel_sad(win + ly * WS + lx, WS, mx, my, src, temp, lane);
  // Out-of-window halo: clamped fetch into scratch (fetch_luma_mb_halo).
  for (int r = 0; r < 21; r++) {
    int y = clampi(hy + r, 0, P.height - 1);
    const uint8_t* row = P.plane + (size_t)y * P.stride;
    if (lane < 21) halo[r * 24 + lane] = row[clampi(hx + lane, 0, P.width - 1)];
  }
  __syncwarp();
  uint32_t s = subpel_sad(halo, 24, mx, my, src, temp, lane);
  return s;
}

__device__ __forceinline__ uint32_t sad_at_mv(const MePlane& P, WarpScratch& S, int wx0, int wy0, int mbx,
                                              int mby, int16_t mv_row, int16_t mv_col, const uint8_t* src,
                                              int lane) {
  return sad_at_mv(P, S.win, S.temp, S.halo, wx0, wy0, mbx, mby, mv_row, mv_col, src, lane);
}

// small_diamond_search_luma (src/motion_search.rs:381-442). Each round
// scores the eight whole-pel neighbours of the round's starting best in
// parallel (four lanes per neighbour), then replays the reference's
// sequential N, S, W, E walk — whose candidates all lie in that 3x3
// neighbourhood — with its strict '<' and collapse skips.
__device__ __forceinline__ vp8a_search_result diamond(const MePlane& P, WarpScratch& S, int wx0, int wy0,
                                                      int mbx, int mby, vp8a_mv center, uint32_t max_iters,
                                                      const uint8_t* src, int lane) {
  vp8a_mv best;
  best.row = snap_whole(clamp_component(center.row));
  best.col = snap_whole(clamp_component(center.col));
  uint32_t best_sad = sad_whole_at(P, S.win, wx0, wy0, mbx + best.col / 4, mby + best.row / 4, src, lane);
  const int k = lane >> 2, q = lane & 3;
  // Neighbour k of the 3x3 ring (row, col) in pixels; index 4 is skipped.
  const int kr = (k < 3) ? -1 : (k < 5 ? 0 : 1);
  const int kc = (k == 0 || k == 3 || k == 5) ? -1 : ((k == 1 || k == 6) ? 0 : 1);
  for (uint32_t it = 0; it < max_iters; it++) {
    const int bx = mbx + best.col / 4, by = mby + best.row / 4;
    const int lx = bx - 1 - wx0, ly = by - 1 - wy0;
    uint32_t tab[8];
    if (lx >= 0 && ly >= 0 && lx + 18 <= WS && ly + 18 <= WS) {
      uint32_t s = 0;
      const uint8_t* base = S.win + (ly + 1 + kr + q * 4) * WS + (lx + 1 + kc);
#pragma unroll
      for (int r = 0; r < 4; r++) {
        uint32_t a0, a1, a2, a3;
        load8u(base + r * WS, a0, a1);
        load8u(base + r * WS + 8, a2, a3);
        const uint32_t* sp = (const uint32_t*)(src + (q * 4 + r) * 16);
        s += __vsadu4(a0, sp[0]) + __vsadu4(a1, sp[1]) + __vsadu4(a2, sp[2]) + __vsadu4(a3, sp[3]);
      }
      s += __shfl_xor_sync(FULL, s, 1);
      s += __shfl_xor_sync(FULL, s, 2);
#pragma unroll
      for (int j = 0; j < 8; j++) tab[j] = __shfl_sync(FULL, s, j * 4);
    } else {
#pragma unroll 1
      for (int j = 0; j < 8; j++) {
        int jr = (j < 3) ? -1 : (j < 5 ? 0 : 1);
        int jc = (j == 0 || j == 3 || j == 5) ? -1 : ((j == 1 || j == 6) ? 0 : 1);
        tab[j] = sad_whole_at(P, S.win, wx0, wy0, bx + jc, by + jr, src, lane);
      }
    }
    // Replay the reference's walk over the 3x3 table.
    vp8a_mv b = best;
    uint32_t bs = best_sad;
    bool improved = false;
    const int dr[4] = {-4, 4, 0, 0}, dc[4] = {0, 0, -4, 4};
#pragma unroll
    for (int d = 0; d < 4; d++) {
      vp8a_mv cand;
      cand.row = snap_whole(clamp_component(b.row + dr[d]));
      cand.col = snap_whole(clamp_component(b.col + dc[d]));
      if (cand.row == b.row && cand.col == b.col) continue;
      int rr = (cand.row - best.row) / 4, rc = (cand.col - best.col) / 4;
      uint32_t s;
      if (rr == 0 && rc == 0) s = best_sad;
      else {
        int idx = (rr + 1) * 3 + (rc + 1);
        s = tab[idx < 4 ? idx : idx - 1];
      }
      if (s < bs) {
        bs = s;
        b = cand;
        improved = true;
      }
    }
    best = b;
    best_sad = bs;
    if (!improved) break;
  }
  vp8a_search_result res;
  res.mv = best;
  res.sad = best_sad;
  return res;
}

// half_pixel_refine_luma / quarter_pixel_refine_luma
// (src/motion_search.rs:564-728): centre plus 8 offsets of `step`
// quarter-pels in the fixed order, strict '<', collapse skips.
// `center_sad` is the SAD at `center` when the caller already has it (the
// previous refinement's result), else ~0u.
__device__ __forceinline__ vp8a_search_result refine(const MePlane& P, WarpScratch& S, int wx0, int wy0, int mbx,
                                                     int mby, vp8a_mv center, int step, const uint8_t* src,
                                                     int lane, uint32_t center_sad = ~0u) {
  vp8a_mv best = center;
  uint32_t best_sad = center_sad != ~0u ? center_sad
                                        : sad_at_mv(P, S, wx0, wy0, mbx, mby, center.row, center.col, src, lane);
#pragma unroll 1
  for (int k = 0; k < 8; k++) {
    // Offsets (-1,-1) (-1,0) (-1,1) (0,-1) (0,1) (1,-1) (1,0) (1,1).
    const int orow = (k < 3) ? -1 : (k < 5 ? 0 : 1);
    const int ocol = (k == 0 || k == 3 || k == 5) ? -1 : ((k == 1 || k == 6) ? 0 : 1);
    vp8a_mv cand;
    cand.row = clamp_component(center.row + orow * step);
    cand.col = clamp_component(center.col + ocol * step);
    if (cand.row == best.row && cand.col == best.col) continue;
    uint32_t s = sad_at_mv(P, S, wx0, wy0, mbx, mby, cand.row, cand.col, src, lane);
    if (s < best_sad) {
      best_sad = s;
      best = cand;
    }
  }
  vp8a_search_result res;
  res.mv = best;
  res.sad = best_sad;
  return res;
}

// Offsets (row, col) of the eight refinement candidates in the reference's
// order: (-1,-1) (-1,0) (-1,1) (0,-1) (0,1) (1,-1) (1,0) (1,1).
__device__ __forceinline__ int cand_dr(int k) { return (k < 3) ? -1 : (k < 5 ? 0 : 1); }
__device__ __forceinline__ int cand_dc(int k) { return (k == 0 || k == 3 || k == 5) ? -1 : ((k == 1 || k == 6) ? 0 : 1); }

// The eight half-pel candidates around a whole-pel centre whose block origin
// in the window is (bx, by) share three planes of half-pel samples: H (22 rows
// x 17, row r = window row by - 3 + r, sample i at bx + i - 1/2), V (17 x 16,
// at by + r - 1/2) and D (17 x 17, vertical over H), so each six-tap output is
// computed once per MB instead of once per candidate; every candidate's
// prediction is a 16 x 16 block of one plane, byte-identical to its own
// two-pass synthesis (same taps, same 8-bit intermediate, same edge-clamped
// source). Rows of 20, 16 and 20 bytes. The functions below give thread t of n
// its share.
constexpr int HP_H = 0, HP_V = HP_H + 22 * 20, HP_D = HP_V + 17 * 16, HP_BYTES = HP_D + 17 * 20;
constexpr int QP_BYTES = 3 * 22 * 16;  // the quarter-pel planes
constexpr int PLANE_BYTES = sizeof(WarpScratch) - offsetof(WarpScratch, temp);
static_assert(HP_BYTES + 16 <= PLANE_BYTES && QP_BYTES <= PLANE_BYTES, "the planes fit behind the window");
static_assert(offsetof(WarpScratch, temp) % 16 == 0, "the planes are read as words");

// H: one (row, word) a thread and round.
__device__ __forceinline__ void half_plane_h(const uint8_t* win, uint8_t* hp, int bx, int by, int t, int n) {
#pragma unroll 1
  for (; t < 22 * 5; t += n) {
    const int r = t / 5, j = t - 5 * r;
    uint32_t u0, u1, u2;
    row_words(win + (by - 3 + r) * WS, bx - 3 + 4 * j, u0, u1, u2);
    *(uint32_t*)(hp + HP_H + t * 4) = filter_row(u0, u1, u2, half6);
  }
}
// V, on one warp: one word column and two or three rows a lane.
__device__ __forceinline__ void half_plane_v(const uint8_t* win, uint8_t* hp, int bx, int by, int lane) {
  {
    const int j = lane & 3, strip = lane >> 2, r0 = 2 * strip + (strip > 0), r1 = 2 * strip + 3;
    const uint8_t* p = win + (by + r0 - 3) * WS;
    uint32_t e[6], o[6];
#pragma unroll
    for (int k = 0; k < 5; k++) {
      const uint32_t w = row_word(p + k * WS, bx + 4 * j);
      e[k] = w & 0x00ff00ffu;
      o[k] = odd_bytes(w);
    }
    for (int r = r0; r < r1; r++, p += WS) {
      const uint32_t w = row_word(p + 5 * WS, bx + 4 * j);
      e[5] = w & 0x00ff00ffu;
      o[5] = odd_bytes(w);
      *(uint32_t*)(hp + HP_V + r * 16 + j * 4) =
          half6(o[0], o[1], o[2], o[3], o[4], o[5]) * 256u + half6(e[0], e[1], e[2], e[3], e[4], e[5]);
#pragma unroll
      for (int k = 0; k < 5; k++) {
        e[k] = e[k + 1];
        o[k] = o[k + 1];
      }
    }
  }
}

// The D plane, from H (after H is complete): one (row, word) a thread and
// round.
__device__ __forceinline__ void half_plane_d(uint8_t* hp, int t, int n) {
#pragma unroll 1
  for (; t < 17 * 5; t += n) {
    const uint8_t* p = hp + HP_H + t * 4;
    uint32_t e[6], o[6];
#pragma unroll
    for (int k = 0; k < 6; k++) {
      const uint32_t w = *(const uint32_t*)(p + k * 20);
      e[k] = w & 0x00ff00ffu;
      o[k] = odd_bytes(w);
    }
    *(uint32_t*)(hp + HP_D + t * 4) =
        half6(o[0], o[1], o[2], o[3], o[4], o[5]) * 256u + half6(e[0], e[1], e[2], e[3], e[4], e[5]);
  }
}

// Sums of the warp's half-warps (each below 65536) in one reduction: lanes 0-15
// in the low half of the result.
__device__ __forceinline__ uint32_t pair_sum(uint32_t s, int lane) {
  return __reduce_add_sync(FULL, lane < 16 ? s : s << 16);
}

// SADs of the half-pel candidates 2 slot and 2 slot + 1 (one warp): row lane
// & 15 of candidate k.
__device__ __forceinline__ uint32_t half_cand_sads(const uint8_t* hp, const uint8_t* src, int slot, int lane) {
  const int k = 2 * slot + (lane >> 4), row = lane & 15, dy = cand_dr(k), dx = cand_dc(k), cx = dx > 0, cy = dy > 0;
  const int at = dy == 0 ? HP_H + (3 + row) * 20 : (dx == 0 ? HP_V + (cy + row) * 16 : HP_D + (cy + row) * 20);
  const uint32_t* w = (const uint32_t*)(hp + at);
  const uint4 sv = *(const uint4*)(src + row * 16);
  const unsigned sh = cx * 8u;
  const uint32_t w1 = w[1], w2 = w[2], w3 = w[3];
  const uint32_t s = __vsadu4(__funnelshift_r(w[0], w1, sh), sv.x) + __vsadu4(__funnelshift_r(w1, w2, sh), sv.y) +
                     __vsadu4(__funnelshift_r(w2, w3, sh), sv.z) + __vsadu4(__funnelshift_r(w3, w[4], sh), sv.w);
  return pair_sum(s, lane);
}

// quarter_pixel_refine_luma's eight candidates around `qc` share three
// horizontal six-tap planes, one per candidate column (qc.col - 1, qc.col,
// qc.col + 1 quarter-pels; fraction 0 is the unfiltered pixel, which the taps 0,
// 0, 128, 0, 0, 0 reproduce). Each candidate's prediction is then its vertical
// pass over its column's plane: the same taps, the same 8-bit intermediate and
// the same edge-clamped source as its own two-pass synthesis.
// Integer position (in the window) and eighth-pel fraction of component v.
__device__ __forceinline__ void quarter_pos(int v, int mb, int w0, int& i, int& f) {
  const int e = eighth(clamp_component(v));
  i = mb + (e >> 3) - w0;
  f = e & 7;
}
// Whether the window covers every candidate's halo.
__device__ __forceinline__ bool quarter_inside(vp8a_mv qc, int mbx, int mby, int wx0, int wy0) {
  int x0, x1, y0, y1, f;
  quarter_pos(qc.col - 1, mbx, wx0, x0, f);
  quarter_pos(qc.col + 1, mbx, wx0, x1, f);
  quarter_pos(qc.row - 1, mby, wy0, y0, f);
  quarter_pos(qc.row + 1, mby, wy0, y1, f);
  return x0 >= 2 && x1 + 19 <= WS && y0 >= 2 && y0 + 20 <= WS && y1 - y0 <= 1;
}
// Horizontal planes: plane k's row rr (window row iy0 + rr) at qh + (k * 22 +
// rr) * 16; one (plane, row, word) a thread and round.
template <class TapsOf>
__device__ __forceinline__ void quarter_planes_h(const uint8_t* win, uint8_t* qh, TapsOf&& taps_of, vp8a_mv qc, int mbx,
                                                 int wx0, int iy0, int t, int n) {
#pragma unroll 1
  for (; t < 3 * 22 * 4; t += n) {
    const int k = t / 88, rr = (t - 88 * k) >> 2, j = t & 3;
    int ix, fx;
    quarter_pos(qc.col + k - 1, mbx, wx0, ix, fx);
    const Taps f = taps_of(fx);
    uint32_t u0, u1, u2;
    row_words(win + (iy0 + rr) * WS, ix - 2 + 4 * j, u0, u1, u2);
    *(uint32_t*)(qh + t * 4) = filter_row(u0, u1, u2, [&](uint32_t a, uint32_t b, uint32_t c, uint32_t d, uint32_t e,
                                                          uint32_t g) { return six(f, a, b, c, d, e, g); });
  }
}

// Vertical passes and SADs of two candidates (one warp), the first in the low half
// of the result: lane (candidate, strip of four rows, word), k the lane's candidate.
template <class TapsOf>
__device__ __forceinline__ uint32_t quarter_pair_sads(const uint8_t* qh, const uint8_t* src, TapsOf&& taps_of,
                                                      vp8a_mv qc, int mby, int wy0, int iy0, int k, int lane) {
  const int strip = (lane >> 2) & 3, j = lane & 3;
  int iy, fy;
  quarter_pos(qc.row + cand_dr(k), mby, wy0, iy, fy);
  const Taps f = taps_of(fy);
  const uint8_t* p = qh + ((cand_dc(k) + 1) * 22 + iy - 2 - iy0 + strip * 4) * 16 + j * 4;
  uint32_t e[6], o[6], s = 0;
#pragma unroll
  for (int i = 0; i < 5; i++) {
    const uint32_t w = *(const uint32_t*)(p + i * 16);
    e[i] = w & 0x00ff00ffu;
    o[i] = odd_bytes(w);
  }
#pragma unroll
  for (int r = 0; r < 4; r++) {
    const uint32_t w = *(const uint32_t*)(p + (r + 5) * 16);
    e[5] = w & 0x00ff00ffu;
    o[5] = odd_bytes(w);
    s += __vsadu4(six(f, o[0], o[1], o[2], o[3], o[4], o[5]) * 256u + six(f, e[0], e[1], e[2], e[3], e[4], e[5]),
                  *(const uint32_t*)(src + (strip * 4 + r) * 16 + j * 4));
#pragma unroll
    for (int i = 0; i < 5; i++) {
      e[i] = e[i + 1];
      o[i] = o[i + 1];
    }
  }
  return pair_sum(s, lane);
}

// Candidates 2 slot and 2 slot + 1.
template <class TapsOf>
__device__ __forceinline__ uint32_t quarter_cand_sads(const uint8_t* qh, const uint8_t* src, TapsOf&& taps_of,
                                                      vp8a_mv qc, int mby, int wy0, int iy0, int slot, int lane) {
  return quarter_pair_sads(qh, src, taps_of, qc, mby, wy0, iy0, 2 * slot + (lane >> 4), lane);
}

// half_pixel_refine_luma's candidates (src/motion_search.rs:589-598; also of
// sub_pixel_refine, src/encoder/inter_search.rs:520-535) on one warp: sads[k] for
// the offsets (row, col) = (-1,-1) (-1,0) (-1,1) (0,-1) (0,1) (1,-1) (1,0) (1,1)
// half-pels; false when the window does not cover the planes.
__device__ __forceinline__ bool half_plane_sads(WarpScratch& S, int wx0, int wy0, int mbx, int mby, vp8a_mv center,
                                                const uint8_t* src, int lane, uint32_t* sads) {
  if ((center.row & 3) || (center.col & 3)) return false;
  const int bx = mbx + center.col / 4 - wx0, by = mby + center.row / 4 - wy0;  // block origin in window
  if (bx < 3 || by < 3 || bx + 19 > WS || by + 19 > WS) return false;
  uint8_t* hp = S.temp;
  half_plane_h(S.win, hp, bx, by, lane, 32);
  half_plane_v(S.win, hp, bx, by, lane);
  __syncwarp();
  half_plane_d(hp, lane, 32);
  __syncwarp();
#pragma unroll
  for (int k = 0; k < 4; k++) {
    const uint32_t both = half_cand_sads(hp, src, k, lane);
    sads[2 * k] = both & 0xffffu;
    sads[2 * k + 1] = both >> 16;
  }
  __syncwarp();
  return true;
}

// quarter_pixel_refine_luma (src/motion_search.rs:666-728) on one warp over the
// shared planes where the window covers them, else candidate by candidate.
// `center_sad` as in refine.
__device__ __forceinline__ vp8a_search_result quarter_refine(const MePlane& P, WarpScratch& S, int wx0, int wy0,
                                                             int mbx, int mby, vp8a_mv center, const uint8_t* src,
                                                             int lane, uint32_t center_sad = ~0u) {
  if (!quarter_inside(center, mbx, mby, wx0, wy0))
    return refine(P, S, wx0, wy0, mbx, mby, center, 1, src, lane, center_sad);
  vp8a_search_result best{center, center_sad};
  if (center_sad == ~0u) best.sad = sad_at_mv(P, S, wx0, wy0, mbx, mby, center.row, center.col, src, lane);
  int iy0, f;
  quarter_pos(center.row - 1, mby, wy0, iy0, f);
  iy0 -= 2;
  auto taps = [](int fr) { return taps_const(fr); };
  quarter_planes_h(S.win, S.temp, taps, center, mbx, wx0, iy0, lane, 32);
  __syncwarp();
#pragma unroll
  for (int k = 0; k < 4; k++) {
    const uint32_t both = quarter_cand_sads(S.temp, src, taps, center, mby, wy0, iy0, k, lane);
#pragma unroll
    for (int i = 0; i < 2; i++) {
      const uint32_t s = i ? both >> 16 : both & 0xffffu;
      if (s < best.sad) {
        best.sad = s;
        best.mv.row = clamp_component(center.row + cand_dr(2 * k + i));
        best.mv.col = clamp_component(center.col + cand_dc(2 * k + i));
      }
    }
  }
  __syncwarp();
  return best;
}

// half_pixel_refine_luma (src/motion_search.rs:564-627) over the shared
// planes; for a whole-pel centre inside [-1020, 1020] no candidate is
// clamped or collapses, so the reference walk is the first strict minimum.
__device__ __forceinline__ bool half_refine_planes(WarpScratch& S, int wx0, int wy0, int mbx, int mby,
                                                   vp8a_mv center, const uint8_t* src, int lane,
                                                   vp8a_search_result* out) {
  if (center.row < -1020 || center.row > 1020 || center.col < -1020 || center.col > 1020) return false;
  uint32_t sads[8];
  if (!half_plane_sads(S, wx0, wy0, mbx, mby, center, src, lane, sads)) return false;
  const int bx = mbx + center.col / 4 - wx0, by = mby + center.row / 4 - wy0;
  vp8a_mv best = center;
  uint32_t best_sad = sad_win16(S.win, bx, by, src, lane);
#pragma unroll
  for (int k = 0; k < 8; k++) {
    const int dy = (k < 3) ? -1 : (k < 5 ? 0 : 1);
    const int dx = (k == 0 || k == 3 || k == 5) ? -1 : ((k == 1 || k == 6) ? 0 : 1);
    if (sads[k] < best_sad) {
      best_sad = sads[k];
      best.row = (int16_t)(center.row + 2 * dy);
      best.col = (int16_t)(center.col + 2 * dx);
    }
  }
  out->mv = best;
  out->sad = best_sad;
  return true;
}

}  // namespace vp8a_dev
