// learned.cu — the learned motion proposal: a 4-layer 3x3 conv net (BF16
// weights and activations, FP32 accumulation) that scores a 32x32 grid of
// whole-pel vectors (2 px apart, -32 .. +30 px) for an MB from a coarse
// cost volume: at each grid vector, the half-resolution SAD of the MB
// against the reference and the reference's texture there. Its top four
// cells seed an exact local search (the plain search's SAD kernels), so
// the net only proposes; every returned vector and SAD is exact.
//
// Kernels (all hand-written; the GEMM-shaped ones on the tensor cores:
// inference and the 32 -> 32 layers and their input gradients with tcgen05 and
// TMEM accumulators, the other training layers with mma.sync BF16 -> FP32):
//   lp_windows_kernel       coarse cost volumes -> NHWC [n, 32, 32, 2] BF16
//   lp_net_kernel           the whole net and the top-k cells per map in one
//                           launch (inference), activations on chip
//   lp_seeded_search_kernel every whole-pel vector near the seed cells,
//                           first smallest SAD
//   lp_conv_tc_kernel       the 32 -> 32 layers, forward and dX, on tcgen05
//   lp_conv_first_kernel, lp_conv_last_kernel   the 2 -> 32 and 32 -> 1 layers
//   lp_conv_bwd_last_kernel dX of the 32 -> 1 layer
//   lp_conv_bwd_w_kernel, lp_conv_bwd_w_edge_kernel   dW = sum over pixels of
//                           dY x shifted X, and db
//   lp_conv_fwd_smem_kernel, lp_conv_bwd_data_kernel, lp_conv_bwd_w_smem_kernel
//                           the same for tensors off the 16-byte boundary and
//                           for other output types, element by element
//   lp_softmax_ce_kernel    softmax over the 1024 cells, cross-entropy,
//                           d(logits) = (p - onehot) / n
//   lp_adam_kernel          Adam on FP32 master weights, BF16 copies
// Layout: activations NHWC, 32x32 pixels per MB, channel count 2 or 32
// (the last layer 1); weights [cout][tap][cin], tap = (dy + 1) * 3 + dx + 1.
#include <cuda.h>
#include <cuda_bf16.h>

#include <algorithm>
#include <mutex>

#include "vp8a_internal.cuh"

namespace {

constexpr int LP_S = 32;          // image side
constexpr int LP_P = LP_S * LP_S; // pixels per image

__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
  const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<const uint32_t*>(&v);
}
__device__ __forceinline__ uint32_t pack_raw(uint16_t lo, uint16_t hi) { return (uint32_t)lo | ((uint32_t)hi << 16); }

__device__ __forceinline__ void mma_bf16(float (&d)[4], const uint32_t (&a)[4], const uint32_t (&b)[2]) {
  asm(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

// Element (pixel q of image img shifted by (dy, dx), channel c) of an NHWC
// BF16 tensor with C channels, 0 outside the image or past C.
__device__ __forceinline__ uint16_t act(const uint16_t* X, int C, int img, int y, int x, int c) {
  if (y < 0 || y >= LP_S || x < 0 || x >= LP_S || c >= C) return 0;
  return X[((size_t)img * LP_P + y * LP_S + x) * C + c];
}

// ---------------------------------------------------------------- windows

// Item i: the MB at (xy[2i], xy[2i+1]). Both pictures are averaged over
// 2x2 (rounded) and edge-clamped: the MB to 8x8, the reference around it
// (80x80 pixels, the MB at [32, 48)) to 40x40. Cell (i, j) is the vector
// (2 (i - 16), 2 (j - 16)) px: channel 0 = (32 - mean |MB - reference block
// at that vector|) / 32, channel 1 = (reference at the block's centre - 128)
// / 64.
__global__ void __launch_bounds__(256) lp_windows_kernel(const uint8_t* src, uint64_t ss, const uint8_t* ref,
                                                         uint64_t rs, int w, int h, const uint32_t* xy, int n,
                                                         uint16_t* out) {
  __shared__ uint32_t rw32[40 * 40 / 4];  // the reference window at half resolution, rows of 10 words
  __shared__ uint32_t mb32[16];           // the MB at half resolution, rows of 2 words
  uint8_t* rw = reinterpret_cast<uint8_t*>(rw32);
  uint8_t* mb = reinterpret_cast<uint8_t*>(mb32);
  const int i = blockIdx.x, t = threadIdx.x;
  if (i >= n) return;
  const int mx = (int)xy[2 * i] * 16, my = (int)xy[2 * i + 1] * 16;
  auto avg2 = [&](const uint8_t* p, uint64_t st, int y, int x) -> int {
    int s = 0;
    for (int a = 0; a < 2; a++)
      for (int b = 0; b < 2; b++) s += p[(size_t)min(max(y + a, 0), h - 1) * st + min(max(x + b, 0), w - 1)];
    return (s + 2) >> 2;
  };
  for (int q = t; q < 40 * 40; q += blockDim.x)
    rw[q] = (uint8_t)avg2(ref, rs, my - 32 + 2 * (q / 40), mx - 32 + 2 * (q % 40));
  if (t < 64) mb[t] = (uint8_t)avg2(src, ss, my + 2 * (t >> 3), mx + 2 * (t & 7));
  __syncthreads();
  // Thread t: cells (oy, 4 j .. 4 j + 3) with oy = t / 8, j = t % 8. Per
  // window row three words hold the 11 bytes the four 8-byte rows need; the
  // byte-shifted rows come from byte permutes and four-byte SADs.
  const int oy = t >> 3, ox0 = (t & 7) * 4;
  uint32_t sad[4] = {0u, 0u, 0u, 0u};
#pragma unroll
  for (int r = 0; r < 8; r++) {
    const uint32_t* row = rw32 + (oy + r) * 10 + (ox0 >> 2);
    const uint32_t w0 = row[0], w1 = row[1], w2 = row[2];
    const uint32_t m0 = mb32[2 * r], m1 = mb32[2 * r + 1];
    sad[0] = __vsadu4(w0, m0) + __vsadu4(w1, m1) + sad[0];
    sad[1] = __vsadu4(__byte_perm(w0, w1, 0x4321), m0) + __vsadu4(__byte_perm(w1, w2, 0x4321), m1) + sad[1];
    sad[2] = __vsadu4(__byte_perm(w0, w1, 0x5432), m0) + __vsadu4(__byte_perm(w1, w2, 0x5432), m1) + sad[2];
    sad[3] = __vsadu4(__byte_perm(w0, w1, 0x6543), m0) + __vsadu4(__byte_perm(w1, w2, 0x6543), m1) + sad[3];
  }
  uint32_t o[4];
#pragma unroll
  for (int c = 0; c < 4; c++) {
    const float c0 = (32.0f - (float)sad[c] * (1.0f / 64.0f)) * (1.0f / 32.0f);
    const float c1 = ((float)rw[(oy + 4) * 40 + ox0 + c + 4] - 128.0f) * (1.0f / 64.0f);
    o[c] = pack_bf16(c0, c1);
  }
  *reinterpret_cast<uint4*>(out + ((size_t)i * LP_P + oy * 32 + ox0) * 2) = make_uint4(o[0], o[1], o[2], o[3]);
}

// ------------------------------------------------------- seeded search

// The exact search around the net's seeds: one CTA per MB, thread t takes
// candidate t = (seed s, row offset dr, column offset dc) in seed, row,
// column order. The source MB and each seed's (16 + 2 radius)-pixel square
// window of the reference (edge-clamped, as every whole-pel SAD reads it)
// sit in shared memory; the first smallest (SAD, order) wins.
constexpr int LP_SEED_MAXC = 128;  // k * (2 radius + 1)^2
constexpr int LP_SEED_MAXW = 16 + 2 * 4;  // window side for radius <= 4
constexpr int LP_SEED_PITCH = 28;         // window row pitch: 7 words, so a row's five words stay in it
__global__ void __launch_bounds__(LP_SEED_MAXC) lp_seeded_search_kernel(const uint8_t* ref, uint64_t rs, int rw,
                                                                        int rh, const uint8_t* src_mbs,
                                                                        const uint32_t* xy, const int32_t* seeds,
                                                                        int k, int radius, vp8a_search_result* out) {
  __shared__ uint32_t win32[4][LP_SEED_MAXW * LP_SEED_PITCH / 4];
  __shared__ uint32_t sm32[64];
  uint8_t* sm = reinterpret_cast<uint8_t*>(sm32);
  __shared__ uint32_t best_w[LP_SEED_MAXC / 32];
  const int i = blockIdx.x, t = threadIdx.x;
  const int mx = (int)xy[2 * i] * 16, my = (int)xy[2 * i + 1] * 16;
  const int side = 16 + 2 * radius, per = (2 * radius + 1) * (2 * radius + 1);
  for (int q = t; q < 256; q += blockDim.x) sm[q] = src_mbs[(size_t)i * 256 + q];
  for (int s = 0; s < k; s++) {
    const int c = seeds[(size_t)i * k + s];
    const int x0 = mx + (c % 32 - 16) * 2 - radius, y0 = my + (c / 32 - 16) * 2 - radius;
    uint8_t* win = reinterpret_cast<uint8_t*>(win32[s]);
    for (int q = t; q < side * side; q += blockDim.x) {
      const int y = min(max(y0 + q / side, 0), rh - 1), x = min(max(x0 + q % side, 0), rw - 1);
      win[(q / side) * LP_SEED_PITCH + q % side] = ref[(size_t)y * rs + x];
    }
  }
  __syncthreads();
  uint32_t key = 0xffffffffu;
  if (t < k * per) {
    const int s = t / per, o = t - s * per, dr = o / (2 * radius + 1), dc = o - dr * (2 * radius + 1);
    // Row r of the candidate: bytes dc .. dc + 15 of window row dr + r, cut
    // from five words by byte permutes, against the MB row's four words.
    const uint32_t* w = win32[s] + dr * (LP_SEED_PITCH / 4) + (dc >> 2);
    const uint32_t sel = 0x3210u + (uint32_t)(dc & 3) * 0x1111u;
    uint32_t sad = 0;
#pragma unroll 4
    for (int r = 0; r < 16; r++) {
      const uint32_t* wr = w + r * (LP_SEED_PITCH / 4);
      const uint32_t w0 = wr[0], w1 = wr[1], w2 = wr[2], w3 = wr[3], w4 = wr[4];
      sad += __vsadu4(__byte_perm(w0, w1, sel), sm32[4 * r]) + __vsadu4(__byte_perm(w1, w2, sel), sm32[4 * r + 1]) +
             __vsadu4(__byte_perm(w2, w3, sel), sm32[4 * r + 2]) + __vsadu4(__byte_perm(w3, w4, sel), sm32[4 * r + 3]);
    }
    key = (sad << 7) | (uint32_t)t;
  }
  key = __reduce_min_sync(0xffffffffu, key);
  if ((t & 31) == 0) best_w[t >> 5] = key;
  __syncthreads();
  if (t == 0) {
    uint32_t b = best_w[0];
    for (int w = 1; w < (int)(blockDim.x >> 5); w++) b = min(b, best_w[w]);
    const int o = (int)(b & 127u), s = o / per, r = o - s * per;
    const int c = seeds[(size_t)i * k + s];
    vp8a_search_result res;
    res.mv.row = (int16_t)((c / 32 - 16) * 8 + 4 * (r / (2 * radius + 1) - radius));
    res.mv.col = (int16_t)((c % 32 - 16) * 8 + 4 * (r % (2 * radius + 1) - radius));
    res.sad = b >> 7;
    out[i] = res;
  }
}

// ------------------------------------------------------------ conv fwd

// Implicit GEMM: A[p][k] = X[p + off(tap)][ci], k = tap * CP + ci (CP = CIN
// rounded up to 16); B[k][n] = W[n][tap][ci].
// Forward pass with the image staged: one CTA (8 warps) per image. The
// 32x32 input gets a zero halo (34x34) in shared memory, one pixel every PS
// halves (channels padded to CP, then 8 spare: a 16-byte-aligned row whose
// 32-bit words fall on distinct banks for the 8 pixels x 4 channel pairs a
// fragment reads); the weights sit beside it ([n][tap][ci], n stride
// 9 CIN + 8). Warp w takes the 16-pixel tiles w, w + 8, ... of the image.
template <int CIN, int NT>
__global__ void __launch_bounds__(256) lp_conv_fwd_smem_kernel(const uint16_t* X, const uint16_t* W, const float* bias,
                                                               int cout, int relu, uint16_t* Y, float* Yf) {
  constexpr int CP = (CIN + 15) / 16 * 16, PS = CP + 8, WS = 9 * CIN + 8, COUTP = NT * 8;
  extern __shared__ __align__(16) uint16_t sm[];
  uint16_t* img_s = sm;                 // 34 * 34 * PS
  uint16_t* w_s = sm + 34 * 34 * PS;    // COUTP * WS
  const int img = blockIdx.x, tid = threadIdx.x;
  // Zero the halo and the channel padding, then copy the image.
  for (int q = tid; q < 34 * 34 * PS / 2; q += blockDim.x) reinterpret_cast<uint32_t*>(img_s)[q] = 0u;
  for (int q = tid; q < COUTP * WS / 2; q += blockDim.x) reinterpret_cast<uint32_t*>(w_s)[q] = 0u;
  __syncthreads();
  const uint16_t* Xi = X + (size_t)img * LP_P * CIN;
  if (CIN % 2 == 0) {
    for (int q = tid; q < LP_P * CIN / 2; q += blockDim.x) {
      const int p = q / (CIN / 2), c = (q % (CIN / 2)) * 2;
      const int sy = (p >> 5) + 1, sx = (p & 31) + 1;
      *reinterpret_cast<uint32_t*>(img_s + (sy * 34 + sx) * PS + c) = reinterpret_cast<const uint32_t*>(Xi)[q];
    }
  }
  for (int q = tid; q < cout * 9 * CIN; q += blockDim.x) w_s[(q / (9 * CIN)) * WS + q % (9 * CIN)] = W[q];
  __syncthreads();
  const int warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  // Warp w takes tiles w, w + 8, ..., four at a time, so each weight
  // fragment loaded from shared memory feeds four MMAs.
  constexpr int TG = 4;
  for (int t0 = warp; t0 < LP_P / 16; t0 += 8 * TG) {
    float d[TG][NT][4];
#pragma unroll
    for (int u = 0; u < TG; u++)
#pragma unroll
      for (int j = 0; j < NT; j++) d[u][j][0] = d[u][j][1] = d[u][j][2] = d[u][j][3] = 0.f;
#pragma unroll
    for (int tap = 0; tap < 9; tap++) {
      const int dy = tap / 3 - 1, dx = tap % 3 - 1;
#pragma unroll
      for (int c0 = 0; c0 < CP; c0 += 16) {
        uint32_t a[TG][4];
#pragma unroll
        for (int u = 0; u < TG; u++) {
          const int tile = t0 + 8 * u, y = tile >> 1, xb = (tile & 1) * 16;
          const uint16_t* r0 = img_s + ((y + dy + 1) * 34 + (xb + g + dx + 1)) * PS;
          const uint16_t* r1 = r0 + 8 * PS;
          a[u][0] = *reinterpret_cast<const uint32_t*>(r0 + c0 + 2 * t);
          a[u][1] = *reinterpret_cast<const uint32_t*>(r1 + c0 + 2 * t);
          a[u][2] = *reinterpret_cast<const uint32_t*>(r0 + c0 + 2 * t + 8);
          a[u][3] = *reinterpret_cast<const uint32_t*>(r1 + c0 + 2 * t + 8);
        }
#pragma unroll
        for (int j = 0; j < NT; j++) {
          const uint16_t* wr = w_s + (j * 8 + g) * WS + tap * CIN + c0 + 2 * t;
          uint32_t b[2];
          if (CIN >= 16) {
            b[0] = *reinterpret_cast<const uint32_t*>(wr);
            b[1] = *reinterpret_cast<const uint32_t*>(wr + 8);
          } else {  // CIN = 2: channels past CIN are zero
            b[0] = (c0 + 2 * t < CIN) ? *reinterpret_cast<const uint32_t*>(wr) : 0u;
            b[1] = 0u;
          }
#pragma unroll
          for (int u = 0; u < TG; u++) mma_bf16(d[u][j], a[u], b);
        }
      }
    }
#pragma unroll
    for (int u = 0; u < TG; u++) {
      const int tile = t0 + 8 * u, y = tile >> 1, xb = (tile & 1) * 16;
#pragma unroll
      for (int j = 0; j < NT; j++)
#pragma unroll
        for (int h = 0; h < 2; h++) {
          const int p = y * LP_S + xb + g + 8 * h, n = j * 8 + 2 * t;
          const size_t o = ((size_t)img * LP_P + p) * cout + n;
          float v0 = d[u][j][2 * h] + (n < cout ? bias[n] : 0.f);
          float v1 = d[u][j][2 * h + 1] + (n + 1 < cout ? bias[n + 1] : 0.f);
          if (relu) {
            v0 = fmaxf(v0, 0.f);
            v1 = fmaxf(v1, 0.f);
          }
          if (Yf) {
            if (n < cout) Yf[o] = v0;
            if (n + 1 < cout) Yf[o + 1] = v1;
          } else if (n + 1 < cout) {
            *reinterpret_cast<uint32_t*>(Y + o) = pack_bf16(v0, v1);
          } else if (n < cout) {
            Y[o] = __bfloat16_as_ushort(__float2bfloat16_rn(v0));
          }
        }
    }
  }
}

// --------------------------------------------------------- conv bwd data

// dX[p][ci] = sum over taps and co of dY[p - off(tap)][co] W[co][tap][ci],
// times (Xa[p][ci] > 0) when `mask` (the ReLU of the layer that produced X).
template <int COUT, int NT>
__global__ void __launch_bounds__(128) lp_conv_bwd_data_kernel(const uint16_t* dY, const uint16_t* W, int cin,
                                                               int n_img, const uint16_t* Xa, uint16_t* dX) {
  constexpr int KP = (COUT + 15) / 16 * 16;
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int tile = blockIdx.x * 4 + (threadIdx.x >> 5);
  if (tile >= n_img * (LP_P / 16)) return;
  const int img = tile / (LP_P / 16), rem = tile % (LP_P / 16), y = rem >> 1, xb = (rem & 1) * 16;
  float d[NT][4];
#pragma unroll
  for (int j = 0; j < NT; j++) d[j][0] = d[j][1] = d[j][2] = d[j][3] = 0.f;
  for (int tap = 0; tap < 9; tap++) {
    const int dy = tap / 3 - 1, dx = tap % 3 - 1;
#pragma unroll
    for (int c0 = 0; c0 < KP; c0 += 16) {
      uint32_t a[4];
      const int ca = c0 + 2 * t, cb = c0 + 2 * t + 8;
      // dY at p - off: the output pixel whose tap `tap` reads p.
      a[0] = pack_raw(act(dY, COUT, img, y - dy, xb + g - dx, ca), act(dY, COUT, img, y - dy, xb + g - dx, ca + 1));
      a[1] = pack_raw(act(dY, COUT, img, y - dy, xb + g + 8 - dx, ca),
                      act(dY, COUT, img, y - dy, xb + g + 8 - dx, ca + 1));
      a[2] = pack_raw(act(dY, COUT, img, y - dy, xb + g - dx, cb), act(dY, COUT, img, y - dy, xb + g - dx, cb + 1));
      a[3] = pack_raw(act(dY, COUT, img, y - dy, xb + g + 8 - dx, cb),
                      act(dY, COUT, img, y - dy, xb + g + 8 - dx, cb + 1));
#pragma unroll
      for (int j = 0; j < NT; j++) {
        const int n = j * 8 + g;  // ci
        auto wv = [&](int co) -> uint16_t {
          return (n < cin && co < COUT) ? W[((size_t)co * 9 + tap) * cin + n] : (uint16_t)0;
        };
        const uint32_t b[2] = {pack_raw(wv(ca), wv(ca + 1)), pack_raw(wv(cb), wv(cb + 1))};
        mma_bf16(d[j], a, b);
      }
    }
  }
#pragma unroll
  for (int j = 0; j < NT; j++)
#pragma unroll
    for (int h = 0; h < 2; h++) {
      const int p = y * LP_S + xb + g + 8 * h;
#pragma unroll
      for (int e = 0; e < 2; e++) {
        const int n = j * 8 + 2 * t + e;
        if (n >= cin) continue;
        const size_t o = ((size_t)img * LP_P + p) * cin + n;
        float v = d[j][2 * h + e];
        if (Xa && !(__bfloat162float(__ushort_as_bfloat16(Xa[o])) > 0.f)) v = 0.f;
        dX[o] = __bfloat16_as_ushort(__float2bfloat16_rn(v));
      }
    }
}

// ------------------------------------------------------- conv bwd weights

// dW[co][tap][ci] += sum over a chunk of pixels of dY[p][co] X[p + off][ci]:
// M = co (16-row tiles), N = tap * CIN + ci (8-column tiles), K = pixels.
constexpr int LP_WCHUNK = 512;  // pixels per staged chunk (half an image)


// ------------------------------------------------------------- loss

// One block per item: softmax over its 1024 logits, the cross-entropy of
// the label cell (added to *loss), and d(logits) = (softmax - onehot) / n
// as BF16. Labels < 0 contribute nothing (zero gradient).
__global__ void __launch_bounds__(256) lp_softmax_ce_kernel(const float* logits, const int32_t* labels, int n,
                                                            uint16_t* dlogits, float* loss, float* top_prob) {
  const int i = blockIdx.x, t = threadIdx.x;
  __shared__ float red[8];
  const float* z = logits + (size_t)i * LP_P;
  float m = -INFINITY;
  for (int q = t; q < LP_P; q += 256) m = fmaxf(m, z[q]);
  for (int o = 16; o; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
  if ((t & 31) == 0) red[t >> 5] = m;
  __syncthreads();
  m = red[0];
  for (int k = 1; k < 8; k++) m = fmaxf(m, red[k]);
  __syncthreads();
  float s = 0.f;
  for (int q = t; q < LP_P; q += 256) s += __expf(z[q] - m);
  for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if ((t & 31) == 0) red[t >> 5] = s;
  __syncthreads();
  s = 0.f;
  for (int k = 0; k < 8; k++) s += red[k];
  const int lab = labels ? labels[i] : -1;
  for (int q = t; q < LP_P; q += 256) {
    const float p = __expf(z[q] - m) / s;
    if (dlogits) {
      const float gr = lab < 0 ? 0.f : (p - (q == lab ? 1.f : 0.f)) / (float)n;
      dlogits[(size_t)i * LP_P + q] = __bfloat16_as_ushort(__float2bfloat16_rn(gr));
    }
    if (top_prob && q == lab) top_prob[i] = p;
  }
  if (t == 0 && loss && lab >= 0) atomicAdd(loss, -(z[lab] - m - __logf(s)));
}

// ------------------------------------------------------------- Adam

__global__ void lp_adam_kernel(float* w, const float* grad, float* m, float* v, int n, float lr, float b1, float b2,
                               float eps, float c1, float c2, uint16_t* w_bf16) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float gr = grad[i];
  const float mi = b1 * m[i] + (1.f - b1) * gr, vi = b2 * v[i] + (1.f - b2) * gr * gr;
  m[i] = mi;
  v[i] = vi;
  const float wi = w[i] - lr * (mi / c1) / (sqrtf(vi / c2) + eps);
  w[i] = wi;
  w_bf16[i] = __bfloat16_as_ushort(__float2bfloat16_rn(wi));
}

// ------------------------------------------------- loop-filter window

// Channel sums of n images' activations ([n][32][32][C] BF16) into
// out[C] (FP32, accumulated): one CTA per image.
__global__ void __launch_bounds__(256) lp_pool_kernel(const uint16_t* X, int C, float* out) {
  __shared__ float part[64];
  const int img = blockIdx.x, t = threadIdx.x;
  if (t < 64) part[t] = 0.f;
  __syncthreads();
  const uint16_t* Xi = X + (size_t)img * LP_P * C;
  // Thread t sums channel t % C over pixels t / C, t / C + 256 / C, ...
  const int c = t % C, step = 256 / C;
  float s = 0.f;
  if (t < step * C)
    for (int p = t / C; p < LP_P; p += step) s += __bfloat162float(__ushort_as_bfloat16(Xi[(size_t)p * C + c]));
  atomicAdd(&part[c], s);
  __syncthreads();
  if (t < C) atomicAdd(&out[t], part[t]);
}

// The head: f = sums / count (C features), z = W f + b (L levels), softmax;
// with a label: loss += CE, dW += (p - onehot) f^T, db += p - onehot. One
// CTA of L threads.
__global__ void lp_lf_head_kernel(const float* sums, float count, int C, const float* W, const float* b, int L,
                                  int label, float* logits, float* dW, float* db, float* loss) {
  __shared__ float f[64], z[128];
  const int t = threadIdx.x;
  if (t < C) f[t] = sums[t] / count;
  __syncthreads();
  float zi = 0.f;
  if (t < L) {
    zi = b[t];
    for (int c = 0; c < C; c++) zi += W[t * C + c] * f[c];
    z[t] = zi;
    if (logits) logits[t] = zi;
  }
  __syncthreads();
  if (label < 0 || t >= L) return;
  float m = -INFINITY;
  for (int k = 0; k < L; k++) m = fmaxf(m, z[k]);
  float s = 0.f;
  for (int k = 0; k < L; k++) s += __expf(z[k] - m);
  const float p = __expf(zi - m) / s, gz = p - (t == label ? 1.f : 0.f);
  for (int c = 0; c < C; c++) dW[t * C + c] += gz * f[c];
  db[t] += gz;
  if (t == label && loss) *loss += -(zi - m - __logf(s));
}

// ------------------------------- tcgen05 convolutions: layout and waits
namespace lptc {
constexpr int NV = 1224;                    // halo pixels per channel group (>= 1151 + 70 + 1)
constexpr int REGION = NV * 16;             // bytes per channel group
constexpr int IMG_BYTES = 4 * REGION;
constexpr int W_BYTES = 36 * 32 * 16;       // 36 k-groups x 32 n x 16 bytes
static_assert(REGION % 128 == 0, "TMA destinations are 128-byte aligned");
constexpr int TILES = 9;                    // ceil(32 * 34 / 128)
// Instruction descriptor (kind::f16): D FP32, A and B BF16, both K-major,
// N = 32, M = 128.
constexpr uint32_t IDESC = (1u << 4) | (1u << 7) | (1u << 10) | ((32u >> 3) << 17) | ((128u >> 4) << 24);

__device__ __forceinline__ uint64_t smem_desc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
  // Unswizzled K-major shared-memory matrix descriptor: start address,
  // leading (K) and stride (M/N) byte offsets in 16-byte units, version 1.
  return (uint64_t)((addr & 0x3FFFF) >> 4) | ((uint64_t)((lbo >> 4) & 0x3FFF) << 16) |
         ((uint64_t)((sbo >> 4) & 0x3FFF) << 32) | (1ull << 46);
}
}  // namespace lptc

// Bounded wait for phase `phase` of the mbarrier at shared address `bar`;
// true when it completed.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t phase, int limit) {
  uint32_t done = 0;
  for (int it = 0; it < limit && !done; it++) {
    asm volatile(
        "{\n\t.reg .pred P1;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 P1, [%1], %2;\n\t"
        "selp.b32 %0, 1, 0, P1;\n\t}\n"
        : "=r"(done)
        : "r"(bar), "r"(phase)
        : "memory");
  }
  return done != 0;
}

// ------------------------------------------ fused net inference (tcgen05)
// The whole proposal net, one image at a time per persistent CTA (one per
// SM, the weights staged once), warp-specialised: the MMA warps (8 on)
// issue the tcgen05.mma of the tiles in turn (lane 0 of each) into a ring
// of 16 TMEM accumulators of 32 columns; warps 0-3 and 4-7, two groups that take
// alternate tiles, read each one back as soon as its MMAs commit, add the bias,
// apply the ReLU, store BF16 into the next layer's activation buffer and mark the
// (layer, tile) written (a tile's read-back is a chain of 500 to 700 cycles, so
// one group of eight warps waits where two overlap). A tile
// u of the next layer reads the halo rows of tiles u - 1 .. u + 1, so its
// MMAs start once those three are written, while the epilogue of the later
// tiles runs. Two activation buffers alternate: B holds the input and layer
// 2's output, A layers 1 and 3. Layouts: a 34-pixel halo pitch, channel-group
// major (8 channels = 16 bytes per pixel), each 3x3 tap a descriptor offset, 9 M
// = 128 tiles of virtual pixels.
//
// One thread issuing tcgen05.mma (M = 128, K = 16) sustains one per ~63
// cycles whatever N up to 128, and between a tile's commit and its next
// tile it waits on the queue for several hundred more; the operands stream
// from shared memory at ~128 B per cycle (4 KB of A and 1 KB of B at N =
// 32: ~40 cycles an MMA). Several issuing warps keep the tensor pipe fed.
// The shapes follow from that:
//  - Layer 1 (2 -> 32): each pixel of B's first group holds the input pairs
//    of (x - 1, x, x + 1) and two zeros, so a kernel row is one K = 8 core
//    matrix; rows dy = -1 and 0 share one K = 16 MMA (leading byte offset
//    34 pixels), dy = +1 shares one with a zero-weight half: 2 MMAs a tile.
//  - Layers 2 and 3 (32 -> 32): 18 MMAs a tile (9 taps x 2 K halves), the
//    taps as row offsets of the A descriptor, so the epilogue only adds the
//    bias (putting taps into N instead makes the epilogue shift rows across
//    lanes, which costs more than the MMAs it saves).
//  - Layer 4 (32 -> 1): a 1 x 1 contraction with the 9 taps as N (= 16),
//    z[h][t] = act[h] . w4[t], 2 MMAs a tile, stored into B's channel
//    groups 1-3 (free once layer 3's MMAs are done; their halo rings and
//    tails are zeroed again after); after the last tile the epilogue forms
//    logit[o] = b4 + sum_t z[o + off_t][t] in one pass.
// The next image's 4 KB input arrives by one bulk copy while this image
// runs; a third group of four warps repacks it into B's first group once layer
// 3's MMAs are done, and makes this image's logits and its top k cells (first
// index on ties) while the others go on with the next image: only z has to be
// read before layer 2 of that image is stored over it.
//
// No read of a buffer is overtaken: the epilogue of layer l + 1's tile u waits
// for MMAs that were issued after layer l's tiles u - 1 .. u + 1 were stored, so
// after every MMA that read those rows of the buffer it stores into; layer 4's z
// and the repacked input go over B once all of layer 3's tiles are stored.
// Measured (8160 images, k = 4): 784 us with one epilogue group that also made the
// outputs, 670 us so; of that the tensor pipe takes one M = 128 MMA per ~63
// cycles, 360 an image.
//
// Every slot's tiles come from one issuer (16 is a multiple of the issuer
// count), and each (layer, tile) barrier completes once an image, so no parity
// wait can run a phase ahead of its barrier. Every wait is bounded; a wait that runs out sets the context's status word,
// the other warps leave at their next wait, and the CTA drains its MMAs
// and copy before freeing TMEM.
namespace lpnet {
constexpr int REGION = lptc::REGION;           // one channel group's halo plane (1224 pixels x 16 B)
constexpr int BUF = 4 * REGION;                // 32 channels
constexpr int OFF_A = 0;
constexpr int OFF_B = OFF_A + BUF;
constexpr int OFF_W1 = OFF_B + BUF;            // 4 k-groups x 32 n x 16 B: dy = -1, 0, +1, zeros
constexpr int OFF_W2 = OFF_W1 + 4 * 32 * 16;   // 36 k-groups (tap, channel group) x 32 n x 16 B
constexpr int OFF_W3 = OFF_W2 + 36 * 32 * 16;
constexpr int OFF_W4 = OFF_W3 + 36 * 32 * 16;  // 4 k-groups x 16 n (taps 0-8, zeros) x 16 B
constexpr int OFF_STAGE = OFF_W4 + 4 * 16 * 16;  // the next image's input, 32 x 32 x 2 BF16
constexpr int OFF_Z = OFF_B + REGION;          // layer 4's z, [9 taps][1152 rows] FP32, in B's groups 1-3
constexpr int OFF_LOG = OFF_STAGE + 4096;      // 1024 FP32 logits
constexpr int OFF_RED = OFF_LOG + 1024 * 4;    // 2 x 4 u64 per-warp maxima (by round parity)
constexpr int OFF_BAR = OFF_RED + 2 * 8 * 8;
constexpr int TILES = 9;                       // ceil(32 * 34 / 128)
constexpr int NSLOT = 16;                      // TMEM accumulators of 32 columns
constexpr int ISSUERS = 4;
constexpr int BAR_FULL = 0;                    // [16] MMAs of a slot committed
constexpr int BAR_EMPTY = BAR_FULL + NSLOT;    // [16] a slot read back (4 warp arrivals)
constexpr int BAR_WRITTEN = BAR_EMPTY + NSLOT; // [3][9] layer l's tile u stored (4 warp arrivals)
constexpr int BAR_INPUT = BAR_WRITTEN + 3 * TILES;  // the image's input repacked (4 warp arrivals)
constexpr int BAR_STAGE = BAR_INPUT + 1;       // the bulk copy landed
constexpr int BAR_FIN = BAR_STAGE + 1;         // [4] an issuer's MMAs all completed
constexpr int NBAR = BAR_FIN + ISSUERS;
constexpr int OFF_BIAS = (OFF_BAR + NBAR * 8 + 15) / 16 * 16;  // layers 1-3, 32 FP32 each
constexpr int OFF_TMEM = OFF_BIAS + 3 * 32 * 4;
constexpr int OFF_ABORT = OFF_TMEM + 4;
constexpr int SMEM = OFF_ABORT + 12;
constexpr int EPI = 256;                       // 8 epilogue warps
constexpr int GRP = 128;                       // in two groups
constexpr int ISSUE_END = EPI / 32 + ISSUERS;  // the output group's first warp
constexpr int THREADS = EPI + 32 * ISSUERS + GRP;
constexpr uint32_t TMEM_COLS = 512;
constexpr int LIMIT = 1 << 22;
constexpr uint32_t IDESC32 = lptc::IDESC;
constexpr uint32_t IDESC16 = (1u << 4) | (1u << 7) | (1u << 10) | ((16u >> 3) << 17) | ((128u >> 4) << 24);
static_assert(SMEM <= 227 * 1024, "fits one CTA per SM");
static_assert(OFF_STAGE % 128 == 0 && OFF_BAR % 8 == 0, "copy and barrier alignment");
static_assert(NSLOT * 32 <= (int)TMEM_COLS && NSLOT % ISSUERS == 0, "TMEM ring; a slot's tiles from one issuer");
static_assert((TILES - 1) * 128 + 127 + 70 < REGION / 16, "tile reads stay in a channel group");
static_assert(9 * TILES * 128 * 4 <= 3 * REGION, "z fits B's groups 1-3");

// A float's order as an unsigned key (finite values).
__device__ __forceinline__ uint32_t fkey(float f) {
  const uint32_t u = __float_as_uint(f);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

__device__ __forceinline__ void mma(uint32_t d, uint64_t ad, uint64_t bd, uint32_t idesc, uint32_t acc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(d),
      "l"(ad), "l"(bd), "r"(idesc), "r"(acc));
}

__device__ __forceinline__ bool try_wait(uint32_t bar, uint32_t parity) {
  uint32_t done;
  asm volatile(
      "{\n\t.reg .pred P1;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 P1, [%1], %2;\n\t"
      "selp.b32 %0, 1, 0, P1;\n\t}\n"
      : "=r"(done)
      : "r"(bar), "r"(parity)
      : "memory");
  return done != 0;
}

// Bounded wait for the phase of parity `parity`; gives up early once another
// warp has set the abort word.
__device__ __forceinline__ bool wait(uint32_t bar, uint32_t parity, const volatile uint32_t* abort) {
  for (int it = 0; it < LIMIT; it++) {
    if (try_wait(bar, parity)) return true;
    if ((it & 255) == 255 && *abort) return false;
  }
  return false;
}

__device__ __forceinline__ void arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}

// Named barrier 3 over the epilogue and output groups' threads; the OR of `p`.
__device__ __forceinline__ bool out_or(bool p) {
  uint32_t r;
  __syncwarp();
  asm volatile(
      "{\n\t.reg .pred q, r;\n\t"
      "setp.ne.b32 q, %1, 0;\n\t"
      "bar.red.or.pred r, 3, %2, q;\n\t"
      "selp.b32 %0, 1, 0, r;\n\t}\n"
      : "=r"(r)
      : "r"((uint32_t)p), "n"(EPI + GRP)
      : "memory");
  return r != 0;
}

// 16 consecutive 32-bit TMEM columns of this warp's 32 lanes.
__device__ __forceinline__ void tmem_ld16(uint32_t addr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, "
      "%14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(addr));
}

// The 4 KB input of one image into `stage` by one bulk copy completing on `bar`.
__device__ __forceinline__ void fetch_input(uint32_t stage, const uint16_t* src, uint32_t bar) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(4096) : "memory");
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], 4096, [%2];" ::"r"(stage),
      "l"(src), "r"(bar)
      : "memory");
}
}  // namespace lpnet

__global__ void __launch_bounds__(lpnet::THREADS, 1) lp_net_kernel(const uint16_t* X, int n, const uint16_t* W1,
                                                                 const float* b1, const uint16_t* W2, const float* b2,
                                                                 const uint16_t* W3, const float* b3,
                                                                 const uint16_t* W4, const float* b4, int k,
                                                                 int32_t* cells, float* logits, uint32_t* status) {
  using namespace lpnet;
  extern __shared__ __align__(128) uint8_t sm_[];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t base = (uint32_t)__cvta_generic_to_shared(sm_);
  const uint32_t a_a = base + OFF_A, b_a = base + OFF_B;
  const uint32_t w1_a = base + OFF_W1, w2_a = base + OFF_W2, w3_a = base + OFF_W3, w4_a = base + OFF_W4;
  const uint32_t stage_a = base + OFF_STAGE;
  auto bar = [&](int i) { return base + (uint32_t)(OFF_BAR + 8 * i); };
  volatile uint32_t* abort_w = reinterpret_cast<volatile uint32_t*>(sm_ + OFF_ABORT);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(sm_ + OFF_TMEM);

  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(base + OFF_TMEM),
                 "r"(TMEM_COLS));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  if (tid == 0) {
    for (int i = 0; i < NBAR; i++) {
      const bool one = (i >= BAR_FULL && i < BAR_FULL + NSLOT) || i == BAR_STAGE || i >= BAR_FIN;
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar(i)), "r"(one ? 1 : GRP / 32));
    }
    *abort_w = 0;
    asm volatile("fence.mbarrier_init.release.cluster;");
  }
  // Zero both activation buffers once (halo rings and tails stay zero: only
  // interior pixels are ever written), and stage the weights as
  // [k-group][n][8] K-major matrices.
  for (int q = tid; q < 2 * BUF / 16; q += THREADS) reinterpret_cast<uint4*>(sm_ + OFF_A)[q] = make_uint4(0, 0, 0, 0);
  uint16_t* w1s = reinterpret_cast<uint16_t*>(sm_ + OFF_W1);
  for (int q = tid; q < 4 * 32 * 8; q += THREADS) {
    // k-group kg = dy + 1 holds the row's taps dx = -1, 0, +1 for both input
    // channels (e = 2 (dx + 1) + c); k-group 3 and e = 6, 7 are zero.
    const int e = q & 7, nn = (q >> 3) & 31, kg = q >> 8;
    w1s[q] = (kg < 3 && e < 6) ? W1[nn * 18 + (kg * 3 + (e >> 1)) * 2 + (e & 1)] : (uint16_t)0;
  }
  uint16_t* w2s = reinterpret_cast<uint16_t*>(sm_ + OFF_W2);
  uint16_t* w3s = reinterpret_cast<uint16_t*>(sm_ + OFF_W3);
  for (int q = tid; q < 36 * 32 * 8; q += THREADS) {
    // k-group kg = 4 tap + channel group.
    const int e = q & 7, nn = (q >> 3) & 31, kg = q >> 8;
    w2s[q] = W2[nn * 288 + kg * 8 + e];
    w3s[q] = W3[nn * 288 + kg * 8 + e];
  }
  if (tid < 96) reinterpret_cast<float*>(sm_ + OFF_BIAS)[tid] = (tid < 32 ? b1 : (tid < 64 ? b2 : b3))[tid & 31];
  uint16_t* w4s = reinterpret_cast<uint16_t*>(sm_ + OFF_W4);
  for (int q = tid; q < 4 * 16 * 8; q += THREADS) {
    // n = tap t (rows 9-15 zero), k = channel.
    const int e = q & 7, t = (q >> 3) & 15, kg = q >> 7;
    w4s[q] = t < 9 ? W4[t * 32 + kg * 8 + e] : (uint16_t)0;
  }
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tmem_slot;
  const int first = blockIdx.x, stride = gridDim.x;

  if (warp >= EPI / 32 && warp < ISSUE_END) {
    // ---- the MMA warps: issuer i takes the tiles t = i, i + ISSUERS, ... of
    // the 36 an image (layers 1-4 x 9); lane 0 issues, the whole warp waits.
    const int iss = warp - EPI / 32;
    bool ok = true;
    int copies = 0;  // bulk copies issued (issuer 0)
    if (iss == 0) {
      if (lane == 0) fetch_input(stage_a, X + (size_t)first * 2048, bar(BAR_STAGE));
      copies = 1;
    }
    int j = 0;
    for (int img = first; img < n && ok; img += stride, j++) {
      ok = __all_sync(0xffffffffu, wait(bar(BAR_INPUT), (uint32_t)j & 1u, abort_w));
      if (!ok) break;
      // The stage is free again (its contents repacked): the next image's copy.
      if (iss == 0 && img + stride < n) {
        if (lane == 0) fetch_input(stage_a, X + (size_t)(img + stride) * 2048, bar(BAR_STAGE));
        copies++;
      }
      for (int t = iss; t < 4 * TILES; t += ISSUERS) {
        const int layer = t / TILES, u = t % TILES;
        bool w_ok = true;
        if (layer > 0) {
          // The previous layer's tiles u - 1 .. u + 1 stored.
          for (int w = u - 1; w <= u + 1 && w_ok; w++)
            if (w >= 0 && w < TILES) w_ok = wait(bar(BAR_WRITTEN + (layer - 1) * TILES + w), (uint32_t)j & 1u, abort_w);
        }
        const uint32_t seq = (uint32_t)j * (4u * TILES) + (uint32_t)t, s = seq % NSLOT, use = seq / NSLOT;
        if (w_ok && use > 0) w_ok = wait(bar(BAR_EMPTY + (int)s), (use - 1) & 1u, abort_w);
        ok = __all_sync(0xffffffffu, w_ok);
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        if (lane == 0) {
          const uint32_t d = tmem + s * 32;
          const uint32_t v0 = (uint32_t)u * 128;
          if (layer == 0) {
            // Rows dy = -1 and 0 (34 pixels apart), then dy = +1 with a
            // zero-weight half one pixel on.
            mma(d, lptc::smem_desc(b_a + (v0 + 1) * 16, 34 * 16, 128), lptc::smem_desc(w1_a, 512, 128), IDESC32, 0u);
            mma(d, lptc::smem_desc(b_a + (v0 + 69) * 16, 16, 128), lptc::smem_desc(w1_a + 2 * 512, 512, 128), IDESC32,
                1u);
          } else if (layer < 3) {
            const uint32_t src = layer == 1 ? a_a : b_a, w_a = layer == 1 ? w2_a : w3_a;
#pragma unroll
            for (int ks = 0; ks < 18; ks++) {
              const int tap = ks >> 1, hh = ks & 1, off = (tap / 3) * 34 + tap % 3;
              mma(d, lptc::smem_desc(src + (uint32_t)(2 * hh * REGION) + (v0 + off) * 16, REGION, 128),
                  lptc::smem_desc(w_a + (uint32_t)((tap * 4 + 2 * hh) * 512), 512, 128), IDESC32, ks > 0 ? 1u : 0u);
            }
          } else {
            // Layer 4 over A: z for the tile's 128 halo pixels.
            mma(d, lptc::smem_desc(a_a + v0 * 16, REGION, 128), lptc::smem_desc(w4_a, 256, 128), IDESC16, 0u);
            mma(d, lptc::smem_desc(a_a + 2 * REGION + v0 * 16, REGION, 128), lptc::smem_desc(w4_a + 512, 256, 128),
                IDESC16, 1u);
          }
          asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                           bar(BAR_FULL + (int)s))
                       : "memory");
        }
        __syncwarp();
      }
    }
    if (!ok && lane == 0) {
      atomicExch(status, 1u);  // DEV_TIMEOUT
      *abort_w = 1;
    }
    // Drain: every MMA this warp issued, and the last bulk copy, complete
    // before the CTA frees TMEM and leaves.
    if (lane == 0)
      asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                       bar(BAR_FIN + iss))
                   : "memory");
    __syncwarp();
    mbar_wait(bar(BAR_FIN + iss), 0, LIMIT);
    if (iss == 0) mbar_wait(bar(BAR_STAGE), (uint32_t)(copies - 1) & 1u, LIMIT);
    __syncwarp();
  } else {
    // ---- the epilogue warps, in two groups of four: warp w reads TMEM lanes 32
    // (w % 4) .. +31, all 32 columns, of its group's accumulators. A third group
    // repacks inputs and makes an image's outputs while they go on.
    const int lq = warp & 3, grp = warp >= ISSUE_END ? 2 : warp >> 2, gt = tid & 127;
    float* z = reinterpret_cast<float*>(sm_ + OFF_Z);
    float* log_s = reinterpret_cast<float*>(sm_ + OFF_LOG);
    unsigned long long* red = reinterpret_cast<unsigned long long*>(sm_ + OFF_RED);
    const float bias4 = __ldg(b4);
    bool ok = true;
    // One image's input from the stage into B's first group (the output group):
    // pixel (y, x) holds the pairs of (x - 1, x, x + 1) (zero outside the image)
    // and two zeros; then the hand-over to the MMA warps.
    auto repack = [&]() {
      const uint32_t* st = reinterpret_cast<const uint32_t*>(sm_ + OFF_STAGE);
      for (int p = gt; p < 1024; p += GRP) {
        const int y = p >> 5, x = p & 31;
        const uint32_t l = x > 0 ? st[p - 1] : 0u, c = st[p], r = x < 31 ? st[p + 1] : 0u;
        *reinterpret_cast<uint4*>(sm_ + OFF_B + ((y + 1) * 34 + x + 1) * 16) = make_uint4(l, c, r, 0u);
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (lane == 0) arrive(bar(BAR_INPUT));
    };
    // A bounded wait by the whole warp; one that runs out stops the other warps'.
    auto wait_warp = [&](int i, uint32_t parity) {
      const bool done = __all_sync(0xffffffffu, wait(bar(i), parity, abort_w));
      if (!done && lane == 0) *abort_w = 1;
      return done;
    };
    auto group_sync = [&]() {
      __syncwarp();
      asm volatile("bar.sync 2, %0;" ::"n"(GRP) : "memory");
    };
    // An image's logits from z, by the output group; then B's groups 1-3 are free.
    auto make_logits = [&]() {
      // The logits (halo rows past the last tile are zero).
      for (int o = gt; o < 32 * 34; o += GRP) {
        const int y = o / 34, x = o % 34;
        if (x < 32) {
          float acc = 0.f;
#pragma unroll
          for (int tap = 0; tap < 9; tap++) {
            const int h = o + (tap / 3) * 34 + tap % 3;
            acc += h < TILES * 128 ? z[tap * (TILES * 128) + h] : 0.f;
          }
          log_s[y * 32 + x] = acc + bias4;
        }
      }
      group_sync();  // z read: B's groups 1-3 get their zero halo rings and tails back
      for (int q = gt; q < 3 * (34 * 34 - 32 * 32 + lptc::NV - 34 * 34); q += GRP) {
        const int g = 1 + q / (lptc::NV - 32 * 32), r = q % (lptc::NV - 32 * 32);
        // r-th non-interior pixel of the group: the ring (34 x 34 minus the
        // 32 x 32 interior), then the tail past 34 x 34.
        int h;
        if (r < 34) h = r;                                    // top row
        else if (r < 68) h = 33 * 34 + (r - 34);              // bottom row
        else if (r < 68 + 64) { const int rr = r - 68; h = (1 + (rr >> 1)) * 34 + ((rr & 1) ? 33 : 0); }
        else h = 34 * 34 + (r - 132);                          // tail
        *reinterpret_cast<uint4*>(sm_ + OFF_B + g * REGION + h * 16) = make_uint4(0, 0, 0, 0);
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    };
    auto outputs = [&](int img) {
      if (logits)
        for (int q = gt; q < 1024; q += GRP) logits[(size_t)img * 1024 + q] = log_s[q];
      // The top k cells, best first, the first index among equal scores:
      // each thread keeps its eight scores in registers; a round publishes
      // the warp maxima (one barrier, the array alternating by round),
      // every thread reduces them alike and the owner drops the chosen cell.
      float mine[8];
#pragma unroll
      for (int i = 0; i < 8; i++) mine[i] = log_s[gt + GRP * i];
      for (int round = 0; round < k; round++) {
        unsigned long long best = 0;
#pragma unroll
        for (int i = 0; i < 8; i++) {
          const unsigned long long key = ((unsigned long long)fkey(mine[i]) << 32) | (uint32_t)(1023 - (gt + GRP * i));
          best = key > best ? key : best;
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
          const unsigned long long other = __shfl_xor_sync(0xffffffffu, best, o);
          best = other > best ? other : best;
        }
        unsigned long long* rr = red + (round & 1) * 4;
        if (lane == 0) rr[lq] = best;
        group_sync();
        unsigned long long b = rr[0];
#pragma unroll
        for (int w = 1; w < 4; w++) b = rr[w] > b ? rr[w] : b;
        const int cell = 1023 - (int)(b & 0x3ffu);
        if (gt == 0) cells[(size_t)img * k + round] = cell;
#pragma unroll
        for (int i = 0; i < 8; i++)
          if (cell == gt + GRP * i) mine[i] = -INFINITY;
      }
    };
    // Tiles u0, u0 + step, ... of layer 1, 2 or 3 (layer = 0, 1, 2) of image j.
    auto tiles = [&](int j, int layer, int u0, int step) {
      const uint32_t dst = layer == 1 ? OFF_B : OFF_A;
      float bb[32];
#pragma unroll
      for (int q = 0; q < 32; q++) bb[q] = reinterpret_cast<const float*>(sm_ + OFF_BIAS)[layer * 32 + q];
      for (int u = u0; u < TILES && ok; u += step) {
        const uint32_t seq = (uint32_t)j * (4u * TILES) + (uint32_t)(layer * TILES + u);
        const uint32_t s = seq % NSLOT, use = seq / NSLOT;
        ok = wait_warp(BAR_FULL + (int)s, use & 1u);
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        uint32_t r[2][16];
        tmem_ld16(tmem + ((uint32_t)(32 * lq) << 16) + s * 32, r[0]);
        tmem_ld16(tmem + ((uint32_t)(32 * lq) << 16) + s * 32 + 16u, r[1]);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncwarp();
        if (lane == 0) arrive(bar(BAR_EMPTY + (int)s));
        const int v = u * 128 + 32 * lq + lane, y = v / 34, x = v % 34;
        if (y < 32 && x < 32) {
          uint8_t* px = sm_ + dst + ((y + 1) * 34 + x + 1) * 16;
#pragma unroll
          for (int g = 0; g < 4; g++) {
            uint32_t o[4];
#pragma unroll
            for (int q = 0; q < 4; q++) {
              const int c = 8 * g + 2 * q;
              o[q] = pack_bf16(fmaxf(__uint_as_float(r[c >> 4][c & 15]) + bb[c], 0.f),
                               fmaxf(__uint_as_float(r[c >> 4][(c & 15) + 1]) + bb[c + 1], 0.f));
            }
            *reinterpret_cast<uint4*>(px + g * REGION) = make_uint4(o[0], o[1], o[2], o[3]);
          }
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncwarp();
        if (lane == 0) arrive(bar(BAR_WRITTEN + layer * TILES + u));
      }
    };
    if (grp == 2) {
      ok = wait_warp(BAR_STAGE, 0u);
      if (ok) repack();
    }
    int j = 0, last = -1;
    for (int img = first; img < n; img += stride, j++) {
      if (grp < 2) tiles(j, 0, grp, 2);
      else if (last >= 0) make_logits();
      ok = !out_or(!ok);  // z is read: B's groups 1-3 are free
      if (!ok) break;
      if (grp < 2) {
        tiles(j, 1, grp, 2);
        tiles(j, 2, grp, 2);
      } else if (last >= 0) {
        outputs(last);
      }
      // Once every layer-3 tile's MMAs are done: the next input into B's first
      // group, layer 4's z into the others.
      for (int u = 0; u < TILES && ok; u++) ok = wait_warp(BAR_WRITTEN + 2 * TILES + u, (uint32_t)j & 1u);
      if (ok && grp == 2 && img + stride < n) {
        ok = wait_warp(BAR_STAGE, (uint32_t)(j + 1) & 1u);
        if (ok) repack();
      }
      for (int u = grp; grp < 2 && u < TILES && ok; u += 2) {
        const uint32_t seq = (uint32_t)j * (4u * TILES) + (uint32_t)(3 * TILES + u);
        const uint32_t s = seq % NSLOT, use = seq / NSLOT;
        ok = wait_warp(BAR_FULL + (int)s, use & 1u);
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        uint32_t r[16];
        tmem_ld16(tmem + ((uint32_t)(32 * lq) << 16) + s * 32, r);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncwarp();
        if (lane == 0) arrive(bar(BAR_EMPTY + (int)s));
        float* zs = z + u * 128 + 32 * lq + lane;
#pragma unroll
        for (int t = 0; t < 9; t++) zs[t * (TILES * 128)] = __uint_as_float(r[t]);
      }
      ok = !out_or(!ok);  // z complete, and layer 4's MMAs: A takes the next layer 1
      if (!ok) break;
      last = img;
    }
    if (ok && grp == 2 && last >= 0) {
      make_logits();
      outputs(last);
    }
    if (!ok && tid == 0) {
      atomicExch(status, 1u);  // DEV_TIMEOUT
      *abort_w = 1;
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TMEM_COLS));
  }
}

// ------------------------------------- training on persistent pipelines
//
// The training pass's convolutions for 16-byte aligned tensors (others take
// lp_conv_fwd_smem_kernel, lp_conv_bwd_data_kernel and lp_conv_bwd_w_smem_kernel).
// All of them are bound by the activations' way through memory (64 KB an
// image and 32-channel tensor, read or written once a kernel) as long as
// neither the loads nor the tensor cores wait: so each kernel is one CTA an SM
// that walks its images with a producer warp issuing the TMA loads of the next
// while the others compute. Every wait is bounded; one that runs out sets the
// context's status word and the abort word, and the CTA leaves once its own
// copies and MMAs are in (bounded again).
//
// Sums grow in the element-wise kernels' order, so results differ from theirs only
// in the order of the atomics (dW of the last layer: in the order of its chain).
//
// Measured at 2048 images, us a launch, with the element-wise kernels and a
// one-image-a-CTA tcgen05 forward, then with these: 2 -> 32 forward 87 -> 55, 32 ->
// 32 forward 129 -> 73, dX 943 -> 86, dW 1397 -> 126, 32 -> 1 forward 115 -> 39, dX
// 153 -> 57, dW 954 -> 28, dW of 2 -> 32 549 -> 69; the training step 6.85 -> 0.89 ms.
namespace lptrain {
using lpnet::arrive;
using lpnet::mma;
using lpnet::tmem_ld16;
using lpnet::wait;
using lptc::smem_desc;
constexpr uint32_t FULL = 0xffffffffu;
constexpr int LIMIT = lpnet::LIMIT;
constexpr int HALF_BYTES = 16 * 32 * 64;  // 16 rows of 32 pixels, 32 channels

__device__ __forceinline__ void bar_init(uint32_t bar, int count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count));
}
// K-major shared-memory matrix descriptor of 64-byte rows in the 64-byte swizzle:
// 8-row atoms 512 bytes apart.
__device__ __forceinline__ uint64_t smem_desc64(uint32_t addr) {
  return (uint64_t)((addr & 0x3FFFF) >> 4) | (1ull << 16) | (32ull << 32) | (1ull << 46) | (4ull << 61);
}
__device__ __forceinline__ void expect(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void tma4(uint32_t dst, const CUtensorMap* tm, int c, int x, int y, int im, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], "
      "[%6];" ::"r"(dst),
      "l"(tm), "r"(c), "r"(x), "r"(y), "r"(im), "r"(bar)
      : "memory");
}
__device__ __forceinline__ void tma3(uint32_t dst, const CUtensorMap* tm, int x, int y, int im, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], "
      "[%5];" ::"r"(dst),
      "l"(tm), "r"(x), "r"(y), "r"(im), "r"(bar)
      : "memory");
}
__device__ __forceinline__ void commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void ldsm4(uint32_t addr, uint32_t (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr)
               : "memory");
}
__device__ __forceinline__ void ldsm4t(uint32_t addr, uint32_t (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr)
               : "memory");
}
__device__ __forceinline__ float bf_lo(uint32_t v) { return __uint_as_float(v << 16); }
__device__ __forceinline__ float bf_hi(uint32_t v) { return __uint_as_float(v & 0xffff0000u); }
// Two channels of `v` where the same channels of x are above zero (the ReLU's
// gradient; NaN is not above).
__device__ __forceinline__ uint32_t relu_mask(uint32_t v, uint32_t x) {
  return (bf_lo(x) > 0.f ? v & 0xffffu : 0u) | (bf_hi(x) > 0.f ? v & 0xffff0000u : 0u);
}
// Byte offset of channel group cg (8 channels, 16 bytes) of pixel p in a tile of
// 64-byte pixels that TMA's 64-byte swizzle wrote (512-byte aligned): 8
// consecutive pixels' groups lie on distinct banks.
__device__ __forceinline__ uint32_t swz(int p, int cg) { return (uint32_t)(p * 64 + (((cg ^ (p >> 1)) & 3) << 4)); }

// db over half an image of dY in a stage at `tile`: lane = channel, pixel after
// pixel. One FP32 chain a group of LP_WCPB halves, the element-wise kernel's: a
// bias gradient is a small difference of large sums, and another order of them
// moves it by up to 2e-4. 512 dependent additions take less time than a stage's
// MMAs, on a warp of their own.
__device__ __forceinline__ void db_chain(uint32_t tile, int lane, float& sum) {
  uint32_t at[4];
#pragma unroll
  for (int r = 0; r < 4; r++) at[r] = tile + (uint32_t)((((lane >> 3) ^ r) & 3) << 4) + (lane & 7) * 2;
  // Each addition sits between the loads of the pixels 32 on.
  uint32_t v[32];
  auto load = [&](int p, int i) {
    asm volatile("ld.shared.u16 %0, [%1];" : "=r"(v[i]) : "r"(at[(i >> 1) & 3] + (uint32_t)(p + i) * 64));
  };
#pragma unroll
  for (int i = 0; i < 32; i++) load(0, i);
#pragma unroll 1
  for (int p = 32; p < 512; p += 32)
#pragma unroll
    for (int i = 0; i < 32; i++) {
      sum += __uint_as_float(v[i] << 16);
      load(p, i);
    }
#pragma unroll
  for (int i = 0; i < 32; i++) sum += __uint_as_float(v[i] << 16);
}
}  // namespace lptrain

// The 32 -> 32 convolution, forward or (BWD) the gradient of its input. An
// implicit GEMM D[pixel][n] = sum over (tap, k) of A[pixel + tap][k] *
// W'[n][tap][k] on the 5th-generation tensor cores: forward A = X, W' = W;
// backward A = dY, W'[ci][tap][co] = W[co][8 - tap][ci], and the result is
// masked by the ReLU of X. An image lies in shared memory with a zero halo on
// a 34-pixel row pitch, 64 bytes a pixel in TMA's 64-byte swizzle, as one tile
// load brings it in: the activations as a 4-D tensor (channel, x, y, image), a
// box of 32 channels x 34 x 34 pixels from (0, -1, -1, image), the halo ring from
// the out-of-bounds zero fill. 8 consecutive "virtual" output pixels v = y * 34 +
// x are the 8 rows of a K-major swizzle atom (512 bytes, the pattern a function
// of the address bits), so a tap (dy, dx) is only a base-address shift of (dy + 1)
// * 34 + dx + 1 pixels. (Channel-group major tiles need no swizzle, but their four
// boxes come as 4624 rows of 16 bytes an image: 99 us a
// launch instead of 72.) The
// virtual grid computes 2 discarded columns per row (x = 32, 33) and is covered
// by 9 M = 128 tiles; each takes 18 MMAs of K = 16 (9 taps x 2 channel halves)
// into a 32-column FP32 accumulator in tensor memory. The weights sit as
// [k-group of 8][n][8] (k = tap * 32 + channel).
//
// Warps 0-7 read accumulators back (warp w: lanes 32 (w % 4) .. +31, columns
// 16 (w / 4) .. +15 of a tile), 8-10 issue the MMAs of three tiles an image
// each (one issuing thread sustains one MMA per ~63 cycles, several one per
// ~40, the rate at which A streams from shared memory), 11 loads. Two image
// buffers; five accumulator slots of three tiles, so the next image's MMAs run
// while this one is read back.
namespace lptc3 {
constexpr int SLOTS = 5, GROUP = 3;                      // accumulator slots of GROUP tiles
constexpr int OFF_W = 2 * lptc::IMG_BYTES;
constexpr int OFF_BAR = OFF_W + lptc::W_BYTES;
constexpr int BAR_FULL = 0, BAR_FREE = 2, BAR_ACC = 4, BAR_READ = BAR_ACC + SLOTS, BAR_FIN = BAR_READ + SLOTS;
constexpr int NBAR = BAR_FIN + 3;
constexpr int OFF_TMEM = OFF_BAR + NBAR * 8;
constexpr int SMEM = OFF_TMEM + 8 + 1024;                // + the abort word, + alignment
constexpr int EPI = 256, THREADS = EPI + 4 * 32;
constexpr uint32_t TMEM_COLS = 512;
static_assert(SLOTS * GROUP * 32 <= (int)TMEM_COLS && 3 * GROUP == lptc::TILES, "slots");
}  // namespace lptc3

template <bool BWD>
__global__ void __launch_bounds__(lptc3::THREADS, 1)
    lp_conv_tc_kernel(const __grid_constant__ CUtensorMap tmx, int n, const uint16_t* W, const float* bias, int relu,
                      const uint16_t* Xa, uint16_t* Y, uint32_t* status) {
  using namespace lptrain;
  using namespace lptc3;
  using lptc::IDESC;
  using lptc::NV;
  extern __shared__ uint8_t sm_raw[];
  uint8_t* smt = sm_raw + ((1024u - ((uint32_t)__cvta_generic_to_shared(sm_raw) & 1023u)) & 1023u);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t base = (uint32_t)__cvta_generic_to_shared(smt);
  const uint32_t w_a = base + OFF_W;
  auto bar = [&](int i) { return base + (uint32_t)(OFF_BAR + 8 * i); };
  volatile uint32_t* abort_w = reinterpret_cast<volatile uint32_t*>(smt + OFF_TMEM + 4);
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(base + OFF_TMEM),
                 "r"(TMEM_COLS));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  if (tid == 0) {
    for (int i = 0; i < NBAR; i++)
      bar_init(bar(i), i == BAR_FREE || i == BAR_FREE + 1 ? 3 : (i >= BAR_READ && i < BAR_FIN ? 8 : 1));
    *abort_w = 0;
    asm volatile("fence.mbarrier_init.release.cluster;");
  }
  uint16_t* w_s = reinterpret_cast<uint16_t*>(smt + OFF_W);
  if (BWD) {
    for (int q = tid; q < 9 * 32 * 32; q += THREADS) {
      const int nn = q & 31, co = (q >> 5) & 31, tap = q >> 10;
      w_s[((tap * 4 + (co >> 3)) * 32 + nn) * 8 + (co & 7)] = W[(co * 9 + 8 - tap) * 32 + nn];
    }
  } else {
    for (int q = tid; q < 32 * 36; q += THREADS)
      reinterpret_cast<uint4*>(w_s)[(q % 36) * 32 + q / 36] = reinterpret_cast<const uint4*>(W)[q];
  }
  // Zeros past the 34 x 34 box, which no load touches.
  constexpr int TAIL = (NV - 34 * 34) * 4;
  for (int q = tid; q < 2 * TAIL; q += THREADS)
    reinterpret_cast<uint4*>(smt + (q / TAIL) * lptc::IMG_BYTES)[34 * 34 * 4 + q % TAIL] = make_uint4(0, 0, 0, 0);
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *reinterpret_cast<uint32_t*>(smt + OFF_TMEM);
  const int first = blockIdx.x, stride = gridDim.x;
  bool ok = true;

  if (warp == 11) {
    if (lane == 0) {
      int j = 0;
      for (int img = first; img < n; img += stride, j++) {
        const int b = j & 1;
        if (j >= 2) ok = wait(bar(BAR_FREE + b), (uint32_t)((j >> 1) - 1) & 1u, abort_w);
        if (!ok) break;
        expect(bar(BAR_FULL + b), 34 * 34 * 64);
        tma4(base + (uint32_t)(b * lptc::IMG_BYTES), &tmx, 0, -1, -1, img, bar(BAR_FULL + b));
      }
      // The last loads are in before the CTA leaves.
      for (int k = j > 2 ? j - 2 : 0; k < j; k++) mbar_wait(bar(BAR_FULL + (k & 1)), (uint32_t)(k >> 1) & 1u, LIMIT);
    }
  } else if (warp >= 8) {
    if (lane == 0) {
      const int s = warp - 8;
      int j = 0;
      for (int img = first; img < n; img += stride, j++) {
        const int b = j & 1;
        const uint32_t q = (uint32_t)(3 * j + s), slot = q % SLOTS, use = q / SLOTS;
        ok = wait(bar(BAR_FULL + b), (uint32_t)(j >> 1) & 1u, abort_w) &&
             (use == 0 || wait(bar(BAR_READ + (int)slot), (use - 1) & 1u, abort_w));
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        for (int u = 0; u < GROUP; u++) {
          const uint32_t a0 = base + (uint32_t)(b * lptc::IMG_BYTES + (s * GROUP + u) * 128 * 64);
          const uint32_t d = tmem + slot * (GROUP * 32) + (uint32_t)(u * 32);
          for (int ks = 0; ks < 18; ks++) {
            const int tap = BWD ? 8 - (ks >> 1) : ks >> 1, hh = ks & 1;
            const int off = (tap / 3) * 34 + tap % 3;
            mma(d, smem_desc64(a0 + (uint32_t)(off * 64 + hh * 32)),
                smem_desc(w_a + (uint32_t)((tap * 4 + 2 * hh) * 512), 512, 128), IDESC, ks > 0 ? 1u : 0u);
          }
        }
        commit(bar(BAR_ACC + (int)slot));
        commit(bar(BAR_FREE + b));
      }
      commit(bar(BAR_FIN + s));
      mbar_wait(bar(BAR_FIN + s), 0, LIMIT);
    }
  } else {
    const int lq = warp & 3, half = warp >> 2;
    float bv[16];
#pragma unroll
    for (int i = 0; i < 16; i++) bv[i] = BWD ? 0.f : bias[half * 16 + i];
    // Where this lane's pixels of group s of an image lie.
    auto place = [&](int img, int s, int u, bool& in) {
      const int v = (s * GROUP + u) * 128 + 32 * lq + lane, y = v / 34, x = v - y * 34;
      in = y < 32 && x < 32;
      return ((size_t)img * LP_P + y * 32 + x) * 32 + half * 16;
    };
    // The ReLU's inputs, a group ahead.
    uint4 ahead[GROUP][2] = {};
    auto fetch = [&](int img, int s) {
#pragma unroll
      for (int u = 0; u < GROUP; u++) {
        bool in;
        const size_t at = place(img, s, u, in);
        if (in) {
          ahead[u][0] = reinterpret_cast<const uint4*>(Xa + at)[0];
          ahead[u][1] = reinterpret_cast<const uint4*>(Xa + at)[1];
        }
      }
    };
    if (BWD && Xa) fetch(first, 0);
    uint32_t q = 0;
    for (int img = first; img < n && ok; img += stride) {
      for (int s = 0; s < 3 && ok; s++, q++) {
        const uint32_t slot = q % SLOTS;
        size_t at[GROUP];
        bool in[GROUP];
        uint4 xm[GROUP][2];
#pragma unroll
        for (int u = 0; u < GROUP; u++) {
          at[u] = place(img, s, u, in[u]);
          xm[u][0] = ahead[u][0];
          xm[u][1] = ahead[u][1];
        }
        if (BWD && Xa && (s < 2 || img + stride < n)) fetch(s < 2 ? img : img + stride, s < 2 ? s + 1 : 0);
        ok = __all_sync(FULL, wait(bar(BAR_ACC + (int)slot), (q / SLOTS) & 1u, abort_w));
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        uint32_t r[GROUP][16];
#pragma unroll
        for (int u = 0; u < GROUP; u++)
          tmem_ld16(tmem + ((uint32_t)(32 * lq) << 16) + slot * (GROUP * 32) + (uint32_t)(u * 32 + half * 16), r[u]);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncwarp();
        if (lane == 0) arrive(bar(BAR_READ + (int)slot));
#pragma unroll
        for (int u = 0; u < GROUP; u++) {
          if (!in[u]) continue;
          uint32_t o[8];
#pragma unroll
          for (int i = 0; i < 8; i++) {
            float a = __uint_as_float(r[u][2 * i]), b = __uint_as_float(r[u][2 * i + 1]);
            if (!BWD) {
              a += bv[2 * i];
              b += bv[2 * i + 1];
              if (relu) {
                a = fmaxf(a, 0.f);
                b = fmaxf(b, 0.f);
              }
            }
            o[i] = pack_bf16(a, b);
          }
          if (BWD && Xa) {
            o[0] = relu_mask(o[0], xm[u][0].x);
            o[1] = relu_mask(o[1], xm[u][0].y);
            o[2] = relu_mask(o[2], xm[u][0].z);
            o[3] = relu_mask(o[3], xm[u][0].w);
            o[4] = relu_mask(o[4], xm[u][1].x);
            o[5] = relu_mask(o[5], xm[u][1].y);
            o[6] = relu_mask(o[6], xm[u][1].z);
            o[7] = relu_mask(o[7], xm[u][1].w);
          }
          uint4* dst = reinterpret_cast<uint4*>(Y + at[u]);
          dst[0] = make_uint4(o[0], o[1], o[2], o[3]);
          dst[1] = make_uint4(o[4], o[5], o[6], o[7]);
        }
      }
    }
  }
  if (!ok) {
    atomicExch(status, 1u);  // DEV_TIMEOUT
    *abort_w = 1;
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncwarp();
  __syncthreads();
  if (warp == 0) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TMEM_COLS));
  }
}

// dW and db of the 32 -> 32 convolution: dW[co][tap][ci] = sum over pixels p of
// dY[p][co] X[p + off(tap)][ci]. M = co, N = (tap, ci), K = pixels, by
// mma.sync with both operands read through ldmatrix.trans from the tiles that
// TMA left in shared memory (half an image a stage: 16 rows of dY, 18 rows of X
// with a zero halo); the contraction is over pixels, so each tap is the same
// tile at another pixel offset. A CTA takes groups of LP_WCPB half images and
// adds a group's sums with one atomic per weight: the FP32 chains (512 MMA steps)
// are lp_conv_bwd_w_smem_kernel's, pixel by pixel, so the partial sums are the
// same bits (four shorter chains a warp each measured 20 % less time and gradients
// 2e-5 apart). That fixes K, so six warps split N: warp w holds 16 input
// channels (w / 3) and (ROWS = 3) kernel row w % 3, or (ROWS = 1: few groups, one
// kernel row a CTA) kernel column w % 3. Two more load the stages and add up db.
// (Twelve warps of 8 channels each keep shared memory busier than the tensor
// cores: 126 us at 2048 images without db and 175 with it, 126 with it so.)
constexpr int LP_WCPB = 16;  // half images whose gradients one FP32 chain adds up
namespace lpdw {
constexpr int X_BYTES = 18 * 34 * 64, X_SPACE = (X_BYTES + 511) / 512 * 512;
constexpr int STAGE = X_SPACE + lptrain::HALF_BYTES;
constexpr int STAGES = 3, WARPS = 6, THREADS = (WARPS + 2) * 32;  // + db, + loads
constexpr int OFF_BAR = STAGES * STAGE;
constexpr int SMEM = OFF_BAR + 2 * STAGES * 8 + 8 + 512;  // + the abort word, + alignment
}  // namespace lpdw

template <int ROWS>
__global__ void __launch_bounds__(lpdw::THREADS, 1)
    lp_conv_bwd_w_kernel(const __grid_constant__ CUtensorMap tmx, const __grid_constant__ CUtensorMap tmd, int n,
                         float* dW, float* db, uint32_t* status) {
  using namespace lptrain;
  using namespace lpdw;
  constexpr int KX = ROWS == 3 ? 3 : 1;  // kernel columns of a warp
  extern __shared__ uint8_t sm_raw[];
  uint8_t* sm = sm_raw + ((512u - ((uint32_t)__cvta_generic_to_shared(sm_raw) & 511u)) & 511u);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const uint32_t base = (uint32_t)__cvta_generic_to_shared(sm);
  auto full = [&](int i) { return base + (uint32_t)(OFF_BAR + 8 * i); };
  auto empty = [&](int i) { return base + (uint32_t)(OFF_BAR + 8 * (STAGES + i)); };
  volatile uint32_t* abort_w = reinterpret_cast<volatile uint32_t*>(sm + OFF_BAR + 16 * STAGES);
  if (tid == 0) {
    for (int i = 0; i < STAGES; i++) {
      bar_init(full(i), 1);
      bar_init(empty(i), WARPS + 1);
    }
    *abort_w = 0;
    asm volatile("fence.mbarrier_init.release.cluster;");
  }
  __syncthreads();
  const int items = 2 * n, first = blockIdx.x * LP_WCPB, stride = gridDim.x * LP_WCPB;
  bool ok = true;
  int j = 0;  // half images so far
  if (warp == WARPS + 1) {
    if (lane == 0) {
      for (int i0 = first; i0 < items && ok; i0 += stride)
        for (int it = i0; it < items && it < i0 + LP_WCPB; it++, j++) {
          const int s = j % STAGES;
          if (j >= STAGES) ok = wait(empty(s), (uint32_t)(j / STAGES - 1) & 1u, abort_w);
          if (!ok) break;
          expect(full(s), X_BYTES + HALF_BYTES);
          tma4(base + (uint32_t)(s * STAGE), &tmx, 0, -1, (it & 1) * 16 - 1, it >> 1, full(s));
          tma4(base + (uint32_t)(s * STAGE + X_SPACE), &tmd, 0, 0, (it & 1) * 16, it >> 1, full(s));
        }
      // The last loads are in before the CTA leaves.
      for (int k = j > STAGES ? j - STAGES : 0; k < j; k++)
        mbar_wait(full(k % STAGES), (uint32_t)(k / STAGES) & 1u, LIMIT);
    }
  } else if (warp == WARPS) {
    for (int i0 = first; i0 < items && ok; i0 += stride) {
      float sum = 0.f;
      for (int it = i0; it < items && it < i0 + LP_WCPB; it++, j++) {
        const int s = j % STAGES;
        ok = __all_sync(FULL, wait(full(s), (uint32_t)(j / STAGES) & 1u, abort_w));
        if (!ok) break;
        db_chain(base + (uint32_t)(s * STAGE + X_SPACE), lane, sum);
        __syncwarp();
        if (lane == 0) arrive(empty(s));
      }
      if (ok && (ROWS == 3 || blockIdx.y == 0)) atomicAdd(db + lane, sum);
    }
  } else {
    const int ky = ROWS == 3 ? warp % 3 : (int)blockIdx.y, kx0 = ROWS == 3 ? 0 : warp % 3, ch = warp / 3;
    // This lane's row of the 8 x 8 matrices a load takes: of dY (pixels 0-7 and
    // 8-15, channel groups 0 and 1; 2 and 3 for co 16-31), of X (the same pixels,
    // groups 2 ch and 2 ch + 1).
    const int pa = (lane & 7) + ((lane >> 4) & 1) * 8, ca = (lane >> 3) & 1;
    const int pb = (lane & 15) + kx0 + ky * 34, cb = 2 * ch + (lane >> 4);
    for (int i0 = first; i0 < items && ok; i0 += stride) {
      float acc[KX][2][2][4] = {};  // [kernel column][8 ci][16 co][fragment]
      for (int it = i0; it < items && it < i0 + LP_WCPB; it++, j++) {
        const int s = j % STAGES;
        ok = __all_sync(FULL, wait(full(s), (uint32_t)(j / STAGES) & 1u, abort_w));
        if (!ok) break;
        const uint32_t xs = base + (uint32_t)(s * STAGE), ds = xs + X_SPACE;
        // Step k = 8 o + i takes pixels 16 k .. + 15: row 4 o + i / 2, columns 16 (i
        // % 2) on. The swizzle depends on that row's place in four (a 34-pixel
        // pitch): four base addresses, the rest is immediate. The next step's
        // fragments load while this one's MMAs run.
        uint32_t xb[KX == 3 ? 2 : 1][4];  // kernel columns 0 and 1; 2 is two pixels on
#pragma unroll
        for (int x = 0; x < (KX == 3 ? 2 : 1); x++)
#pragma unroll
          for (int r = 0; r < 4; r++)
            xb[x][r] = xs + (uint32_t)((pb + x) * 64 + (((cb ^ (r + ((pb + x) >> 1))) & 3) << 4));
        uint32_t aa = ds + swz(pa, ca), ab = aa ^ 32u;
        uint32_t a[2][2][4], b[2][KX][4];
        auto load = [&](int i) {
          const int u = i & 1, r = i >> 1, q = (r * 34 + (i & 1) * 16) * 64;
          ldsm4t(aa + i * 1024, a[u][0]);
          ldsm4t(ab + i * 1024, a[u][1]);
          ldsm4t(xb[0][r & 3] + q, b[u][0]);
          if (KX == 3) {
            ldsm4t(xb[KX == 3 ? 1 : 0][r & 3] + q, b[u][KX / 2]);
            ldsm4t(xb[0][(r + 1) & 3] + q + 128, b[u][KX - 1]);
          }
        };
        load(0);
#pragma unroll 1
        for (int o = 0; o < 4; o++) {
#pragma unroll
          for (int i = 0; i < 8; i++) {
            const int u = i & 1;
            if (i < 7) {
              load(i + 1);
            } else if (o < 3) {
              // Four rows on.
              aa += 8 * 1024;
              ab += 8 * 1024;
#pragma unroll
              for (int r = 0; r < (KX == 3 ? 8 : 4); r++) xb[r >> 2][r & 3] += 4 * 34 * 64;
              load(0);
            }
#pragma unroll
            for (int m = 0; m < 2; m++)
#pragma unroll
              for (int x = 0; x < KX; x++) {
                mma_bf16(acc[x][0][m], a[u][m], {b[u][x][0], b[u][x][1]});
                mma_bf16(acc[x][1][m], a[u][m], {b[u][x][2], b[u][x][3]});
              }
          }
        }
        __syncwarp();
        if (lane == 0) arrive(empty(s));
      }
      if (!ok) break;
#pragma unroll
      for (int q = 0; q < KX * 16; q++) {
        const int x = q >> 4, i = (q >> 3) & 1, m = (q >> 2) & 1, f = q & 3;
        atomicAdd(dW + (m * 16 + g + 8 * (f >> 1)) * 288 + (ky * 3 + kx0 + x) * 32 + ch * 16 + i * 8 + 2 * t + (f & 1),
                  acc[x][i][m][f]);
      }
    }
  }
  if (!ok) {
    atomicExch(status, 1u);  // DEV_TIMEOUT
    *abort_w = 1;
  }
  __syncwarp();
  __syncthreads();
}

// dW and db where one side has C channels, 1 or 2, and the other 32. C = 2 (the
// first layer, 2 -> 32): dW[co][tap][c] = sum of dY[p][co] X[p + off][c]. C = 1
// (the last, 32 -> 1): dW[tap][ci] = sum of X[q][ci] dY[q - off]. Either way M =
// the 32 channels, read through ldmatrix.trans from half an image a stage, N =
// (tap, c) gathered from the small tensor's 18 rows (8 elements of zero halo
// beside each, so that the TMA box starts on 16 bytes), K = pixels; a warp holds
// one 16 x 8 tile of dW, its FP32 chain as long as the element-wise kernel's. Bound
// by reading the 32-channel tensor once.
namespace lpdws {
constexpr int STAGE = lptrain::HALF_BYTES + 4096, STAGES = 3;  // two CTAs an SM
constexpr int OFF_BAR = STAGES * STAGE;
constexpr int SMEM = OFF_BAR + 2 * STAGES * 8 + 8 + 512;
template <int C>
constexpr int WARPS_OF = 2 * ((9 * C + 7) / 8);  // 16 x 8 tiles of dW
template <int C>
constexpr int THREADS_OF = 32 * (WARPS_OF<C> + C);  // + loads, + db (C = 2)
}  // namespace lpdws

// One half image of dW of the last layer at (channel, tap), pixel by pixel, added to
// `sum`. A matrix instruction multiplies every X of its tile with every column's dY, a
// halo's zeros among them, which an infinity or NaN in X would turn into NaN where
// that pixel and tap have no pixel of dY between them; and a pixel of dY whose own X
// lies outside does not count there, where the element-wise kernel multiplies it with
// a zero. So a half image that leaves a tile's sums not finite is summed this way
// instead, as the element-wise kernel's zeros have it.
__device__ __noinline__ float lp_edge_sum(const uint8_t* xt, const uint16_t* small, int half, int ch, int tap,
                                          float sum) {
  constexpr int RP = 32 + 16;
  const int dy = tap / 3 - 1, dx = tap % 3 - 1;
  auto in = [](int v) { return v >= 0 && v < 32; };
  auto value = [](uint16_t b) { return __uint_as_float((uint32_t)b << 16); };
#pragma unroll 1
  for (int p = 0; p < 512; p++) {
    const int r = p >> 5, x = p & 31, y = half * 16 + r;
    if (in(y - dy) && in(x - dx))
      sum += value(*reinterpret_cast<const uint16_t*>(xt + lptrain::swz(p, ch >> 3) + (ch & 7) * 2)) *
             value(small[(r + 1 - dy) * RP + 8 + x - dx]);
    if (!in(y + dy) || !in(x + dx)) sum += value(small[(r + 1) * RP + 8 + x]) * 0.f;
  }
  return sum;
}

template <int C>
__global__ void __launch_bounds__(lpdws::THREADS_OF<C>, 2)
    lp_conv_bwd_w_edge_kernel(const __grid_constant__ CUtensorMap tm32, const __grid_constant__ CUtensorMap tms, int n,
                              float* dW, float* db, uint32_t* status) {
  using namespace lptrain;
  using namespace lpdws;
  constexpr int RP = 32 * C + 16, SMALL = 18 * RP * 2, N = 9 * C, WARPS = WARPS_OF<C>, S = C == 2 ? 1 : -1;
  static_assert(SMALL <= 4096, "the small tensor's rows fit");
  extern __shared__ uint8_t sm_raw[];
  uint8_t* sm = sm_raw + ((512u - ((uint32_t)__cvta_generic_to_shared(sm_raw) & 511u)) & 511u);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const uint32_t base = (uint32_t)__cvta_generic_to_shared(sm);
  auto full = [&](int i) { return base + (uint32_t)(OFF_BAR + 8 * i); };
  auto empty = [&](int i) { return base + (uint32_t)(OFF_BAR + 8 * (STAGES + i)); };
  volatile uint32_t* abort_w = reinterpret_cast<volatile uint32_t*>(sm + OFF_BAR + 16 * STAGES);
  if (tid == 0) {
    for (int i = 0; i < STAGES; i++) {
      bar_init(full(i), 1);
      bar_init(empty(i), C == 2 ? WARPS + 1 : WARPS);
    }
    *abort_w = 0;
    asm volatile("fence.mbarrier_init.release.cluster;");
  }
  __syncthreads();
  const int items = 2 * n, first = blockIdx.x * LP_WCPB, stride = gridDim.x * LP_WCPB;
  bool ok = true;
  int j = 0;
  if (warp == WARPS) {
    if (lane == 0) {
      for (int i0 = first; i0 < items && ok; i0 += stride)
        for (int it = i0; it < items && it < i0 + LP_WCPB; it++, j++) {
          const int s = j % STAGES;
          if (j >= STAGES) ok = wait(empty(s), (uint32_t)(j / STAGES - 1) & 1u, abort_w);
          if (!ok) break;
          expect(full(s), HALF_BYTES + SMALL);
          tma4(base + (uint32_t)(s * STAGE), &tm32, 0, 0, (it & 1) * 16, it >> 1, full(s));
          tma3(base + (uint32_t)(s * STAGE + HALF_BYTES), &tms, -8, (it & 1) * 16 - 1, it >> 1, full(s));
        }
      for (int k = j > STAGES ? j - STAGES : 0; k < j; k++)
        mbar_wait(full(k % STAGES), (uint32_t)(k / STAGES) & 1u, LIMIT);
    }
  } else if (C == 2 && warp == WARPS + 1) {
    for (int i0 = first; i0 < items && ok; i0 += stride) {
      float sum = 0.f;
      for (int it = i0; it < items && it < i0 + LP_WCPB; it++, j++) {
        const int s = j % STAGES;
        ok = __all_sync(FULL, wait(full(s), (uint32_t)(j / STAGES) & 1u, abort_w));
        if (!ok) break;
        db_chain(base + (uint32_t)(s * STAGE), lane, sum);
        __syncwarp();
        if (lane == 0) arrive(empty(s));
      }
      if (ok) atomicAdd(db + lane, sum);
    }
  } else {
    const int m = warp & 1, i = warp >> 1;  // 16 channels, 8 columns
    const int pa = (lane & 7) + ((lane >> 4) & 1) * 8, ca = ((lane >> 3) & 1) + 2 * m;
    // This lane's column's element at pixel 2 t of a row's first 16 (columns past N,
    // not stored, take the middle tap's).
    const int nn = i * 8 + g < N ? i * 8 + g : N / 2, tap = nn / C;
    const int nb = (1 + S * (tap / 3 - 1)) * RP + 8 + (2 * t + S * (tap % 3 - 1)) * C + nn % C;
    float bs = 0.f;  // C = 1: db
    for (int i0 = first; i0 < items && ok; i0 += stride) {
      float acc[4] = {};
      for (int it = i0; it < items && it < i0 + LP_WCPB; it++, j++) {
        const int s = j % STAGES;
        ok = __all_sync(FULL, wait(full(s), (uint32_t)(j / STAGES) & 1u, abort_w));
        if (!ok) break;
        const uint32_t as = base + (uint32_t)(s * STAGE);
        const uint16_t* small = reinterpret_cast<const uint16_t*>(sm + s * STAGE + HALF_BYTES);
        const float before[4] = {acc[0], acc[1], acc[2], acc[3]};
        // Four steps' fragments load while the four before run.
        uint32_t a[2][4][4], b[2][4][2];
        auto load = [&](int v) {
#pragma unroll
          for (int w = 0; w < 4; w++) {
            const int k = v * 4 + w;
            ldsm4t(as + swz(pa, ca) + (uint32_t)k * 1024u, a[v & 1][w]);
            const uint16_t* e = small + (k >> 1) * RP + (k & 1) * 16 * C + nb;
            b[v & 1][w][0] = pack_raw(e[0], e[C]);
            b[v & 1][w][1] = pack_raw(e[8 * C], e[9 * C]);
          }
        };
        load(0);
#pragma unroll 2
        for (int v = 0; v < 8; v++) {
          const int u = v & 1;
          if (v < 7) load(v + 1);
#pragma unroll
          for (int w = 0; w < 4; w++) {
            mma_bf16(acc, a[u][w], b[u][w]);
            const int k = v * 4 + w;
            if (C == 1 && lane < 16 && warp == w)
              bs += __uint_as_float((uint32_t)small[((k >> 1) + 1) * RP + 8 + (k & 1) * 16 + lane] << 16);
          }
        }
        if (C == 1) {
          // Every not finite element reaches the sums of its channel's row or, through
          // the middle tap, a column of every tile.
          const float most = fmaxf(fmaxf(fabsf(acc[0]), fabsf(acc[1])), fmaxf(fabsf(acc[2]), fabsf(acc[3])));
          const bool nan = acc[0] != acc[0] || acc[1] != acc[1] || acc[2] != acc[2] || acc[3] != acc[3];
          if (__any_sync(FULL, nan || most == INFINITY)) {
#pragma unroll
            for (int f = 0; f < 4; f++) {
              const int c = i * 8 + 2 * t + (f & 1);
              acc[f] = lp_edge_sum(sm + s * STAGE, small, it & 1, m * 16 + g + 8 * (f >> 1), c < N ? c : N / 2, before[f]);
            }
          }
        }
        __syncwarp();
        if (lane == 0) arrive(empty(s));
      }
      if (!ok) break;
#pragma unroll
      for (int f = 0; f < 4; f++) {
        const int ch = m * 16 + g + 8 * (f >> 1), c = i * 8 + 2 * t + (f & 1);
        if (c < N) atomicAdd(dW + (C == 2 ? ch * N + c : c * 32 + ch), acc[f]);
      }
    }
    if (C == 1 && ok) {
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) bs += __shfl_xor_sync(FULL, bs, o);
      if (lane == 0) atomicAdd(db, bs);
    }
  }
  if (!ok) {
    atomicExch(status, 1u);  // DEV_TIMEOUT
    *abort_w = 1;
  }
  __syncwarp();
  __syncthreads();
}

// The first layer, 2 -> 32: a tile of 16 pixels takes one K = 8 step a tap (its
// first pair of columns is the pixel's channel pair, the others zero): the sums
// grow tap by tap as in lp_conv_fwd_smem_kernel, so the BF16 results are the same
// ones; eight taps in one K = 16 step would round differently and costs only the
// tensor time that the stores hide. The weights stay in registers, their columns
// ordered so that a lane ends up with 8 consecutive channels of a pixel: column c
// of block j is channel 8 (c / 2) + 2 j + c % 2. One CTA an image; bound by
// writing the 64 KB of its output.
__device__ __forceinline__ void mma_bf16_k8(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t b) {
  asm(
      "mma.sync.aligned.m16n8k8.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a0), "r"(a1), "r"(b));
}
__global__ void __launch_bounds__(256) lp_conv_first_kernel(const uint16_t* X, const uint16_t* W, const float* bias,
                                                            int relu, uint16_t* Y) {
  constexpr int RP = 40;  // words a row: 3 unused, the halo, 32 pixels, the halo
  __shared__ uint32_t xs[34 * RP];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const size_t img = blockIdx.x;
  const uint32_t* Xi = reinterpret_cast<const uint32_t*>(X) + img * LP_P;
  uint32_t v[4];
#pragma unroll
  for (int i = 0; i < 4; i++) v[i] = Xi[tid + 256 * i];
  if (tid < 2 * 34) xs[(tid / 34) * 33 * RP + 3 + tid % 34] = 0;
  else if (tid < 2 * 34 + 64) xs[(1 + ((tid - 68) >> 1)) * RP + 3 + ((tid - 68) & 1) * 33] = 0;
#pragma unroll
  for (int i = 0; i < 4; i++) {
    const int p = tid + 256 * i;
    xs[((p >> 5) + 1) * RP + 4 + (p & 31)] = v[i];
  }
  uint32_t b[4][9];
#pragma unroll
  for (int j = 0; j < 4; j++) {
    const uint16_t* w = W + (8 * (g >> 1) + 2 * j + (g & 1)) * 18;
#pragma unroll
    for (int tap = 0; tap < 9; tap++) b[j][tap] = t == 0 ? pack_raw(w[2 * tap], w[2 * tap + 1]) : 0u;
  }
  float bv[8];
#pragma unroll
  for (int i = 0; i < 8; i++) bv[i] = bias[8 * t + i];
  __syncthreads();
#pragma unroll 2
  for (int u = 0; u < 8; u++) {
    const int tile = warp * 8 + u, y = tile >> 1, xb = (tile & 1) * 16;
    const uint32_t* r = xs + y * RP + xb + g + 3;
    float d[4][4] = {};
#pragma unroll
    for (int tap = 0; tap < 9; tap++) {
      const uint32_t* q = r + (tap / 3) * RP + tap % 3;
      const uint32_t a0 = t == 0 ? q[0] : 0u, a1 = t == 0 ? q[8] : 0u;
#pragma unroll
      for (int j = 0; j < 4; j++) mma_bf16_k8(d[j], a0, a1, b[j][tap]);
    }
#pragma unroll
    for (int h = 0; h < 2; h++) {
      uint32_t o[4];
#pragma unroll
      for (int j = 0; j < 4; j++) {
        float p = d[j][2 * h] + bv[2 * j], q = d[j][2 * h + 1] + bv[2 * j + 1];
        if (relu) {
          p = fmaxf(p, 0.f);
          q = fmaxf(q, 0.f);
        }
        o[j] = pack_bf16(p, q);
      }
      *reinterpret_cast<uint4*>(Y + (img * LP_P + y * 32 + xb + g + 8 * h) * 32 + 8 * t) =
          make_uint4(o[0], o[1], o[2], o[3]);
    }
  }
}

// The gradient of the last layer's input, 1 -> 32: one K = 8 step a tap (its first
// column is dY's pixel), the sums growing tap by tap as the element-wise kernel's;
// masked by the ReLU of X; weights in registers in lp_conv_first_kernel's column
// order. Bound by reading X and writing dX.
__global__ void __launch_bounds__(256) lp_conv_bwd_last_kernel(const uint16_t* dY, const uint16_t* W,
                                                               const uint16_t* Xa, uint16_t* dX) {
  using lptrain::relu_mask;
  constexpr int RP = 40;
  __shared__ uint16_t ys[34 * RP];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const size_t img = blockIdx.x;
  uint32_t v[2];
#pragma unroll
  for (int i = 0; i < 2; i++) v[i] = reinterpret_cast<const uint32_t*>(dY + img * LP_P)[tid + 256 * i];
  if (tid < 2 * 34) ys[(tid / 34) * 33 * RP + 3 + tid % 34] = 0;
  else if (tid < 2 * 34 + 64) ys[(1 + ((tid - 68) >> 1)) * RP + 3 + ((tid - 68) & 1) * 33] = 0;
#pragma unroll
  for (int i = 0; i < 2; i++) {
    const int p = 2 * (tid + 256 * i);
    *reinterpret_cast<uint32_t*>(&ys[((p >> 5) + 1) * RP + 4 + (p & 31)]) = v[i];
  }
  uint32_t b[4][9];
#pragma unroll
  for (int j = 0; j < 4; j++)
#pragma unroll
    for (int tap = 0; tap < 9; tap++)
      b[j][tap] = t == 0 ? (uint32_t)W[tap * 32 + 8 * (g >> 1) + 2 * j + (g & 1)] : 0u;
  __syncthreads();
#pragma unroll 2
  for (int u = 0; u < 8; u++) {
    const int tile = warp * 8 + u, y = tile >> 1, xb = (tile & 1) * 16;
    const size_t at = (img * LP_P + y * 32 + xb + g) * 32 + 8 * t;
    uint4 xm[2];
    if (Xa) {
      xm[0] = *reinterpret_cast<const uint4*>(Xa + at);
      xm[1] = *reinterpret_cast<const uint4*>(Xa + at + 8 * 32);
    }
    // dY at p - off(tap).
    const uint16_t* r = ys + y * RP + xb + g + 3;
    float d[4][4] = {};
#pragma unroll
    for (int tap = 0; tap < 9; tap++) {
      const uint16_t* q = r + (2 - tap / 3) * RP + 2 - tap % 3;
      const uint32_t a0 = t == 0 ? (uint32_t)q[0] : 0u, a1 = t == 0 ? (uint32_t)q[8] : 0u;
#pragma unroll
      for (int j = 0; j < 4; j++) mma_bf16_k8(d[j], a0, a1, b[j][tap]);
    }
#pragma unroll
    for (int h = 0; h < 2; h++) {
      uint32_t o[4];
#pragma unroll
      for (int j = 0; j < 4; j++) o[j] = pack_bf16(d[j][2 * h], d[j][2 * h + 1]);
      if (Xa) {
        o[0] = relu_mask(o[0], xm[h].x);
        o[1] = relu_mask(o[1], xm[h].y);
        o[2] = relu_mask(o[2], xm[h].z);
        o[3] = relu_mask(o[3], xm[h].w);
      }
      *reinterpret_cast<uint4*>(dX + at + (size_t)h * 8 * 32) = make_uint4(o[0], o[1], o[2], o[3]);
    }
  }
}

// The last layer, 32 -> 1: an implicit GEMM over a staged image with its halo,
// one column of N = 8 in use, A through ldmatrix. The sums grow tap by tap and
// channel half by half as in lp_conv_fwd_smem_kernel, so the scores are the same
// bits. (A contraction with the taps as N takes 4 MMAs a tile instead of 18 and the
// same time, 25 us at 2048 images, but scores 3e-7 away, which the softmax's
// BF16 gradient passes on.) Bound by reading X.
namespace lplast {
constexpr int SPACE = (34 * 34 * 64 + 511) / 512 * 512, STAGES = 3, WARPS = 8, THREADS = (WARPS + 1) * 32;
constexpr int OFF_BAR = STAGES * SPACE;
constexpr int SMEM = OFF_BAR + 2 * STAGES * 8 + 8 + 512;
}  // namespace lplast

__global__ void __launch_bounds__(lplast::THREADS, 1)
    lp_conv_last_kernel(const __grid_constant__ CUtensorMap tmx, int n, const uint16_t* W, const float* bias, int relu,
                        float* Y, uint32_t* status) {
  using namespace lptrain;
  using namespace lplast;
  extern __shared__ uint8_t sm_raw[];
  uint8_t* sm = sm_raw + ((512u - ((uint32_t)__cvta_generic_to_shared(sm_raw) & 511u)) & 511u);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const uint32_t base = (uint32_t)__cvta_generic_to_shared(sm);
  auto full = [&](int i) { return base + (uint32_t)(OFF_BAR + 8 * i); };
  auto empty = [&](int i) { return base + (uint32_t)(OFF_BAR + 8 * (STAGES + i)); };
  volatile uint32_t* abort_w = reinterpret_cast<volatile uint32_t*>(sm + OFF_BAR + 16 * STAGES);
  if (tid == 0) {
    for (int i = 0; i < STAGES; i++) {
      bar_init(full(i), 1);
      bar_init(empty(i), WARPS);
    }
    *abort_w = 0;
    asm volatile("fence.mbarrier_init.release.cluster;");
  }
  __syncthreads();
  const int first = blockIdx.x, stride = gridDim.x;
  bool ok = true;
  int j = 0;
  if (warp == WARPS) {
    if (lane == 0) {
      for (int img = first; img < n; img += stride, j++) {
        const int s = j % STAGES;
        if (j >= STAGES) ok = wait(empty(s), (uint32_t)(j / STAGES - 1) & 1u, abort_w);
        if (!ok) break;
        expect(full(s), 34 * 34 * 64);
        tma4(base + (uint32_t)(s * SPACE), &tmx, 0, -1, -1, img, full(s));
      }
      for (int k = j > STAGES ? j - STAGES : 0; k < j; k++)
        mbar_wait(full(k % STAGES), (uint32_t)(k / STAGES) & 1u, LIMIT);
    }
  } else {
    const int pa = (lane & 7) + ((lane >> 3) & 1) * 8, ca = (lane >> 4) & 1;
    uint32_t b[18][2];  // [tap, 16 channels][fragment]: column 0 only
#pragma unroll
    for (int k = 0; k < 18; k++) {
      const uint16_t* w = W + k * 16 + 2 * t;
      b[k][0] = g == 0 ? pack_raw(w[0], w[1]) : 0u;
      b[k][1] = g == 0 ? pack_raw(w[8], w[9]) : 0u;
    }
    const float bv = bias[0];
    for (int img = first; img < n; img += stride, j++) {
      const int s = j % STAGES;
      ok = __all_sync(FULL, wait(full(s), (uint32_t)(j / STAGES) & 1u, abort_w));
      if (!ok) break;
      const uint32_t xs = base + (uint32_t)(s * SPACE);
#pragma unroll 1
      for (int h = 0; h < 2; h++) {
        // Four tiles of 16 pixels: rows 4 warp + 2 h and the next.
        const int y = 4 * warp + 2 * h;
        float d[4][4] = {};
#pragma unroll
        for (int tap = 0; tap < 9; tap++) {
#pragma unroll
          for (int u = 0; u < 4; u++) {
            const int p = (y + (u >> 1) + tap / 3) * 34 + (u & 1) * 16 + tap % 3 + pa;
            const uint32_t aa = xs + swz(p, ca);
            uint32_t a[2][4];
            ldsm4(aa, a[0]);
            ldsm4(aa ^ 32u, a[1]);
            mma_bf16(d[u], a[0], b[2 * tap]);
            mma_bf16(d[u], a[1], b[2 * tap + 1]);
          }
        }
        if (t == 0) {
#pragma unroll
          for (int u = 0; u < 4; u++)
#pragma unroll
            for (int e = 0; e < 2; e++) {
              const float v = d[u][2 * e] + bv;
              Y[(size_t)img * LP_P + (y + (u >> 1)) * 32 + (u & 1) * 16 + g + 8 * e] = relu ? fmaxf(v, 0.f) : v;
            }
        }
      }
      __syncwarp();
      if (lane == 0) arrive(empty(s));
    }
  }
  if (!ok) {
    atomicExch(status, 1u);  // DEV_TIMEOUT
    *abort_w = 1;
  }
  __syncwarp();
  __syncthreads();
}

// cuTensorMapEncodeTiled, taken from the driver once.
using EncodeTiledFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                   const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                   CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeTiledFn encode_tiled() {
  static EncodeTiledFn fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(p);
    else
      cudaGetLastError();
  });
  return fn;
}

vp8a_status encode_map(const uint16_t* x, int rank, const cuuint64_t* dim, const cuuint64_t* stride,
                       const cuuint32_t* box, CUtensorMapSwizzle swizzle, CUtensorMap* tm) {
  const EncodeTiledFn enc = encode_tiled();
  if (!enc) {
    vp8a::set_error("the driver does not provide cuTensorMapEncodeTiled");
    return VP8A_E_CUDA;
  }
  const cuuint32_t estride[4] = {1, 1, 1, 1};
  const CUresult r = enc(tm, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, rank, const_cast<uint16_t*>(x), dim, stride, box,
                         estride, CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                         CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    vp8a::set_error("cuTensorMapEncodeTiled rejected the activation map (error " + std::to_string((int)r) + ")");
    return VP8A_E_CUDA;
  }
  return VP8A_OK;
}

// The TMA map of n NHWC [32][32][32] BF16 images: a 4-D tensor (channel, x, y,
// image) with boxes of 32 channels x w x h x 1 in the 64-byte swizzle.
vp8a_status image_map(const uint16_t* x, uint32_t n, uint32_t w, uint32_t h, CUtensorMap* tm) {
  const cuuint64_t dim[4] = {32, 32, 32, n};
  const cuuint64_t stride[3] = {32 * 2, 32 * 32 * 2, 32 * 32 * 32 * 2};  // bytes, dims 1..3
  const cuuint32_t box[4] = {32, w, h, 1};
  return encode_map(x, 4, dim, stride, box, CU_TENSOR_MAP_SWIZZLE_64B, tm);
}

// The TMA map of n NHWC [32][32][C] images as (x * C + c, y, image): boxes of 18
// rows with 8 elements beside each.
vp8a_status row_map(const uint16_t* x, uint32_t n, uint32_t c, CUtensorMap* tm) {
  const cuuint64_t dim[3] = {32 * c, 32, n};
  const cuuint64_t stride[2] = {64 * c, 2048 * c};
  const cuuint32_t box[3] = {32 * c + 16, 18, 1};
  return encode_map(x, 3, dim, stride, box, CU_TENSOR_MAP_SWIZZLE_NONE, tm);
}

template <typename K>
vp8a_status use_smem(K* kernel, int bytes) {
  VP8A_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
  return VP8A_OK;
}

// The persistent kernels' launches (16-byte aligned tensors, n > 0).
template <bool BWD>
vp8a_status conv_tc(vp8a_ctx* ctx, const uint16_t* a, const uint16_t* W, const float* bias, int n, int relu,
                    const uint16_t* Xa, uint16_t* Y) {
  CUtensorMap tm;
  vp8a_status s = image_map(a, (uint32_t)n, 34, 34, &tm);
  if (s == VP8A_OK) s = use_smem(lp_conv_tc_kernel<BWD>, lptc3::SMEM);
  if (s != VP8A_OK) return s;
  lp_conv_tc_kernel<BWD><<<std::min(n, ctx->sm_count), lptc3::THREADS, lptc3::SMEM, ctx->stream>>>(
      tm, n, W, bias, relu, Xa, Y, ctx->d_status);
  VP8A_CUDA(cudaGetLastError());
  ctx->launches++;
  return VP8A_OK;
}

vp8a_status conv_last(vp8a_ctx* ctx, const uint16_t* X, const uint16_t* W, const float* bias, int n, int relu,
                      float* Y) {
  CUtensorMap tm;
  vp8a_status s = image_map(X, (uint32_t)n, 34, 34, &tm);
  if (s == VP8A_OK) s = use_smem(lp_conv_last_kernel, lplast::SMEM);
  if (s != VP8A_OK) return s;
  lp_conv_last_kernel<<<std::min(n, ctx->sm_count), lplast::THREADS, lplast::SMEM, ctx->stream>>>(
      tm, n, W, bias, relu, Y, ctx->d_status);
  VP8A_CUDA(cudaGetLastError());
  ctx->launches++;
  return VP8A_OK;
}

// All kernel rows in one CTA a group, each byte staged once (512 images 60 us,
// 2048 122 us; a row a CTA 87 and 254), or a row a CTA while three a group find an
// SM each (256 images 46 us; one a group 60).
vp8a_status conv_bwd_w_32(vp8a_ctx* ctx, const uint16_t* dY, const uint16_t* X, int n, float* dW, float* db) {
  CUtensorMap tmx, tmd;
  const int groups = (2 * n + LP_WCPB - 1) / LP_WCPB;
  const bool split = 3 * groups <= ctx->sm_count;
  const auto kernel = split ? lp_conv_bwd_w_kernel<1> : lp_conv_bwd_w_kernel<3>;
  vp8a_status s = image_map(X, (uint32_t)n, 34, 18, &tmx);
  if (s == VP8A_OK) s = image_map(dY, (uint32_t)n, 32, 16, &tmd);
  if (s == VP8A_OK) s = use_smem(kernel, lpdw::SMEM);
  if (s != VP8A_OK) return s;
  kernel<<<dim3(std::min(groups, ctx->sm_count), split ? 3 : 1), lpdw::THREADS, lpdw::SMEM, ctx->stream>>>(
      tmx, tmd, n, dW, db, ctx->d_status);
  VP8A_CUDA(cudaGetLastError());
  ctx->launches++;
  return VP8A_OK;
}

template <int C>
vp8a_status conv_bwd_w_edge(vp8a_ctx* ctx, const uint16_t* t32, const uint16_t* small, int n, float* dW, float* db) {
  CUtensorMap tm, tms;
  const int groups = (2 * n + LP_WCPB - 1) / LP_WCPB;
  vp8a_status s = image_map(t32, (uint32_t)n, 32, 16, &tm);
  if (s == VP8A_OK) s = row_map(small, (uint32_t)n, C, &tms);
  if (s == VP8A_OK) s = use_smem(lp_conv_bwd_w_edge_kernel<C>, lpdws::SMEM);
  if (s != VP8A_OK) return s;
  lp_conv_bwd_w_edge_kernel<C>
      <<<std::min(groups, 2 * ctx->sm_count), lpdws::THREADS_OF<C>, lpdws::SMEM, ctx->stream>>>(tm, tms, n, dW, db,
                                                                                                ctx->d_status);
  VP8A_CUDA(cudaGetLastError());
  ctx->launches++;
  return VP8A_OK;
}

bool aligned16(const void* a, const void* b = nullptr, const void* c = nullptr) {
  return (((uintptr_t)a | (uintptr_t)b | (uintptr_t)c) & 15) == 0;
}

template <int CIN, int NT>
vp8a_status conv_fwd(vp8a_ctx* ctx, const uint16_t* X, const uint16_t* W, const float* b, int cout, int n, int relu,
                     uint16_t* Y, float* Yf) {
  if (n == 0) return VP8A_OK;
  constexpr int CP = (CIN + 15) / 16 * 16, PS = CP + 8, WS = 9 * CIN + 8;
  const size_t smem = sizeof(uint16_t) * (34 * 34 * PS + NT * 8 * WS);
  VP8A_CUDA(cudaFuncSetAttribute(lp_conv_fwd_smem_kernel<CIN, NT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)smem));
  lp_conv_fwd_smem_kernel<CIN, NT><<<n, 256, smem, ctx->stream>>>(X, W, b, cout, relu, Y, Yf);
  VP8A_CUDA(cudaGetLastError());
  ctx->launches++;
  return VP8A_OK;
}

template <int COUT, int NT>
vp8a_status conv_bwd_data(vp8a_ctx* ctx, const uint16_t* dY, const uint16_t* W, int cin, int n, const uint16_t* Xa,
                          uint16_t* dX) {
  const int tiles = n * (LP_P / 16);
  lp_conv_bwd_data_kernel<COUT, NT><<<(tiles + 3) / 4, 128, 0, ctx->stream>>>(dY, W, cin, n, Xa, dX);
  VP8A_CUDA(cudaGetLastError());
  ctx->launches++;
  return VP8A_OK;
}

// Weight gradient with staged chunks: each CTA walks LP_WCPB chunks of 512
// pixels (half an image each), staging the chunk's dY ([pixel][co], co
// padded to 16 * MT) and its 18 input rows with a zero halo ([row][col][ci])
// in shared memory; warp w accumulates the n-tiles w, w + 4, ... of
// dW = dY^T x im2col(X) in registers across all its chunks, and the CTA
// adds its partial sums with one atomic per weight at the end.
template <int CIN, int MT>
__global__ void __launch_bounds__(128) lp_conv_bwd_w_smem_kernel(const uint16_t* dY, const uint16_t* X, int cout,
                                                                 long n_chunks, float* dW, float* db) {
  constexpr int NTOT = (9 * CIN + 7) / 8, NPW = (NTOT + 3) / 4;
  constexpr int DS = 16 * MT + 8, PS = CIN + (CIN >= 16 ? 8 : 0) + (CIN < 16 ? 2 : 0);
  extern __shared__ __align__(16) uint16_t smw[];
  uint16_t* dy_s = smw;                        // 512 * DS
  uint16_t* x_s = smw + LP_WCHUNK * DS;        // 18 * 34 * PS
  const int tid = threadIdx.x, lane = tid & 31, g = lane >> 2, t = lane & 3, warp = tid >> 5;
  float d[NPW][MT][4];
#pragma unroll
  for (int a = 0; a < NPW; a++)
#pragma unroll
    for (int m = 0; m < MT; m++) d[a][m][0] = d[a][m][1] = d[a][m][2] = d[a][m][3] = 0.f;
  float bsum = 0.f;
  for (long ch = (long)blockIdx.x * LP_WCPB; ch < n_chunks && ch < (long)(blockIdx.x + 1) * LP_WCPB; ch++) {
    const long p0 = ch * LP_WCHUNK;
    const int img = (int)(p0 / LP_P), row0 = (int)(p0 % LP_P) / 32;
    __syncthreads();  // the previous chunk's fragments are read
    for (int q = tid; q < LP_WCHUNK * DS; q += 128) {
      const int pp = q / DS, co = q % DS;
      dy_s[q] = co < cout ? dY[(p0 + pp) * cout + co] : (uint16_t)0;
    }
    for (int q = tid; q < 18 * 34 * PS; q += 128) {
      const int ci = q % PS, c = (q / PS) % 34, r = q / (PS * 34);
      const int y = row0 + r - 1, x = c - 1;
      x_s[q] = (ci < CIN && y >= 0 && y < 32 && x >= 0 && x < 32)
                   ? X[((size_t)img * LP_P + y * 32 + x) * CIN + ci]
                   : (uint16_t)0;
    }
    __syncthreads();
    if (tid < cout)
      for (int pp = 0; pp < LP_WCHUNK; pp++) bsum += __bfloat162float(__ushort_as_bfloat16(dy_s[pp * DS + tid]));
#pragma unroll
    for (int a = 0; a < NPW; a++) {
      const int nt = warp + 4 * a;
      if (nt >= NTOT) break;
      const int n = nt * 8 + g;
      const bool nv = n < 9 * CIN;
      const int tap = nv ? n / CIN : 0, ci = nv ? n % CIN : 0, oy = tap / 3, ox = tap % 3;
      for (int k0 = 0; k0 < LP_WCHUNK; k0 += 16) {
        auto xv = [&](int pp) -> uint32_t {
          return nv ? x_s[(((pp >> 5) + oy) * 34 + (pp & 31) + ox) * PS + ci] : 0u;
        };
        const uint32_t b[2] = {xv(k0 + 2 * t) | (xv(k0 + 2 * t + 1) << 16),
                               xv(k0 + 2 * t + 8) | (xv(k0 + 2 * t + 9) << 16)};
#pragma unroll
        for (int m = 0; m < MT; m++) {
          const int m0 = m * 16 + g, m1 = m0 + 8;
          auto dv = [&](int co, int pp) -> uint32_t { return dy_s[pp * DS + co]; };
          const uint32_t av[4] = {dv(m0, k0 + 2 * t) | (dv(m0, k0 + 2 * t + 1) << 16),
                                  dv(m1, k0 + 2 * t) | (dv(m1, k0 + 2 * t + 1) << 16),
                                  dv(m0, k0 + 2 * t + 8) | (dv(m0, k0 + 2 * t + 9) << 16),
                                  dv(m1, k0 + 2 * t + 8) | (dv(m1, k0 + 2 * t + 9) << 16)};
          mma_bf16(d[a][m], av, b);
        }
      }
    }
  }
#pragma unroll
  for (int a = 0; a < NPW; a++) {
    const int nt = warp + 4 * a;
    if (nt >= NTOT) break;
#pragma unroll
    for (int m = 0; m < MT; m++)
#pragma unroll
      for (int h = 0; h < 2; h++)
#pragma unroll
        for (int e = 0; e < 2; e++) {
          const int co = m * 16 + g + 8 * h, n = nt * 8 + 2 * t + e;
          if (co < cout && n < 9 * CIN) atomicAdd(&dW[(size_t)co * 9 * CIN + n], d[a][m][2 * h + e]);
        }
  }
  if (tid < cout) atomicAdd(&db[tid], bsum);
}

template <int CIN>
vp8a_status conv_bwd_w(vp8a_ctx* ctx, const uint16_t* dY, const uint16_t* X, int cout, int n, float* dW, float* db) {
  const long n_chunks = (long)n * LP_P / LP_WCHUNK;
  const unsigned grid = (unsigned)((n_chunks + LP_WCPB - 1) / LP_WCPB);
  if (grid == 0) return VP8A_OK;
  constexpr int PS = CIN + (CIN >= 16 ? 8 : 0) + (CIN < 16 ? 2 : 0);
  if (cout > 16) {
    const size_t smem = sizeof(uint16_t) * (LP_WCHUNK * (32 + 8) + 18 * 34 * PS);
    VP8A_CUDA(cudaFuncSetAttribute(lp_conv_bwd_w_smem_kernel<CIN, 2>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   (int)smem));
    lp_conv_bwd_w_smem_kernel<CIN, 2><<<grid, 128, smem, ctx->stream>>>(dY, X, cout, n_chunks, dW, db);
  } else {
    const size_t smem = sizeof(uint16_t) * (LP_WCHUNK * (16 + 8) + 18 * 34 * PS);
    VP8A_CUDA(cudaFuncSetAttribute(lp_conv_bwd_w_smem_kernel<CIN, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   (int)smem));
    lp_conv_bwd_w_smem_kernel<CIN, 1><<<grid, 128, smem, ctx->stream>>>(dY, X, cout, n_chunks, dW, db);
  }
  VP8A_CUDA(cudaGetLastError());
  ctx->launches++;
  return VP8A_OK;
}

}  // namespace

extern "C" {

vp8a_status vp8a_lp_windows(vp8a_ctx* ctx, const vp8a_luma_ref* src, const vp8a_luma_ref* ref, const uint32_t* mb_xy,
                            uint32_t n, uint16_t* out) {
  if (!ctx || !src || !ref || (n && (!mb_xy || !out))) {
    vp8a::set_error("null argument");
    return VP8A_E_INVALID_ARGUMENT;
  }
  if (src->width != ref->width || src->height != ref->height || !src->width || !src->height) {
    vp8a::set_error("source and reference planes differ in size");
    return VP8A_E_REFERENCE_DIMENSIONS_MISMATCH;
  }
  if (n == 0) return VP8A_OK;
  if ((uintptr_t)out & 15) {
    vp8a::set_error("out must be 16-byte aligned");
    return VP8A_E_INVALID_ARGUMENT;
  }
  VP8A_CUDA(cudaSetDevice(ctx->device));
  lp_windows_kernel<<<n, 256, 0, ctx->stream>>>(src->plane, src->stride, ref->plane, ref->stride, (int)src->width,
                                                 (int)src->height, mb_xy, (int)n, out);
  VP8A_CUDA(cudaGetLastError());
  ctx->launches++;
  return VP8A_OK;
}

vp8a_status vp8a_lp_seeded_search(vp8a_ctx* ctx, const vp8a_luma_ref* ref, const uint8_t* src_mbs,
                                  const uint32_t* mb_xy, const int32_t* seeds, uint32_t k, uint32_t radius, uint32_t n,
                                  vp8a_search_result* out) {
  if (!ctx || !ref || (n && (!src_mbs || !mb_xy || !seeds || !out))) {
    vp8a::set_error("null argument");
    return VP8A_E_INVALID_ARGUMENT;
  }
  if (k < 1 || k > 4 || radius > 4 || k * (2 * radius + 1) * (2 * radius + 1) > (uint32_t)LP_SEED_MAXC) {
    vp8a::set_error("seeded search: 1 <= k <= 4, radius <= 4 and k * (2 radius + 1)^2 <= 128");
    return VP8A_E_INVALID_ARGUMENT;
  }
  if (!ref->plane || ref->width < 16 || ref->height < 16 || ref->stride < ref->width) {
    vp8a::set_error("bad reference plane");
    return VP8A_E_INVALID_ARGUMENT;
  }
  if (n == 0) return VP8A_OK;
  VP8A_CUDA(cudaSetDevice(ctx->device));
  lp_seeded_search_kernel<<<n, LP_SEED_MAXC, 0, ctx->stream>>>(ref->plane, ref->stride, (int)ref->width,
                                                                (int)ref->height, src_mbs, mb_xy, seeds, (int)k,
                                                                (int)radius, out);
  VP8A_CUDA(cudaGetLastError());
  ctx->launches++;
  return VP8A_OK;
}

vp8a_status vp8a_lp_net_propose(vp8a_ctx* ctx, const uint16_t* x, uint32_t n, const uint16_t* w1, const float* b1,
                                const uint16_t* w2, const float* b2, const uint16_t* w3, const float* b3,
                                const uint16_t* w4, const float* b4, uint32_t k, int32_t* cells, float* logits) {
  if (!ctx || (n && (!x || !w1 || !b1 || !w2 || !b2 || !w3 || !b3 || !w4 || !b4 || !cells))) {
    vp8a::set_error("null argument");
    return VP8A_E_INVALID_ARGUMENT;
  }
  if (k < 1 || k > 16) {
    vp8a::set_error("k must be 1..16");
    return VP8A_E_INVALID_ARGUMENT;
  }
  if ((((uintptr_t)x) & 15) || (((uintptr_t)w1 | (uintptr_t)w2 | (uintptr_t)w3 | (uintptr_t)w4) & 1)) {
    vp8a::set_error("the input must be 16-byte aligned, the weights 2-byte aligned");
    return VP8A_E_INVALID_ARGUMENT;
  }
  if (n == 0) return VP8A_OK;
  VP8A_CUDA(cudaSetDevice(ctx->device));
  VP8A_CUDA(cudaFuncSetAttribute(lp_net_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, lpnet::SMEM));
  const unsigned grid = (unsigned)std::min<uint32_t>(n, (uint32_t)ctx->sm_count);
  lp_net_kernel<<<grid, lpnet::THREADS, lpnet::SMEM, ctx->stream>>>(x, (int)n, w1, b1, w2, b2, w3, b3, w4, b4, (int)k, cells,
                                                          logits, ctx->d_status);
  VP8A_CUDA(cudaGetLastError());
  ctx->launches++;
  return VP8A_OK;
}

vp8a_status vp8a_lp_conv_forward(vp8a_ctx* ctx, const uint16_t* x, uint32_t cin, const uint16_t* w, const float* bias,
                                 uint32_t cout, uint32_t n, uint32_t relu, uint16_t* y, float* y_f32) {
  if (!ctx || !x || !w || !bias || (!y && !y_f32)) {
    vp8a::set_error("null argument");
    return VP8A_E_INVALID_ARGUMENT;
  }
  VP8A_CUDA(cudaSetDevice(ctx->device));
  if (cin == 2 && cout == 32 && y && !y_f32 && n > 0 && aligned16(y)) {
    lp_conv_first_kernel<<<n, 256, 0, ctx->stream>>>(x, w, bias, (int)relu, y);
    VP8A_CUDA(cudaGetLastError());
    ctx->launches++;
    return VP8A_OK;
  }
  if (cin == 2 && cout == 32) return conv_fwd<2, 4>(ctx, x, w, bias, 32, (int)n, relu, y, y_f32);
  if (cin == 32 && cout == 32 && y && !y_f32 && n > 0) {
    // The tensor-core path: 16-byte aligned activations and weights.
    if (((uintptr_t)x | (uintptr_t)w | (uintptr_t)y) & 15) {
      vp8a::set_error("tensor-core conv needs 16-byte aligned buffers");
      return VP8A_E_INVALID_ARGUMENT;
    }
    return conv_tc<false>(ctx, x, w, bias, (int)n, (int)relu, nullptr, y);
  }
  if (cin == 32 && cout == 32) return conv_fwd<32, 4>(ctx, x, w, bias, 32, (int)n, relu, y, y_f32);
  if (cin == 32 && cout == 1 && y_f32 && n > 0 && aligned16(x) && encode_tiled())
    return conv_last(ctx, x, w, bias, (int)n, (int)relu, y_f32);
  if (cin == 32 && cout == 1) return conv_fwd<32, 1>(ctx, x, w, bias, 1, (int)n, relu, y, y_f32);
  vp8a::set_error("conv shape must be 2->32, 32->32 or 32->1");
  return VP8A_E_INVALID_ARGUMENT;
}

vp8a_status vp8a_lp_conv_backward(vp8a_ctx* ctx, const uint16_t* x, uint32_t cin, const uint16_t* w, uint32_t cout,
                                  uint32_t n, const uint16_t* dy, uint32_t x_relu, uint16_t* dx, float* dw,
                                  float* db) {
  if (!ctx || !x || !w || !dy || !dw || !db) {
    vp8a::set_error("null argument");
    return VP8A_E_INVALID_ARGUMENT;
  }
  VP8A_CUDA(cudaSetDevice(ctx->device));
  vp8a_status s;
  const uint16_t* mask = x_relu ? x : nullptr;
  // The persistent kernels read whole 16-byte groups; any other alignment takes
  // the element-wise ones.
  const bool wide = n > 0 && aligned16(x, dy, dx) && encode_tiled();
  if (cin == 2 && cout == 32) {
    s = wide ? conv_bwd_w_edge<2>(ctx, dy, x, (int)n, dw, db) : conv_bwd_w<2>(ctx, dy, x, 32, (int)n, dw, db);
    if (s != VP8A_OK) return s;
    if (dx) return conv_bwd_data<32, 1>(ctx, dy, w, 2, (int)n, mask, dx);
    return VP8A_OK;
  }
  if (cin == 32 && cout == 32) {
    s = wide ? conv_bwd_w_32(ctx, dy, x, (int)n, dw, db) : conv_bwd_w<32>(ctx, dy, x, 32, (int)n, dw, db);
    if (s != VP8A_OK) return s;
    if (dx && wide) return conv_tc<true>(ctx, dy, w, nullptr, (int)n, 0, mask, dx);
    if (dx) return conv_bwd_data<32, 4>(ctx, dy, w, 32, (int)n, mask, dx);
    return VP8A_OK;
  }
  if (cin == 32 && cout == 1) {
    s = wide ? conv_bwd_w_edge<1>(ctx, x, dy, (int)n, dw, db) : conv_bwd_w<32>(ctx, dy, x, 1, (int)n, dw, db);
    if (s != VP8A_OK) return s;
    if (dx && wide) {
      lp_conv_bwd_last_kernel<<<n, 256, 0, ctx->stream>>>(dy, w, mask, dx);
      VP8A_CUDA(cudaGetLastError());
      ctx->launches++;
      return VP8A_OK;
    }
    if (dx) return conv_bwd_data<1, 4>(ctx, dy, w, 32, (int)n, mask, dx);
    return VP8A_OK;
  }
  vp8a::set_error("conv shape must be 2->32, 32->32 or 32->1");
  return VP8A_E_INVALID_ARGUMENT;
}

vp8a_status vp8a_lp_softmax_ce(vp8a_ctx* ctx, const float* logits, const int32_t* labels, uint32_t n,
                               uint16_t* dlogits, float* loss, float* label_prob) {
  if (!ctx || !logits) {
    vp8a::set_error("null argument");
    return VP8A_E_INVALID_ARGUMENT;
  }
  if (n == 0) return VP8A_OK;
  VP8A_CUDA(cudaSetDevice(ctx->device));
  lp_softmax_ce_kernel<<<n, 256, 0, ctx->stream>>>(logits, labels, (int)n, dlogits, loss, label_prob);
  VP8A_CUDA(cudaGetLastError());
  ctx->launches++;
  return VP8A_OK;
}

vp8a_status vp8a_lp_adam(vp8a_ctx* ctx, float* w, const float* grad, float* m, float* v, uint32_t n, float lr,
                         float beta1, float beta2, float eps, uint32_t step, uint16_t* w_bf16) {
  if (!ctx || !w || !grad || !m || !v || !w_bf16 || step == 0) {
    vp8a::set_error("null argument or step 0");
    return VP8A_E_INVALID_ARGUMENT;
  }
  if (n == 0) return VP8A_OK;
  VP8A_CUDA(cudaSetDevice(ctx->device));
  const float c1 = 1.f - powf(beta1, (float)step), c2 = 1.f - powf(beta2, (float)step);
  lp_adam_kernel<<<(n + 255) / 256, 256, 0, ctx->stream>>>(w, grad, m, v, (int)n, lr, beta1, beta2, eps, c1, c2,
                                                            w_bf16);
  VP8A_CUDA(cudaGetLastError());
  ctx->launches++;
  return VP8A_OK;
}

vp8a_status vp8a_lp_pool(vp8a_ctx* ctx, const uint16_t* x, uint32_t c, uint32_t n, float* sums) {
  if (!ctx || !sums || (n && !x) || c == 0 || c > 64 || 256 % c != 0) {
    vp8a::set_error("null argument or channel count not a divisor of 256 up to 64");
    return VP8A_E_INVALID_ARGUMENT;
  }
  if (n == 0) return VP8A_OK;
  VP8A_CUDA(cudaSetDevice(ctx->device));
  lp_pool_kernel<<<n, 256, 0, ctx->stream>>>(x, (int)c, sums);
  VP8A_CUDA(cudaGetLastError());
  ctx->launches++;
  return VP8A_OK;
}

vp8a_status vp8a_lp_lf_head(vp8a_ctx* ctx, const float* sums, float count, uint32_t c, const float* w,
                            const float* b, uint32_t levels, int32_t label, float* logits, float* dw, float* db,
                            float* loss) {
  if (!ctx || !sums || !w || !b || c == 0 || c > 64 || levels == 0 || levels > 128 || !(count > 0.f) ||
      (label >= 0 && (!dw || !db || label >= (int32_t)levels))) {
    vp8a::set_error("bad loop-filter head arguments");
    return VP8A_E_INVALID_ARGUMENT;
  }
  VP8A_CUDA(cudaSetDevice(ctx->device));
  lp_lf_head_kernel<<<1, 128, 0, ctx->stream>>>(sums, count, (int)c, w, b, (int)levels, label, logits, dw, db, loss);
  VP8A_CUDA(cudaGetLastError());
  ctx->launches++;
  return VP8A_OK;
}

}  // extern "C"
