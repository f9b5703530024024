// encode.cu — a whole P frame from host planes (encode_p_frame_multi_ref_auto_
// loop_filter, src/encoder.rs:9373, with intra picking off): the analysis, the
// reconstruction, the loop-filter choice and pass on the device, the bitstream on
// the host.
//
// The stages are the library's own entry points, called on device copies. What
// bounds the frame is their chain, so what is not on it runs beside it: the
// source and the references go up once (chroma, which the analysis does not read,
// on a second stream while it runs), the caller's output pages are touched
// meanwhile, decisions, coefficients and the reconstruction come down on the second
// stream while the device chooses the loop-filter level, and a thread codes the
// token partitions, which do not depend on that level. Measured through
// encode_p_frame (QI 56, three references, the same planes again and again): stage
// by stage through host buffers 2.5 ms at 640x360, 1.43 ms so; 1920x1080 12.8 and
// 5.9-6.6 ms, 3840x2160 40 and 21.6 ms. (On a faster host 9.6 and 4.7, 25.7 and 14.0;
// the first frames from planes never seen before take 0.2 ms longer at 640x360.)
#include <algorithm>
#include <cstring>
#include <exception>
#include <memory>
#include <system_error>
#include <thread>
#include <vector>

#include "emit.h"
#include "vp8a_internal.cuh"

namespace {

// A plane bundle in one device allocation.
struct DevPlanes {
  uint8_t* y = nullptr;
  size_t ys = 0, yh = 0, cs = 0, ch = 0;
  size_t bytes() const { return ys * yh + 2 * cs * ch; }
  uint8_t* u() const { return y + ys * yh; }
  uint8_t* v() const { return u() + cs * ch; }
};

// The second stream's work is over, and the token thread's, before anything that
// they use goes away.
struct Beside {
  cudaStream_t stream;
  std::thread tokens;
  void join() {
    if (tokens.joinable()) tokens.join();
  }
  ~Beside() {
    join();
    cudaStreamSynchronize(stream);
  }
};

vp8a_status second_stream(vp8a_ctx* ctx) {
  if (!ctx->aux) VP8A_CUDA(cudaStreamCreateWithFlags(&ctx->aux, cudaStreamNonBlocking));
  if (!ctx->aux_ev) VP8A_CUDA(cudaEventCreateWithFlags(&ctx->aux_ev, cudaEventDisableTiming));
  return VP8A_OK;
}

// `to` waits for what is on `from` now.
vp8a_status follow(vp8a_ctx* ctx, cudaStream_t from, cudaStream_t to) {
  VP8A_CUDA(cudaEventRecord(ctx->aux_ev, from));
  VP8A_CUDA(cudaStreamWaitEvent(to, ctx->aux_ev, 0));
  return VP8A_OK;
}

vp8a_status rows_up(uint8_t* d, size_t pitch, const uint8_t* h, size_t stride, size_t w, size_t rows, cudaStream_t s) {
  if (stride == pitch)
    VP8A_CUDA(cudaMemcpyAsync(d, h, stride * (rows - 1) + w, cudaMemcpyHostToDevice, s));
  else
    VP8A_CUDA(cudaMemcpy2DAsync(d, pitch, h, stride, w, rows, cudaMemcpyHostToDevice, s));
  return VP8A_OK;
}
void rows_out(uint8_t* to, size_t stride, const uint8_t* from, size_t w, size_t rows) {
  if (stride == w)
    std::memcpy(to, from, w * rows);
  else
    for (size_t r = 0; r < rows; r++) std::memcpy(to + r * stride, from + r * w, w);
}
// A bundle's planes, one after another at `from`, into the caller's.
void planes_out(const vp8a_planes* to, const DevPlanes& p, const uint8_t* from) {
  rows_out(to->y, to->y_stride, from, p.ys, p.yh);
  rows_out(to->u, to->uv_stride, from + p.ys * p.yh, p.cs, p.ch);
  rows_out(to->v, to->uv_stride, from + p.ys * p.yh + p.cs * p.ch, p.cs, p.ch);
}

// `bytes` of host memory for results: the context's pinned block, whose copies run
// at the link's rate without the driver's own staging, or, for more than it may
// hold, `own`.
uint8_t* result_memory(vp8a_ctx* ctx, size_t bytes, std::unique_ptr<uint8_t[]>& own) {
  if (bytes > ctx->down_bytes && bytes <= vp8a_ctx::DOWN_MAX) {
    if (ctx->down_host) cudaFreeHost(ctx->down_host);
    ctx->down_host = nullptr;
    ctx->down_bytes = 0;
    if (cudaHostAlloc((void**)&ctx->down_host, bytes, cudaHostAllocDefault) == cudaSuccess)
      ctx->down_bytes = bytes;
    else
      cudaGetLastError();
  }
  if (bytes <= ctx->down_bytes) return ctx->down_host;
  own.reset(new uint8_t[bytes]);
  return own.get();
}

// The first touch of fresh memory is the kernel's work, done while the device is
// busy: a write a page, of what is there (an output that the call leaves alone, at a
// chosen level of 0 or on an error return, keeps its bytes).
void touch(void* p, size_t bytes) {
  uint8_t* b = static_cast<uint8_t*>(p);
  for (size_t i = 0; i < bytes; i += 4096) __atomic_fetch_or(b + i, 0, __ATOMIC_RELAXED);
}
// A plane's rows; what lies between them is not the call's.
void touch_rows(uint8_t* p, size_t stride, size_t w, size_t rows) {
  for (size_t at = 0; at < stride * rows;) {
    touch(p + at, 1);
    // A page on, or the next row where that byte lies between rows.
    const size_t next = at + 4096, y = next / stride;
    at = next - y * stride < w ? next : (y + 1) * stride;
  }
}

#define TRY(call)                          \
  do {                                     \
    const vp8a_status _s = (call);         \
    if (_s != VP8A_OK) return _s;          \
  } while (0)

vp8a_status encode(vp8a_ctx* ctx, const vp8a_i420* frame, const vp8a_planes* refs, const uint8_t* ref_ids,
                   uint32_t n_refs, const vp8a_mv_contexts* mv_contexts, double lambda, const vp8a_mv* proposals,
                   const vp8a_frame_header* header, uint32_t auto_lf, vp8a_mb_decision* decisions, int16_t* coeffs,
                   uint8_t* mb_flags, vp8a_mb_lf_info* lf_info, const vp8a_planes* recon, const vp8a_planes* filtered,
                   uint8_t* level_out, uint8_t* sharpness_out, uint8_t* out, uint64_t out_capacity,
                   uint64_t* out_size) {
  vp8a_frame_header h = *header;
  const size_t cols = (h.width + 15) / 16, rows = (h.height + 15) / 16, n = cols * rows;
  TRY(second_stream(ctx));
  vp8a::Stager st(ctx);
  const size_t cw = (h.width + 1) / 2, ch = (h.height + 1) / 2;
  auto device = [&](size_t bytes, uint8_t** d) {
    void* p;
    const vp8a_status s = st.scratch(bytes, &p);
    *d = static_cast<uint8_t*>(p);
    return s;
  };
  DevPlanes src, ref[3], rec, fil;
  src.ys = (h.width + 15) / 16 * 16;
  src.cs = src.ys / 2;
  src.yh = h.height;
  src.ch = ch;
  auto padded = [&](DevPlanes& p) {
    p.ys = cols * 16;
    p.yh = rows * 16;
    p.cs = cols * 8;
    p.ch = rows * 8;
    return device(p.bytes(), &p.y);
  };
  uint8_t *d_dec, *d_cf, *d_fl, *d_lf, *d_lv;
  TRY(device(src.bytes(), &src.y));
  for (uint32_t k = 0; k < n_refs; k++) TRY(padded(ref[k]));
  TRY(padded(rec));
  TRY(padded(fil));
  // The records lie behind one another, on the device and on the host.
  auto after = [](size_t at, size_t bytes) { return (at + bytes + 255) / 256 * 256; };
  const size_t o_cf = after(0, sizeof(vp8a_mb_decision) * n), o_lf = after(o_cf, sizeof(int16_t) * 400 * n);
  const size_t o_fl = after(o_lf, sizeof(vp8a_mb_lf_info) * n), records = after(o_fl, n);
  TRY(device(records, &d_dec));
  d_cf = d_dec + o_cf;
  d_lf = d_dec + o_lf;
  d_fl = d_dec + o_fl;
  TRY(device(2, &d_lv));
  std::unique_ptr<uint8_t[]> own;
  uint8_t* down = result_memory(ctx, records + 2 * rec.bytes(), own);
  const vp8a_mb_decision* h_dec = reinterpret_cast<const vp8a_mb_decision*>(down);
  const int16_t* h_cf = reinterpret_cast<const int16_t*>(down + o_cf);
  vp8a_emit::FrameTokens t;
  vp8a_status coded = VP8A_OK;
  std::exception_ptr failed;
  // Declared after what the second stream and the token thread use.
  Beside beside{ctx->aux, {}};
  TRY(follow(ctx, ctx->stream, ctx->aux));  // the allocations are in place

  // The analysis reads luma.
  TRY(rows_up(src.y, src.ys, frame->y, frame->y_stride, h.width, h.height, ctx->stream));
  for (uint32_t k = 0; k < n_refs; k++)
    TRY(rows_up(ref[k].y, ref[k].ys, refs[k].y, refs[k].y_stride, cols * 16, rows * 16, ctx->stream));
  vp8a_i420 f = *frame;
  f.y = src.y;
  f.u = src.u();
  f.v = src.v();
  f.y_stride = src.ys;
  f.uv_stride = src.cs;
  auto bundle = [&](const DevPlanes& p) {
    vp8a_planes b{};
    b.y = p.y;
    b.u = p.u();
    b.v = p.v();
    b.y_stride = p.ys;
    b.uv_stride = p.cs;
    b.mb_rows = (uint32_t)rows;
    b.mb_cols = (uint32_t)cols;
    return b;
  };
  vp8a_planes rp[3];
  for (uint32_t k = 0; k < n_refs; k++) rp[k] = bundle(ref[k]);
  vp8a_mb_decision* dec = reinterpret_cast<vp8a_mb_decision*>(d_dec);
  TRY(proposals ? vp8a_analyse_inter_frame_proposals(ctx, &f, rp, ref_ids, n_refs, mv_contexts, lambda, proposals, dec,
                                                     nullptr)
                : vp8a_analyse_inter_frame(ctx, &f, rp, ref_ids, n_refs, mv_contexts, lambda, dec, nullptr));
  TRY(rows_up(src.u(), src.cs, frame->u, frame->uv_stride, cw, ch, ctx->aux));
  TRY(rows_up(src.v(), src.cs, frame->v, frame->uv_stride, cw, ch, ctx->aux));
  for (uint32_t k = 0; k < n_refs; k++) {
    TRY(rows_up(ref[k].u(), ref[k].cs, refs[k].u, refs[k].uv_stride, cols * 8, rows * 8, ctx->aux));
    TRY(rows_up(ref[k].v(), ref[k].cs, refs[k].v, refs[k].uv_stride, cols * 8, rows * 8, ctx->aux));
  }
  touch(decisions, sizeof(vp8a_mb_decision) * n);
  touch(coeffs, sizeof(int16_t) * 400 * n);
  for (const vp8a_planes* p : {recon, filtered}) {
    touch_rows(p->y, p->y_stride, cols * 16, rows * 16);
    touch_rows(p->u, p->uv_stride, cols * 8, rows * 8);
    touch_rows(p->v, p->uv_stride, cols * 8, rows * 8);
  }
  touch(out, std::min<uint64_t>(out_capacity, 600 * n));  // more than any but the finest quantisers take
  TRY(follow(ctx, ctx->aux, ctx->stream));
  TRY(vp8a::check_device_status(ctx));  // the decisions are whole, or the call ends here

  vp8a_planes recp = bundle(rec);
  vp8a_mb_lf_info* lf = reinterpret_cast<vp8a_mb_lf_info*>(d_lf);
  TRY(vp8a_reconstruct_inter_frame(ctx, &f, rp, ref_ids, n_refs, dec, &h.quant, nullptr, nullptr, 0, 0,
                                   VP8A_FILTER_SIXTAP, &recp, reinterpret_cast<int16_t*>(d_cf), d_fl, lf));
  TRY(follow(ctx, ctx->stream, ctx->aux));
  // The results so far down and the tokens coded, beside the device's choice of
  // the level (which waits for it).
  auto code = [&] {
    auto run = [&]() -> vp8a_status {
      VP8A_CUDA(cudaSetDevice(ctx->device));
      VP8A_CUDA(cudaStreamSynchronize(ctx->aux));
      TRY(vp8a_emit::scan_frame(header, h_dec, h_cf, nullptr, t));
      vp8a_emit::code_tokens(header, h_dec, h_cf, nullptr, t);
      return VP8A_OK;
    };
    try {
      coded = run();
    } catch (...) {
      failed = std::current_exception();
    }
  };
  VP8A_CUDA(cudaMemcpyAsync(down, d_dec, records, cudaMemcpyDeviceToHost, ctx->aux));
  VP8A_CUDA(cudaMemcpyAsync(down + records, rec.y, rec.bytes(), cudaMemcpyDeviceToHost, ctx->aux));
  try {
    beside.tokens = std::thread(code);
  } catch (const std::system_error&) {
    code();  // no thread to be had
  }
  vp8a_filter_config cfg{};
  cfg.loop_filter_level = h.loop_filter_level;
  cfg.sharpness_level = h.sharpness_level;
  cfg.simple = h.filter_type;
  // The header's deltas, as a decoder of the frame adds them.
  cfg.delta_enabled = h.lf_delta_enabled;
  cfg.ref_delta_current = h.lf_ref_delta[0];
  cfg.ref_delta_last = h.lf_ref_delta[1];
  cfg.ref_delta_golden = h.lf_ref_delta[2];
  cfg.ref_delta_altref = h.lf_ref_delta[3];
  cfg.bpred_mode_delta = h.lf_mode_delta[0];
  cfg.zero_mv_mode_delta = h.lf_mode_delta[1];
  cfg.other_mv_mode_delta = h.lf_mode_delta[2];
  cfg.split_mv_mode_delta = h.lf_mode_delta[3];
  if (auto_lf) {
    vp8a_filter_config base = cfg;
    base.loop_filter_level = 0;
    vp8a_source s{};
    s.y = f.y;
    s.u = f.u;
    s.v = f.v;
    s.y_stride = f.y_stride;
    s.uv_stride = f.uv_stride;
    s.width = f.width;
    s.height = f.height;
    TRY(vp8a_select_filter_params(ctx, &recp, lf, &base, &s, d_lv, d_lv + 1));
    uint8_t lv[2];
    VP8A_CUDA(cudaMemcpyAsync(lv, d_lv, 2, cudaMemcpyDeviceToHost, ctx->stream));
    TRY(vp8a::check_device_status(ctx));
    h.loop_filter_level = cfg.loop_filter_level = lv[0];
    h.sharpness_level = cfg.sharpness_level = lv[1];
  }
  if (cfg.loop_filter_level) {
    VP8A_CUDA(cudaMemcpyAsync(fil.y, rec.y, rec.bytes(), cudaMemcpyDeviceToDevice, ctx->stream));
    vp8a_planes fp = bundle(fil);
    TRY(vp8a_filter_frame(ctx, &fp, lf, &cfg));
  }
  uint8_t* h_fil = down + records + rec.bytes();
  if (cfg.loop_filter_level)
    VP8A_CUDA(cudaMemcpyAsync(h_fil, fil.y, fil.bytes(), cudaMemcpyDeviceToHost, ctx->stream));
  // The caller's copies, while the filter runs and the tokens are coded.
  VP8A_CUDA(cudaStreamSynchronize(ctx->aux));
  planes_out(recon, rec, down + records);
  std::memcpy(decisions, h_dec, sizeof(vp8a_mb_decision) * n);
  std::memcpy(coeffs, h_cf, sizeof(int16_t) * 400 * n);
  std::memcpy(lf_info, down + o_lf, sizeof(vp8a_mb_lf_info) * n);
  std::memcpy(mb_flags, down + o_fl, n);
  TRY(vp8a::check_device_status(ctx));
  if (cfg.loop_filter_level) planes_out(filtered, fil, h_fil);
  beside.join();
  if (failed) std::rethrow_exception(failed);
  TRY(coded);
  std::vector<uint8_t> first;
  TRY(vp8a_emit::first_partition(&h, h_dec, nullptr, t, first));
  *level_out = h.loop_filter_level;
  *sharpness_out = h.sharpness_level;
  return vp8a_emit::assemble(first, t, out, out_capacity, out_size);
}

}  // namespace

extern "C" vp8a_status vp8a_encode_inter_frame(
    vp8a_ctx* ctx, const vp8a_i420* frame, const vp8a_planes* refs, const uint8_t* ref_ids, uint32_t n_refs,
    const vp8a_mv_contexts* mv_contexts, double lambda, const vp8a_mv* proposals, const vp8a_frame_header* header,
    uint32_t auto_lf, vp8a_mb_decision* decisions, int16_t* coeffs, uint8_t* mb_flags, vp8a_mb_lf_info* lf_info,
    const vp8a_planes* recon, const vp8a_planes* filtered, uint8_t* level_out, uint8_t* sharpness_out, uint8_t* out,
    uint64_t out_capacity, uint64_t* out_size) {
  if (!ctx || !frame || !refs || !ref_ids || !header || !decisions || !coeffs || !mb_flags || !lf_info || !recon ||
      !filtered || !level_out || !sharpness_out || !out || !out_size) {
    vp8a::set_error("null argument");
    return VP8A_E_INVALID_ARGUMENT;
  }
  *out_size = 0;
  if (n_refs == 0 || n_refs > 3 || header->segmentation) {
    vp8a::set_error("n_refs must be 1..3, segmentation off");
    return VP8A_E_INVALID_ARGUMENT;
  }
  const vp8a_status s = vp8a_emit::check_header(header, nullptr);
  if (s != VP8A_OK) {
    vp8a::set_error("bad frame header");
    return s;
  }
  if (frame->width != header->width || frame->height != header->height) {
    vp8a::set_error("the frame is not the header's size");
    return VP8A_E_INVALID_DIMENSIONS;
  }
  const uint32_t cols = (header->width + 15) / 16, rows = (header->height + 15) / 16;
  auto fits = [&](const vp8a_planes& p) {
    return p.y && p.u && p.v && p.mb_cols == cols && p.mb_rows == rows && p.y_stride >= cols * 16 &&
           p.uv_stride >= cols * 8;
  };
  bool ok = fits(*recon) && fits(*filtered);
  for (uint32_t k = 0; k < n_refs; k++) ok = ok && fits(refs[k]);
  if (!ok) {
    vp8a::set_error("reference or output planes do not match the frame's MB grid");
    return VP8A_E_REFERENCE_DIMENSIONS_MISMATCH;
  }
  if (!frame->y || !frame->u || !frame->v || frame->y_stride < frame->width ||
      frame->uv_stride < (frame->width + 1) / 2) {
    vp8a::set_error("bad source plane");
    return VP8A_E_INVALID_ARGUMENT;
  }
  VP8A_CUDA(cudaSetDevice(ctx->device));
  try {
    return encode(ctx, frame, refs, ref_ids, n_refs, mv_contexts, lambda, proposals, header, auto_lf, decisions, coeffs,
                  mb_flags, lf_info, recon, filtered, level_out, sharpness_out, out, out_capacity, out_size);
  } catch (const std::exception& e) {
    vp8a::set_error(e.what());
    return VP8A_E_OUT_OF_MEMORY;
  }
}
