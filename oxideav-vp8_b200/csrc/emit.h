// emit.h — the bitstream writer's parts, for callers that have a frame's
// coefficients before its loop-filter level is known.
#pragma once
#include <cstdint>
#include <vector>

#include "../../include/vp8a.h"

namespace vp8a_emit {

// What the writer derives from a frame's decisions and coefficients, and the
// coded token partitions.
struct FrameTokens {
  std::vector<uint8_t> skip, seg;   // per MB: nothing coded; wire segment
  std::vector<uint32_t> nzmask;     // per MB: bit b = coding-order block b has a coded nonzero
  uint32_t n_skip = 0, n_ref[4] = {0, 0, 0, 0}, seg_count[4] = {0, 0, 0, 0};
  std::vector<std::vector<uint8_t>> parts;
};

// The header's range checks; the levels among them.
vp8a_status check_header(const vp8a_frame_header* h, const int8_t* mb_segment);
// The per-MB flags (VP8A_E_* for decisions or coefficients that cannot be coded).
vp8a_status scan_frame(const vp8a_frame_header* h, const vp8a_mb_decision* decisions, const int16_t* coeffs,
                       const int8_t* mb_segment, FrameTokens& t);
// The token partitions: nothing of the header but the size and the count.
void code_tokens(const vp8a_frame_header* h, const vp8a_mb_decision* decisions, const int16_t* coeffs,
                 const uint8_t* token_prob_updates, FrameTokens& t);
// The first partition (header and modes) from scan_frame's counts.
vp8a_status first_partition(const vp8a_frame_header* h, const vp8a_mb_decision* decisions,
                            const uint8_t* token_prob_updates, const FrameTokens& t, std::vector<uint8_t>& first);
// The frame: tag, first partition, size table, token partitions.
vp8a_status assemble(const std::vector<uint8_t>& first, const FrameTokens& t, uint8_t* out, uint64_t out_capacity,
                     uint64_t* out_size);

}  // namespace vp8a_emit
