// How a frame launch hands its samples out to the lanes of its warps.
#pragma once
#include <algorithm>
#include <cstdint>

namespace fdk {

struct LaunchShape {
  uint32_t idle_lanes;  // lanes of each warp that take no sample
  uint32_t tail;        // queue slots left from which a warp takes only what its idle lanes need
};

// Warps an SM that a launch of few samples is spread over, instead of filling the first warps: a
// warp of 32 lanes that diverge runs every lane's branches and waits for every lane's table
// loads. Kernel ms at full warps / 2 4 8 12 16 warps an SM: 64x36 shallow 0.42 / 0.38 0.37 0.35
// 0.35 0.35, 64x36 at 1e-100 with blocks 1.08 / 0.90 0.93 0.92 0.91 0.85. The extended tier
// without a table: a deep view's samples step together, and more warps only run the same
// instructions more often (59x88 at 2e-331 1.82 / 1.82 2.37 2.95 2.95 2.95, 77x21 at 6e-778
// 6.87 / 6.85 7.45 8.52 8.52 8.56; a shallow 161x91 0.54 / 0.51 0.50 0.46 0.49 0.50; 48x27 at 1e-60
// 0.79 0.66 0.99 at 2 4 12).
constexpr uint32_t SPREAD_WARPS = 12, SPREAD_WARPS_EXT_PLAIN = 4;

// slots: the launch's queue slots. frame_slots: those of the frame whose launch it stands for
// (FDC_BAND; its own otherwise). blocks: 128-thread blocks an SM that are launched, so that no
// lane idles for warps that are not there; resident: those the kernel is compiled for. Over the
// last three waves of the grid a warp reserves no slots ahead (401x227 without a table 1.15 ->
// 0.86 ms, 480x270 2.72 -> 2.49), or over an eighth of the queue where that is more; a band's
// tail is the same part of its own slots.
inline LaunchShape launch_shape(uint64_t slots, uint64_t frame_slots, uint32_t sms, uint32_t blocks, uint32_t resident,
                                uint32_t spread) {
  const uint64_t warps = (uint64_t)sms * std::max(1u, std::min(spread, 4 * blocks));
  const uint64_t lanes = (frame_slots + warps - 1) / warps;
  const uint64_t tail = std::max<uint64_t>(frame_slots / 8, 3ull * sms * std::min(blocks, resident) * 128);
  LaunchShape s;
  s.idle_lanes = lanes < 32 ? (uint32_t)(32 - std::max<uint64_t>(lanes, 1)) : 0;
  uint64_t own = tail;
  if (slots != frame_slots) own = tail >= frame_slots ? slots : (uint64_t)((double)slots * ((double)tail / (double)frame_slots));
  s.tail = (uint32_t)std::min<uint64_t>(own, 0xffffffffu);
  return s;
}

}  // namespace fdk
