// launch_shape (launch_shape.hpp) for the CPU tests. TEST INFRASTRUCTURE ONLY.
#include "launch_shape.hpp"

extern "C" void launch_shape_of(uint64_t slots, uint64_t frame_slots, uint32_t sms, uint32_t blocks, uint32_t resident,
                                uint32_t spread, uint32_t *out) {
  const fdk::LaunchShape s = fdk::launch_shape(slots, frame_slots, sms, blocks, resident, spread);
  out[0] = s.idle_lanes;
  out[1] = s.tail;
}
extern "C" uint32_t spread_warps(int ext_plain) { return ext_plain ? fdk::SPREAD_WARPS_EXT_PLAIN : fdk::SPREAD_WARPS; }
