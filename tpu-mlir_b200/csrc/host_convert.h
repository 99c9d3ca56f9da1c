// The interpreter keeps every tensor as float: its integers in float buffers <-> their storage types, on host memory.
#pragma once
#include <stddef.h>
#include <stdint.h>

namespace b200q {

// y[i] = (uint8_t)(int)x[i]: integral by contract, so the low byte is the int8 or uint8 value (what does not fit an int32 is
// taken to its nearest end and NaN to 0, as the device's conversion does)
void host_f32_to_bytes(const float* x, uint8_t* y, size_t n);
// y[i] = (float)x[i] for the storage type `dt` (b200q_dtype); past_cache: y is large and not read soon
void host_q_to_f32(const void* x, int dt, float* y, size_t n, bool past_cache);
// a short rest in a polling loop
void host_pause();

}  // namespace b200q
