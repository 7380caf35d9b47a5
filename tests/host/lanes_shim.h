// device_shim.h with the lanes of a group one after the other: in a first pass a shuffle notes its argument,
// in a second it returns what the other lane noted at the same call; reductions are noted, not carried out.
#pragma once
#define __shfl_xor_sync shim_shfl_one_lane
#define atomicAdd shim_add_at
#include "device_shim.h"
#undef __shfl_xor_sync
#undef atomicAdd
#include <utility>
#include <vector>
struct Lanes {
    bool record = false;
    int lane = 0;
    size_t next = 0;
    std::vector<std::vector<uint32_t>> args;
    std::vector<std::pair<float *, float>> adds;
    std::vector<std::pair<int64_t, uint32_t>> all;
} static lanes;
template <typename T> inline T __shfl_xor_sync(unsigned, T v, int mask, int) {
    static_assert(sizeof(T) == 4, "32-bit shuffles");
    uint32_t b;
    std::memcpy(&b, &v, 4);
    if (lanes.record) lanes.args[lanes.lane].push_back(b);
    else b = lanes.args[lanes.lane ^ mask].at(lanes.next++);
    std::memcpy(&v, &b, 4);
    return v;
}
inline void atomicAdd(float *p, float v) { lanes.adds.push_back({p, v}); }
