// pv_barrier.cuh — the word of the cooperative steps' grid barrier (pv_stepping.cu), apart from the waiting.
//
// One 64-bit word, zero before the launch:
//   bits 0-10, 11-21   CTAs that arrived with an error, by the barrier's parity
//   bits 22, 23        the barrier was broken by a wait that gave up, by its parity
//   bits 24-63         arrivals since the launch, whose carry leaves at the top
// Barrier r is open once the arrivals reach r times the grid. Both sides of that comparison may pass 2^40
// (148 CTAs, four barriers an RK4 step: after 1.9e9 steps of one launch), so it is made on their difference
// modulo 2^64, which is right while they are less than 2^39 arrivals apart: two barriers at most are. The
// functions are __host__ __device__ so that the same source can be checked on the CPU.
#pragma once

#include <stdint.h>

#if defined(__CUDACC__)
#define PVB_HD __host__ __device__ __forceinline__
#else
#define PVB_HD inline
#endif

namespace pvb {
namespace barrier {

constexpr unsigned kMaxCtas = 2047;  // an error field's largest count
constexpr int kArrivalShift = 24;

PVB_HD int error_shift(unsigned parity) { return parity ? 11 : 0; }

// What a CTA adds when it arrives.
PVB_HD unsigned long long arrival(bool error, unsigned parity) {
    return (1ull << kArrivalShift) + (error ? 1ull << error_shift(parity) : 0ull);
}
// Arrivals of `ctas` CTAs: what the point of opening moves by from one barrier to the next.
PVB_HD unsigned long long arrivals(unsigned ctas) {
    return static_cast<unsigned long long>(ctas) << kArrivalShift;
}
PVB_HD bool open(unsigned long long word, unsigned long long open_at) {
    return static_cast<long long>(word - open_at) >= 0;
}
PVB_HD bool errors(unsigned long long word, unsigned parity) {
    return ((word >> error_shift(parity)) & kMaxCtas) != 0;
}
PVB_HD unsigned long long broken(unsigned parity) { return 1ull << (parity ? 23 : 22); }

} // namespace barrier
} // namespace pvb
