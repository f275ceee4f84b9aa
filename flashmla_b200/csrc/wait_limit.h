// Limits of the kernels' barrier waits, in the unit the waiting threads count in: 2^8 SM cycles, so that 32 bits hold
// limits of up to 1.1e12 cycles (about nine minutes; longer ones count as that).  Plain C++, no CUDA.
#pragma once
#include <stdint.h>
#include <stdlib.h>

namespace mla {

constexpr int WAIT_UNIT_LOG2 = 8;
constexpr long long WAIT_LIMIT_DEFAULT = 2000000000LL;    // SM cycles (about one second)

constexpr uint32_t wait_units(long long cycles) {
    const long long units = ((cycles - 1) >> WAIT_UNIT_LOG2) + 1;
    return units < 0xffffffffLL ? (uint32_t)units : 0xffffffffu;
}

// MLA_WAIT_LIMIT_CYCLES as the environment gives it (null: not set); the default unless it is a positive number.
inline uint32_t wait_units_from(const char* cycles) {
    const long long x = cycles ? atoll(cycles) : 0;
    return wait_units(x > 0 ? x : WAIT_LIMIT_DEFAULT);
}

}  // namespace mla
