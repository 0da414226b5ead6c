// wait_value.cuh -- values that are their own signal, passed between the
// CTAs of one cooperative launch.
#pragma once
#include "ecg_internal.h"

namespace ecg {

// The value that stands for "not computed yet" in the vectors the cooperative
// solves pass between CTAs: a quiet NaN with a payload no arithmetic makes
// (hardware NaNs are 0x7fff...).
constexpr unsigned long long UNSET = 0xfff8c0de5eedfaceULL;
__device__ __forceinline__ cd unset() { return cd{__longlong_as_double(UNSET), __longlong_as_double(UNSET)}; }

__device__ __forceinline__ void look_value(const cd* p, unsigned long long& a, unsigned long long& b)
{
    asm volatile("ld.relaxed.gpu.global.v2.b64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "l"(p) : "memory");
}

// The computed value at *p; ok turns false when this thread gives up: after
// `limit` polls (abort_word[1]: SOLVE_SPIN_LIMIT unless a caller set another
// through ecg_set_wait_limit), or when the abort word is set, which is looked
// at every 64th poll (its load would otherwise stand between the polls).
__device__ __forceinline__ double2 wait_value(const cd* p, int* status, int* abort_word, int limit, bool& ok)
{
    unsigned long long a, b;
    int spins = 0;
    for (;;) {
        look_value(p, a, b);
        if ((a != UNSET && b != UNSET) || !ok) break;
        ++spins;
        if (spins > limit || ((spins & 63) == 0 && *((volatile int*)abort_word) != 0)) {
            atomicExch(status + ST_SOLVE_TIMEOUT, 1);
            atomicExch(abort_word, 1);
            ok = false;
        }
    }
    return make_double2(__longlong_as_double((long long)a), __longlong_as_double((long long)b));
}

}  // namespace ecg
