// Waiting on the host for results that arrive one by one in pinned memory (plain C++, no CUDA).
#pragma once
#include <stdint.h>
#include <string.h>

namespace rstq {

// A NaN that no arithmetic on the device produces: what a word holds before its result has arrived.
constexpr uint32_t kNotYet = 0x7FE5A5A5u;

// Copies the n words of res to y as they arrive.  Every so often (some 50 us) `query` says whether the work that writes
// them is over: 0 = it is, > 0 = it is not, < 0 = it failed; the wait ends with it, and the words are taken as
// they are.  Returns query's failure, else 0; *missing: whether a word still held kNotYet then.
template <typename Query>
inline int32_t await_results(const uint32_t* res, int64_t n, void* y, Query query, bool* missing) {
    *missing = false;
    int64_t i = 0;
    for (uint32_t spins = 1;; ++spins) {
        while (i < n) {   // 32 results at a time
            asm volatile("" ::: "memory");
            uint32_t r[32];
            const int m = n - i < 32 ? (int)(n - i) : 32;
            if (m == 32) memcpy(r, res + i, 128);
            else
                for (int j = 0; j < 32; ++j) r[j] = j < m ? res[i + j] : 0u;
            uint32_t waiting = 0;
            for (int j = 0; j < 32; ++j) waiting |= r[j] == kNotYet ? 1u : 0u;
            if (waiting) break;
            memcpy((uint32_t*)y + i, r, (size_t)m * 4);
            i += m;
        }
        if (i == n) return 0;
        if ((spins & 0x3FFF) == 0) {
            const int32_t q = query();
            if (q > 0) continue;
            if (q < 0) return q;
            asm volatile("" ::: "memory");
            memcpy(y, res, (size_t)n * 4);
            for (int64_t j = i; j < n; ++j) *missing |= ((const uint32_t*)y)[j] == kNotYet;
            return 0;
        }
    }
}

}  // namespace rstq
