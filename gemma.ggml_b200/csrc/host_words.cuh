// host_words.cuh — results that a kernel leaves in page-locked host memory: each a word of eight bytes, the number of the call above the result, for which the host
// looks.  Plain C++.
#pragma once

#include <stdint.h>
#include <string.h>

struct host_words {
    uint64_t *words = nullptr; // [n], zero when they are new
    int64_t n = 0;
    uint32_t call = 0;

    // The number of the next call, never zero.  A word that only large calls use keeps its number while 2^32 small ones go by: when the numbers begin again, the words
    // are cleared, once `drained` says that no kernel of an earlier call can still store (false: not this time)
    template <typename F> bool next(F drained) {
        if (call != UINT32_MAX) {
            call++;
            return true;
        }
        if (!drained()) return false;
        memset(words, 0, (size_t)n * 8);
        call = 1;
        return true;
    }

    // `count` results of this call from word `first` on, each as soon as it is there.  `state`: 1 while the kernel may be under way, 0 when it is done, -1 when it has
    // failed.  false: a result will never be there
    template <typename F> bool take(float *dst, int64_t first, int64_t count, F state) const {
        for (int64_t i = 0; i < count; i++) {
            uint64_t w;
            for (int turns = 0; (w = at(first + i)) >> 32 != call;) {
                if (++turns < 2000) continue;
                turns = 0;
                const int s = state();
                if (s < 0 || (s == 0 && at(first + i) >> 32 != call)) return false;
            }
            const uint32_t v = (uint32_t)w;
            memcpy(dst + i, &v, 4);
        }
        return true;
    }

private:
    uint64_t at(int64_t i) const { return __atomic_load_n(words + i, __ATOMIC_ACQUIRE); }
};
