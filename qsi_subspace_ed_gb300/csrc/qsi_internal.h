// Internal helpers shared by the host (.cpp) and device (.cu) translation units.
#pragma once
#include <cstdint>
#include <cstdio>
#include <cstdarg>
#include <string>
#include "../../include/qsi_ed.h"

namespace qsi {

// Sets the calling thread's last-error text and returns the status unchanged.
qsi_status fail(qsi_status st, const char* fmt, ...);

using u128 = unsigned __int128;

inline u128 make_u128(uint64_t lo, uint64_t hi) { return ((u128)hi << 64) | lo; }
inline uint64_t lo64(u128 v) { return (uint64_t)v; }
inline uint64_t hi64(u128 v) { return (uint64_t)(v >> 64); }
inline int popc128(u128 v) { return __builtin_popcountll(lo64(v)) + __builtin_popcountll(hi64(v)); }

// For a call that ran out of device memory: asks the solves under way for the lookup caches they built for themselves and
// waits until those are free.  Whether there were any.
bool reclaim_solve_caches();

// Exceptions never leave an extern "C" function: this wrapper turns them into statuses.  A call that ran out of device
// memory has changed nothing yet that counts, and runs again once the caches of other threads' solves are gone.
template <class F>
qsi_status guarded(F&& f) {
    try {
        qsi_status s = f();
        for (int again = 0; again < 3 && s == QSI_OOM && reclaim_solve_caches(); ++again) s = f();
        return s;
    } catch (const std::bad_alloc&) {
        return fail(QSI_OOM, "host allocation failed");
    } catch (const std::exception& e) {
        return fail(QSI_INVALID_ARG, "%s", e.what());
    } catch (...) {
        return fail(QSI_INVALID_ARG, "unknown exception");
    }
}

}  // namespace qsi
