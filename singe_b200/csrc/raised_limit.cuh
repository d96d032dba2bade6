// A limit that calls raise to what they need and none lowers.  Host code only.
#pragma once

#include <mutex>

namespace singe {

// Raises a limit that is known to stand at `done` or above; `set(needed)` sets it and returns 0 on success.  Threads that ask
// for different amounts at once end with the largest.
template <typename Set>
inline int raise_limit(int needed, int &done, std::mutex &mutex, Set set) {
    if (__atomic_load_n(&done, __ATOMIC_ACQUIRE) >= needed) return 0;
    std::lock_guard<std::mutex> guard(mutex);
    if (done >= needed) return 0;
    const int error = set(needed);
    if (error == 0) __atomic_store_n(&done, needed, __ATOMIC_RELEASE);
    return error;
}

}  // namespace singe
