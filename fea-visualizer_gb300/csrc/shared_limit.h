// shared_limit.h -- a limit that belongs to the process, raised by any thread.
#pragma once

#include <cstddef>
#include <mutex>

namespace fea {

inline std::mutex& limit_mutex() {
    static std::mutex m;
    return m;
}

// Raises the limit to `want` when read() is below it.  Read and write are one
// step for all threads: two handles that ask for different sizes at once must
// not leave the smaller one behind.
template <typename Read, typename Write>
void raise_shared_limit(std::size_t want, Read read, Write write) {
    const std::lock_guard<std::mutex> hold(limit_mutex());
    if (read() < want) write(want);
}

}  // namespace fea
