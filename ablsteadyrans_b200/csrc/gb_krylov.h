// The book-keeping of a solver's Krylov vectors that came from allocations
// made during a solve (host only).
#pragma once

#include <algorithm>
#include <cstdint>
#include <functional>
#include <vector>

namespace gb {

//! One allocation of Krylov vectors: its first double and how many it holds
//! (the last one of a restart is shorter than the others).
struct KrylovChunk {
    double* base;
    int64_t count;
};

//! Takes the vectors that lie in the chunks off a list; the others stay, in order.
inline void forget_chunks(const std::vector<KrylovChunk>& chunks, std::vector<double*>& list)
{
    const std::less<const double*> before;
    auto ours = [&](const double* p) {
        return std::any_of(chunks.begin(), chunks.end(),
                           [&](const KrylovChunk& c) { return !before(p, c.base) && before(p, c.base + c.count); });
    };
    list.erase(std::remove_if(list.begin(), list.end(), ours), list.end());
}

}  // namespace gb
