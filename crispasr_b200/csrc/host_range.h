// host_range.h — address questions of the host-buffer entry point (plain C++: no CUDA).
#pragma once
#include <cstddef>
#include <cstdint>

namespace b200 {

// Whether [p, p + bytes) lies inside one allocation.  `query(p, &start, &size)` gives the allocation that holds the address p,
// or false.  Asking for the two ends only would accept a range whose ends are in two allocations with a hole between them.
template <typename Query>
bool inside_one_allocation(Query query, uintptr_t p, size_t bytes) {
    uintptr_t start = 0;
    size_t size = 0;
    return query(p, &start, &size) && start <= p && p - start <= size && bytes <= size - (p - start);
}

// How a result [dst, dst + n * stride) of n entries meets an operand of m entries, [p, p + (m - 1) * entry_stride + entry_bytes).
// kByEntry: entry i of the operand lies inside entry i of the result (an update in place): entries stay independent.
enum class Meets { kNot, kByEntry, kAnyhow };
inline Meets result_meets(uintptr_t dst, size_t stride, size_t n, uintptr_t p, size_t entry_stride, size_t entry_bytes, size_t m) {
    const size_t span = (m - 1) * entry_stride + entry_bytes;
    if (p >= dst + n * stride || dst >= p + span) return Meets::kNot;
    return m == n && p >= dst && p - dst + entry_bytes <= stride && (n == 1 || entry_stride == stride) ? Meets::kByEntry : Meets::kAnyhow;
}

}  // namespace b200
