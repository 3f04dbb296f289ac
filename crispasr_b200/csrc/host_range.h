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

}  // namespace b200
