// Whether a kernel can reach a range of host memory from end to end.
#pragma once
#include <stddef.h>
#include <stdint.h>

namespace smat {

// The pinned host memory that an address belongs to, as the driver mapped it.
struct HostMapping {
    uintptr_t base = 0;      // first address of the mapping
    size_t size = 0;
    char* device = nullptr;  // what the device calls the address asked for
};

// The device's address of host memory [p, p + bytes), or null where any of it is not pinned or the device does not see it in
// one piece.  query(address, &mapping) says false for memory that is not pinned.  Mapping after mapping up to the end: two
// pinned ends say nothing about the pages between them, and a kernel that stores to a pageable one faults.
template <class Query>
char* device_view_of_range(const void* p, size_t bytes, Query&& query) {
    constexpr int kMostMappings = 16;
    const uintptr_t begin = reinterpret_cast<uintptr_t>(p);
    char* view = nullptr;
    size_t done = 0;
    for (int i = 0; done < bytes; i++) {
        HostMapping m;
        if (i == kMostMappings || !query(begin + done, &m) || !m.device) return nullptr;
        if (begin + done < m.base || begin + done - m.base >= m.size) return nullptr;
        if (!view) view = m.device;
        if (m.device != view + done) return nullptr;
        done = m.base + m.size - begin;
    }
    return view;
}

}  // namespace smat
