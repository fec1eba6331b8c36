// Device buffers that are made and replaced together, for host code; the caller passes the allocator.
#pragma once
#include <cstddef>
#include <cstring>
#include <vector>

namespace mi {

// Every buffer belongs to a pointer variable of its owner.  As long as a buffer lives its pointer is set, and a pointer never outlives
// its buffer: release() clears the variables, so that after an allocation that failed half-way nothing refers to freed memory.
class BufferSet {
    struct Slot { void* variable; void* buffer; };       // address of the owner's pointer variable, of whatever type
    std::vector<Slot> slots;

public:
    // alloc(void**, bytes) -> true on success; false leaves the set as it was, with *variable null
    template <class T, class Alloc>
    bool take(T** variable, size_t bytes, Alloc alloc) {
        void* p = nullptr;
        *variable = nullptr;
        if (!alloc(&p, bytes)) return false;
        *variable = static_cast<T*>(p);
        slots.push_back(Slot{variable, p});
        return true;
    }
    template <class Free>
    void release(Free free_one) {
        for (const Slot& s : slots) { std::memset(s.variable, 0, sizeof(void*)); free_one(s.buffer); }
        slots.clear();
    }
};

}  // namespace mi
