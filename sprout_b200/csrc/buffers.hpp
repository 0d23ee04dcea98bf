// Replacing a set of device buffers by larger ones (render.cu); host code only.
#pragma once

#include <cstddef>
#include <vector>

namespace spb::render {

struct Buffer {
    void** at;
    size_t bytes;  // 0: none, the pointer stays null
};

template <class T>
Buffer buffer(T*& p, size_t bytes) {
    return {reinterpret_cast<void**>(&p), bytes};
}

// Releases all buffers of the set, then allocates each anew.  alloc(pointer, bytes) returns an error
// code (0: none); release(pointer) takes null.  Returns the first error, after which every buffer of
// the set is released and null: the caller's record of what they hold must be empty before the call and
// set after it, or a later, smaller request would find room in buffers that are not there.
template <class Alloc, class Release>
int replace_buffers(std::vector<Buffer> const& set, Alloc&& alloc, Release&& release) {
    auto const clear = [&] {
        for (Buffer const& b : set) {
            release(*b.at);
            *b.at = nullptr;
        }
    };
    clear();
    for (Buffer const& b : set) {
        if (b.bytes == 0) {
            continue;
        }
        if (int const e = int(alloc(b.at, b.bytes))) {
            *b.at = nullptr;
            clear();
            return e;
        }
    }
    return 0;
}

}  // namespace spb::render
