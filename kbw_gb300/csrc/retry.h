// Allocations that may ask for idle memory back.
#pragma once

namespace kbwg {

// alloc(); once more if it ended in `out_of_memory` and release() gave
// something back.
template <class E, class Alloc, class Release>
E alloc_or_release(E out_of_memory, Alloc &&alloc, Release &&release) {
    const E e = alloc();
    return e == out_of_memory && release() ? alloc() : e;
}

}  // namespace kbwg
