// Arrays that a call allocates when it first needs them: all of a set or none,
// so that a call that ran out of memory can be made again and finds either the
// whole set or nothing.  Plain C++; the allocator is the caller's.
#pragma once
#include <stddef.h>

struct MpmgPiece {
    void **ptr;
    size_t bytes;
};

// Allocates every piece (at least a byte each) with alloc(void **, size_t),
// which returns whether it succeeded.  On a failure what was allocated is given
// back through release(void *) and every pointer is null.
template <class Alloc, class Release>
bool mpmg_alloc_all(const MpmgPiece *pieces, size_t count, Alloc alloc, Release release)
{
    size_t have = 0;
    while (have < count && alloc(pieces[have].ptr, pieces[have].bytes > 0 ? pieces[have].bytes : 1)) have++;
    if (have == count) return true;
    for (size_t k = 0; k < have; k++) release(*pieces[k].ptr);
    for (size_t k = 0; k < count; k++) *pieces[k].ptr = nullptr;
    return false;
}
