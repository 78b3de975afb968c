// Sizes of the FP64 step's element rows.  Plain C++, checked on the host.
#pragma once
#include <limits.h>
#include <stddef.h>

#include <new>

// Slots a row and filled elements for the initial element map emap[n] (-1:
// outside the grid) of ne elements.  A row holds at least twice the mean count
// of the filled elements (a power of two from 16), since a flow packs elements
// unevenly.  Rows above 16 slots have no more than 128 slots a particle in all:
// a crowd on a large empty grid goes beyond its rows (64 slots on 4096^2 elements
// are 8.6 GB in the two buffers, 16 are 2.1).  False without the memory to count
// (a bit an element).
inline bool mpmg_row_width(const int *emap, size_t n, size_t ne, int *cap, size_t *filled)
{
    constexpr size_t bits = CHAR_BIT * sizeof(unsigned long);
    unsigned long *seen = new (std::nothrow) unsigned long[ne / bits + 1]();
    if (seen == nullptr) return false;
    size_t inside = 0;
    *filled = 0;
    for (size_t i = 0; i < n; i++) {
        if (emap[i] < 0) continue;
        const size_t e = (size_t)emap[i];
        const unsigned long bit = 1ul << (e % bits);
        inside++;
        if ((seen[e / bits] & bit) == 0) {
            seen[e / bits] |= bit;
            (*filled)++;
        }
    }
    delete[] seen;
    *cap = 16;
    while (*filled > 0 && (size_t)*cap * *filled < 2 * inside && 2 * (size_t)*cap * ne <= 128 * n) *cap *= 2;
    return true;
}
