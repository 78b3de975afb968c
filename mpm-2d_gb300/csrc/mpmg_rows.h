// Sizes of the FP64 step's element rows.  Plain C++, checked on the host.
#pragma once
#include <limits.h>
#include <stddef.h>

#include <new>

// Counts the particles inside the grid and the elements that hold one, a bit an
// element.  Kept free of branches: it runs in the loop that forms the element
// map, beside its divisions (1 048 576 particles: a loop of its own took 0.74
// ms of a create of 5.6).
class MpmgFilled {
public:
    // False without the memory.
    bool begin(size_t ne)
    {
        words = ne / kBits + 1;
        seen = new (std::nothrow) unsigned long[words]();
        return seen != nullptr;
    }
    ~MpmgFilled() { delete[] seen; }
    MpmgFilled() = default;
    MpmgFilled(const MpmgFilled &) = delete;
    MpmgFilled &operator=(const MpmgFilled &) = delete;
    // A particle in element e, or outside the grid (-1).
    void add(int e)
    {
        const bool in = e >= 0;
        const size_t at = in ? (size_t)e : 0;
        inside += in;
        seen[at / kBits] |= (unsigned long)in << (at % kBits);
    }
    size_t filled() const
    {
        size_t n = 0;
        for (size_t k = 0; k < words; k++) n += (size_t)__builtin_popcountl(seen[k]);
        return n;
    }
    size_t inside = 0;

private:
    static constexpr size_t kBits = CHAR_BIT * sizeof(unsigned long);
    unsigned long *seen = nullptr;
    size_t words = 0;
};

// Slots a row, for n particles of which `inside` lie in `filled` of the ne
// elements.  A row holds at least twice the mean count of the filled elements (a
// power of two from 16), since a flow packs elements unevenly.  Rows above 16
// slots have no more than 128 slots a particle in all: a crowd on a large empty
// grid goes beyond its rows (64 slots on 4096^2 elements are 8.6 GB in the two
// buffers, 16 are 2.1).
inline int mpmg_row_slots(size_t inside, size_t filled, size_t n, size_t ne)
{
    int cap = 16;
    while (filled > 0 && (size_t)cap * filled < 2 * inside && 2 * (size_t)cap * ne <= 128 * n) cap *= 2;
    return cap;
}

// Whether the FP64 step keeps its corner sums and coefficients (288 bytes) for
// the elements on the list of filled ones, at most one a particle, or for every
// element of the grid.  By list, an element of an empty grid takes 200 bytes with
// its node instead of 480, and the place is one more load (1 048 576 particles on
// 262 144 elements 5570 us a pass of 20 steps, 5517 by element; 125k 2246 and
// 2198; 7 million on 2^24 3983 us a step and 3825): so only grids whose size is a
// matter of memory, 8 GB by element here.
inline bool mpmg_sums_by_list(size_t n, size_t ne)
{
    return ne >= ((size_t)1 << 24) && ne > 2 * n;
}
