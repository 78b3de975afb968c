// Test-only: MpmgFilled and mpmg_row_slots (mpmg_rows.h), with a non-throwing
// operator new[] that can be made to fail.  Built by tests/test_rows.py with g++ into a
// temporary shared library.
#include <stdlib.h>

#include "../../mpm-2d_gb300/csrc/mpmg_rows.h"

static bool out_of_memory = false;

void *operator new[](size_t n, const std::nothrow_t &) noexcept
{
    return out_of_memory ? nullptr : malloc(n);
}
void operator delete[](void *p) noexcept
{
    free(p);
}
void operator delete[](void *p, size_t) noexcept
{
    free(p);
}

// 0, or 1 where the count found no memory.
extern "C" int row_width(const int *emap, size_t n, size_t ne, int no_memory, int *cap, size_t *filled)
{
    out_of_memory = no_memory != 0;
    MpmgFilled count;
    const bool ok = count.begin(ne);
    out_of_memory = false;
    if (!ok) return 1;
    for (size_t i = 0; i < n; i++) count.add(emap[i]);
    *filled = count.filled();
    *cap = mpmg_row_slots(count.inside, *filled, n, ne);
    return 0;
}

extern "C" int sums_by_list(size_t n, size_t ne)
{
    return mpmg_sums_by_list(n, ne) ? 1 : 0;
}
