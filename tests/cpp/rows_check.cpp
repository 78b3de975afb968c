// Test-only: mpmg_row_width (mpmg_rows.h), with a non-throwing operator new[]
// that can be made to fail.  Built by tests/test_rows.py with g++ into a
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
    const bool ok = mpmg_row_width(emap, n, ne, cap, filled);
    out_of_memory = false;
    return ok ? 0 : 1;
}
