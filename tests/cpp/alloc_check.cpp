// Test-only: mpmg_alloc_all (mpmg_alloc.h) with an allocator that fails at a
// given call.  Built by tests/test_alloc.py with g++ into a temporary shared
// library.
#include <stdlib.h>

#include <set>

#include "../../mpm-2d_gb300/csrc/mpmg_alloc.h"

namespace {

std::set<void *> live;

bool attempt(void **p, size_t count, const size_t *bytes, int fail_at)
{
    MpmgPiece pieces[16];
    for (size_t k = 0; k < count; k++) pieces[k] = MpmgPiece{p + k, bytes[k]};
    int calls = 0;
    return mpmg_alloc_all(
        pieces, count,
        [&](void **q, size_t n) {
            if (calls++ == fail_at || n == 0) return false;
            *q = malloc(n);
            live.insert(*q);
            return true;
        },
        [](void *q) {
            live.erase(q);
            free(q);
        });
}

}  // namespace

// A set of `count` arrays whose allocation fails at call fail_at, then is made
// again.  Returns 0 where the failed attempt left nothing (no memory held, every
// pointer null) and the second one all.
extern "C" int fail_then_succeed(int count, const size_t *bytes, int fail_at)
{
    void *p[16];
    for (void *&q : p) q = (void *)0x10;       // what an earlier owner left
    live.clear();
    if (attempt(p, (size_t)count, bytes, fail_at)) return 1;
    for (int k = 0; k < count; k++)
        if (p[k] != nullptr) return 2;
    if (!live.empty()) return 3;
    if (!attempt(p, (size_t)count, bytes, -1)) return 4;
    if (live.size() != (size_t)count) return 5;
    for (int k = 0; k < count; k++) {
        if (live.count(p[k]) != 1) return 6;
        free(p[k]);
    }
    return 0;
}
