// Stable LSD radix sort of (element key, particle index) pairs, and the
// per-element start offsets of the sorted order.  The allocation-free entry
// point (mpmg_sort_noalloc.cu) runs it on its fixed scratch, mpmg_get_sort of
// the FP64 form on the context's; the mixed step bins particles with the
// counting sort of mpmg_bin.cu, which gives the same order.
//
// The reference groups particles by element in find_filled_elements
// (libmpm/process_usl.c:677-723): for each element, its particles in
// ascending particle index.  A stable sort of the keys over particle indices
// 0..n-1 reproduces exactly those groups, so the permutation is bit-exact
// against the reference's lists.
//
// Keys need ceil(log2(num_elements + 1)) bits (18 for 512^2 elements); they
// are sorted in ceil(bits / 10) passes of at most 10 bits.  Each pass:
//   upsweep    per-tile digit histogram (shared atomics); the first pass's also
//              clamps the caller's keys into the scratch
//   scan       one warp per digit: exclusive prefix of that digit's counts
//              over the tiles, and the digit's total
//   downsweep  every warp ranks its 128 or 256 contiguous keys stably (match_any +
//              a warp-private digit histogram), the block turns the per-warp
//              counts into offsets (digit prefix over the whole input + this
//              tile's prefix + earlier warps), and keys and values scatter
// Integer-only and deterministic for any launch order.
//
// Bound by latency: 125k keys are seven short kernels.  So each is launched
// before its predecessor has finished (programmatic dependent launch), a tile
// is 1024 keys where 2048 would leave SMs without one, and the offsets come
// from 32-way searches of block ranges: 125k keys of 262 144 elements 49 -> 27
// us, of 40 000 elements 19.4 (35.0 without the early launches).
#include "mpmg_internal.cuh"

namespace {

constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;
constexpr int kMaxRounds = 8;                    // keys per lane: 4 or 8, 1024 or 2048 a block
constexpr int kMaxBits = 10;
constexpr int kMaxRadix = 1 << kMaxBits;

// FIRST: the keys are the caller's; a key outside [0, ne] becomes ne, and the
// clamped keys go to `clamped` for the rest of the sort.
template <int ROUNDS, bool FIRST>
__global__ void __launch_bounds__(kThreads) upsweep_kernel(const uint32_t *__restrict__ keys, int n, uint32_t ne,
                                                           int shift, int bits, int num_tiles,
                                                           uint32_t *__restrict__ clamped,
                                                           uint32_t *__restrict__ tile_hist)
{
    __shared__ uint32_t hist[kMaxRadix];
    const int radix = 1 << bits;
    for (int d = threadIdx.x; d < radix; d += kThreads) hist[d] = 0;
    __syncthreads();
    const uint32_t mask = (uint32_t)radix - 1u;
    const int base = blockIdx.x * (kThreads * ROUNDS);
    mpmg_pdl_wait();
    mpmg_pdl_trigger();
#pragma unroll
    for (int k = 0; k < ROUNDS; k++) {
        int idx = base + k * kThreads + threadIdx.x;
        if (idx >= n) continue;
        uint32_t key = keys[idx];
        if (FIRST) {
            if (key > ne) key = ne;             // a negative key is above every element
            clamped[idx] = key;
        }
        atomicAdd(&hist[(key >> shift) & mask], 1u);
    }
    __syncthreads();
    for (int d = threadIdx.x; d < radix; d += kThreads)
        tile_hist[(size_t)d * num_tiles + blockIdx.x] = hist[d];
}

// One warp per digit: exclusive scan of tile_hist[d][0..num_tiles) in place,
// total of digit d into digit_total[d].
__global__ void __launch_bounds__(kThreads) scan_tiles_kernel(uint32_t *__restrict__ tile_hist,
                                                              int num_tiles, int radix,
                                                              uint32_t *__restrict__ digit_total)
{
    const int lane = threadIdx.x & 31;
    const int d = blockIdx.x * kWarps + (threadIdx.x >> 5);
    if (d >= radix) return;
    uint32_t *row = tile_hist + (size_t)d * num_tiles;
    uint32_t run = 0;
    mpmg_pdl_wait();
    mpmg_pdl_trigger();
    for (int base = 0; base < num_tiles; base += 32) {
        int t = base + lane;
        uint32_t v = (t < num_tiles) ? row[t] : 0u;
        uint32_t incl = v;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            uint32_t u = __shfl_up_sync(0xffffffffu, incl, off);
            if (lane >= off) incl += u;
        }
        if (t < num_tiles) row[t] = run + incl - v;
        run += __shfl_sync(0xffffffffu, incl, 31);
    }
    if (lane == 0) digit_total[d] = run;
}

// FIRST: the values are the index sequence.
template <int ROUNDS, bool FIRST>
__global__ void __launch_bounds__(kThreads) downsweep_kernel(
    const uint32_t *__restrict__ keys_in, const uint32_t *__restrict__ vals_in, int n, int shift,
    int bits, int num_tiles, const uint32_t *__restrict__ tile_prefix,
    const uint32_t *__restrict__ digit_total, uint32_t *__restrict__ keys_out,
    uint32_t *__restrict__ vals_out)
{
    __shared__ uint32_t warp_hist[kWarps][kMaxRadix];   // counts, then per-warp bases
    __shared__ uint32_t digit_base[kMaxRadix];
    __shared__ uint32_t warp_sums[kWarps];
    const int radix = 1 << bits;
    const uint32_t mask = (uint32_t)radix - 1u;
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    const uint32_t lt_mask = (1u << lane) - 1u;

    for (int k = threadIdx.x; k < kWarps * kMaxRadix; k += kThreads) (&warp_hist[0][0])[k] = 0;
    mpmg_pdl_wait();
    mpmg_pdl_trigger();

    // Exclusive prefix of the digit totals (the digit's start in the output).
    {
        const int per = kMaxRadix / kThreads;            // 4 digits per thread
        uint32_t local[per];
        uint32_t s = 0;
#pragma unroll
        for (int j = 0; j < per; j++) {
            int d = threadIdx.x * per + j;
            local[j] = (d < radix) ? digit_total[d] : 0u;
            s += local[j];
        }
        uint32_t incl = s;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            uint32_t u = __shfl_up_sync(0xffffffffu, incl, off);
            if (lane >= off) incl += u;
        }
        if (lane == 31) warp_sums[warp] = incl;
        __syncthreads();
        uint32_t wbase = 0;
        for (int w = 0; w < warp; w++) wbase += warp_sums[w];
        uint32_t run = wbase + incl - s;
#pragma unroll
        for (int j = 0; j < per; j++) {
            int d = threadIdx.x * per + j;
            if (d < radix) digit_base[d] = run + tile_prefix[(size_t)d * num_tiles + blockIdx.x];
            run += local[j];
        }
    }
    __syncthreads();

    // Each warp ranks its contiguous keys in order (stable).
    const int wbase_idx = blockIdx.x * (kThreads * ROUNDS) + warp * (ROUNDS * 32);
    uint32_t key[ROUNDS], val[ROUNDS], rank[ROUNDS];
#pragma unroll
    for (int r = 0; r < ROUNDS; r++) {
        const int idx = wbase_idx + r * 32 + lane;
        key[r] = idx < n ? keys_in[idx] : 0xffffffffu;
        val[r] = FIRST ? (uint32_t)idx : idx < n ? vals_in[idx] : 0u;
    }
#pragma unroll
    for (int r = 0; r < ROUNDS; r++) {
        const bool valid = wbase_idx + r * 32 + lane < n;
        const uint32_t d = (key[r] >> shift) & mask;
        const uint32_t vmask = __ballot_sync(0xffffffffu, valid);
        const uint32_t peers = __match_any_sync(0xffffffffu, valid ? d : 0xffffffffu) & vmask;
        uint32_t before = 0;
        if (valid) before = warp_hist[warp][d];
        __syncwarp();
        rank[r] = before + __popc(peers & lt_mask);
        if (valid && (peers & lt_mask) == 0) warp_hist[warp][d] = before + __popc(peers);
        __syncwarp();
    }
    __syncthreads();
    // Per digit: exclusive prefix over warps, offset by the digit's base.
    for (int d = threadIdx.x; d < radix; d += kThreads) {
        uint32_t run = digit_base[d];
#pragma unroll
        for (int w = 0; w < kWarps; w++) {
            uint32_t c = warp_hist[w][d];
            warp_hist[w][d] = run;
            run += c;
        }
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < ROUNDS; r++) {
        const int idx = wbase_idx + r * 32 + lane;
        if (idx < n) {
            const uint32_t d = (key[r] >> shift) & mask;
            const uint32_t dst = warp_hist[warp][d] + rank[r];
            keys_out[dst] = key[r];
            vals_out[dst] = val[r];
        }
    }
}

// The first sorted position whose key is >= e, by a whole warp: 32 probes a
// round, so that a million keys take four dependent loads.
__device__ __forceinline__ int lower_bound_warp(const uint32_t *__restrict__ keys, int n, uint32_t e)
{
    const int lane = threadIdx.x & 31;
    int lo = 0, hi = n;                      // the answer is in [lo, hi]
    while (lo < hi) {
        const int step = (hi - lo + 31) / 32;
        const int at = lo + (lane + 1) * step - 1;
        const uint32_t below = __ballot_sync(0xffffffffu, at < hi && keys[at] < e);
        const int count = __popc(below);     // the probes are ordered: lanes 0 .. count - 1
        const int next = lo + (count + 1) * step - 1;
        lo += count * step;
        if (next < hi) hi = next;
    }
    return lo;
}

// The first position in [lo, hi) whose key is >= e (hi if none), by one thread:
// three probes a round.
__device__ __forceinline__ int lower_bound_in(const uint32_t *__restrict__ keys, int lo, int hi, uint32_t e)
{
    while (lo < hi) {
        const int q = (hi - lo) >> 2, a = lo + q, b = a + q, c = b + q;    // c < hi
        const bool ka = keys[a] < e, kb = keys[b] < e, kc = keys[c] < e;
        if (kc) lo = c + 1;
        else if (kb) { lo = b + 1; hi = c; }
        else if (ka) { lo = a + 1; hi = b; }
        else hi = a;
    }
    return lo;
}

// cell_start[e] = first sorted position whose key is >= e, for e in [0, ne].  A
// block of kStartElems elements finds its range of the sorted keys, and each
// thread the first entries there of the elements between its key and the one
// before; or, where the range is long, each thread its element's by a search in
// it (full elements: a few blocks would read nearly all of the keys).
constexpr int kStartElems = 256;            // 1024: 125k keys of 40 000 elements 23.2 us instead of 19.4
constexpr int kSweepKeys = 8 * kThreads;     // eight keys a thread, about a search's ten dependent loads

__global__ void __launch_bounds__(kThreads) cell_start_kernel(const uint32_t *__restrict__ sorted_keys, int n, int ne,
                                                              int *__restrict__ cell_start)
{
    __shared__ int range[2];
    __shared__ int first[kStartElems];
    const long long e0 = (long long)blockIdx.x * kStartElems;
    const int w = threadIdx.x >> 5;
    mpmg_pdl_wait();
    if (w < 2) {
        // up to the keys outside the grid, in the last block
        const long long e = w == 0 ? e0 : e0 + kStartElems < ne ? e0 + kStartElems : ne;
        const int at = lower_bound_warp(sorted_keys, n, (uint32_t)e);
        if ((threadIdx.x & 31) == 0) range[w] = at;
    }
    __syncthreads();
    const int lo = range[0], hi = range[1];
    if (hi - lo > kSweepKeys) {
        for (int t = threadIdx.x; t < kStartElems; t += kThreads)
            if (e0 + t <= ne) cell_start[e0 + t] = lower_bound_in(sorted_keys, lo, hi, (uint32_t)(e0 + t));
        return;
    }
    for (int t = threadIdx.x; t < kStartElems; t += kThreads) first[t] = hi;
    __syncthreads();
    for (int i = lo + threadIdx.x; i < hi; i += kThreads) {
        const int k = (int)((long long)sorted_keys[i] - e0);
        const int before = i > lo ? (int)((long long)sorted_keys[i - 1] - e0) : -1;
        for (int e = before + 1; e <= k; e++) first[e] = i;
    }
    __syncthreads();
    for (int t = threadIdx.x; t < kStartElems; t += kThreads)
        if (e0 + t <= ne) cell_start[e0 + t] = first[t];
}

}  // namespace

// Sorts the caller's n keys (clamped to [0, ne], ne < 2^key_bits) with their
// indices into sorted_keys and perm using the given scratch, then fills
// cell_start[0..ne].  A tile is 1024 keys up to 1024 a multiprocessor (a tile
// of 2048 leaves half of them idle: 125k keys 19.4 us, 22.3 with it) and 2048
// beyond (300k keys 29.4 us, 31.3 with tiles of 1024, and the scratch holds 512
// tiles).
cudaError_t mpmg_sort_run(const uint32_t *keys, int n, int ne, int key_bits, int sms, const SortScratch &sc,
                          uint32_t *sorted_keys, uint32_t *perm, int *cell_start, cudaStream_t s)
{
    const dim3 block(kThreads);
    if (n > 0) {
        const bool small = n <= sms * kThreads * 4;
        const int passes = (key_bits + kMaxBits - 1) / kMaxBits;
        const int base_bits = key_bits / passes, extra = key_bits % passes;
        const int tile = kThreads * (small ? 4 : kMaxRounds), tiles = (n + tile - 1) / tile;
        const uint32_t *src_k = sc.keys, *src_v = nullptr;
        int shift = 0;
        for (int p = 0; p < passes; p++) {
            const int bits = base_bits + (p < extra ? 1 : 0);
            const int radix = 1 << bits;
            const bool to_out = ((passes - 1 - p) % 2) == 0, first = p == 0;
            uint32_t *dst_k = to_out ? sorted_keys : sc.keys_alt;
            uint32_t *dst_v = to_out ? perm : sc.vals_alt;
            cudaError_t e = mpmg_launch_pdl(
                true, first ? (small ? upsweep_kernel<4, true> : upsweep_kernel<8, true>)
                            : (small ? upsweep_kernel<4, false> : upsweep_kernel<8, false>),
                dim3(tiles), block, 0, s, first ? keys : src_k, n, (uint32_t)ne, shift, bits, tiles, sc.keys, sc.tile_hist);
            if (e == cudaSuccess)
                e = mpmg_launch_pdl(true, scan_tiles_kernel, dim3((radix + kWarps - 1) / kWarps), block, 0, s,
                                    sc.tile_hist, tiles, radix, sc.digit_total);
            if (e == cudaSuccess)
                e = mpmg_launch_pdl(true, first ? (small ? downsweep_kernel<4, true> : downsweep_kernel<8, true>)
                                                : (small ? downsweep_kernel<4, false> : downsweep_kernel<8, false>),
                                    dim3(tiles), block, 0, s, src_k, src_v, n, shift, bits, tiles,
                                    (const uint32_t *)sc.tile_hist, (const uint32_t *)sc.digit_total, dst_k, dst_v);
            if (e != cudaSuccess) return e;
            src_k = dst_k;
            src_v = dst_v;
            shift += bits;
        }
    }
    return mpmg_launch_pdl(true, cell_start_kernel, dim3(ne / kStartElems + 1), block, 0, s,
                           (const uint32_t *)sorted_keys, n, ne, cell_start);
}
