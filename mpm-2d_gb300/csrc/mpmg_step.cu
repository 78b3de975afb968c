// The explicit USL step on the GPU (reference: explicit_mpm_step_usl_threaded,
// libmpm/process_usl.c:465-592, plus the driver's time_varying_loads tail,
// src/main.c:975 and libmpm/loading.c:34-54).
//
//   rows      each element's particle indices, in a row of the element's own
//             (find_filled_elements, :677-723).  The G2P bins every particle it
//             moves for the next step (WHICH_ELEMENT4, :43-44 and :631-674), so
//             a step needs no pass of its own for it; keys_kernel does it where
//             positions came from outside (the first step, a set field)
//   p2g       one thread (or two) per element puts its row in particle order
//             and sums the contributions to its four corners
//             (map_to_grid_explicit_split, :812-910); advances t and the
//             gravity scalar in the device StepParams
//   grid      one thread per node adds the four adjacent elements' corner
//             sums in colour order 0..3, applies the box / square-silo
//             conditions and the nodal update (bc_momentum, bc_force,
//             move_grid_split :596-625); then one per element forms the
//             bilinear coefficients of the nodal acceleration and velocity
//   g2p       one thread per particle: velocity and position update, strain
//             rate, volume and the material law (move_particles :914-957,
//             calculate_strainrate :764-808, update_densities :961-970,
//             calculate_stress_threaded), and the next step's rows
//
// The kernels are launched with programmatic dependent launch: each waits for
// the one before it at its start, and lets the next one launch at its end, or
// right after that wait where every kernel is at most a warp an SM (`early`):
// there the next one's launch overlaps this one's work (block of 4096
// particles: 15.7 against 17.3 us a step), while in larger grids blocks that
// launch beside working ones are placed unevenly (125 k particles: 97 against
// 76 us).
//
// Shape functions (tent / grad_tent, interpolate.c:23-65) are recomputed in
// registers from the start-of-step position wherever they are needed.  No
// floating-point atomics are used; every sum has a fixed order.
#include <math.h>

#include "mpmg_fp64_common.cuh"
#include "mpmg_internal.cuh"
#include "mpmg_materials.cuh"

namespace {

using fp64::BcParams;
using fp64::GridGeom;
using fp64::ShapeFns;
using fp64::bc_mask;
using fp64::make_bc;
using fp64::make_geom;
using fp64::shape;

// Whether the step's kernels let their successors launch early (see above).
inline int early_launch(const mpmg_ctx *ctx)
{
    return ctx->np <= (size_t)ctx->sms * 32;
}

// ---------------------------------------------------------------------------
// rows

struct RowsOut {
    uint32_t *count, *rows, *filled, *pos, *n_filled, *head, *next;
    int cap;
};

// Adds particle i to element key's row (every lane of the warp calls it; valid
// marks lanes with a particle inside the grid).  Runs of equal keys in
// consecutive lanes share one atomic.
__device__ __forceinline__ void bin_particle(const RowsOut &R, int i, uint32_t key, bool valid)
{
    const int lane = threadIdx.x & 31;
    const uint32_t k = valid ? key : 0xffffffffu;
    const uint32_t prev = __shfl_up_sync(0xffffffffu, k, 1);
    const bool start = valid && (lane == 0 || prev != k);
    const uint32_t starts = __ballot_sync(0xffffffffu, start);
    const uint32_t invalid = ~__ballot_sync(0xffffffffu, valid);
    uint32_t base = 0;
    if (start) {
        const uint32_t above = lane == 31 ? 0u : (starts | invalid) & (0xfffffffeu << lane);
        const int end = above ? __ffs(above) - 1 : 32;
        base = atomicAdd(&R.count[key], (uint32_t)(end - lane));
    }
    const uint32_t below = starts & (0xffffffffu >> (31 - lane));
    const int leader = below ? 31 - __clz(below) : lane;
    // the first particle of an element puts it on the list
    const uint32_t firsts = __ballot_sync(0xffffffffu, start && base == 0);
    if (firsts) {
        uint32_t at = 0;
        if (lane == 0) at = atomicAdd(R.n_filled, (uint32_t)__popc(firsts));
        at = __shfl_sync(0xffffffffu, at, 0);
        if (start && base == 0) {
            at += (uint32_t)__popc(firsts & ((1u << lane) - 1u));
            R.filled[at] = key;
            if (R.pos != nullptr) R.pos[key] = at;
        }
    }
    base = __shfl_sync(0xffffffffu, base, leader);
    if (!valid) return;
    const uint32_t slot = base + (uint32_t)(lane - leader);
    if (slot < (uint32_t)R.cap) R.rows[(size_t)key * R.cap + slot] = (uint32_t)i;
    else R.next[i] = atomicExch(&R.head[key], (uint32_t)i);
}

// The rows of the current positions, where no G2P has left them: keys[i] is
// the element, or the sentinel for a particle that is inactive or outside.
__global__ void __launch_bounds__(256) keys_kernel(GridGeom g, float inv_hf, int n, const double *__restrict__ x,
                                                   const double *__restrict__ y, const int *__restrict__ active,
                                                   uint32_t *__restrict__ keys, uint32_t sentinel, RowsOut R)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    uint32_t key = sentinel;
    if (i < n) {
        if (active[i]) {
            const int e = mpmg_which_element_fast(x[i], y[i], g.h, g.inv_h, inv_hf, g.xmax, g.ymax,
                                                  __double_as_longlong(g.xmax), __double_as_longlong(g.ymax), g.Ex,
                                                  g.Ey);
            if (e >= 0) key = (uint32_t)e;
        }
        keys[i] = key;
    }
    bin_particle(R, i, key, key != sentinel);
}

// ---------------------------------------------------------------------------
// p2g: per-element corner sums over the element's row, in particle order.
//
// The corner weights are bilinear in the local coordinates (x, y):
// N = {(1-x)(1-y), x(1-y), xy, (1-x)y}, dN/dx h = {-(1-y), 1-y, y, -y},
// dN/dy h = {-(1-x), -x, x, 1-x}.  So the element's four corner sums of a
// particle quantity q follow from four moments, A = sum q, X = sum x q,
// Y = sum y q, Z = sum xy q:  corners A - X - Y + Z, X - Z, Z, Y - Z; and the
// eight internal-force sums from seven moments of the stress terms.  The
// particle loop costs 26 FP64 operations; 1 / h of the gradients and the body
// force are applied once per node (grid_kernel).
//
// The loop is bound by the FP64 pipe, where an instruction costs a sub-partition
// 64 cycles whatever the number of active lanes: a warp costs its fullest
// element's count.  So a block takes EB of the filled elements from the list
// (empty ones cost nothing, and a sparse grid's work spreads over all SMs),
// sorts them by count, so that each warp holds about equal counts, and rotates
// the sorted warps with the block index, so that no sub-partition gets the
// full ones of every block.  SPLIT = 2 gives the two halves of an element's
// moments to two threads in different warps, which shortens the serial chain
// where there are too few elements to fill the chip.  The sums are stored a run
// an element, by element or in the list's order (RowBins::pos): 4 corners x (m,
// mx, my, h fx), then 4 x h fy.

constexpr int kCell = 20;                  // doubles an element
constexpr int kStage = 16;                 // staged row entries an element, at most a row's slots

// Puts the lists of a block's elements with more than kStage particles in
// ascending order, a warp to a list: by rank in registers up to 128 particles,
// beyond by a bitonic network in place whose pairs past the end are left out
// (all of its exchanges put the larger entry last).  A list longer than its row
// is first gathered in over_list from the row and its chain, a thread to a
// chain, and its place left in row[0] and sh_base.  In a thread's insertion sort
// instead, the random order of 64 entries took most of the P2G (1 048 576
// particles, 64 to an element: 2118 -> 328 us a step).  Called by the whole block.
__device__ __noinline__ void order_long_lists(RowView rv, int lists, const int *sh_elem, const int *sh_count,
                                              uint32_t *sh_base, const uint32_t *head, const uint32_t *next,
                                              uint32_t *cursor)
{
    const unsigned all = 0xffffffffu;
    const int lane = threadIdx.x & 31, warps = blockDim.x / 32;
    if ((int)threadIdx.x < lists && sh_count[threadIdx.x] > rv.cap) {
        const int cnt = sh_count[threadIdx.x], e = sh_elem[threadIdx.x];
        const uint32_t base = atomicAdd(cursor, (uint32_t)cnt);
        sh_base[threadIdx.x] = base;
        uint32_t i = head[e];
        for (int j = rv.cap; j < cnt; j++) {
            rv.over_list[base + j] = i;
            if (j + 1 < cnt) i = next[i];      // the first one's has no meaning
        }
    }
    __syncthreads();
    for (int le = threadIdx.x / 32; le < lists; le += warps) {
        const int cnt = sh_count[le], e = sh_elem[le];
        if (cnt <= kStage) continue;
        uint32_t *lst = rv.rows + (size_t)e * rv.cap;
        if (cnt > rv.cap) {
            uint32_t *row = lst;
            lst = rv.over_list + sh_base[le];
            for (int j = lane; j < rv.cap; j += 32) lst[j] = row[j];
            __syncwarp();
            if (lane == 0) row[0] = sh_base[le];
        }
        if (cnt <= 128) {
            uint32_t q[4];
            int rank[4] = {0, 0, 0, 0};
#pragma unroll
            for (int r = 0; r < 4; r++) q[r] = lane + 32 * r < cnt ? lst[lane + 32 * r] : 0xffffffffu;
#pragma unroll
            for (int b = 0; b < 4; b++) {
                if (32 * b >= cnt) break;
#pragma unroll 8
                for (int k = 0; k < 32; k++) {
                    const uint32_t w = __shfl_sync(all, q[b], k);
#pragma unroll
                    for (int r = 0; r < 4; r++) rank[r] += w < q[r] ? 1 : 0;
                }
            }
            __syncwarp();
#pragma unroll
            for (int r = 0; r < 4; r++)
                if (lane + 32 * r < cnt) lst[rank[r]] = q[r];
        } else {
            for (long long size = 2; size < 2ll * cnt; size *= 2) {
                for (long long d = size / 2; d > 0; d /= 2) {
                    const bool flip = d == size / 2;      // the first pass of a size pairs mirrored places
                    for (long long i = lane;; i += 32) {
                        const long long a0 = i / d * (2 * d), t = i % d, a = a0 + t;
                        if (a >= cnt) break;
                        const long long b = flip ? a0 + 2 * d - 1 - t : a + d;
                        if (b >= cnt) continue;
                        const uint32_t u = lst[a], w = lst[b];
                        if (u > w) {
                            lst[a] = w;
                            lst[b] = u;
                        }
                    }
                    __syncwarp();
                }
            }
        }
        __syncwarp();
    }
}

template <int EB, int SPLIT, bool LIST>
__global__ void __launch_bounds__(EB * SPLIT) p2g_cells_kernel(
    GridGeom g, RowView rv, const uint32_t *__restrict__ filled, const uint32_t *__restrict__ n_filled,
    const uint32_t *__restrict__ head, const uint32_t *__restrict__ next, uint32_t *__restrict__ cursor,
    int keep_order, int early, const double *__restrict__ x, const double *__restrict__ y,
    const double *__restrict__ m,
    const double *__restrict__ vx, const double *__restrict__ vy, const double *__restrict__ v,
    const double *__restrict__ sxx, const double *__restrict__ sxy, const double *__restrict__ syy, StepParams *sp,
    double dt, int gravity_mode, double gravity_const, double *__restrict__ cell_sums)
{
    constexpr int NB = 17;                 // count classes 0..15 and 16 or more
    constexpr int kSumStride = kCell + 1;
    __shared__ double sh_sum[EB * kSumStride];
    __shared__ uint32_t sh_idx[kStage * EB];
    __shared__ int sh_bin[NB];
    __shared__ int sh_order[EB], sh_count[EB], sh_elem[EB];
    __shared__ uint32_t sh_base[EB];
    __shared__ double sh_const[3];         // constants as registers (mat::Unit)
    const int tid = threadIdx.x;
    if (tid == 0) {
        sh_const[0] = mat::opaque(1.0);
        sh_const[1] = mat::opaque(-0.0);
        sh_const[2] = g.inv_h;
    }
    if (tid < NB) sh_bin[tid] = 0;
    mpmg_pdl_wait();
    if (early) mpmg_pdl_trigger();
    if (blockIdx.x == 0 && tid == 0) {
        // time_varying_loads (loading.c:34-54) of the previous step's tail, or
        // initial_loads (loading.c:21-30) before the first step; then t += dt
        // (process_usl.c:522).
        double t = sp->t;
        double grav;
        if (gravity_mode == MPMG_GRAVITY_CONSTANT) {
            grav = gravity_const;
        } else if (sp->step_count == 0) {
            grav = 0.0;
        } else if ((0.1 + sp->step_start_time) > t) {
            grav = -9.8 * ((t - sp->step_start_time) / 0.1);
        } else {
            grav = -9.8;
        }
        sp->gravity = grav;
        sp->t = t + dt;
        sp->step_count += 1;
    }
    const int total = (int)*n_filled;
    const int first = blockIdx.x * EB;
    if (first >= total) return;
    int le = tid % EB;
    if (tid < EB) {
        const int e0 = first + tid < total ? (int)filled[first + tid] : -1;
        sh_elem[tid] = e0;
        sh_count[tid] = e0 >= 0 ? (int)rv.count[e0] : 0;
    }
    if (__syncthreads_or(tid < EB && sh_count[tid] > kStage)) {
        order_long_lists(rv, EB, sh_elem, sh_count, sh_base, head, next, cursor);
        __syncthreads();
    }
    constexpr int WB = EB / 32;            // warps an element set
    const int half = SPLIT == 2 ? tid / EB : 0;
    if (WB > 1) {
        // elements by descending count; this thread's: sorted warps rotated
        int cls = 0, at = 0;
        if (tid < EB) {
            cls = NB - 1 - min(sh_count[tid], NB - 1);
            at = atomicAdd(&sh_bin[cls], 1);
        }
        __syncthreads();
        if (tid < 32) {
            int c = tid < NB ? sh_bin[tid] : 0, incl = c;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const int w = __shfl_up_sync(0xffffffffu, incl, d);
                if (tid >= d) incl += w;
            }
            if (tid < NB) sh_bin[tid] = incl - c;
        }
        __syncthreads();
        if (tid < EB) sh_order[sh_bin[cls] + at] = tid;
        __syncthreads();
        le = sh_order[(((tid % EB) / 32 + (int)blockIdx.x) % WB) * 32 + (tid & 31)];
    }
    const int cnt = sh_count[le], e = sh_elem[le];
    const uint32_t *list = nullptr;        // a long element's list in global memory
    if (half == 0 && cnt > 0 && cnt <= kStage) {
        uint32_t *row = rv.rows + (size_t)e * rv.cap;
        // ascending particle index, as the reference's lists (insertion
        // sort of a handful of entries in this thread's shared column)
        uint32_t *col = sh_idx + le;
        uint4 r4[kStage / 4];              // all of the row's loads in flight
#pragma unroll
        for (int j = 0; j < kStage / 4; j++)
            if (4 * j < cnt) r4[j] = reinterpret_cast<const uint4 *>(row)[j];
#pragma unroll
        for (int j = 0; j < kStage; j++) {
            if (j >= cnt) break;
            const uint4 v4 = r4[j / 4];
            const uint32_t q = j % 4 == 0 ? v4.x : j % 4 == 1 ? v4.y : j % 4 == 2 ? v4.z : v4.w;
            int t = j - 1;
            while (t >= 0 && col[t * EB] > q) {
                col[(t + 1) * EB] = col[t * EB];
                t--;
            }
            col[(t + 1) * EB] = q;
        }
        if (keep_order)
            for (int j = 0; j < cnt; j++) row[j] = col[j * EB];
    }
    if (SPLIT == 2) __syncthreads();
    if (cnt > kStage)
        list = cnt <= rv.cap ? rv.rows + (size_t)e * rv.cap : rv.over_list + sh_base[le];
    const int ci = e % g.Ex, cj = e / g.Ex;
    const double cx = mat::small_int(ci), cy = mat::small_int(cj);   // the element's column and row (element.c:10-19)
    // moments [A, X, Y, Z] of m, m vx, m vy; stress-term moments
    double mm[4] = {0, 0, 0, 0}, mx[4] = {0, 0, 0, 0}, my[4] = {0, 0, 0, 0};
    double P0 = 0, Py0 = 0, P1 = 0, Px1 = 0, Py1 = 0, P2 = 0, Px2 = 0;
    const bool do_a = SPLIT == 1 || half == 0, do_b = SPLIT == 1 || half == 1;
    const mat::Unit u{sh_const[0], sh_const[1]};
    const double inv_h = sh_const[2];
    // integer products where the FP64 pipe is the bound, not a thread's chain
    auto prod = [&](double a, double b) { return SPLIT == 1 ? mat::imul(a, b) : u.mul(a, b); };
    // the next particle's loads are in flight during this one's arithmetic
    double nx = 0, ny = 0, nm = 0, nvx = 0, nvy = 0, nv = 0, n0 = 0, n1 = 0, n2 = 0;
    auto fetch = [&](int k) {
        const int i = (int)(list ? list[k] : sh_idx[k * EB + le]);
        nx = x[i];
        ny = y[i];
        nm = m[i];
        if (do_a) nvx = vx[i];
        if (do_b) {
            nvy = vy[i];
            nv = v[i];
            n0 = sxx[i];
            n1 = sxy[i];
            n2 = syy[i];
        }
    };
    if (cnt > 0) fetch(0);
    for (int k = 0; k < cnt; k++) {
        const double px = nx, py = ny, pm = nm, pvx = nvx, pvy = nvy, vol = nv, t0 = n0, t1 = n1, t2 = n2;
        if (k + 1 < cnt) fetch(k + 1);
        const double xl = mpmg_local_coord_fma(px, cx, inv_h);
        const double yl = mpmg_local_coord_fma(py, cy, inv_h);
        const double xy = prod(xl, yl);
        if (do_a) {
            const double pmx = prod(pvx, pm);
            mm[0] = u.add(pm, mm[0]);
            mm[1] = fma(xl, pm, mm[1]);
            mm[2] = fma(yl, pm, mm[2]);
            mm[3] = fma(xy, pm, mm[3]);
            mx[0] = u.add(pmx, mx[0]);
            mx[1] = fma(xl, pmx, mx[1]);
            mx[2] = fma(yl, pmx, mx[2]);
            mx[3] = fma(xy, pmx, mx[3]);
        }
        if (do_b) {
            const double pmy = prod(pvy, pm);
            const double vlx = prod(vol, xl), vly = prod(vol, yl);
            my[0] = u.add(pmy, my[0]);
            my[1] = fma(xl, pmy, my[1]);
            my[2] = fma(yl, pmy, my[2]);
            my[3] = fma(xy, pmy, my[3]);
            P0 = fma(t0, vol, P0);
            Py0 = fma(t0, vly, Py0);
            P1 = fma(t1, vol, P1);
            Px1 = fma(t1, vlx, Px1);
            Py1 = fma(t1, vly, Py1);
            P2 = fma(t2, vol, P2);
            Px2 = fma(t2, vlx, Px2);
        }
    }
    // corners BL, BR, TR, TL (process_usl.c:140-143); an element's sums leave
    // as one run through shared memory
    double *out = sh_sum + le * kSumStride;
    if (do_a && cnt > 0) {
        const double dm = u.sub(mm[2], mm[3]), dx = u.sub(mx[2], mx[3]);
        out[0] = u.sub(u.sub(mm[0], mm[1]), dm);
        out[4] = u.sub(mm[1], mm[3]);
        out[8] = mm[3];
        out[12] = dm;
        out[1] = u.sub(u.sub(mx[0], mx[1]), dx);
        out[5] = u.sub(mx[1], mx[3]);
        out[9] = mx[3];
        out[13] = dx;
    }
    if (do_b && cnt > 0) {
        const double dy = u.sub(my[2], my[3]);
        out[2] = u.sub(u.sub(my[0], my[1]), dy);
        out[6] = u.sub(my[1], my[3]);
        out[10] = my[3];
        out[14] = dy;
        // h times the internal force, -V T grad N
        const double a0 = u.sub(P0, Py0), a1 = u.sub(P1, Px1), b1 = u.sub(P1, Py1), b2 = u.sub(P2, Px2);
        out[3] = u.add(a0, a1);
        out[7] = u.sub(Px1, a0);
        out[11] = -u.add(Py0, Px1);
        out[15] = u.sub(Py0, a1);
        out[16] = u.add(b1, b2);
        out[17] = u.sub(Px2, b1);
        out[18] = -u.add(Py1, Px2);
        out[19] = u.sub(Py1, b2);
    }
    __syncthreads();
    const int here = min(EB, total - first);
    for (int q = tid; q < kCell * here; q += EB * SPLIT) {
        const int l = q / kCell, f = q - l * kCell;
        cell_sums[(size_t)(LIST ? first + l : sh_elem[l]) * kCell + f] = sh_sum[l * kSumStride + f];
    }
    mpmg_pdl_trigger();
}

// ---------------------------------------------------------------------------
// grid: finish P2G per node, boundary conditions, nodal update; then per
// element the bilinear coefficients of the nodal fields.
//
// A block of 32 x TY threads finishes a tile of 32 x TY nodes (tiles share one
// column and row of nodes, computed by both to the same bits and stored by
// one) and then the elements between them.  With node values q0..q3
// (BL, BR, TR, TL) the field on the element is
// c0 + c1 x + c2 y + c3 xy, c0 = q0, c1 = q1 - q0, c2 = q3 - q0,
// c3 = (q2 - q3) - c1: four FP64 operations per element and field here save
// the G2P about six per particle, and an element's sixteen doubles are one
// 128-byte line for its gathers instead of sixteen loads from eight lines.
// Flat tiles: TY = 4 recomputes 39 % of the nodes (16: 10 %), but a block is one
// warp a sub-partition, and a sparse grid's filled tiles spread over all SMs
// (125k particles on 261k nodes: 54.0 us a step, 56.3 with TY = 8, 58.2 with 16;
// 1 048 576 particles on 263k: 253.3, 252.3, 253.8).  Narrow grids take 8 x 16
// (launch_grid).

// The corner (BL, BR, TR, TL) that node (i, j) is of its colour-c element.
__device__ __forceinline__ int c_corner(int c, int i, int j)
{
    const bool right = (i & 1) == (c & 1), up = (j & 1) == (c >> 1);   // the element lies right of, above the node
    return right ? (up ? 0 : 3) : (up ? 1 : 2);
}

template <int TX, int TY, bool LIST>
__global__ void __launch_bounds__(TX * TY) grid_kernel(
    GridGeom g, BcParams bc, int tiles_x, const uint32_t *__restrict__ count, const uint32_t *__restrict__ pos,
    uint32_t *__restrict__ count_next,
    uint32_t *__restrict__ n_filled_next, uint32_t *__restrict__ cursor,
    const double *__restrict__ cell_sums, const StepParams *__restrict__ sp, double dt,
    double *__restrict__ node_m, double *__restrict__ node_ax, double *__restrict__ node_ay,
    double *__restrict__ node_vx, double *__restrict__ node_vy, double *__restrict__ node_mx,
    double *__restrict__ node_my, double *__restrict__ node_fx, double *__restrict__ node_fy,
    double2 *__restrict__ coef, int early)
{
    __shared__ double sh[4][TY][TX];
    __shared__ double sh_const[4];         // constants as registers (mat::Unit)
    if (threadIdx.x == 0) {
        sh_const[0] = mat::opaque(1.0);
        sh_const[1] = mat::opaque(-0.0);
        sh_const[2] = g.inv_h;
        sh_const[3] = dt;
    }
    const int tx = threadIdx.x % TX, ty = threadIdx.x / TX;
    const int i = (int)(blockIdx.x % tiles_x) * (TX - 1) + tx, j = (int)(blockIdx.x / tiles_x) * (TY - 1) + ty;
    const bool node = i < g.Nx && j < g.Ny;
    // Colour c = 2 * (row % 2) + (col % 2) (process_usl.c:158); the four
    // elements around a node have the four colours, summed in order 0..3.
    // The counts are the previous step's work: read before the wait.
    const double *src[4];
    bool filled = false;                   // the element whose BL node this is holds particles
    uint32_t place = 0;                    // its place on the list
    if (node) {
#pragma unroll
        for (int c = 0; c < 4; c++) {
            src[c] = nullptr;
            const int ci = ((i & 1) == (c & 1)) ? i : i - 1;
            const int cj = ((j & 1) == (c >> 1)) ? j : j - 1;
            if (ci < 0 || cj < 0 || ci >= g.Ex || cj >= g.Ey) continue;
            const int e = cj * g.Ex + ci;
            if (count[e] == 0) continue;
            const uint32_t at = LIST ? pos[e] : (uint32_t)e;
            const int corner = c_corner(c, i, j);
            if (corner == 0) {
                filled = true;
                place = at;
            }
            src[c] = cell_sums + (size_t)at * kCell + corner * 4;
        }
    }
    const bool own = node && (tx < TX - 1 || i == g.Nx - 1) && (ty < TY - 1 || j == g.Ny - 1);
    mpmg_pdl_wait();
    if (early) mpmg_pdl_trigger();
    __syncthreads();
    const mat::Unit u{sh_const[0], sh_const[1]};
    // the next step's rows start empty (the G2P fills them)
    if (own && i < g.Ex && j < g.Ey) count_next[j * g.Ex + i] = 0;
    if (blockIdx.x == 0 && threadIdx.x == 0) *n_filled_next = *cursor = 0;
    double ax = 0, ay = 0, vxn = 0, vyn = 0;
    double m = 0, mx = 0, my = 0, fx = 0, fy = 0;
    if (node && (src[0] || src[1] || src[2] || src[3])) {
        double sum[5] = {0, 0, 0, 0, 0};
        // a corner's m, mx, my, h fx as two loads, and its h fy (16 - 3 corner
        // doubles further on)
        double2 q0[4], q1[4];
        double q2[4];
#pragma unroll
        for (int c = 0; c < 4; c++) {
            if (src[c] == nullptr) continue;
            q0[c] = *reinterpret_cast<const double2 *>(src[c]);
            q1[c] = *reinterpret_cast<const double2 *>(src[c] + 2);
            const int corner = c_corner(c, i, j);
            q2[c] = src[c][16 - 3 * corner];
        }
        if (src[0] && src[1] && src[2] && src[3]) {
            sum[0] = u.add(u.add(u.add(q0[0].x, q0[1].x), q0[2].x), q0[3].x);
            sum[1] = u.add(u.add(u.add(q0[0].y, q0[1].y), q0[2].y), q0[3].y);
            sum[2] = u.add(u.add(u.add(q1[0].x, q1[1].x), q1[2].x), q1[3].x);
            sum[3] = u.add(u.add(u.add(q1[0].y, q1[1].y), q1[2].y), q1[3].y);
            sum[4] = u.add(u.add(u.add(q2[0], q2[1]), q2[2]), q2[3]);
        } else {
#pragma unroll
            for (int c = 0; c < 4; c++) {
                if (src[c] == nullptr) continue;
                sum[0] = u.add(sum[0], q0[c].x);
                sum[1] = u.add(sum[1], q0[c].y);
                sum[2] = u.add(sum[2], q1[c].x);
                sum[3] = u.add(sum[3], q1[c].y);
                sum[4] = u.add(sum[4], q2[c]);
            }
        }
        m = sum[0];
        mx = sum[1];
        my = sum[2];
        // body force bx is zero (loading.c:48); by = g acts on the node's mass
        const double inv_h = sh_const[2], dtr = sh_const[3];
        fx = u.mul(sum[3], inv_h);
        fy = fma(sp->gravity, m, u.mul(sum[4], inv_h));
        bool bx, by;
        bc_mask(bc, g, i, j, sp->t, bx, by);
        if (bx) { mx = 0; fx = 0; }
        if (by) { my = 0; fy = 0; }
        // m > MPMG_TOL on the bit patterns
        if (__double_as_longlong(m) > __double_as_longlong(MPMG_TOL) && !mat::is_nan(m)) {
            // one division: the four quotients by m differ from IEEE division
            // by at most an ulp
            const double inv_m = mat::quot(u.one, m);
            ax = u.mul(fx, inv_m);
            ay = u.mul(fy, inv_m);
            mx = fma(dtr, fx, mx);
            my = fma(dtr, fy, my);
            vxn = u.mul(mx, inv_m);
            vyn = u.mul(my, inv_m);
        }
    }
    if (own) {
        const int n = j * g.Nx + i;
        node_m[n] = m;
        node_ax[n] = ax;
        node_ay[n] = ay;
        node_vx[n] = vxn;
        node_vy[n] = vyn;
        if (node_mx != nullptr) {
            node_mx[n] = mx;
            node_my[n] = my;
            node_fx[n] = fx;
            node_fy[n] = fy;
        }
    }
    sh[0][ty][tx] = ax;
    sh[1][ty][tx] = ay;
    sh[2][ty][tx] = vxn;
    sh[3][ty][tx] = vyn;
    __syncthreads();
    if (filled && tx < TX - 1 && ty < TY - 1) {
        double2 *out = coef + (size_t)place * 8;
#pragma unroll
        for (int f = 0; f < 4; f++) {
            const double q0 = sh[f][ty][tx], q1 = sh[f][ty][tx + 1], q2 = sh[f][ty + 1][tx + 1], q3 = sh[f][ty + 1][tx];
            const double c1 = u.sub(q1, q0);
            out[2 * f] = make_double2(q0, c1);
            out[2 * f + 1] = make_double2(u.sub(q3, q0), u.sub(u.sub(q2, q3), c1));
        }
    }
    mpmg_pdl_trigger();
}

template <int TX, int TY>
cudaError_t launch_grid_t(mpmg_ctx *ctx, const GridGeom &g)
{
    const RowBins &r = ctx->row;
    const int tiles_x = (g.Nx + TX - 2) / (TX - 1), tiles_y = (g.Ny + TY - 2) / (TY - 1);
    return mpmg_launch_pdl(true, r.pos[0] != nullptr ? grid_kernel<TX, TY, true> : grid_kernel<TX, TY, false>,
                           dim3(tiles_x * tiles_y), dim3(TX * TY), 0, ctx->stream, g,
                           make_bc(ctx), tiles_x, (const uint32_t *)r.count[r.cur], (const uint32_t *)r.pos[r.cur],
                           r.count[1 - r.cur],
                           r.n_filled + (1 - r.cur), r.cursor, (const double *)ctx->cell_sums,
                           (const StepParams *)ctx->d_params, ctx->cfg.dt,
                           ctx->node_m, ctx->node_ax, ctx->node_ay, ctx->node_vx, ctx->node_vy, ctx->node_mx,
                           ctx->node_my, ctx->node_fx, ctx->node_fy, (double2 *)ctx->elem_coef, early_launch(ctx));
}

// Tiles of 8 x 16 nodes on a grid of up to 8 columns, where rows of 32 are
// mostly idle (3 x 20001 nodes: 62 us a step, 126 with rows).
cudaError_t launch_grid(mpmg_ctx *ctx, const GridGeom &g)
{
    return g.Nx <= 8 ? launch_grid_t<8, 16>(ctx, g) : launch_grid_t<32, 4>(ctx, g);
}

// ---------------------------------------------------------------------------
// g2p + material

// The arithmetic's constants, copied to shared memory (mat::Unit).
struct G2PConst {
    mat::SoftElastic el;
    mat::Mu2Params mu2;
    double inv_h, half_inv_h;
};

struct G2PArgs {
    GridGeom g;
    int n;
    int early;
    G2PConst k;
    mat::NonlocalParams nl;
    uint32_t *keys;        // element of this step in, of the next step out (sentinel: none)
    uint32_t sentinel;
    float inv_hf;
    RowsOut next;          // the next step's rows
    int *in_element;
    int *active;
    const double2 *coef;   // element coefficients (grid_kernel) at their places (pos)
    const double *node_vx, *node_vy;
    double *x, *y, *vx, *vy, *ux, *uy, *v, *m;
    double *sxx, *sxy, *syy, *Tzz;
    double *st0, *st1, *st3, *st4, *st5, *st6, *st9, *st10;
    double *ax, *ay, *exx, *exy, *eyy, *wxy, *xl_out, *yl_out;
    // g_nonlocal_mu2: the trial stress the stress update reads after the
    // fluidity solve, 5 per particle, value-major (p_d, t0xx, t0xy, t0yy, tau)
    double *trial;
    const uint32_t *pos;   // places of the filled elements (RowBins::pos)
};

// G2P phases.  USL (process_usl.c:465-592) runs them all in one pass; MUSL
// (process_usl.c:284-462) runs the move first, maps the moved particles'
// momentum to the nodes again (p2g_momentum_kernel, node_velocity_kernel),
// then the strain phase with the nodal velocities of that second projection.
enum { G2P_FULL = 0, G2P_MOVE = 1, G2P_STRAIN = 2 };

// A particle's state in registers, loaded before the kernel waits for the grid
// update (all of it is the previous step's work, or the move phase's).
struct Particle {
    double x, y, vx, vy, ux, uy, v, m, sxx, sxy, syy, Tzz, st1, st5, st9, st10, st0, xl, yl;
};

template <int MATERIAL, int PHASE>
__device__ __forceinline__ Particle load_particle(const G2PArgs &A, int i)
{
    Particle p = {};
    p.x = A.x[i];
    p.y = A.y[i];
    if (PHASE != G2P_STRAIN) {
        p.vx = A.vx[i];
        p.vy = A.vy[i];
        p.ux = A.ux[i];
        p.uy = A.uy[i];
    } else {
        // the start-of-step local coordinates the move phase kept
        p.xl = A.xl_out[i];
        p.yl = A.yl_out[i];
    }
    if (PHASE == G2P_MOVE) return p;
    p.v = A.v[i];
    if (MATERIAL != MPMG_G_NONLOCAL) {
        p.sxx = A.sxx[i];
        p.sxy = A.sxy[i];
        p.syy = A.syy[i];
    }
    if (MATERIAL != MPMG_ISOLIN && MATERIAL != MPMG_G_NONLOCAL) p.m = A.m[i];
    if (MATERIAL == MPMG_G_LOCAL_MU2) p.Tzz = A.Tzz[i];
    if (MATERIAL == MPMG_DP_RI_MT || MATERIAL == MPMG_G_LOCAL_MU2_PLANE_STRAIN) p.st1 = A.st1[i];
    if (MATERIAL == MPMG_G_LOCAL_MU2_PLANE_STRAIN || MATERIAL == MPMG_G_LOCAL_MU2_TRUE_2D ||
        MATERIAL == MPMG_G_LOCAL_MU2_REVERSE)
        p.st5 = A.st5[i];
    if (MATERIAL != MPMG_ISOLIN && MATERIAL != MPMG_G_NONLOCAL && MATERIAL != MPMG_G_NONLOCAL_MU2 &&
        MATERIAL != MPMG_G_LOCAL_MU2_EXT)
        p.st9 = A.st9[i];
    if (MATERIAL == MPMG_G_LOCAL_MU2_REVERSE || MATERIAL == MPMG_G_LOCAL_MU2_EXT) p.st10 = A.st10[i];
    if (MATERIAL == MPMG_G_LOCAL_MU2_EXT) p.st0 = A.st0[i];
    return p;
}

// The in-plane local returns on particle i (mat::plane_return): szz in
// state[1] (dp_ri_mt.c:27, g_local_mu2_plane_strain.c:43), beta in state[5],
// gammap in state[9], gammadotp in state[10].
template <class E, int MATERIAL>
__device__ __forceinline__ void plane_return_particle(const G2PArgs &A, const G2PConst &C, int i, const Particle &p,
                                                      double vol, double exx, double exy, double eyy, double wxy)
{
    constexpr bool trial3d = MATERIAL != MPMG_G_LOCAL_MU2_TRUE_2D;
    constexpr bool mu_i = MATERIAL != MPMG_DP_RI_MT;
    constexpr bool beta = MATERIAL != MPMG_DP_RI_MT;
    const mat::ReturnParams rp = {C.mu2.mu_s, C.mu2.mu_2, C.mu2.I0, C.mu2.grains_rho, C.mu2.grains_d,
                                  C.mu2.rho_critical};
    double sxx = p.sxx, sxy = p.sxy, syy = p.syy, szz = p.st1, b = p.st5, gp = p.st9, gdp;
    mat::plane_return<trial3d, mu_i, beta>(static_cast<const E &>(C.el), rp, p.m, vol, exx, exy, eyy, wxy, sxx, sxy, syy, szz, b, gp, gdp);
    A.sxx[i] = sxx;
    A.sxy[i] = sxy;
    A.syy[i] = syy;
    if (trial3d) A.st1[i] = szz;
    if (beta) A.st5[i] = b;
    A.st9[i] = gp;
    A.st10[i] = gdp;
}

// g_local_mu2_reverse on particle i: beta in state[5], gammap in state[9],
// gammadotp in state[10] (g_local_mu2_reverse.c:57-64).
template <class E>
__device__ __forceinline__ void reverse_particle(const G2PArgs &A, const G2PConst &C, int i, const Particle &p,
                                                 double vol, double exx, double exy, double eyy, double wxy)
{
    double sxx = p.sxx, sxy = p.sxy, syy = p.syy, b = p.st5, gp = p.st9, gdp = p.st10;
    mat::g_local_mu2_reverse(static_cast<const E &>(C.el), C.mu2, p.m, vol, exx, exy, eyy, wxy, sxx, sxy, syy, b, gp, gdp);
    A.sxx[i] = sxx;
    A.sxy[i] = sxy;
    A.syy[i] = syy;
    A.st5[i] = b;
    A.st9[i] = gp;
    A.st10[i] = gdp;
}

template <class E>
__device__ __forceinline__ void isolin_particle(const G2PArgs &A, const G2PConst &C, int i, const Particle &p,
                                                double exx, double exy, double eyy, double wxy)
{
    double sxx = p.sxx, sxy = p.sxy, syy = p.syy;
    mat::isolin(static_cast<const E &>(C.el), exx, exy, eyy, wxy, sxx, sxy, syy);
    A.sxx[i] = sxx;
    A.sxy[i] = sxy;
    A.syy[i] = syy;
}

template <class E>
__device__ __forceinline__ void mu2_particle(const G2PArgs &A, const G2PConst &C, int i, const Particle &p, double vol,
                                             double exx, double eyy, double d2, double w2)
{
    double Txx = p.sxx, Txy = p.sxy, Tyy = p.syy, Tzz = p.Tzz, gp = p.st9, gdp;
    mat::g_local_mu2(static_cast<const E &>(C.el), C.mu2, p.m, vol, exx, eyy, d2, w2, Txx, Txy, Tyy, Tzz, gp, gdp);
    A.sxx[i] = Txx;
    A.sxy[i] = Txy;
    A.syy[i] = Tyy;
    A.Tzz[i] = Tzz;
    A.st9[i] = gp;
    A.st10[i] = gdp;
}

// A field on an element from its coefficients: value at (x, y), and h times
// its gradient.
struct Field {
    double val, gx, gy;
};
__device__ __forceinline__ Field field_at(double2 c01, double2 c23, double x, double y)
{
    Field f;
    f.gy = fma(x, c23.y, c23.x);
    f.val = fma(y, f.gy, fma(x, c01.y, c01.x));
    f.gx = fma(y, c23.y, c01.y);
    return f;
}

// One particle inside the grid, element e (its sums at `place`) at the step's
// start; p.x, p.y leave as the moved position.
template <class E, int MATERIAL, int PHASE>
__device__ __forceinline__ void g2p_particle(const G2PArgs &A, const G2PConst &C, int i, int e, uint32_t place,
                                             Particle &p)
{
    const GridGeom &g = A.g;
    const E &u = C.el;
    const int cj = e / g.Ex, ci = e - cj * g.Ex;
    const double dt = C.el.dt, inv_h = C.inv_h;
    Field vx, vy;
    if (PHASE == G2P_STRAIN) {
        // the nodal velocities of the second projection: h grad N is
        // ((-oy, -ox), (oy, -x), (y, x), (-y, ox)), grouped by node differences
        const int n0 = cj * g.Nx + ci;
        const int nd[4] = {n0, n0 + 1, n0 + 1 + g.Nx, n0 + g.Nx};
        double nvx[4], nvy[4];
#pragma unroll
        for (int a = 0; a < 4; a++) {
            nvx[a] = A.node_vx[nd[a]];
            nvy[a] = A.node_vy[nd[a]];
        }
        const double ox = u.sub(u.one, p.xl), oy = u.sub(u.one, p.yl);
        vx.gx = fma(oy, u.sub(nvx[1], nvx[0]), u.mul(p.yl, u.sub(nvx[2], nvx[3])));
        vy.gx = fma(oy, u.sub(nvy[1], nvy[0]), u.mul(p.yl, u.sub(nvy[2], nvy[3])));
        vx.gy = fma(ox, u.sub(nvx[3], nvx[0]), u.mul(p.xl, u.sub(nvx[2], nvx[1])));
        vy.gy = fma(ox, u.sub(nvy[3], nvy[0]), u.mul(p.xl, u.sub(nvy[2], nvy[1])));
    } else {
        const double xl = mpmg_local_coord_fma(p.x, mat::small_int(ci), inv_h);
        const double yl = mpmg_local_coord_fma(p.y, mat::small_int(cj), inv_h);
        const double2 *c = A.coef + (size_t)place * 8;
        vx = field_at(c[4], c[5], xl, yl);
        vy = field_at(c[6], c[7], xl, yl);
        // move_particles_explicit_usl_split (process_usl.c:914-957); light
        // nodes (m <= 1e-10) carry zero acceleration and velocity.
        const double xtt = field_at(c[0], c[1], xl, yl).val, ytt = field_at(c[2], c[3], xl, yl).val;
        p.x = fma(dt, vx.val, p.x);
        p.y = fma(dt, vy.val, p.y);
        A.vx[i] = fma(dt, xtt, p.vx);
        A.vy[i] = fma(dt, ytt, p.vy);
        A.x[i] = p.x;
        A.y[i] = p.y;
        A.ux[i] = fma(dt, vx.val, p.ux);
        A.uy[i] = fma(dt, vy.val, p.uy);
        if (A.ax != nullptr) {
            A.ax[i] = xtt;
            A.ay[i] = ytt;
        }
        if (A.xl_out != nullptr) {
            A.xl_out[i] = xl;
            A.yl_out[i] = yl;
        }
        if (PHASE == G2P_MOVE) return;
    }
    // calculate_strainrate_split (process_usl.c:796-803): the sums of
    // grad N_a v_a, scaled by 1 / h once
    const double exx = u.mul(vx.gx, inv_h), eyy = u.mul(vy.gy, inv_h);
    const double gsum = u.add(vx.gy, vy.gx), gdiff = u.sub(vx.gy, vy.gx);
    double exy = 0, wxy = 0;
    if (MATERIAL != MPMG_G_LOCAL_MU2 || A.exx != nullptr) {
        exy = u.mul(C.half_inv_h, gsum);
        wxy = u.mul(C.half_inv_h, gdiff);
    }
    // update_particle_densities_split (process_usl.c:961-970)
    const double vol = u.mul(p.v, mat::exp_small(u.mul(dt, u.add(exx, eyy))));
    A.v[i] = vol;
    if (A.exx != nullptr) {
        A.exx[i] = exx;
        A.exy[i] = exy;
        A.eyy[i] = eyy;
        A.wxy[i] = wxy;
    }

    if (MATERIAL == MPMG_ISOLIN) {
        isolin_particle<E>(A, C, i, p, exx, exy, eyy, wxy);
    } else if (MATERIAL == MPMG_G_LOCAL_MU2) {
        mu2_particle<E>(A, C, i, p, vol, exx, eyy, u.mul(inv_h, gsum), u.mul(inv_h, gdiff));
    } else if (MATERIAL == MPMG_DP_RI_MT || MATERIAL == MPMG_G_LOCAL_MU2_PLANE_STRAIN ||
               MATERIAL == MPMG_G_LOCAL_MU2_TRUE_2D) {
        plane_return_particle<E, MATERIAL>(A, C, i, p, vol, exx, exy, eyy, wxy);
    } else if (MATERIAL == MPMG_G_LOCAL_MU2_REVERSE) {
        reverse_particle<E>(A, C, i, p, vol, exx, exy, eyy, wxy);
    } else if (MATERIAL == MPMG_G_LOCAL_MU2_EXT) {
        // first phase only; the stress waits for the nodal Laplacian
        double mu_t = p.st0, gfl;
        mat::ext_local_fluidity(C.mu2, p.sxx, p.syy, p.st10, mu_t, gfl);
        A.st0[i] = mu_t;
        A.st4[i] = gfl;
    } else if (MATERIAL == MPMG_G_NONLOCAL_MU2) {
        double p_tr, t0xx, t0xy, t0yy, tau_tr, dense, gfl, xisq;
        mat::nonlocal_mu2_trial(u, exx, exy, eyy, wxy, p.sxx, p.sxy, p.syy, p_tr, t0xx, t0xy, t0yy, tau_tr);
        mat::nonlocal_mu2_bulk(u, C.mu2, p.m, vol, p_tr, tau_tr, dense, gfl, xisq);
        A.st0[i] = dense;
        A.st5[i] = gfl;
        A.st6[i] = xisq;
        const size_t n = (size_t)A.n;
        A.trial[i] = dense != 0 ? p_tr : 0.0;
        A.trial[n + i] = t0xx;
        A.trial[2 * n + i] = t0xy;
        A.trial[3 * n + i] = t0yy;
        A.trial[4 * n + i] = tau_tr;
    }
    // MPMG_G_NONLOCAL computes its bulk fluidity over every particle in the
    // fluidity phase (g_nonlocal.c:306-352).
}

// Copies the constants to shared memory (the caller synchronises).
__device__ __forceinline__ void stage_const(G2PConst &C, const G2PConst &param)
{
    static_assert(sizeof(G2PConst) % 8 == 0, "copied as 64-bit words");
    const unsigned long long *src = reinterpret_cast<const unsigned long long *>(&param);
    unsigned long long *dst = reinterpret_cast<unsigned long long *>(&C);
    for (int k = threadIdx.x; k < (int)(sizeof(G2PConst) / 8); k += blockDim.x) dst[k] = src[k];
}

// The block's size and E are the launch's (g2p_pipe_bound).  Every thread stays to the
// end: the binning is a warp's work.
template <class E, int MATERIAL, int PHASE, bool LIST>
__global__ void __launch_bounds__(128) g2p_kernel(const __grid_constant__ G2PArgs A)
{
    __shared__ G2PConst C;
    stage_const(C, A.k);
    const GridGeom &g = A.g;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t key = i < A.n ? A.keys[i] : A.sentinel;
    Particle p;
    uint32_t place = 0;
    if (key != A.sentinel) {
        place = LIST ? A.pos[key] : key;
        p = load_particle<MATERIAL, PHASE>(A, i);
    }
    __syncthreads();
    mpmg_pdl_wait();
    if (A.early) mpmg_pdl_trigger();
    uint32_t next = A.sentinel;
    if (key != A.sentinel) {
        if (PHASE != G2P_STRAIN) A.in_element[i] = (int)key;
        g2p_particle<E, MATERIAL, PHASE>(A, C, i, (int)key, place, p);
        if (PHASE != G2P_MOVE) {
            const int e = mpmg_which_element_fast(p.x, p.y, g.h, g.inv_h, A.inv_hf, g.xmax, g.ymax,
                                                  __double_as_longlong(g.xmax), __double_as_longlong(g.ymax), g.Ex,
                                                  g.Ey);
            if (e >= 0) next = (uint32_t)e;
            A.keys[i] = next;
        }
    } else if (PHASE != G2P_STRAIN && i < A.n && A.active[i]) {
        A.active[i] = 0;       // process_usl.c:660-666: outside the grid for good
        A.in_element[i] = -1;
    }
    if (PHASE != G2P_MOVE) bin_particle(A.next, i, next, next != A.sentinel);
    mpmg_pdl_trigger();
}

// g_local_mu2_ext's second phase (g_local_mu2_ext.c:232-265): per element,
// each particle's -v gflocal |grad N_j|^2 summed per corner in the binned
// order of the step, with the start-of-step shape-function gradients.
__global__ void __launch_bounds__(128) ext_cells_kernel(
    int ne, double inv_h, RowView rv, const uint32_t *__restrict__ pos,
    const double *__restrict__ xl, const double *__restrict__ yl, const double *__restrict__ v,
    const double *__restrict__ gflocal, double *__restrict__ cell_sums)
{
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= ne) return;
    const int cnt = (int)rv.count[e];
    if (cnt == 0) return;
    const uint32_t *list = rv.list(e, cnt);
    double *out = pos != nullptr ? cell_sums + (size_t)pos[e] * 4 : cell_sums + e;
    const size_t step = pos != nullptr ? 1 : (size_t)ne;
    double acc[4] = {0, 0, 0, 0};
    for (int k = 0; k < cnt; k++) {
        const int i = (int)list[k];
        const ShapeFns f = shape(xl[i], yl[i], inv_h);
        const double q = mat::mul(-v[i], gflocal[i]);
#pragma unroll
        for (int a = 0; a < 4; a++) {
            const double sj = mat::add(mat::mul(f.gx[a], f.gx[a]), mat::mul(f.gy[a], f.gy[a]));
            acc[a] = mat::add(acc[a], mat::mul(q, sj));
        }
    }
#pragma unroll
    for (int a = 0; a < 4; a++) out[a * step] = acc[a];
}

// The nodal sums of ext_cells_kernel's corners in colour order.
__global__ void __launch_bounds__(256) ext_nodes_kernel(GridGeom g, int ne, const uint32_t *__restrict__ count,
                                                        const uint32_t *__restrict__ pos, const double *__restrict__ cell_sums,
                                                        double *__restrict__ d2)
{
    const int nn = g.Nx * g.Ny;
    const int n = blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= nn) return;
    const int i = n % g.Nx, j = n / g.Nx;
    double sum = 0;
#pragma unroll
    for (int c = 0; c < 4; c++) {
        const int ci = ((i & 1) == (c & 1)) ? i : i - 1;
        const int cj = ((j & 1) == (c >> 1)) ? j : j - 1;
        if (ci < 0 || cj < 0 || ci >= g.Ex || cj >= g.Ey) continue;
        const int e = cj * g.Ex + ci;
        if (count[e] == 0) continue;
        const int corner = (ci == i) ? ((cj == j) ? 0 : 3) : ((cj == j) ? 1 : 2);
        sum = mat::add(sum, cell_sums[pos != nullptr ? (size_t)pos[e] * 4 + corner : (size_t)corner * ne + e]);
    }
    d2[n] = sum;
}

// g_local_mu2_ext's gf and gammadotp correction (g_local_mu2_ext.c:268-290)
// and the stress (mat::ext_stress).
__global__ void __launch_bounds__(256) ext_stress_kernel(const __grid_constant__ G2PArgs A,
                                                         const double *__restrict__ d2)
{
    const G2PConst &C = A.k;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= A.n || !A.active[i]) return;
    const GridGeom &g = A.g;
    const int e = A.in_element[i];
    const int ci = e % g.Ex, cj = e / g.Ex;
    const int n0 = cj * g.Nx + ci;
    const int nd[4] = {n0, n0 + 1, n0 + 1 + g.Nx, n0 + g.Nx};
    double gf = 0;
#pragma unroll
    for (int a = 0; a < 4; a++) gf = mat::add(gf, mat::mul(0.25, d2[nd[a]]));
    double mu_t = A.st0[i], gdp = A.st10[i];
    const double Ad = C.mu2.A, d = C.mu2.grains_d;
    gf = mat::mul(mat::mul(mat::mul(mat::mul(mat::mul(Ad, Ad), d), d), mu_t), gf);
    if (mu_t > C.mu2.mu_s) gdp = mat::sub(gdp, mat::quot(gf, fabs(mat::sub(mu_t, C.mu2.mu_s))));
    if (gdp < 0) gdp = 0;
    A.st3[i] = gf;
    double sxx = A.sxx[i], sxy = A.sxy[i], syy = A.syy[i], beta = A.st5[i], gp = A.st9[i];
    mat::ext_stress(C.el, C.mu2, A.nl.E, A.nl.nu, A.m[i], A.v[i], A.exx[i], A.exy[i], A.eyy[i], A.wxy[i], sxx, sxy,
                    syy, mu_t, beta, gp, gdp);
    A.sxx[i] = sxx;
    A.sxy[i] = sxy;
    A.syy[i] = syy;
    A.st0[i] = mu_t;
    A.st5[i] = beta;
    A.st9[i] = gp;
    A.st10[i] = gdp;
}

// MUSL's second projection (process_usl.c:424-431): per element, the moved
// particles' mass and momentum with their start-of-step shape functions, in
// the step's particle order, from the same moments as the P2G.
template <bool LIST>
__global__ void __launch_bounds__(128) p2g_momentum_kernel(
    int ne, RowView rv, const uint32_t *__restrict__ pos, const double *__restrict__ xl,
    const double *__restrict__ yl, const double *__restrict__ m, const double *__restrict__ vx, const double *__restrict__ vy,
    double *__restrict__ cell_sums)
{
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    // The counts are the previous step's work.  A warp of empty elements leaves
    // without waiting; block 0 waits always, so that this kernel ends after the
    // one before it (4000 particles on 2048^2 elements: 187 us a step, 206 with a
    // wait in every warp).
    const int cnt = e < ne ? (int)rv.count[e] : 0;
    if (!__any_sync(0xffffffffu, cnt != 0) && blockIdx.x != 0) return;
    mpmg_pdl_wait();
    mpmg_pdl_trigger();
    if (cnt == 0) return;
    const uint32_t *list = rv.list(e, cnt);
    // by element value-major, by list a run a place (they come in no order)
    double *out = LIST ? cell_sums + (size_t)pos[e] * 12 : cell_sums + e;
    const size_t step = LIST ? 1 : (size_t)ne;
    double q[3][4];
#pragma unroll
    for (int f = 0; f < 3; f++)
#pragma unroll
        for (int a = 0; a < 4; a++) q[f][a] = 0.0;
    for (int k = 0; k < cnt; k++) {
        const int i = (int)list[k];
        const double a = xl[i], b = yl[i], ab = a * b;
        const double pm = m[i], p[3] = {pm, vx[i] * pm, vy[i] * pm};
#pragma unroll
        for (int f = 0; f < 3; f++) {
            q[f][0] += p[f];
            q[f][1] = fma(a, p[f], q[f][1]);
            q[f][2] = fma(b, p[f], q[f][2]);
            q[f][3] = fma(ab, p[f], q[f][3]);
        }
    }
#pragma unroll
    for (int f = 0; f < 3; f++) {
        out[(0 * 3 + f) * step] = (q[f][0] - q[f][1]) - (q[f][2] - q[f][3]);
        out[(1 * 3 + f) * step] = q[f][1] - q[f][3];
        out[(2 * 3 + f) * step] = q[f][3];
        out[(3 * 3 + f) * step] = q[f][2] - q[f][3];
    }
}

// MUSL nodal velocities of the second projection (process_usl.c:433-447):
// v = p / m where m > 1e-10, else 0.  The reference zeroes the constrained
// momenta only after forming v, so the boundary conditions do not reach v;
// the zeroed momenta are what it keeps in the nodes (node_mx, node_my).
template <bool LIST>
__global__ void __launch_bounds__(256) node_velocity_kernel(
    GridGeom g, BcParams bc, int ne, const uint32_t *__restrict__ count, const uint32_t *__restrict__ pos,
    const double *__restrict__ cell_sums,
    const StepParams *__restrict__ sp, double *__restrict__ node_m, double *__restrict__ node_vx,
    double *__restrict__ node_vy, double *__restrict__ node_mx, double *__restrict__ node_my)
{
    mpmg_pdl_wait();
    mpmg_pdl_trigger();
    const int nn = g.Nx * g.Ny;
    const int n = blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= nn) return;
    const int i = n % g.Nx, j = n / g.Nx;
    double sum[3] = {0, 0, 0};
#pragma unroll
    for (int c = 0; c < 4; c++) {
        const int ci = ((i & 1) == (c & 1)) ? i : i - 1;
        const int cj = ((j & 1) == (c >> 1)) ? j : j - 1;
        if (ci < 0 || cj < 0 || ci >= g.Ex || cj >= g.Ey) continue;
        const int e = cj * g.Ex + ci;
        if (count[e] == 0) continue;
        const int corner = (ci == i) ? ((cj == j) ? 0 : 3) : ((cj == j) ? 1 : 2);
        const double *src = LIST ? cell_sums + (size_t)pos[e] * 12 + corner * 3 : cell_sums + (size_t)(corner * 3) * ne + e;
#pragma unroll
        for (int q = 0; q < 3; q++) sum[q] += src[LIST ? q : (size_t)q * ne];
    }
    const double m = sum[0];
    double vxn = 0, vyn = 0;
    if (m > MPMG_TOL) {
        vxn = mat::quot(sum[1], m);
        vyn = mat::quot(sum[2], m);
    }
    node_m[n] = m;
    node_vx[n] = vxn;
    node_vy[n] = vyn;
    if (node_mx != nullptr) {
        bool bx, by;
        bc_mask(bc, g, i, j, sp->t, bx, by);
        node_mx[n] = bx ? 0.0 : sum[1];
        node_my[n] = by ? 0.0 : sum[2];
    }
}

__global__ void material_only_kernel(const __grid_constant__ G2PArgs A, int material)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= A.n || !A.active[i]) return;
    const G2PConst &C = A.k;
    const double exx = A.exx[i], exy = A.exy[i], eyy = A.eyy[i], wxy = A.wxy[i], vol = A.v[i];
    if (material == MPMG_ISOLIN) {
        isolin_particle<mat::Elastic>(A, C, i, load_particle<MPMG_ISOLIN, G2P_FULL>(A, i), exx, exy, eyy, wxy);
    } else if (material == MPMG_DP_RI_MT) {
        plane_return_particle<mat::Elastic, MPMG_DP_RI_MT>(A, C, i, load_particle<MPMG_DP_RI_MT, G2P_FULL>(A, i), vol, exx, exy,
                                             eyy, wxy);
    } else if (material == MPMG_G_LOCAL_MU2_PLANE_STRAIN) {
        plane_return_particle<mat::Elastic, MPMG_G_LOCAL_MU2_PLANE_STRAIN>(
            A, C, i, load_particle<MPMG_G_LOCAL_MU2_PLANE_STRAIN, G2P_FULL>(A, i), vol, exx, exy, eyy, wxy);
    } else if (material == MPMG_G_LOCAL_MU2_TRUE_2D) {
        plane_return_particle<mat::Elastic, MPMG_G_LOCAL_MU2_TRUE_2D>(
            A, C, i, load_particle<MPMG_G_LOCAL_MU2_TRUE_2D, G2P_FULL>(A, i), vol, exx, exy, eyy, wxy);
    } else if (material == MPMG_G_LOCAL_MU2_REVERSE) {
        reverse_particle<mat::Elastic>(A, C, i, load_particle<MPMG_G_LOCAL_MU2_REVERSE, G2P_FULL>(A, i), vol, exx, exy, eyy, wxy);
    } else {
        // L's off-diagonal entries, g_local_mu2.c:191-199
        const double Lxy = mat::add(exy, wxy), Lyx = mat::sub(exy, wxy);
        mu2_particle<mat::Elastic>(A, C, i, load_particle<MPMG_G_LOCAL_MU2, G2P_FULL>(A, i), vol, exx, eyy, mat::add(Lxy, Lyx),
                     mat::sub(Lxy, Lyx));
    }
}

// The key each particle's last element map gives (mpmg_fp64_sort).
__global__ void __launch_bounds__(256) map_keys_kernel(int n, const int *__restrict__ in_element,
                                                       const int *__restrict__ active, uint32_t sentinel,
                                                       uint32_t *__restrict__ keys)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) keys[i] = active[i] ? (uint32_t)in_element[i] : sentinel;
}

RowsOut rows_out(const mpmg_ctx *ctx, int b)
{
    const RowBins &r = ctx->row;
    return RowsOut{r.count[b], r.rows[b], r.filled[b], r.pos[b], r.n_filled + b, r.head, r.next, r.cap};
}

RowView row_view(const mpmg_ctx *ctx)
{
    const RowBins &r = ctx->row;
    return RowView{r.count[r.cur], r.rows[r.cur], r.over_list, r.cap};
}

G2PArgs make_g2p_args(mpmg_ctx *ctx)
{
    G2PArgs A;
    const mpmg_config &c = ctx->cfg;
    A.g = make_geom(ctx);
    A.n = (int)ctx->np;
    A.early = early_launch(ctx);
    static_cast<mat::Elastic &>(A.k.el) = mat::make_elastic(ctx->G, ctx->K, ctx->lambda, c.dt);
    A.k.inv_h = ctx->inv_h;
    A.k.half_inv_h = 0.5 * ctx->inv_h;
    A.k.mu2.mu_s = c.mp[MPMG_MP_MU_S];
    A.k.mu2.mu_2 = c.mp[MPMG_MP_MU_2];
    A.k.mu2.I0 = c.mp[MPMG_MP_I0];
    A.k.mu2.grains_rho = c.mp[MPMG_MP_GRAINS_RHO];
    A.k.mu2.grains_d = c.mp[MPMG_MP_GRAINS_D];
    A.k.mu2.rho_critical = c.mp[MPMG_MP_RHO_CRITICAL];
    A.k.mu2.A = c.mp[MPMG_MP_A];
    A.k.mu2.krho = mat::make_known(A.k.mu2.grains_rho);
    A.k.mu2.kd = mat::make_known(A.k.mu2.grains_d);
    const bool bracket = A.k.mu2.rho_critical >= 0x1p-60 && A.k.mu2.rho_critical <= 0x1p60;
    A.k.mu2.rho_lo = bracket ? A.k.mu2.rho_critical * (1.0 - 0x1p-47) : -1.0;
    A.k.mu2.rho_hi = bracket ? A.k.mu2.rho_critical * (1.0 + 0x1p-47) : (double)INFINITY;
    A.k.mu2.kAAdd = mat::make_known(((A.k.mu2.A * A.k.mu2.A) * A.k.mu2.grains_d) * A.k.mu2.grains_d);
    A.k.mu2.alpha_c = (((ctx->G * A.k.mu2.I0) * c.dt) / A.k.mu2.grains_d) / sqrt(A.k.mu2.grains_rho);
    A.k.mu2.GI0dt = (ctx->G * A.k.mu2.I0) * c.dt;
    A.nl.E = c.mp[MPMG_MP_E];
    A.nl.nu = c.mp[MPMG_MP_NU];
    A.nl.mu_s = c.mp[MPMG_MP_MU_S];
    A.nl.grains_rho = c.mp[MPMG_MP_GRAINS_RHO];
    A.nl.B = c.mp[MPMG_MP_B];
    A.nl.A = c.mp[MPMG_MP_A];
    A.nl.grains_d = c.mp[MPMG_MP_GRAINS_D];
    A.nl.cohesion = c.mp[MPMG_MP_COHESION];
    A.keys = ctx->keys;
    A.sentinel = (uint32_t)ctx->ne;
    A.inv_hf = (float)ctx->inv_h;
    A.next = rows_out(ctx, 1 - ctx->row.cur);
    A.in_element = ctx->in_element;
    A.active = ctx->active;
    A.pos = ctx->row.pos[ctx->row.cur];
    A.coef = (const double2 *)ctx->elem_coef;
    A.node_vx = ctx->node_vx;
    A.node_vy = ctx->node_vy;
    A.x = ctx->x; A.y = ctx->y; A.vx = ctx->vx; A.vy = ctx->vy; A.ux = ctx->ux; A.uy = ctx->uy;
    A.v = ctx->v; A.m = ctx->m;
    A.sxx = ctx->sxx; A.sxy = ctx->sxy; A.syy = ctx->syy; A.Tzz = ctx->Tzz;
    A.st0 = ctx->state[0]; A.st1 = ctx->state[1]; A.st3 = ctx->state[3]; A.st4 = ctx->state[4]; A.st5 = ctx->state[5];
    A.st6 = ctx->state[6]; A.st9 = ctx->state[9]; A.st10 = ctx->state[10];
    A.ax = ctx->ax; A.ay = ctx->ay;
    A.exx = ctx->exx; A.exy = ctx->exy; A.eyy = ctx->eyy; A.wxy = ctx->wxy;
    A.xl_out = ctx->xl; A.yl_out = ctx->yl;
    A.trial = ctx->nl_trial;
    return A;
}

inline int blocks_for(size_t n, int threads)
{
    size_t b = (n + (size_t)threads - 1) / (size_t)threads;
    return (int)(b > 0 ? b : 1);
}

}  // namespace

// More than two warps of particles a sub-partition: the G2P is then bound by
// the FP64 pipe and takes larger blocks and integer products
// (mat::SoftElastic; g_local_mu2, 1 048 576 particles: 287 -> 254 us a step,
// 125k: 67 -> 62; isolin, 65k: 40.5 -> 38.8).  Up to there a sub-partition's
// one or two warps run a serial chain, through an instruction cache that the
// integer products' longer code overflows: one-warp blocks (a larger one would
// leave most SMs idle) and FP64 products (31k: 30.7 us, 31.5 with integer ones;
// 4k: 15.5 and 16.3).
static bool g2p_pipe_bound(const mpmg_ctx *ctx)
{
    return ctx->np > (size_t)ctx->sms * 4 * 32 * 2;
}

// The arithmetic of a pipe-bound phase; the move phase has no products.
template <int PHASE>
struct BoundArith {
    using E = mat::SoftElastic;
};
template <>
struct BoundArith<G2P_MOVE> {
    using E = mat::Elastic;
};

template <int MATERIAL, int PHASE>
static cudaError_t launch_g2p(mpmg_ctx *ctx, const G2PArgs &A)
{
    const bool bound = g2p_pipe_bound(ctx);
    // blocks of two warps up to sixteen warps a sub-partition, where a block of
    // four more or less on an SM still shows (125k: 58.2 us with four, 56.4 with
    // two; 1 048 576: 253.8 and 255.6)
    const int t = !bound ? 32 : ctx->np <= (size_t)ctx->sms * 4 * 32 * 16 ? 64 : 128;
    ctx->launches += 1;
    using E = typename BoundArith<PHASE>::E;
    const bool list = PHASE != G2P_STRAIN && ctx->row.pos[0] != nullptr;
    return mpmg_launch_pdl(true,
                           list ? (bound ? g2p_kernel<E, MATERIAL, PHASE, PHASE != G2P_STRAIN>
                                         : g2p_kernel<mat::Elastic, MATERIAL, PHASE, PHASE != G2P_STRAIN>)
                                : (bound ? g2p_kernel<E, MATERIAL, PHASE, false>
                                         : g2p_kernel<mat::Elastic, MATERIAL, PHASE, false>),
                           dim3(blocks_for(ctx->np, t)), dim3(t), 0, ctx->stream, A);
}

template <int EB, int SPLIT>
static cudaError_t launch_p2g(mpmg_ctx *ctx, const GridGeom &g, bool keep_order)
{
    const mpmg_config &c = ctx->cfg;
    RowBins &r = ctx->row;
    ctx->launches += 1;
    // blocks for the most elements that can be filled; the rest leave at once
    const size_t most = ctx->np < ctx->ne ? ctx->np : ctx->ne;
    return mpmg_launch_pdl(true, r.pos[0] != nullptr ? p2g_cells_kernel<EB, SPLIT, true> : p2g_cells_kernel<EB, SPLIT, false>,
                           dim3(blocks_for(most, EB)), dim3(EB * SPLIT), 0, ctx->stream, g, row_view(ctx),
                           (const uint32_t *)r.filled[r.cur],
                           (const uint32_t *)(r.n_filled + r.cur), (const uint32_t *)r.head,
                           (const uint32_t *)r.next, r.cursor, keep_order ? 1 : 0, early_launch(ctx),
                           (const double *)ctx->x, (const double *)ctx->y, (const double *)ctx->m, (const double *)ctx->vx,
                           (const double *)ctx->vy, (const double *)ctx->v, (const double *)ctx->sxx,
                           (const double *)ctx->sxy, (const double *)ctx->syy, ctx->d_params, c.dt, c.gravity_mode,
                           c.gravity, ctx->cell_sums);
}

int mpmg_fp64_ready(mpmg_ctx *ctx)
{
    RowBins &r = ctx->row;
    if (r.ready) return MPMG_OK;
    cudaStream_t s = ctx->stream;
    const int n = (int)ctx->np;
    MPMG_CHECK(cudaMemsetAsync(r.count[r.cur], 0, ctx->ne * sizeof(uint32_t), s));
    MPMG_CHECK(cudaMemsetAsync(r.n_filled, 0, 2 * sizeof(uint32_t), s));
    MPMG_CHECK(cudaMemsetAsync(r.cursor, 0, sizeof(uint32_t), s));
    keys_kernel<<<blocks_for(n, 256), 256, 0, s>>>(make_geom(ctx), (float)ctx->inv_h, n, ctx->x, ctx->y, ctx->active,
                                                   ctx->keys, (uint32_t)ctx->ne, rows_out(ctx, r.cur));
    ctx->launches += 1;
    MPMG_CHECK(cudaGetLastError());
    r.ready = true;
    return MPMG_OK;
}

// A radix sort, whose time does not depend on how the particles crowd: 262 144
// of them, 64 to an element, 83 us with the read-back (234 with a counting sort
// that left each element's entries to one thread); 900 to an element 75 (2834).
int mpmg_fp64_sort(mpmg_ctx *ctx)
{
    const int n = (int)ctx->np, ne = (int)ctx->ne;
    cudaStream_t s = ctx->stream;
    if (ctx->sort_keys == nullptr) {
        SortScratch &sc = ctx->sort_scratch;
        const size_t keys = ctx->np * sizeof(uint32_t), digits = 1024 * sizeof(uint32_t);
        const size_t tiles = ctx->np / 1024 + 1;       // tiles of 1024 keys or more
        const int rc = mpmg_dalloc_all({{(void **)&sc.keys, keys},
                                        {(void **)&sc.keys_alt, keys},
                                        {(void **)&sc.vals_alt, keys},
                                        {(void **)&sc.tile_hist, digits * tiles},
                                        {(void **)&sc.digit_total, digits},
                                        {(void **)&ctx->sort_keys, keys}});
        if (rc != MPMG_OK) return rc;
    }
    map_keys_kernel<<<blocks_for(n, 256), 256, 0, s>>>(n, ctx->in_element, ctx->active, (uint32_t)ne, ctx->sort_keys);
    MPMG_CHECK(cudaGetLastError());
    MPMG_CHECK(mpmg_sort_run(ctx->sort_keys, n, ne, ctx->key_bits, ctx->sms, ctx->sort_scratch, ctx->sorted_keys,
                             ctx->perm, ctx->cell_start, s));
    ctx->launches += 1 + 3 * (n > 0 ? (ctx->key_bits + 9) / 10 : 0) + 1;
    return MPMG_OK;
}

int mpmg_launch_step(mpmg_ctx *ctx)
{
    cudaStream_t s = ctx->stream;
    const mpmg_config &c = ctx->cfg;
    const GridGeom g = make_geom(ctx);
    const int n = (int)ctx->np;
    const int ne = (int)ctx->ne;
    const int nn = (int)ctx->nn;
    const uint32_t *pos = ctx->row.pos[ctx->row.cur];   // null: sums by element
    const bool list = pos != nullptr;
    const bool nonlocal = c.material == MPMG_G_NONLOCAL_MU2 || c.material == MPMG_G_NONLOCAL ||
                          c.material == MPMG_G_NONLOCAL_AVG;
    const bool musl = c.scheme == MPMG_SCHEME_MUSL;

    mpmg_phase_begin(ctx, PH_P2G);
    // later phases of these read the ordered rows
    const bool keep_order = nonlocal || musl || c.material == MPMG_G_LOCAL_MU2_EXT || ctx->row.record;
    // two threads an element in single-warp sets, where that leaves every
    // sub-partition at most one warp (of the initial positions: a run that
    // spreads from one form's range into the other's keeps its form, 262 144
    // particles 87.7 us a step where they began packed, 83.5 where spread)
    MPMG_CHECK((ctx->row.filled0 <= (size_t)ctx->sms * 4 * 16 ? launch_p2g<32, 2>(ctx, g, keep_order)
                                                              : launch_p2g<64, 1>(ctx, g, keep_order)));
    mpmg_phase_end(ctx, PH_P2G);

    mpmg_phase_begin(ctx, PH_GRID);
    MPMG_CHECK(launch_grid(ctx, g));
    ctx->launches += 1;
    mpmg_phase_end(ctx, PH_GRID);

    mpmg_phase_begin(ctx, PH_G2P);
    G2PArgs A = make_g2p_args(ctx);
    if (musl) {
        // move, second projection of the moved momentum, then strain
        // the move phase does not depend on the material
        MPMG_CHECK((launch_g2p<MPMG_ISOLIN, G2P_MOVE>(ctx, A)));
        MPMG_CHECK(mpmg_launch_pdl(true, list ? p2g_momentum_kernel<true> : p2g_momentum_kernel<false>, dim3(blocks_for(ne, 128)), dim3(128), 0, s, ne,
                                   row_view(ctx), pos, (const double *)ctx->xl, (const double *)ctx->yl,
                                   (const double *)ctx->m, (const double *)ctx->vx, (const double *)ctx->vy,
                                   ctx->cell_sums));
        MPMG_CHECK(mpmg_launch_pdl(true, list ? node_velocity_kernel<true> : node_velocity_kernel<false>, dim3(blocks_for(nn, 256)), dim3(256), 0, s, g,
                                   make_bc(ctx), ne, (const uint32_t *)ctx->row.count[ctx->row.cur], pos,
                                   (const double *)ctx->cell_sums, (const StepParams *)ctx->d_params, ctx->node_m,
                                   ctx->node_vx, ctx->node_vy, ctx->node_mx, ctx->node_my));
        ctx->launches += 2;
        switch (c.material) {
        case MPMG_ISOLIN: MPMG_CHECK((launch_g2p<MPMG_ISOLIN, G2P_STRAIN>(ctx, A))); break;
        case MPMG_DP_RI_MT: MPMG_CHECK((launch_g2p<MPMG_DP_RI_MT, G2P_STRAIN>(ctx, A))); break;
        case MPMG_G_LOCAL_MU2_PLANE_STRAIN:
            MPMG_CHECK((launch_g2p<MPMG_G_LOCAL_MU2_PLANE_STRAIN, G2P_STRAIN>(ctx, A)));
            break;
        case MPMG_G_LOCAL_MU2_TRUE_2D: MPMG_CHECK((launch_g2p<MPMG_G_LOCAL_MU2_TRUE_2D, G2P_STRAIN>(ctx, A))); break;
        case MPMG_G_LOCAL_MU2_REVERSE: MPMG_CHECK((launch_g2p<MPMG_G_LOCAL_MU2_REVERSE, G2P_STRAIN>(ctx, A))); break;
        default: MPMG_CHECK((launch_g2p<MPMG_G_LOCAL_MU2, G2P_STRAIN>(ctx, A))); break;
        }
    } else {
        switch (c.material) {
        case MPMG_ISOLIN: MPMG_CHECK((launch_g2p<MPMG_ISOLIN, G2P_FULL>(ctx, A))); break;
        case MPMG_G_LOCAL_MU2: MPMG_CHECK((launch_g2p<MPMG_G_LOCAL_MU2, G2P_FULL>(ctx, A))); break;
        case MPMG_DP_RI_MT: MPMG_CHECK((launch_g2p<MPMG_DP_RI_MT, G2P_FULL>(ctx, A))); break;
        case MPMG_G_LOCAL_MU2_PLANE_STRAIN:
            MPMG_CHECK((launch_g2p<MPMG_G_LOCAL_MU2_PLANE_STRAIN, G2P_FULL>(ctx, A)));
            break;
        case MPMG_G_LOCAL_MU2_TRUE_2D: MPMG_CHECK((launch_g2p<MPMG_G_LOCAL_MU2_TRUE_2D, G2P_FULL>(ctx, A))); break;
        case MPMG_G_LOCAL_MU2_REVERSE: MPMG_CHECK((launch_g2p<MPMG_G_LOCAL_MU2_REVERSE, G2P_FULL>(ctx, A))); break;
        case MPMG_G_LOCAL_MU2_EXT:
            MPMG_CHECK((launch_g2p<MPMG_G_LOCAL_MU2_EXT, G2P_FULL>(ctx, A)));
            ext_cells_kernel<<<blocks_for(ne, 128), 128, 0, s>>>(ne, ctx->inv_h, row_view(ctx), pos, ctx->xl, ctx->yl,
                                                                ctx->v, ctx->state[4], ctx->cell_sums);
            ext_nodes_kernel<<<blocks_for(nn, 256), 256, 0, s>>>(g, ne, ctx->row.count[ctx->row.cur], pos,
                                                                ctx->cell_sums, ctx->node_gf);
            ext_stress_kernel<<<blocks_for(n, 256), 256, 0, s>>>(A, ctx->node_gf);
            ctx->launches += 3;
            break;
        case MPMG_G_NONLOCAL_MU2: MPMG_CHECK((launch_g2p<MPMG_G_NONLOCAL_MU2, G2P_FULL>(ctx, A))); break;
        default: MPMG_CHECK((launch_g2p<MPMG_G_NONLOCAL, G2P_FULL>(ctx, A))); break;
        }
    }
    mpmg_phase_end(ctx, PH_G2P);
    MPMG_CHECK(cudaGetLastError());

    if (nonlocal) {
        mpmg_phase_begin(ctx, PH_FLUIDITY);
        const int rc = mpmg_launch_fluidity(ctx);
        if (rc != MPMG_OK) return rc;
        mpmg_phase_end(ctx, PH_FLUIDITY);
    }
    ctx->row.cur = 1 - ctx->row.cur;
    return MPMG_OK;
}

int mpmg_launch_material_only(mpmg_ctx *ctx)
{
    G2PArgs A = make_g2p_args(ctx);
    if (A.exx == nullptr) {
        mpmg_set_error("material-only update needs store_transients (strain-rate inputs)");
        return MPMG_ERR_INVALID;
    }
    material_only_kernel<<<blocks_for(ctx->np, 256), 256, 0, ctx->stream>>>(A, ctx->cfg.material);
    ctx->launches += 1;
    MPMG_CHECK(cudaGetLastError());
    return MPMG_OK;
}
