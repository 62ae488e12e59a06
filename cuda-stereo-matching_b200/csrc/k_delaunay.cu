// GPU Delaunay triangulation of the support points of both views
// (algorithm and predicates: delaunay_core.h).  Replaces the reference's
// device->host copy, Triangle call and host->device copy
// (src/Elas.cu:282-328, called twice from :89-90).
//
// Both views run as two independent problems inside the same launches:
// problem 0 triangulates (u, v), problem 1 triangulates (u - d, v).
#include <algorithm>
#include <climits>
#include <cooperative_groups.h>
#include <type_traits>
#include <cuda_runtime.h>
#include "common.cuh"
#include "launch.cuh"
#include "delaunay_core.h"
#include "kernels.h"

namespace elas {

using namespace del;
namespace cg = cooperative_groups;

namespace {

constexpr int SORT_CAP = 2048;   // max candidates per lattice row
constexpr int FLIP_THREADS = 1024;

__device__ __forceinline__ void set_err(unsigned* err, unsigned f) { atomicOr(err, f); }

// Exclusive scan of one int per thread over a 1024-thread block; *total
// receives the sum.  `warp_sums` has 32 entries.
__device__ int block_scan(int v, int* warp_sums, int* total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) warp_sums[warp] = x;
    __syncthreads();
    if (warp == 0) {
        int w = lane < (blockDim.x >> 5) ? warp_sums[lane] : 0;
        int ws = w;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            int y = __shfl_up_sync(0xffffffffu, ws, o);
            if (lane >= o) ws += y;
        }
        warp_sums[lane] = ws - w;
        if (lane == 31) warp_sums[32] = ws;
    }
    __syncthreads();
    int r = x - v + warp_sums[warp];
    *total = warp_sums[32];
    __syncthreads();
    return r;
}

// Reserve one slot per calling lane in a list whose length counter `ctr`
// is shared by many threads: one atomic per converged group of lanes
// instead of one per lane (shared-memory atomics on one address serialise).
// The order of entries within a list carries no meaning.
__device__ __forceinline__ int agg_inc(int* ctr) {
    const unsigned mask = __activemask();
    const int lane = threadIdx.x & 31;
    const int leader = __ffs(mask) - 1;
    int base = 0;
    if (lane == leader) base = atomicAdd(ctr, __popc(mask));
    base = __shfl_sync(mask, base, leader);
    return base + __popc(mask & ((1u << lane) - 1u));
}

// As agg_inc, for lanes whose counters may differ (grouped by address).
__device__ __forceinline__ int agg_inc_keyed(int* ctr) {
    const unsigned mask = __activemask();
    const unsigned peers = __match_any_sync(mask, reinterpret_cast<unsigned long long>(ctr));
    const int lane = threadIdx.x & 31;
    const int leader = __ffs(peers) - 1;
    int base = 0;
    if (lane == leader) base = atomicAdd(ctr, __popc(peers));
    base = __shfl_sync(mask, base, leader);
    return base + __popc(peers & ((1u << lane) - 1u));
}

// Worklists hold every interior edge at most once per round, as its lower
// half-edge c = min(x, r) (x a half-edge, r its twin; hull edges, r < 0,
// never flip).  `mark` is the round's bitset over half-edges, cleared before
// the round's pushes; the lane that sets c's bit queues it.  With one entry
// per edge, no edge is proposed twice in a round.
__device__ __forceinline__ bool claim_edge(uint32_t* mark, int x, int r, int& c) {
    if (r < 0) return false;
    c = min(x, r);
    const uint32_t bit = 1u << (c & 31);
    return (atomicOr(mark + (c >> 5), bit) & bit) == 0u;
}

// Round 0 of a flip kernel: propose every interior edge of the half-edges
// [h0, h1) once (the owner rule: the half-edge whose triangle has the
// smaller index).  Each warp compacts its owned half-edges through a
// 64-entry ring in shared memory (`ring`, per warp) and proposes them 32 at
// a time, so no lane idles on a twin.  `opp_of(h)` reads a link, `prop(h)`
// proposes; all 32 lanes of every warp of the block must call this.
template <class Opp, class Prop>
__device__ __forceinline__ void propose_owned(int h0, int h1, int32_t* ring, Opp opp_of, Prop prop) {
    const int lane = threadIdx.x & 31;
    int head = 0, cnt = 0;
    for (int base = h0 + int(threadIdx.x & ~31u); base < h1; base += int(blockDim.x)) {
        const int h = base + lane;
        bool own = false;
        if (h < h1) {
            const int o = opp_of(h);
            own = o >= 0 && o / 3 > h / 3;
        }
        const unsigned bal = __ballot_sync(0xffffffffu, own);
        if (own) ring[(head + cnt + __popc(bal & ((1u << lane) - 1u))) & 63] = h;
        cnt += __popc(bal);
        __syncwarp();
        if (cnt >= 32) {
            const int hh = ring[(head + lane) & 63];
            __syncwarp();
            prop(hh);
            head = (head + 32) & 63;
            cnt -= 32;
        }
    }
    __syncwarp();
    if (lane < cnt) prop(ring[(head + lane) & 63]);
}

// Per lattice row: sort the row's points by (x, index), drop repeated x
// (keeps the lowest index), write the unique list to srt[row_off[r] ..]
// (with the packed coordinates beside it in sxy) and its length to rcnt[r];
// pxy[i] gets point i's packed coordinates, or PXY_NONE if it was dropped.
// The left view's rows come sorted (the support list is in raster order;
// only add_corners breaks it) and need no sort; up to ROW_RANK points every
// thread counts the keys below its own (one pass without barriers, where a
// bitonic sort of 64 keys has 21 stages with one each).
// xbs > 0 (star construction): also the row's index by 8-pixel column
// bucket, xb[r * xbs + k] = the position in srt of the row's first point at
// or right of column 8 k (bucket 0 also holds the columns below 0, the last
// entry is the row's end), with which the star searches find a column range
// by two independent loads.
constexpr int ROW_THREADS = 256;
constexpr int ROW_RANK = 2 * ROW_THREADS;
__global__ void __launch_bounds__(ROW_THREADS) k_rowsort(DelDev d0, DelDev d1, const int32_t* __restrict__ row_off,
                                                         int nrows, int xbs, unsigned* err) {
    grid_dep_wait();
    // x biased to 16 bits (the right view's corner points of add_corners
    // lie left of x = 0) above the 12-bit position in the row
    __shared__ uint32_t key[SORT_CAP];
    __shared__ int cx[SORT_CAP];        // x of the points kept
    __shared__ int wcnt[ROW_THREADS / 32 + 1];
    const DelDev& D = blockIdx.y ? d1 : d0;
    const int r = blockIdx.x, tid = threadIdx.x;
    if (r >= nrows) return;
    const int b = row_off[r], n = row_off[r + 1] - b;
    if (n > SORT_CAP) {
        if (tid == 0) { set_err(err, ERRF_BOUNDS); D.rcnt[r] = 0; }
        for (int k = tid; k < xbs; k += ROW_THREADS) D.xb[size_t(r) * xbs + k] = b;
        return;
    }
    int np = 1;
    while (np < n) np <<= 1;
    for (int i = tid; i < np; i += ROW_THREADS)
        key[i] = i < n ? uint32_t(D.x[b + i] + 32768) << 12 | uint32_t(i) : 0xffffffffu;
    const int32_t yr = n > 0 ? D.y[b] : 0;      // the row's y
    __syncthreads();
    bool unsorted = false;
    for (int i = tid + 1; i < n; i += ROW_THREADS) unsorted = unsorted || key[i] < key[i - 1];
    if (__syncthreads_or(unsorted)) {
        if (n <= ROW_RANK) {
            const uint32_t k0 = tid < n ? key[tid] : 0u, k1 = tid + ROW_THREADS < n ? key[tid + ROW_THREADS] : 0u;
            int r0 = 0, r1 = 0;
            for (int j = 0; j < n; ++j) {
                const uint32_t kj = key[j];
                r0 += kj < k0;
                r1 += kj < k1;
            }
            __syncthreads();
            if (tid < n) key[r0] = k0;
            if (tid + ROW_THREADS < n) key[r1] = k1;
            __syncthreads();
        } else {
            for (int k = 2; k <= np; k <<= 1)
                for (int j = k >> 1; j > 0; j >>= 1) {
                    for (int i = tid; i < np; i += ROW_THREADS) {
                        const int ixj = i ^ j;
                        if (ixj > i) {
                            const bool up = (i & k) == 0;
                            const uint32_t a = key[i], c = key[ixj];
                            if ((a > c) == up) { key[i] = c; key[ixj] = a; }
                        }
                    }
                    __syncthreads();
                }
        }
    }
    // compaction: each warp counts its span, every thread sums the counts before its own
    const int lane = tid & 31, warp = tid >> 5, nw = ROW_THREADS >> 5;
    const int span = ((n + nw - 1) / nw + 31) & ~31;
    const int w0 = imin(n, warp * span), w1 = imin(n, w0 + span);
    auto kept = [&](int i) { return i == 0 || (key[i] >> 12) != (key[i - 1] >> 12); };
    int c = 0;
    for (int i = w0 + lane; i < w1; i += 32) c += kept(i);
    c = __reduce_add_sync(0xffffffffu, c);
    if (lane == 0) wcnt[warp] = c;
    __syncthreads();
    int base = 0, nu = 0;
#pragma unroll
    for (int w = 0; w < nw; ++w) {
        base += w < warp ? wcnt[w] : 0;
        nu += wcnt[w];
    }
    if (tid == 0) D.rcnt[r] = nu;
    for (int i0 = w0; i0 < w1; i0 += 32) {
        const int i = i0 + lane;
        const bool in = i < w1;
        const bool k = in && kept(i);
        const unsigned m = __ballot_sync(0xffffffffu, k);
        if (in) {
            const int32_t idx = b + int32_t(key[i] & 0xfffu);
            const uint32_t xy = pack_xy(int32_t(key[i] >> 12) - 32768, yr);
            // packed coordinates by point (the star searches), PXY_NONE for a dropped duplicate
            D.pxy[idx] = k ? xy : PXY_NONE;
            D.hnext[idx] = -1;
            D.hprev[idx] = -1;
            if (k) {
                const int pos = base + __popc(m & ((1u << lane) - 1));
                D.srt[b + pos] = idx;
                D.sxy[b + pos] = xy;
                cx[pos] = px_of(xy);
            }
        }
        base += __popc(m);
    }
    if (xbs == 0) return;
    __syncthreads();
    for (int k = tid; k < xbs; k += ROW_THREADS) {
        int lo = 0, hi = nu;
        if (k == 0) hi = 0;
        if (k == xbs - 1) lo = nu;
        while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            if (cx[mid] < 8 * k) lo = mid + 1;
            else hi = mid;
        }
        D.xb[size_t(r) * xbs + k] = b + lo;
    }
}

// Lattice rows: row r lies at y = r * step; with add_corners the extra row
// `crow` (-1: none) holds the corner points at y = H - 1.
struct RowGeom {
    int step, crow, H;
    float inv;          // 1 / step
    __device__ __forceinline__ int y(int r) const { return r == crow ? H - 1 : r * step; }
    // floor(y / step): (y + 0.5) / step is at least 0.5 / step away from a
    // whole number, far more than the rounding for y <= 16384
    __device__ __forceinline__ int row(int y) const { return int((float(y) + 0.5f) * inv); }
};

// For the star construction, in the block of k_plan once the non-empty
// rows (ne, with their y in ney, both in shared memory) are known: the box
// of all points (box[0..3]) and the window half-size (box[4], star_r0), and
// the hull boundary (hnext / hprev of every boundary point).  roff and cnt:
// the rows' offsets and unique counts, also in shared memory.  The rows'
// extreme points are staged in shared memory.  Point i leaves its chain
// exactly when it lies strictly inside the segment of two other chain points
// above and below it (strictly right of it on the left chain, left on the
// right one).  With coordinates relative to i, x mirrored for the right
// chain, that holds iff min_{above} x / -y + min_{below} x / y < 0.  |x| <=
// 18094 and |y| <= 16383 (the limits of orient_p), so every cross product
// is below 2^29 and the final sum below 2^30: exact in int32.  HULL_LANES
// lanes decide one point together (the two minima over the other rows, each
// lane a share of them, then merged), both chains at once: first against the
// HULL_GROUP rows around it, then what is left (a third) against what is
// left, as a point inside the hull is inside the hull of the points that
// their own groups keep.  One SM does this, bound by instruction issue:
// against all rows at once the kernel took 7.2 us for 73 rows and 17.4 for
// 214, now 6.7 and 10.2.
constexpr int HULL_LANES = 8, HULL_GROUP = 16;
__device__ void star_setup(const DelDev& D, const int32_t* roff, const int32_t* cnt, const int32_t* ne,
                           const int32_t* ney, int R, int npts, uint32_t* xyf, uint32_t* xyl, int32_t* lstk,
                           int32_t* rstk, int32_t* flag, int* ws) {
    __shared__ int box_s[2], left[2];
    const int tid = threadIdx.x, nt = blockDim.x, lane = tid & 31;
    if (tid == 0) {
        box_s[0] = INT_MAX;
        box_s[1] = INT_MIN;
        left[0] = left[1] = 0;
    }
    __syncthreads();
    for (int s0 = tid - lane; s0 < R; s0 += nt) {
        const int s = s0 + lane;
        int x0 = INT_MAX, x1 = INT_MIN;
        if (s < R) {
            const int r = ne[s], b = roff[r];
            const uint32_t f = D.sxy[b], l = D.sxy[b + cnt[r] - 1];
            xyf[s] = f;
            xyl[s] = l;
            flag[s] = 0;
            x0 = px_of(f);
            x1 = px_of(l);
        }
        x0 = __reduce_min_sync(0xffffffffu, x0);
        x1 = __reduce_max_sync(0xffffffffu, x1);
        if (lane == 0) {
            atomicMin(&box_s[0], x0);
            atomicMax(&box_s[1], x1);
        }
    }
    __syncthreads();
    if (tid == nt - 1) {
        const int32_t b[4] = {R ? box_s[0] : 0, R ? ney[0] : 0, R ? box_s[1] : 0, R ? ney[R - 1] : 0};
        for (int k = 0; k < 4; ++k) D.box[k] = b[k];
        D.box[4] = star_r0(b, npts);
    }
    if (R < 2) return;
    // flag[i]: bit 0 on the left chain, bit 16 on the right one
    const int hl = tid % HULL_LANES;
    // whether row i stays on a side's chain against n rows, row(k) the k-th
    auto on_chain = [&](int side, int i, int n, auto row) {
        const uint32_t* xy = side ? xyl : xyf;
        const uint32_t c = xy[i];
        const int sg = side ? -1 : 1;
        int32_t n0 = 1, e0 = 0, n1 = 1, e1 = 0;         // rows above and below; 1/0: +infinity
#pragma unroll 2
        for (int k = hl; k < n; k += HULL_LANES) {
            const uint32_t v = xy[row(k)];
            const int32_t x = sg * dx_p(v, c), y = dy_p(v, c);
            if (y < 0 && (e0 == 0 || x * e0 < n0 * -y)) { n0 = x; e0 = -y; }
            if (y > 0 && (e1 == 0 || x * e1 < n1 * y)) { n1 = x; e1 = y; }
        }
#pragma unroll
        for (int o = 1; o < HULL_LANES; o <<= 1) {
            const int32_t m0 = __shfl_xor_sync(0xffffffffu, n0, o), f0 = __shfl_xor_sync(0xffffffffu, e0, o);
            const int32_t m1 = __shfl_xor_sync(0xffffffffu, n1, o), f1 = __shfl_xor_sync(0xffffffffu, e1, o);
            if (f0 != 0 && (e0 == 0 || m0 * e0 < n0 * f0)) { n0 = m0; e0 = f0; }
            if (f1 != 0 && (e1 == 0 || m1 * e1 < n1 * f1)) { n1 = m1; e1 = f1; }
        }
        return e0 == 0 || e1 == 0 || n0 * e1 + n1 * e0 >= 0;
    };
    for (int it = tid / HULL_LANES; it < ((2 * R + 3) & ~3); it += nt / HULL_LANES) {   // whole warps
        const int side = it & 1, i = imin(it >> 1, R - 1), b = i & ~(HULL_GROUP - 1);
        const bool on = on_chain(side, i, imin(HULL_GROUP, R - b), [&](int k) { return b + k; });
        if (hl == 0 && it < 2 * R && on) (side ? rstk : lstk)[atomicAdd(&left[side], 1)] = i;
    }
    __syncthreads();
    const int n0 = left[0], n1 = left[1];
    for (int it = tid / HULL_LANES; it < ((n0 + n1 + 3) & ~3); it += nt / HULL_LANES) {
        const int side = it >= n0 && n1 > 0, q = imin(it, n0 + n1 - 1) - (side ? n0 : 0);
        const int32_t* rows = side ? rstk : lstk;
        const int i = rows[q];
        const bool on = on_chain(side, i, side ? n1 : n0, [&](int k) { return rows[k]; });
        if (hl == 0 && it < n0 + n1 && on) atomicOr(&flag[i], side ? 1 << 16 : 1);
    }
    __syncthreads();
    int nl = 0, nr = 0;
    for (int b = 0; b < R; b += nt) {
        const int i = b + tid, f = i < R ? flag[i] : 0;
        int tot = 0;
        const int pos = block_scan(f, ws, &tot);        // both chains' counts in one scan (below 2^16 each)
        if (f & 0xffff) lstk[nl + (pos & 0xffff)] = i;
        if (f >> 16) rstk[nr + (pos >> 16)] = i;
        nl += tot & 0xffff;
        nr += tot >> 16;
    }
    __syncthreads();
    const int tl = cnt[ne[0]], bl = cnt[ne[R - 1]];
    const int C = hull_cycle_len(tl, bl, nl, nr);
    auto at = [&](int j) {
        int row, pos;
        bool last;
        hull_cycle_at(j, R, tl, bl, lstk, nl, rstk, nr, &row, &pos, &last);
        const int r = ne[row];
        return D.srt[roff[r] + (last ? cnt[r] - 1 : pos)];
    };
    for (int j = tid; j < C; j += nt) {
        const int v = at(j), a = at(j + 1 == C ? 0 : j + 1), b = at(j == 0 ? C - 1 : j - 1);
        D.hnext[v] = a;
        D.hprev[v] = b;
    }
}

// Non-empty rows, then either the star set-up (stars) or the strip offsets
// (flips).  One 1024-thread block per problem; the per-row arrays are staged
// in shared memory (PLAN_ARRAYS arrays of nrows entries).  ctr[7] = 1 when
// the strip plan holds (two non-empty rows at least, strips and pockets
// within Tmax); the strips and pockets are then built by k_strips, which
// also sets the triangle count ctr[0].
constexpr int PLAN_ARRAYS = 9;
static_assert(size_t(PLAN_ARRAYS) * sizeof(int32_t) * (LATTICE_ROWS_MAX + 1) + 1024 <= SMEM_PER_CTA,
              "the rows of the tallest lattice and the corners' row fit");
__global__ void __launch_bounds__(1024) k_plan(DelDev d0, DelDev d1, const int32_t* __restrict__ row_off,
                                               int nrows, RowGeom rg, int flips, unsigned* err) {
    grid_dep_wait();
    __shared__ int ws[33];
    extern __shared__ int32_t psm[];
    int32_t* roff = psm;
    int32_t* cnt = psm + nrows;
    int32_t* ne = psm + 2 * nrows;
    int32_t* ney = psm + 3 * nrows;
    DelDev D = blockIdx.x ? d1 : d0;
    const int tid = threadIdx.x, nt = blockDim.x;
    const int npts = row_off[nrows];
    int R = 0, total = 0;
    // non-empty rows in order
    for (int r0 = 0; r0 < nrows; r0 += nt) {
        const int r = r0 + tid;
        int f = 0;
        if (r < nrows) {
            const int c = D.rcnt[r];
            roff[r] = row_off[r];
            cnt[r] = c;
            f = c > 0 ? 1 : 0;
        }
        const int pos = block_scan(f, ws, &total);
        if (f) {
            ne[R + pos] = r;
            ney[R + pos] = rg.y(r);
            if (flips) D.ne[R + pos] = r;
        }
        R += total;
    }
    __syncthreads();
    int off = 0;
    if (!flips) {
        star_setup(D, roff, cnt, ne, ney, R, npts, reinterpret_cast<uint32_t*>(psm + 4 * nrows),
                   reinterpret_cast<uint32_t*>(psm + 5 * nrows), psm + 6 * nrows, psm + 7 * nrows, psm + 8 * nrows,
                   ws);
    } else {
        // strip s between ne[s] and ne[s+1] holds cnt[ne[s]] + cnt[ne[s+1]] - 2 triangles
        for (int s0 = 0; s0 < R - 1; s0 += nt) {
            const int s2 = s0 + tid;
            const int c = s2 < R - 1 ? cnt[ne[s2]] + cnt[ne[s2 + 1]] - 2 : 0;
            const int pos = block_scan(c, ws, &total);
            if (s2 < R - 1) D.soff[s2] = off + pos;
            off += total;
        }
    }
    if (tid == 0) {
        const bool fits = off + 2 * R <= D.Tmax;
        if (flips && R >= 2 && !fits) set_err(err, ERRF_TRI_COUNT);
        D.ctr[0] = 0;
        D.ctr[1] = off;
        D.ctr[2] = 0;    // pocket triangles of both sides
        D.ctr[3] = 0;
        D.ctr[6] = R;
        D.ctr[7] = (flips && R >= 2 && fits) ? 1 : 0;
        D.ctr[8] = 0;    // set to 1 by the flip kernel that handles the problem
        D.ctr[9] = npts;  // support points (vertex ids) of the problem
        D.ctr[4] = 0;    // flip rounds and flips (the flip kernels set them)
        D.ctr[5] = 0;
        D.ctr[10] = 0;   // points left to k_star_far
        D.ctr[11] = 0;   // star construction: overflow pool cursor, (unused), window doublings
        D.ctr[12] = 0;
        D.ctr[13] = 0;
    }
}

// ---------------------------------------------------------------------------
// Star construction (delaunay_core.h, "Stars"): every point's Delaunay
// neighbours are found directly, with no initial triangulation and no
// flips.  Every search is a minimum under a strict total order, so its
// answer does not depend on how threads split the candidates, nor on which
// points beyond the necessary ones were looked at.
//
// Bound by latency: a walk is a chain of some ten dependent steps, and the
// slowest point's chain is the construction's time.  Nine points in ten have
// their whole star within a small square, the others border large empty
// regions and need points from far away.  Hence two kernels:
//   * k_star, a warp per point: the candidates are the at most 64 points
//     nearest around p, two per lane in registers, gathered once (a square
//     of half-size R0, smaller where points are dense, larger where they are
//     sparse).  The walk runs to its end on these alone, in fp32 (exact at
//     such distances), then each lane proves one triangle.  A star that is
//     not proven goes to a list.
//   * k_star_far, a CTA per listed point: the certain triangles are kept,
//     every other step looks at every point of the view.
// One warp per point for everything, with a staged window and searches of
// growing squares, took 54 us at 1242x375 and 399 us with the corner points
// of add_corners; the two kernels 11 + 20 and 12 + 51 us.

constexpr int STAR_WARPS = 8;      // points in flight per CTA
constexpr int STAR_SLOT = 12;      // owned triangles kept in a point's own slot; more go to the pool
constexpr int STAR_LANE = 2;       // candidates per lane
constexpr int STAR_CAND = 32 * STAR_LANE;
constexpr int FAR_REC = DelDev::FAR_REC;   // ints of a listed point's record: point, counts, proofs, neighbours

struct StarSmem {
    int32_t nb[STAR_NB];           // the star's neighbours in counter-clockwise order
    uint32_t nxy[STAR_NB];
};

struct StarEdge {                  // the walk's current edge p -> q
    int p, q;
    uint32_t pp, pq;
    int32_t ux, uy;
};
struct StarBest {                  // best next neighbour so far (i < 0: none)
    int i;
    uint32_t xy;
    float k;
};

// The star order as a float key: for the edge p->q (u = q - p) and a
// candidate s (relative to p) strictly left of it, the centre of the circle
// through p, q, s lies at q/2 + t (-uy, ux) with t = (|s|^2 - u.s) /
// (2 cross(u, s)); the next neighbour has the smallest t.  Numerator and
// denominator are exact in int32 (below 2^31 at the coordinate limits of
// orient_p); the key carries at most three roundings (two conversions, one
// division of at most 2 ulp), a relative error below 4e-7, so keys further
// apart than 4e-6 of the larger order their points correctly and closer
// ones are compared exactly.
constexpr float STAR_KEY_TOL = 4e-6f;

// Out of line: rarely reached and long, and the kernels' chains wait for
// instruction fetches as well as for data.
__device__ __noinline__ bool star_exact(int p, uint32_t pp, int q, uint32_t pq, int a, uint32_t axy, int b,
                                        uint32_t bxy) {
    return star_better_left(p, pp, q, pq, a, axy, b, bxy);
}

__device__ __forceinline__ void star_take(const StarEdge& e, StarBest& best, int s, uint32_t sxy) {
    const int32_t sx = dx_p(sxy, e.pp), sy = dy_p(sxy, e.pp);
    const int32_t cr = e.ux * sy - e.uy * sx;           // orient(p, q, s)
    if (cr <= 0) return;
    const float k = __fdividef(__int2float_rn(sx * sx + sy * sy - (e.ux * sx + e.uy * sy)), __int2float_rn(cr));
    if (best.i >= 0) {
        const float tol = STAR_KEY_TOL * fmaxf(fabsf(best.k), fabsf(k));
        if (k > best.k + tol) return;
        if (k >= best.k - tol &&
            (sxy == best.xy || !star_exact(e.p, e.pp, e.q, e.pq, best.i, best.xy, s, sxy)))
            return;
    }
    best.i = s;
    best.xy = sxy;
    best.k = k;
}

// The minimum over the lanes' bests, in every lane: the smallest key (one
// reduction over order-preserving key bits), then the lanes within the
// keys' rounding of it one by one, exactly.  A lane's other candidates need
// no look: each is worse than its lane's best.
__device__ __forceinline__ void star_reduce(const StarEdge& e, StarBest& best, int lane) {
    const uint32_t kb = __float_as_uint(best.k);
    const uint32_t u = best.i < 0 ? 0xffffffffu : ((kb & 0x80000000u) ? ~kb : (kb | 0x80000000u));
    const uint32_t umin = __reduce_min_sync(0xffffffffu, u);
    if (umin == 0xffffffffu) return;            // no lane holds a candidate
    const int wl = __ffs(__ballot_sync(0xffffffffu, u == umin)) - 1;
    StarBest w;
    w.i = __shfl_sync(0xffffffffu, best.i, wl);
    w.xy = __shfl_sync(0xffffffffu, best.xy, wl);
    w.k = __shfl_sync(0xffffffffu, best.k, wl);
    const bool tie = best.i >= 0 && best.xy != w.xy &&
                     fabsf(best.k - w.k) <= STAR_KEY_TOL * fmaxf(fabsf(best.k), fabsf(w.k));
    for (unsigned m = __ballot_sync(0xffffffffu, tie); m; m &= m - 1) {
        const int j = __ffs(m) - 1;
        const int ci = __shfl_sync(0xffffffffu, best.i, j);
        const uint32_t cxy = __shfl_sync(0xffffffffu, best.xy, j);
        const float ck = __shfl_sync(0xffffffffu, best.k, j);
        if (cxy != w.xy && star_exact(e.p, e.pp, e.q, e.pq, w.i, w.xy, ci, cxy)) {
            w.i = ci;
            w.xy = cxy;
            w.k = ck;
        }
    }
    best = w;
}

// circle_inside in 64-bit floats, for the few triangles that need it (its
// dependent 64-bit operations take over a thousand cycles).
__device__ __noinline__ bool star_proven(uint32_t pp, uint32_t pq, uint32_t pr, int R, const int32_t* box) {
    return circle_inside(pp, pq, pr, R, box);
}

// In fp32: 1 when the whole circle through p, q and r lies in the square of
// half-size R by more than the rounding, -1 when it leaves it by more than
// the rounding, 0 otherwise.  With |q|, |r| <= 2 rho, |q - r| >= 1 the centre
// is off by less than 5e-7 rho^2 (two products of a coordinate and a squared
// length, each rounded once, over the exact determinant) and the rest by
// 1e-6 of the extent.
__device__ __forceinline__ int star_circle_fits(uint32_t pp, uint32_t pq, uint32_t pr, int R) {
    const int32_t qx = dx_p(pq, pp), qy = dy_p(pq, pp), rx = dx_p(pr, pp), ry = dy_p(pr, pp);
    const float q2 = float(qx * qx + qy * qy), r2 = float(rx * rx + ry * ry);
    const float d = 2.0f * float(qx * ry - qy * rx);
    const float cx = __fdividef(float(ry) * q2 - float(qy) * r2, d);
    const float cy = __fdividef(float(qx) * r2 - float(rx) * q2, d);
    const float rho2 = cx * cx + cy * cy;
    const float ext = fmaxf(fabsf(cx), fabsf(cy)) + sqrtf(rho2);
    const float mg = 0.25f + 2e-6f * ext + 1e-6f * rho2;
    return ext + mg <= float(R) ? 1 : (ext - mg > float(R) ? -1 : 0);
}
// circle_inside: a circle that leaves the square can only be proven by its
// part inside the box of all points, which needs a square that reaches past
// the box (rim).
__device__ __forceinline__ bool star_inside(uint32_t pp, uint32_t pq, uint32_t pr, int R, bool rim,
                                            const int32_t* box) {
    const int fit = star_circle_fits(pp, pq, pr, R);
    return fit > 0 || ((fit == 0 || rim) && star_proven(pp, pq, pr, R, box));
}

// One row's points between columns x0 and x1 (and at most seven columns
// more on either side, the buckets' width): first position and count.
__device__ __forceinline__ void star_cols(const DelDev& D, int xbs, int row, int x0, int x1, int* b, int* n) {
    const int32_t* xb = D.xb + size_t(row) * xbs;
    *b = xb[imin(imax(x0 >> 3, 0), xbs - 2)];
    *n = xb[imin(imax(x1 >> 3, 0), xbs - 2) + 1] - *b;
}

__device__ __forceinline__ int warp_excl_scan(int n, int lane) {
    int incl = n;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += y;
    }
    return incl - n;
}

__device__ __forceinline__ float redux_min_f32(float v) {
    float r;
    asm volatile("redux.sync.min.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
    return r;
}

// Store the owned triangles of p's star (a warp; the nt triangles of the
// list nb of deg neighbours of which p is the smallest vertex): their number
// in tcnt[p], their vertex pairs in p's slot, or in the pool when more than
// STAR_SLOT.
__device__ __forceinline__ void star_output(const DelDev& D, int p, const int32_t* nb, int deg, int nt, int lane,
                                            unsigned* err) {
    auto owned = [&](int i, int* a, int* c) {
        if (i >= nt) return false;
        *a = nb[i];
        *c = nb[i + 1 == deg ? 0 : i + 1];
        return p < *a && p < *c;
    };
    int a = 0, c = 0;
    bool o = owned(lane, &a, &c);
    unsigned bal = __ballot_sync(0xffffffffu, o);
    int own = __popc(bal);
    for (int t = 32; t < nt; t += 32) {
        int a2, c2;
        own += __popc(__ballot_sync(0xffffffffu, owned(t + lane, &a2, &c2)));
    }
    int32_t* dst = D.sown + size_t(p) * 2 * STAR_SLOT;
    if (own > STAR_SLOT) {
        int base = 0;
        if (lane == 0) base = atomicAdd(&D.ctr[11], own);
        base = __shfl_sync(0xffffffffu, base, 0);
        if (base + own > D.Tmax) {
            if (lane == 0) set_err(err, ERRF_BOUNDS);
            own = 0;
        } else {
            if (lane == 0) dst[0] = base;
            dst = D.spool + 2 * size_t(base);
        }
    }
    if (own > 0) {
        int pos = 0;
        for (int t = 0;;) {
            if (o) {
                const int j = pos + __popc(bal & ((1u << lane) - 1u));
                *reinterpret_cast<int2*>(dst + 2 * j) = make_int2(a, c);
            }
            t += 32;
            if (t >= nt) break;
            pos += __popc(bal);
            o = owned(t + lane, &a, &c);
            bal = __ballot_sync(0xffffffffu, o);
        }
    }
    if (lane == 0) D.tcnt[p] = own;
}

// The doublings of the window's half-size R0 until the square proves p's
// whole star (what a search by growing squares would have made), by a warp:
// its nt triangles of the deg neighbours at nxy, the start at squared
// distance qd2 (0: a hull point's successor, which needs no proof) and, with
// `open`, a hull edge that only a square over the whole box proves.  Lane =
// item * 4 + level: eight items at four sizes at a time, as a test in 64-bit
// floats takes over a thousand cycles.
__device__ int star_doublings(const DelDev& D, uint32_t pp, const uint32_t* nxy, int deg, int nt, uint32_t qd2,
                              bool open, int lane) {
    const int px = px_of(pp), py = py_of(pp);
    int most = 0;
    for (int t = 0; t <= nt; t += 8) {
        const int i = t + (lane >> 2);
        for (int l0 = 0;; l0 += 4) {
            const int R = D.box[4] << (l0 + (lane & 3));
            const bool w = px - R <= D.box[0], n = py - R <= D.box[1], e = px + R >= D.box[2], s = py + R >= D.box[3];
            bool pass = (w && n && e && s) || i > nt;
            if (!pass)
                pass = i == nt ? !open && qd2 <= uint32_t(R) * uint32_t(R)
                               : star_inside(pp, nxy[i], nxy[i + 1 == deg ? 0 : i + 1], R, w || n || e || s, D.box);
            const unsigned nib = (__ballot_sync(0xffffffffu, pass) >> (lane & 28)) & 15u;
            if (nib) most = imax(most, l0 + __ffs(nib) - 1);
            if (__all_sync(0xffffffffu, nib != 0u)) break;
        }
    }
    return __reduce_max_sync(0xffffffffu, most);
}

// Grid-stride over (point, view) with one warp per point: the star from the
// points around p, stored if it is proven, else p joins the list of
// k_star_far.
__global__ void __launch_bounds__(STAR_WARPS * 32, 3) k_star(DelDev d0, DelDev d1, int nrows, RowGeom rg, int xbs,
                                                             unsigned* err) {
    grid_dep_wait();
    __shared__ StarSmem smem[STAR_WARPS];
    // blockIdx.x is the view, so that the two views' first blocks (the ones
    // with points) are dispatched side by side
    const DelDev& D = blockIdx.x ? d1 : d0;
    const int N = D.ctr[9];
    const int32_t box[4] = {D.box[0], D.box[1], D.box[2], D.box[3]};
    const int R0 = D.box[4];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    StarSmem& sm = smem[warp];
    for (int p = blockIdx.y * STAR_WARPS + warp; p < N; p += gridDim.y * STAR_WARPS) {
        const uint32_t pp = D.pxy[p];
        if (pp == PXY_NONE) {
            if (lane == 0) D.tcnt[p] = 0;
            continue;
        }
        const int hn = D.hnext[p], hp = D.hprev[p];
        const uint32_t hnxy = hn >= 0 ? D.pxy[hn] : PXY_NONE, hpxy = hp >= 0 ? D.pxy[hp] : PXY_NONE;
        const int px = px_of(pp), py = py_of(pp);
        auto covers = [&](int Rs) {
            return px - Rs <= box[0] && px + Rs >= box[2] && py - Rs <= box[1] && py + Rs >= box[3];
        };
        // The candidates: the points of a square of half-size r (a lane per
        // row), r found from R0 by the points it holds.
        int r = R0, b = 0, n = 0, K = 0;
        bool shrunk = false, trusted = true;
        for (int it = 0;; ++it) {
            // the rows from py - r to py + r (and the corners' extra row when it may be one of them)
            const int s0 = imin(rg.row(imax(py - r, 0) + rg.step - 1), nrows - 1);
            const int s1 = rg.crow >= 0 && py + r >= rg.H - 1 ? nrows : imin(rg.row(py + r) + 1, nrows);
            n = 0;
            if (s1 - s0 <= 32) {
                if (s0 + lane < s1) {
                    star_cols(D, xbs, s0 + lane, px - r, px + r, &b, &n);
                    if (r <= 8) {               // the buckets' width counts here
                        while (n > 0 && px_of(D.sxy[b]) < px - r) { ++b; --n; }
                        while (n > 0 && px_of(D.sxy[b + n - 1]) > px + r) --n;
                    }
                }
                K = __reduce_add_sync(0xffffffffu, n);
            } else {
                K = STAR_CAND + 1;
            }
            if (K > STAR_CAND) {
                if (it >= 24 || r <= 2) { trusted = false; break; }
                const int rs = s1 - s0 > 32 ? r * 3 / 5 : int(float(r) * sqrtf(44.0f / float(K)));
                r = imax(2, imin(rs, r - 1));
                shrunk = true;
            } else if (K < 20 && !shrunk && it < 3 && !covers(r)) {
                r *= 2;
            } else {
                break;
            }
        }
        // dealt out over the lanes, two slots each (slot = lane + 32 c): the
        // rows' positions are laid end to end in shared memory
        int cid[STAR_LANE];
        uint32_t cxy[STAR_LANE];
        float fx[STAR_LANE], fy[STAR_LANE], fn[STAR_LANE];     // relative to p; squared length, 0 for p and empty slots
        {
            const int excl = warp_excl_scan(n, lane);
            if (!trusted) K = n = 0;
            for (int i = 0; i < n; ++i) sm.nb[excl + i] = b + i;
            __syncwarp();
#pragma unroll
            for (int c = 0; c < STAR_LANE; ++c) {
                const int k = lane + 32 * c;
                const bool in = k < K;
                const int pos = in ? sm.nb[k] : 0;
                cid[c] = in ? D.srt[pos] : -1;
                cxy[c] = in ? D.sxy[pos] : pp;
                const int dx = dx_p(cxy[c], pp), dy = dy_p(cxy[c], pp);
                fx[c] = float(dx);
                fy[c] = float(dy);
                fn[c] = float(dx * dx + dy * dy);
            }
            __syncwarp();
        }
        auto slot_of = [&](uint32_t xy) {       // the candidates' slot of a point, -1: not among them
            const unsigned m0 = __ballot_sync(0xffffffffu, cid[0] >= 0 && cxy[0] == xy);
            const unsigned m1 = __ballot_sync(0xffffffffu, cid[1] >= 0 && cxy[1] == xy);
            return m0 ? __ffs(m0) - 1 : (m1 ? 31 + __ffs(m1) : -1);
        };
        auto id_at = [&](int slot) { return __shfl_sync(0xffffffffu, slot & 32 ? cid[1] : cid[0], slot & 31); };
        auto xy_at = [&](int slot) { return __shfl_sync(0xffffffffu, slot & 32 ? cxy[1] : cxy[0], slot & 31); };
        const bool whole = trusted && covers(r);
        // the square reaches past the box of all points: a circle that leaves
        // the square may still be proven by its part inside the box
        const bool rim = px - r < box[0] || px + r > box[2] || py - r < box[1] || py + r > box[3];
        // The walk's start.  A hull point whose successor is not among the
        // candidates cannot be finished here; it walks from its nearest
        // neighbour for the record's sake.
        int q0slot = hn >= 0 ? slot_of(hnxy) : -1;
        const bool adrift = hn >= 0 && q0slot < 0;
        if (q0slot < 0) {
            // nearest neighbour, the lowest index among equals
            const float l0 = fn[0] > 0.0f ? fn[0] : INFINITY, l1 = fn[1] > 0.0f ? fn[1] : INFINITY;
            const float lm = redux_min_f32(fminf(l0, l1));
            if (lm < INFINITY && (whole || lm <= float(r * r))) {
                const int i0 = l0 == lm ? cid[0] : INT_MAX, i1 = l1 == lm ? cid[1] : INT_MAX;
                const int q0 = __reduce_min_sync(0xffffffffu, imin(i0, i1));
                const unsigned m0 = __ballot_sync(0xffffffffu, i0 == q0), m1 = __ballot_sync(0xffffffffu, i1 == q0);
                q0slot = m0 ? __ffs(m0) - 1 : 31 + __ffs(m1);
            }
        }
        // The walk on the candidates: lane i keeps neighbour i (up to 32).
        // Coordinates within the square are small enough (r stays below
        // 2048) that cross products and numerators are exact in fp32, so a
        // step is two keys, one reduction and a vote.
        int m = 0, nb = 0;                  // neighbours listed; the lane's: its slot, then its index
        bool closed = false, full = false;
        if (q0slot >= 0 && trusted) {
            const int hpslot = hp >= 0 ? slot_of(hpxy) : -1;
            int slot = q0slot;
            for (;;) {
                if (lane == m) nb = slot;
                ++m;
                if (m > 1 && slot == hpslot) { full = !adrift; break; }
                if (m == 32) break;
                const float ux = __shfl_sync(0xffffffffu, slot & 32 ? fx[1] : fx[0], slot & 31);
                const float uy = __shfl_sync(0xffffffffu, slot & 32 ? fy[1] : fy[0], slot & 31);
                float k[STAR_LANE];
#pragma unroll
                for (int c = 0; c < STAR_LANE; ++c) {
                    const float cr = ux * fy[c] - uy * fx[c];
                    const float num = fn[c] - (ux * fx[c] + uy * fy[c]);
                    k[c] = cr > 0.0f ? __fdividef(num, cr) : INFINITY;
                }
                const float km = redux_min_f32(fminf(k[0], k[1]));
                if (km == INFINITY) break;
                const float lim = km + 2.0f * STAR_KEY_TOL * fabsf(km);
                unsigned m0 = __ballot_sync(0xffffffffu, k[0] <= lim), m1 = __ballot_sync(0xffffffffu, k[1] <= lim);
                int ws = m0 ? __ffs(m0) - 1 : 31 + __ffs(m1);
                if (__popc(m0) + __popc(m1) > 1) {
                    // equal within the keys' rounding: exactly, one by one
                    const int q = id_at(slot);
                    const uint32_t pq = xy_at(slot);
                    if (m0) m0 &= m0 - 1;
                    else m1 &= m1 - 1;
                    int wi = id_at(ws);
                    uint32_t wxy = xy_at(ws);
                    while (m0 | m1) {
                        const int cs = m0 ? __ffs(m0) - 1 : 31 + __ffs(m1);
                        if (m0) m0 &= m0 - 1;
                        else m1 &= m1 - 1;
                        const int ci = id_at(cs);
                        const uint32_t cx = xy_at(cs);
                        if (star_exact(p, pp, q, pq, wi, wxy, ci, cx)) { ws = cs; wi = ci; wxy = cx; }
                    }
                }
                slot = ws;
                if (slot == q0slot) { closed = full = hn < 0; break; }
            }
        }
        // every triangle's proof at once
        uint32_t nxy, sure;
        {
            const int li = nb & 31;
            const int i0 = __shfl_sync(0xffffffffu, cid[0], li), i1 = __shfl_sync(0xffffffffu, cid[1], li);
            const uint32_t x0 = __shfl_sync(0xffffffffu, cxy[0], li), x1 = __shfl_sync(0xffffffffu, cxy[1], li);
            const bool up = (nb & 32) != 0;
            nb = up ? i1 : i0;
            nxy = up ? x1 : x0;
            const uint32_t next = __shfl_sync(0xffffffffu, nxy, lane + 1 == m ? 0 : lane + 1);
            const int nt = star_tris(m, closed);
            const bool in = lane < nt;
            sure = __ballot_sync(0xffffffffu, in && (whole || star_inside(pp, nxy, next, r, rim, D.box)));
            full = full && sure == (nt >= 32 ? 0xffffffffu : (1u << nt) - 1u);
        }
        if (full) {
            sm.nb[lane] = nb;
            sm.nxy[lane] = nxy;
            __syncwarp();
            const int nt = star_tris(m, closed);
            if (r > R0) {
                const uint32_t q = __shfl_sync(0xffffffffu, nxy, 0);
                const int dx = dx_p(q, pp), dy = dy_p(q, pp);
                const uint32_t qd2 = hn >= 0 ? 0u : uint32_t(dx * dx + dy * dy);
                const int g = star_doublings(D, pp, sm.nxy, m, nt, qd2, false, lane);
                if (lane == 0 && g) atomicAdd(&D.ctr[13], g);
            }
            star_output(D, p, sm.nb, m, nt, lane, err);
        } else {
            // what is known of the star goes along: the neighbours listed and which triangles are certain
            int at = 0;
            if (lane == 0) at = atomicAdd(&D.ctr[10], 1);
            at = __shfl_sync(0xffffffffu, at, 0);
            int32_t* rec = D.far + size_t(at) * FAR_REC;
            const int known = m <= FAR_REC - 3 ? m : 0;
            if (lane == 0) {
                rec[0] = p;
                rec[1] = known | (closed ? 1 << 8 : 0) | (adrift ? 1 << 9 : 0);
                rec[2] = int32_t(sure);
            }
            if (lane < known) rec[3 + lane] = nb;
        }
        __syncwarp();
    }
}

// The minimum of a step over the CTA's lanes, in every thread: per warp,
// then over the warps' results in `part`, which the caller alternates
// between two arrays from step to step (so one barrier a step is enough).
template <class Reduce, class T>
__device__ __forceinline__ void star_cta_min(T& v, T* part, int lane, int warp, int nwarps, const T& none,
                                             Reduce reduce) {
    reduce(v);
    if (lane == 0) part[warp] = v;
    __syncthreads();
    v = lane < nwarps ? part[lane] : none;
    reduce(v);
}

// The listed points, a CTA each: a certain triangle of the record is taken
// as it is; every other step starts from a guess (the record's next
// neighbour, or none) and looks at every point of the view; only if one is
// better than the guess are the threads' results merged.  A thread keeps its
// first FAR_KEEP points in registers.  Looking at fewer points was slower
// each time (at 1242x375, against 21 us): only the rows that the guess's
// circle reaches 27, in them only the columns inside it 48, every point
// tested against the circle first 24, as the instructions that choose
// lengthen a step more than the points left out shorten it.  On dense
// lattices a step looks at many points, but the searches over growing
// squares that this replaced did not gain there either: a 1920x1080 pair at
// candidate step 1 (165514 points a view) takes 17.6 ms, 27.6 with them.
constexpr int FAR_THREADS = 512, FAR_KEEP = 8;
__global__ void __launch_bounds__(FAR_THREADS, 2) k_star_far(DelDev d0, DelDev d1, unsigned* err) {
    grid_dep_wait();
    constexpr int NW = FAR_THREADS / 32;
    __shared__ StarSmem sm;
    __shared__ StarBest part[2][NW];
    __shared__ uint2 near[NW];
    const DelDev& D = blockIdx.x ? d1 : d0;
    const int count = D.ctr[10], N = D.ctr[9], R = D.ctr[6];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (int(blockIdx.y) >= count) return;
    uint32_t keep[FAR_KEEP];
#pragma unroll
    for (int k = 0; k < FAR_KEEP; ++k) {
        const int i = tid + k * FAR_THREADS;
        keep[k] = i < N ? D.pxy[i] : PXY_NONE;
    }
    int flip = 0;
    for (int q = blockIdx.y; q < count; q += gridDim.y) {
        const int32_t* rec = D.far + size_t(q) * FAR_REC;
        const int p = rec[0], lm = rec[1] & 0xff;
        const bool lclosed = ((rec[1] >> 8) & 1) != 0, adrift = ((rec[1] >> 9) & 1) != 0;
        const uint32_t sure = uint32_t(rec[2]);
        const int lz = lane < lm ? rec[3 + lane] : -1;
        const uint32_t lzxy = lz >= 0 ? D.pxy[lz] : PXY_NONE;
        const uint32_t pp = D.pxy[p];
        const int hn = D.hnext[p], hp = D.hprev[p];
        const uint32_t hpxy = hp >= 0 ? D.pxy[hp] : PXY_NONE;
        int q0 = lm > 0 && !adrift ? __shfl_sync(0xffffffffu, lz, 0) : hn;
        __syncthreads();                        // the previous point is done with
        if (q0 < 0) {
            // nearest neighbour, the lowest index among equals
            uint2 best = make_uint2(0xffffffffu, 0xffffffffu);     // squared distance, index
            for (int i = tid; i < N; i += FAR_THREADS) {
                const uint32_t xy = D.pxy[i];
                if (xy == PXY_NONE || i == p) continue;
                const int dx = dx_p(xy, pp), dy = dy_p(xy, pp);
                const uint32_t d = uint32_t(dx * dx + dy * dy);
                if (d < best.x) best = make_uint2(d, uint32_t(i));
            }
            star_cta_min(best, near, lane, warp, NW, make_uint2(0xffffffffu, 0xffffffffu), [](uint2& v) {
                const uint32_t d = __reduce_min_sync(0xffffffffu, v.x);
                v.y = __reduce_min_sync(0xffffffffu, v.x == d ? v.y : 0xffffffffu);
                v.x = d;
            });
            q0 = int(best.y);                   // -1: no other point
        }
        int m = 0;
        uint32_t qd2 = 0;
        bool closed = false, open = false, ok = true;
        if (q0 >= 0) {
            const uint32_t q0xy = D.pxy[q0];
            if (tid == 0) { sm.nb[0] = q0; sm.nxy[0] = q0xy; }
            m = 1;
            StarEdge e{p, q0, pp, q0xy, dx_p(q0xy, pp), dy_p(q0xy, pp)};
            if (hn < 0) qd2 = uint32_t(e.ux * e.ux + e.uy * e.uy);
            int j = lm > 0 && !adrift ? 0 : -1; // the current neighbour's place in the record (-1: not in it)
            for (;;) {
                StarBest best{-1, 0u, 0.0f};
                const int jn = j < 0 ? -1 : (j + 1 < lm ? j + 1 : (lclosed ? 0 : -1));
                const int gi = __shfl_sync(0xffffffffu, lz, jn < 0 ? 0 : jn);
                const uint32_t gxy = __shfl_sync(0xffffffffu, lzxy, jn < 0 ? 0 : jn);
                if (jn >= 0 && ((sure >> j) & 1u) != 0u) {
                    best.i = gi;
                    best.xy = gxy;
                } else {
                    if (jn >= 0) star_take(e, best, gi, gxy);
                    const int guess = best.i;
#pragma unroll
                    for (int k = 0; k < FAR_KEEP; ++k)
                        if (keep[k] != PXY_NONE) star_take(e, best, tid + k * FAR_THREADS, keep[k]);
#pragma unroll 1
                    for (int i = tid + FAR_KEEP * FAR_THREADS; i < N; i += FAR_THREADS) {
                        const uint32_t xy = D.pxy[i];
                        if (xy != PXY_NONE) star_take(e, best, i, xy);
                    }
                    if (__syncthreads_or(best.i != guess)) {
                        star_cta_min(best, part[flip], lane, warp, NW, StarBest{-1, 0u, 0.0f},
                                     [&](StarBest& v) { star_reduce(e, v, lane); });
                        flip ^= 1;
                    }
                }
                if (best.i < 0) {
                    open = true;                // a hull edge
                    ok = hn >= 0 || R < 2;
                    break;
                }
                if (best.xy == q0xy) {
                    closed = ok = hn < 0;
                    break;
                }
                if (m >= STAR_NB) {
                    ok = false;
                    break;
                }
                if (tid == 0) { sm.nb[m] = best.i; sm.nxy[m] = best.xy; }
                ++m;
                if (best.xy == hpxy) break;
                j = __ffs(__ballot_sync(0xffffffffu, lzxy == best.xy)) - 1;
                e.q = best.i;
                e.pq = best.xy;
                e.ux = dx_p(best.xy, pp);
                e.uy = dy_p(best.xy, pp);
            }
        }
        __syncthreads();
        if (warp == 0) {
            const int nt = ok ? star_tris(m, closed) : 0;
            const int g = star_doublings(D, pp, sm.nxy, m, nt, qd2, open, lane);
            if (lane == 0) {
                if (g) atomicAdd(&D.ctr[13], g);
                if (!ok) set_err(err, ERRF_BOUNDS);
            }
            star_output(D, p, sm.nb, m, nt, lane, err);
        }
    }
}

// 256 points per CTA, both problems: each point's owned triangles (p, a,
// b) at its offset, the exclusive prefix sum of the owned counts in point
// order, so the list is in point order and the same on every run.  A CTA
// finds the sum of all points before its range itself (the star
// construction runs up to 2^21 pixels, some 10^4 points a view, so the
// repeated sums are cheap and save a separate scan launch); CTA 0 also
// sums every point and writes the triangle count ctr[0].
constexpr int EMIT_THREADS = 256;
__global__ void __launch_bounds__(EMIT_THREADS) k_star_emit(DelDev d0, DelDev d1, unsigned* err) {
    grid_dep_wait();
    __shared__ int ws[33];
    const DelDev& D = blockIdx.y ? d1 : d0;
    const int N = D.ctr[9];
    const int start = blockIdx.x * EMIT_THREADS, tid = threadIdx.x;
    if (start >= N && blockIdx.x != 0) return;
    const int lim = blockIdx.x == 0 ? N : start;     // CTA 0 sums everything (the total), the others their prefix
    int pre = 0, total = 0, tmp = 0;
    for (int i = tid; i < lim; i += EMIT_THREADS) {
        if (i < start) pre += D.tcnt[i];
        total += D.tcnt[i];
    }
    block_scan(pre, ws, &tmp);
    pre = tmp;
    block_scan(total, ws, &tmp);
    total = tmp;
    const int p = start + tid;
    const int c = p < N ? D.tcnt[p] : 0;
    int mine = 0;
    const int off = pre + block_scan(c, ws, &mine);
    if (blockIdx.x == 0 && tid == 0) {
        const bool fits = total <= D.Tmax;
        if (!fits) set_err(err, ERRF_TRI_COUNT);
        D.ctr[0] = fits ? total : 0;
    }
    if (c == 0) return;
    if (off + c > D.Tmax) {
        set_err(err, ERRF_TRI_COUNT);
        return;
    }
    const int32_t* slot = D.sown + size_t(p) * 2 * STAR_SLOT;
    const int32_t* src = c <= STAR_SLOT ? slot : D.spool + 2 * size_t(slot[0]);
    int32_t* t = D.tri + 3 * size_t(off);
    for (int j = 0; j < c; ++j) {
        t[3 * j] = p;
        t[3 * j + 1] = src[2 * j];
        t[3 * j + 2] = src[2 * j + 1];
    }
}

// The two hull pockets of one problem: the triangles, in its order, of the
// monotone-chain stack walk over the rows' first (last) points, every point
// on its own.  In the walk a point j is pushed onto
// pred(j), the point above it whose direction from j is outermost (the
// nearest of collinear ones), and pred(j) stays beneath it; j is popped by
// the first later point i that lies strictly outside the line pred(j) -> j
// (the chain being convex, such an i has popped everything above j before),
// which makes the triangle (pred(j), j, i).  Triangles come in order of i
// and, for one i, of falling j: a triangle's place is the number of smaller
// keys (i, -j).  pocket_points finds every row's pred and key, POCKET_LANES
// lanes a point, in blocks of k_strips; pocket_triangles places them in
// blocks of the next kernel, which also sets the triangle count ctr[0].
// Bound by latency (a chain of compares per point).  The walk itself, one
// thread a side, took k_strips to 120 us at 2880x1988 (398 rows), all points
// in one block 63; now 13.
constexpr int POCKET_LANES = 8;
struct PocketRows {                     // per side and row, in D.chain
    int32_t *key, *pred, *idx;
    __device__ PocketRows(const DelDev& D, int nrows, int side)
        : key(D.chain + side * nrows), pred(D.chain + (2 + side) * nrows), idx(D.chain + (4 + side) * nrows) {}
};
// The points of block `part`; sh: the coordinates of both sides' rows.
__device__ void pocket_points(const DelDev& D, const int32_t* __restrict__ row_off, int nrows, int part, int32_t* sh) {
    const int R = D.ctr[6], lane = threadIdx.x & 31, pl = threadIdx.x % POCKET_LANES;
    const int it = (part * int(blockDim.x) + int(threadIdx.x)) / POCKET_LANES;
    if (part * int(blockDim.x) >= 2 * R * POCKET_LANES) return;
    for (int e = threadIdx.x; e < 2 * R; e += blockDim.x) {
        const int side = e >= R, s = e - side * R, r = D.ne[s];
        const int pos = row_off[r] + (side ? D.rcnt[r] - 1 : 0);
        sh[e] = int32_t(D.sxy[pos]);
        if (part == 0) PocketRows(D, nrows, side).idx[s] = D.srt[pos];
    }
    __syncthreads();
    const int e = imin(it, 2 * R - 1), side = e >= R, j = e - side * R;
    const int32_t* xy = sh + side * R;
    const int sg = side ? -1 : 1;
    const uint32_t c = uint32_t(xy[j]);
    int pred = -1;
    int32_t px = 0, ph = 0;                 // pred's offset (mirrored x) and height above j
#pragma unroll 4
    for (int a = pl; a < j; a += POCKET_LANES) {
        const int32_t x = sg * dx_p(uint32_t(xy[a]), c), h = -dy_p(uint32_t(xy[a]), c);
        if (pred < 0 || x * ph <= px * h) { pred = a; px = x; ph = h; }
    }
#pragma unroll
    for (int o = 1; o < POCKET_LANES; o <<= 1) {
        const int qa = __shfl_xor_sync(0xffffffffu, pred, o);
        const int32_t qx = __shfl_xor_sync(0xffffffffu, px, o), qh = __shfl_xor_sync(0xffffffffu, ph, o);
        const int32_t l = qx * ph, g = px * qh;
        if (qa >= 0 && (pred < 0 || l < g || (l == g && qa > pred))) { pred = qa; px = qx; ph = qh; }
    }
    // orient(pred, j, i) on the outer side, relative to j: pred is at (px, -ph)
    int i = R;
    for (int i0 = j + 1; __any_sync(0xffffffffu, pred >= 0 && i == R && i0 < R); i0 += POCKET_LANES) {
        const int q = i0 + pl;
        bool out = false;
        if (pred >= 0 && q < R) {
            const int32_t x = sg * dx_p(uint32_t(xy[q]), c), y = dy_p(uint32_t(xy[q]), c);
            out = -px * y - ph * x > 0;
        }
        const unsigned all = __ballot_sync(0xffffffffu, out) >> (lane & ~(POCKET_LANES - 1));
        const unsigned m = all & ((1u << POCKET_LANES) - 1u);
        if (m && i == R) i = i0 + __ffs(m) - 1;
    }
    if (pl != 0 || it >= 2 * R) return;
    const PocketRows P(D, nrows, side);
    P.pred[j] = pred;
    static_assert(LATTICE_ROWS_MAX + 1 <= 8192, "a row takes 13 bits");
    P.key[j] = i < R ? (i << 13 | (8191 - j)) : INT_MAX;
    if (i < R) atomicAdd(&D.ctr[2 + side], 1);
}
// Each thread group places its point's triangle; sh: both sides' keys.
__device__ void pocket_triangles(const DelDev& D, int nrows, int part, int32_t* sh) {
    const int R = D.ctr[6], pl = threadIdx.x % POCKET_LANES;
    const int it = (part * int(blockDim.x) + int(threadIdx.x)) / POCKET_LANES;
    if (part * int(blockDim.x) >= 2 * R * POCKET_LANES) return;
    for (int e = threadIdx.x; e < 2 * R; e += blockDim.x) sh[e] = D.chain[(e >= R) * nrows + e - (e >= R ? R : 0)];
    __syncthreads();
    const int e = imin(it, 2 * R - 1), side = e >= R, j = e - side * R;
    const int32_t mine = sh[e];
    int k = 0;
#pragma unroll 4
    for (int q = pl; q < R; q += POCKET_LANES) k += sh[side * R + q] < mine;
#pragma unroll
    for (int o = 1; o < POCKET_LANES; o <<= 1) k += __shfl_xor_sync(0xffffffffu, k, o);
    if (it >= 2 * R || mine == INT_MAX || pl != 0) return;
    const PocketRows P(D, nrows, side);
    const int32_t ia = P.idx[P.pred[j]], ib = P.idx[j], ii = P.idx[mine >> 13];
    int32_t* t = D.tri + 3 * (size_t(D.ctr[1]) + (side ? D.ctr[2] : 0) + k);
    t[0] = ia;
    t[1] = side ? ii : ib;
    t[2] = side ? ib : ii;
}

// Block s < R: the points of non-empty row s, each placing its triangle in
// the strip below the row (as the upper row A) and in the strip above (as
// the lower row B).  Walking the merge of A[1..m) and B[1..n) by x (A first
// on equal x), each element advances its row by one point and creates one
// counter-clockwise triangle, whose other row's point and place in the strip
// a search finds for each element on its own (merge path).  The x of the
// two neighbouring rows are staged in shared memory, so the binary searches
// do not chase loads (a thread finding its row and both places through
// global memory: some fifty dependent loads).  The blocks from nrows on
// find the hull pockets' points meanwhile.
constexpr int STRIP_THREADS = 512;
__global__ void __launch_bounds__(STRIP_THREADS) k_strips(DelDev d0, DelDev d1, const int32_t* __restrict__ row_off,
                                                          int nrows) {
    grid_dep_wait();
    extern __shared__ int32_t sh[];
    const DelDev& D = blockIdx.y ? d1 : d0;
    if (D.ctr[7] == 0) return;
    if (int(blockIdx.x) >= nrows) {
        pocket_points(D, row_off, nrows, blockIdx.x - nrows, sh);
        return;
    }
    const int R = D.ctr[6], s = blockIdx.x;
    if (s >= R) return;
    const int r = D.ne[s], b = row_off[r], n = D.rcnt[r];
    const int ra = s > 0 ? D.ne[s - 1] : -1, rb = s + 1 < R ? D.ne[s + 1] : -1;
    const int ba = ra >= 0 ? row_off[ra] : 0, na = ra >= 0 ? D.rcnt[ra] : 0;
    const int bb = rb >= 0 ? row_off[rb] : 0, nb = rb >= 0 ? D.rcnt[rb] : 0;
    int32_t* xa = sh;
    int32_t* xb = sh + SORT_CAP;
    for (int i = threadIdx.x; i < na; i += STRIP_THREADS) xa[i] = px_of(D.sxy[ba + i]);
    for (int i = threadIdx.x; i < nb; i += STRIP_THREADS) xb[i] = px_of(D.sxy[bb + i]);
    __syncthreads();
    // how many of the sorted x[0..cnt) lie below v (or at it)
    auto below = [](const int32_t* x, int cnt, int32_t v) {
        int lo = 0, hi = cnt;
        while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            if (x[mid] < v) lo = mid + 1;
            else hi = mid;
        }
        return lo;
    };
    for (int k = 1 + threadIdx.x; k < n; k += STRIP_THREADS) {
        const int x = px_of(D.sxy[b + k]), ik = D.srt[b + k], ip = D.srt[b + k - 1];
        if (rb >= 0) {          // as the upper row of strip s: points below strictly left of x
            const int j = imax(below(xb, nb, x) - 1, 0);
            int32_t* o = D.tri + 3 * (size_t(D.soff[s]) + (k - 1) + j);
            o[0] = ip;
            o[1] = ik;
            o[2] = D.srt[bb + j];
        }
        if (ra >= 0) {          // as the lower row of strip s - 1: points above at or left of x
            const int i = imax(below(xa, na, x + 1) - 1, 0);
            int32_t* o = D.tri + 3 * (size_t(D.soff[s - 1]) + i + (k - 1));
            o[0] = D.srt[ba + i];
            o[1] = ik;
            o[2] = ip;
        }
    }
}

__device__ __forceinline__ uint32_t hash_cap(int T) {
    uint32_t need = uint32_t(imax(64, 6 * T));
    uint32_t c = 64;
    while (c < need) c <<= 1;
    return c;
}

// The last pocket_blocks blocks place the hull pockets' triangles.
constexpr int CLEAR_THREADS = 256;
__global__ void __launch_bounds__(CLEAR_THREADS) k_hash_clear(DelDev d0, DelDev d1, int nrows, int pocket_blocks) {
    grid_dep_wait();
    extern __shared__ int32_t sh[];
    const DelDev& D = blockIdx.y ? d1 : d0;
    const int T = D.ctr[7] ? D.ctr[1] + D.ctr[2] + D.ctr[3] : 0, clear = gridDim.x - pocket_blocks;
    if (blockIdx.x == 0 && threadIdx.x == 0) D.ctr[0] = T;
    if (int(blockIdx.x) >= clear) {
        if (T) pocket_triangles(D, nrows, blockIdx.x - clear, sh);
        return;
    }
    uint32_t cap = hash_cap(T);
    for (uint32_t i = blockIdx.x * CLEAR_THREADS + threadIdx.x; i < cap && i < D.Hmax; i += clear * CLEAR_THREADS) {
        D.hkey[i] = HASH_EMPTY;
        D.hcnt[i] = 0;
    }
}

__global__ void k_hash_insert(DelDev d0, DelDev d1, unsigned* err) {
    grid_dep_wait();
    const DelDev& D = blockIdx.y ? d1 : d0;
    const int T = D.ctr[0];
    const uint32_t cap = hash_cap(T), mask = cap - 1;
    if (cap > D.Hmax) { if (blockIdx.x == 0 && threadIdx.x == 0) set_err(err, ERRF_HASH); return; }
    for (int h = blockIdx.x * blockDim.x + threadIdx.x; h < 3 * T; h += gridDim.x * blockDim.x) {
        int t = h / 3, s = h % 3;
        uint64_t key = edge_key(D.tri[3 * t + s], D.tri[3 * t + (s + 1) % 3]);
        uint32_t slot = hash64(key) & mask;
        bool done = false;
        for (uint32_t probe = 0; probe < cap; ++probe) {
            unsigned long long prev = atomicCAS(&D.hkey[slot], HASH_EMPTY, (unsigned long long)key);
            if (prev == HASH_EMPTY || prev == key) {
                int pos = atomicAdd(&D.hcnt[slot], 1);
                if (pos < 2) D.hval[2 * slot + pos] = h;
                else set_err(err, ERRF_HASH);
                D.hslot[h] = int(slot);
                done = true;
                break;
            }
            slot = (slot + 1) & mask;
        }
        if (!done) set_err(err, ERRF_HASH);
    }
}

// Neighbour links from the hash, and the per-triangle flip state.
__global__ void k_link(DelDev d0, DelDev d1, unsigned* err) {
    grid_dep_wait();
    const DelDev& D = blockIdx.y ? d1 : d0;
    const int T = D.ctr[0];
    for (int h = blockIdx.x * blockDim.x + threadIdx.x; h < 3 * T; h += gridDim.x * blockDim.x) {
        int slot = D.hslot[h];
        if (slot < 0 || uint32_t(slot) >= D.Hmax) { set_err(err, ERRF_BOUNDS); D.opp[h] = -1; continue; }
        int c = D.hcnt[slot];
        int o = -1;
        if (c == 2) o = D.hval[2 * slot] == h ? D.hval[2 * slot + 1] : D.hval[2 * slot];
        else if (c != 1) set_err(err, ERRF_HASH);
        if (o >= 3 * T) { set_err(err, ERRF_BOUNDS); o = -1; }
        D.opp[h] = o;
    }
}

struct GAMin {
    __device__ void operator()(uint32_t* p, uint32_t v) const { atomicMin(p, v); }
};

// Shared round driver: one "group" (a CTA, or a cluster of CTAs) runs the
// rounds; `Sync` is its barrier.  Lists live in global memory; their
// counters in shared memory of the owning CTA.
//
// Fallback: one 1024-thread CTA per problem on global memory, for
// triangulations larger than the cluster kernel holds.  Every loop is
// bounded: `max_rounds` rounds at most (ERRF_FLIP_LIMIT).
__global__ void __launch_bounds__(FLIP_THREADS) k_flip_global(DelDev d0, DelDev d1, int max_rounds, unsigned* err) {
    grid_dep_wait();
    __shared__ int n_cand, n_flip, n_next, n_cur, stop;
    const DelDev& D = blockIdx.x ? d1 : d0;
    if (D.ctr[8] != 0) return;            // the cluster kernel handled this problem
    const int T = D.ctr[0];
    FlatTri<GAMin> m{D.tri, D.txy, D.opp, D.lock, D.fround, GAMin()};
    const int cand_cap = 3 * D.Tmax, wl_cap = 6 * D.Tmax;
    const int tid = threadIdx.x;
    // the two per-round push bitsets live in hslot, which k_link was the last to read
    const int mark_words = (3 * D.Tmax + 31) / 32, used_words = (3 * T + 31) / 32;
    uint32_t* const mark0 = reinterpret_cast<uint32_t*>(D.hslot);
    uint32_t* const mark1 = mark0 + mark_words;
    for (int t = tid; t < T; t += FLIP_THREADS) { D.lock[t] = LOCK_FREE; D.fround[t] = -1; }
    for (int i = tid; i < 3 * T; i += FLIP_THREADS) {     // packed corner coordinates of the flat storage
        const int v = D.tri[i];
        D.txy[i] = pack_xy(D.x[v], D.y[v]);
    }
    if (tid == 0) { n_cur = 3 * T; stop = 0; }
    __syncthreads();
    int round = 0, flips_total = 0;
    for (; round < max_rounds; ++round) {
        const int32_t* cur = (round & 1) ? D.wl1 : D.wl0;
        int32_t* nxt = (round & 1) ? D.wl0 : D.wl1;
        if (tid == 0) { n_cand = 0; n_next = 0; n_flip = 0; }
        __syncthreads();
        const int items = n_cur;
        for (int k = tid; k < items; k += FLIP_THREADS) {
            int h = round == 0 ? k : cur[k];
            if (!flip_propose(m, h, T, uint32_t(round), round == 0, [&](int hh, int nn) {
                    int idx = agg_inc(&n_cand);
                    if (idx < cand_cap) { D.cand[2 * idx] = hh; D.cand[2 * idx + 1] = nn; }
                }))
                set_err(err, ERRF_BOUNDS);
        }
        // this round's push bitset was last used two rounds ago
        uint32_t* const mark_nxt = (round & 1) ? mark0 : mark1;
        for (int i = tid; i < used_words; i += FLIP_THREADS) mark_nxt[i] = 0u;
        __syncthreads();
        const int nc = n_cand;
        if (tid == 0 && nc > cand_cap) { set_err(err, ERRF_BOUNDS); stop = 1; }
        __syncthreads();
        if (nc == 0 || stop) break;
        for (int c = tid; c < nc; c += FLIP_THREADS) {
            int h = D.cand[2 * c], n = D.cand[2 * c + 1];
            if (flip_apply(m, h, n, uint32_t(round))) {
                int f = agg_inc(&n_flip);
                D.flips[6 * f] = h / 3;
                D.flips[6 * f + 1] = n;
            }
        }
        __syncthreads();
        const int nf = n_flip;
        for (int f = tid; f < nf; f += FLIP_THREADS) {
            int t = D.flips[6 * f], n = D.flips[6 * f + 1];
            for (int k = 0; k < 4; ++k) {
                int r = flip_resolve_slot(m, outer_slot(t, n, k), uint32_t(round), T);
                if (r == -2) { set_err(err, ERRF_BOUNDS); r = -1; }
                D.flips[6 * f + 2 + k] = r;
            }
        }
        __syncthreads();
        auto push = [&](int x, int r) {
            int c;
            if (!claim_edge(mark_nxt, x, r, c)) return;
            int idx = agg_inc(&n_next);
            if (idx < wl_cap) nxt[idx] = c;
        };
        for (int f = tid; f < nf; f += FLIP_THREADS) {
            int t = D.flips[6 * f], n = D.flips[6 * f + 1];
            flip_relink(m, t, n, D.flips + 6 * f + 2);
            for (int k = 0; k < 4; ++k) push(outer_slot(t, n, k), D.flips[6 * f + 2 + k]);
        }
        for (int c = tid; c < nc; c += FLIP_THREADS) {
            int h = D.cand[2 * c], n = D.cand[2 * c + 1], t = h / 3;
            D.lock[t] = LOCK_FREE;
            D.lock[n] = LOCK_FREE;
            if (D.fround[t] != round && D.fround[n] != round) push(h, D.opp[h]);
        }
        flips_total += nf;
        __syncthreads();
        if (tid == 0) {
            if (n_next > wl_cap) { set_err(err, ERRF_BOUNDS); stop = 1; }
            n_cur = min(n_next, wl_cap);
        }
        __syncthreads();
        if (stop) break;
    }
    __syncthreads();
    for (int t = tid; t < T; t += FLIP_THREADS) normalise(D.tri + 3 * size_t(t));
    if (tid == 0) {
        D.ctr[4] = round + 1;
        D.ctr[5] = flips_total;
        if (round >= max_rounds) set_err(err, ERRF_FLIP_LIMIT);
    }
}

// ---------------------------------------------------------------------------
// Cluster kernel: the triangulation of one problem lives in the distributed
// shared memory of a cluster of CL_MAX CTAs.  Triangle t sits in CTA
// t >> shift at slot t & mask (a power-of-two slice); a record is 48 bytes
// (3 vertex indices, 3 packed coordinates, 3 links, two locks, flip round), so a
// cluster of 16 CTAs holds up to 65536 triangles.  Every access to another
// CTA's triangle is a distributed-shared-memory load, store or atomic; the
// phases are separated by cluster barriers.
constexpr int CL_THREADS = 1024;
constexpr int SLICE_MAX_LOG2 = 12;                 // 4096 triangles per CTA
constexpr int SLICE_MAX = 1 << SLICE_MAX_LOG2;
constexpr int WL_PER_CTA = 6 * SLICE_MAX;           // worklist entries per CTA and round
constexpr int CAND_PER_CTA = 6 * SLICE_MAX;         // proposals per CTA and round
constexpr int FLIP_PER_CTA = SLICE_MAX;             // flipped pairs per CTA and round
constexpr int CL_MARK = 3 * SLICE_MAX / 32;         // words of a per-round half-edge bitset
constexpr int CL_CAND = 864, CL_FLIP = 768;         // entries of a round's lists kept in shared memory
// shared memory: the triangle slice (48 bytes a triangle), two push bitsets
// and the heads of the round lists
constexpr size_t CL_SMEM = size_t(SLICE_MAX) * 48 + size_t(8) * CL_MARK + size_t(16) * CL_CAND + size_t(24) * CL_FLIP;
static_assert(CL_SMEM + 256 <= 227 * 1024, "one CTA's shared memory");
// round 0 stages each warp's owned half-edges (64 entries) in the flip list's
// shared part, which is unused until the first flips
static_assert(6 * CL_FLIP >= 64 * (CL_THREADS / 32), "round-0 staging does not fit");

// Shared-memory addresses of the cluster (32 bits): a word of CTA `rank`,
// its loads, stores and atomics.  (Through generic 64-bit pointers the rounds
// of k_flip_smem took 281 us at 2880x1988, so 271.)
__device__ __forceinline__ uint32_t cl_map(uint32_t addr, int rank) {
    uint32_t r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
__device__ __forceinline__ uint32_t cl_ld(uint32_t a) {
    uint32_t v;
    asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ void cl_st(uint32_t a, uint32_t v) {
    asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(a), "r"(v) : "memory");
}
__device__ __forceinline__ void cl_min(uint32_t a, uint32_t v) {
    asm volatile("red.relaxed.cluster.shared::cluster.min.u32 [%0], %1;" ::"r"(a), "r"(v) : "memory");
}
__device__ __forceinline__ uint32_t cl_or(uint32_t a, uint32_t v) {
    uint32_t o;
    asm volatile("atom.relaxed.cluster.shared::cluster.or.b32 %0, [%1], %2;" : "=r"(o) : "r"(a), "r"(v) : "memory");
    return o;
}
__device__ __forceinline__ int cl_add(uint32_t a, int v) {
    int o;
    asm volatile("atom.relaxed.cluster.shared::cluster.add.s32 %0, [%1], %2;" : "=r"(o) : "r"(a), "r"(v) : "memory");
    return o;
}

struct ClusterTri {
    uint32_t lv, lxy, lopp, llock, lround;   // addresses in the own CTA: vertices, coordinates and links
                                             // [3 * SLICE_MAX], locks and flip rounds [SLICE_MAX]
    int shift, mask;
    // word 3 t + k of an array of three words a triangle, word t of one
    __device__ __forceinline__ uint32_t at3(uint32_t base, int t, int k) const {
        return cl_map(base + 4u * uint32_t(3 * (t & mask) + k), t >> shift);
    }
    __device__ __forceinline__ uint32_t at1(uint32_t base, int t) const {
        return cl_map(base + 4u * uint32_t(t & mask), t >> shift);
    }
    __device__ int v(int t, int k) const { return int(cl_ld(at3(lv, t, k))); }
    __device__ uint32_t xy(int t, int k) const { return cl_ld(at3(lxy, t, k)); }
    __device__ int opp(int h) const { int t = h / 3; return int(cl_ld(at3(lopp, t, h - 3 * t))); }
    __device__ uint32_t lock(int t) const { return cl_ld(at1(llock, t)); }
    __device__ int32_t fround(int t) const { return int32_t(cl_ld(at1(lround, t))); }
    __device__ void lock_min(int t, uint32_t p) { cl_min(at1(llock, t), p); }
    __device__ void set_v(int t, int a, int b, int c, uint32_t pa, uint32_t pb, uint32_t pc) {
        const uint32_t V = at3(lv, t, 0), X = at3(lxy, t, 0);
        cl_st(V, a); cl_st(V + 4, b); cl_st(V + 8, c);
        cl_st(X, pa); cl_st(X + 4, pb); cl_st(X + 8, pc);
    }
    __device__ void set_opp(int h, int o) { int t = h / 3; cl_st(at3(lopp, t, h - 3 * t), uint32_t(o)); }
    __device__ void set_fround(int t, int32_t r) { cl_st(at1(lround, t), uint32_t(r)); }
};

// Point-table accessor for a problem that fits one SM: corner coordinates
// are looked up per vertex (4 bytes per support point instead of 12 per
// triangle), which leaves shared memory for the round lists.
struct PtTri {
    int32_t* lv;
    const uint32_t* pxy;
    int32_t* lopp;
    uint32_t* llock;
    int32_t* lround;
    __device__ int v(int t, int k) const { return lv[3 * t + k]; }
    __device__ uint32_t xy(int t, int k) const { return pxy[lv[3 * t + k]]; }
    __device__ int opp(int h) const { return lopp[h]; }
    __device__ uint32_t lock(int t) const { return *((volatile uint32_t*)llock + t); }
    __device__ int32_t fround(int t) const { return lround[t]; }
    __device__ void lock_min(int t, uint32_t p) { atomicMin(llock + t, p); }
    __device__ void set_v(int t, int a, int b, int c, uint32_t, uint32_t, uint32_t) {
        lv[3 * t] = a; lv[3 * t + 1] = b; lv[3 * t + 2] = c;
    }
    __device__ void set_opp(int h, int o) { lopp[h] = o; }
    __device__ void set_fround(int t, int32_t r) { lround[t] = r; }
};

// A round list whose first entries live in shared memory and the rest in
// global memory (records of `width` ints).
struct List2 {
    int32_t* s;
    int32_t* g;
    int scap, gcap, width;
    __device__ int32_t* slot(int i) const { return i < scap ? s + width * i : g + width * (i - scap); }
    __device__ int cap() const { return scap + gcap; }
};

constexpr int LOC_T = 4096;        // triangles of a one-SM problem
constexpr int LOC_PTS = 4096;      // support points (vertex ids) of a one-SM problem
constexpr int LOC_CAND = 1536;     // proposals of a round in shared memory (two round lists)
constexpr int LOC_FLIP = 1280;     // flipped pairs in shared memory
constexpr int LOC_MARK = (3 * LOC_T + 31) / 32;   // words of a per-round half-edge bitset
constexpr int FLIP_TAIL = 64;      // rounds with at most this many proposals run on one warp
constexpr size_t LOC_SMEM = size_t(36) * LOC_T + size_t(4) * LOC_PTS + size_t(16) * LOC_CAND +
                            size_t(24) * LOC_FLIP + size_t(8) * LOC_MARK;
// round 0 stages each warp's owned half-edges (64 entries) in the flip list's
// shared part, which is unused until the first flips
static_assert(6 * LOC_FLIP >= 64 * (1024 / 32), "round-0 staging does not fit");

// Flip rounds of one problem in one CTA: triangles, points and the round
// lists in shared memory.  Problems with more triangles or points are left
// (ctr[8] stays 0) to the cluster kernel.
//
// A round is three phases between barriers:
//   B   flip the proposals that won both locks; release the locks of the
//       round before; clear the next round's edge bitset;
//   C1  resolve the outer neighbours of every flipped pair (read only) and
//       propose, for the next round, each outer edge that is not locally
//       Delaunay (vertices are final once B is over, so the test needs no
//       links);
//   C2  write the links; re-propose the proposals that lost a lock while
//       neither of their triangles flipped (their test result is unchanged).
// Proposals of consecutive rounds use two lock arrays, so the next round's
// locks fill while this round's are still held.  The rounds, proposals and
// flips are those of the propose / flip / resolve / relink formulation with
// a worklist (the host emulation): only the tests move forward a phase.
__global__ void __launch_bounds__(1024) k_flip_local(DelDev d0, DelDev d1, int max_rounds, unsigned* err) {
    grid_dep_wait();
    extern __shared__ __align__(16) uint8_t lsm[];
    __shared__ int n_cand[2], n_flip;
    const DelDev& D = blockIdx.x ? d1 : d0;
    const int T = D.ctr[0], NP = D.ctr[9];
    if (D.ctr[8] != 0 || T > LOC_T || NP > LOC_PTS) return;
    const int tid = threadIdx.x, NT = blockDim.x;
    PtTri m;
    m.lv = reinterpret_cast<int32_t*>(lsm);
    m.lopp = m.lv + 3 * LOC_T;
    uint32_t* const lock0 = reinterpret_cast<uint32_t*>(m.lopp + 3 * LOC_T);
    uint32_t* const lock1 = lock0 + LOC_T;
    m.lround = reinterpret_cast<int32_t*>(lock1 + LOC_T);
    uint32_t* pxy = reinterpret_cast<uint32_t*>(m.lround + LOC_T);
    m.pxy = pxy;
    int32_t* sw = reinterpret_cast<int32_t*>(pxy + LOC_PTS);
    const List2 cand0{sw, D.ccand, LOC_CAND, CAND_PER_CTA, 2};
    const List2 cand1{sw + 2 * LOC_CAND, D.ccand + 2 * CAND_PER_CTA, LOC_CAND, CAND_PER_CTA, 2};
    const List2 flips{sw + 4 * LOC_CAND, D.cflips, LOC_FLIP, FLIP_PER_CTA, 6};
    uint32_t* const mark0 = reinterpret_cast<uint32_t*>(sw + 4 * LOC_CAND + 6 * LOC_FLIP);
    uint32_t* const mark1 = mark0 + LOC_MARK;
    for (int i = tid; i < NP; i += NT) pxy[i] = pack_xy(D.x[i], D.y[i]);
    for (int t = tid; t < T; t += NT) {
        for (int k = 0; k < 3; ++k) {
            m.lv[3 * t + k] = D.tri[3 * t + k];
            m.lopp[3 * t + k] = D.opp[3 * t + k];
        }
        lock0[t] = LOCK_FREE;
        lock1[t] = LOCK_FREE;
        m.lround[t] = -1;
    }
    if (tid == 0) { n_cand[0] = 0; n_cand[1] = 0; n_flip = 0; }
    __syncthreads();
    // round 0's proposals: every interior edge once
    m.llock = lock0;
    {
        auto add0 = [&](int hh, int nn) {
            int idx = agg_inc(&n_cand[0]);
            if (idx < cand0.cap()) { int32_t* c = cand0.slot(idx); c[0] = hh; c[1] = nn; }
        };
        propose_owned(0, 3 * T, flips.s + 64 * (tid >> 5), [&](int h) { return m.lopp[h]; }, [&](int h) {
            if (!flip_propose(m, h, T, 0u, false, add0)) set_err(err, ERRF_BOUNDS);
        });
    }
    __syncthreads();
    int round = 0, flips_total = 0, nc_prev = 0;
    bool converged = false;
    // One round with threads [0, nt) of the CTA (index `me`), `sync` the
    // barrier among them.  Returns 0 to continue, 1 when converged, 2 on
    // an overflow.
    auto flip_round = [&](const int me, const int nt, auto&& sync) -> int {
        const int cur = round & 1, nxt = cur ^ 1;
        // selected by value: a dynamically indexed pair would live in local memory
        const List2 cand_cur = cur ? cand1 : cand0, cand_nxt = cur ? cand0 : cand1;
        uint32_t* const lock_cur = cur ? lock1 : lock0;
        uint32_t* const lock_nxt = cur ? lock0 : lock1;
        uint32_t* const mark_nxt = cur ? mark0 : mark1;
        const int nc = n_cand[cur];             // final since the last barrier; equal in every thread
        if (nc == 0) { converged = true; return 1; }
        if (nc > cand_cur.cap()) {
            if (me == 0) set_err(err, ERRF_BOUNDS);
            return 2;
        }
        // B: flip the winners; release the previous round's locks; clear the next round's bitset
        m.llock = lock_cur;
        for (int c = me; c < nc; c += nt) {
            const int32_t* cc = cand_cur.slot(c);
            int h = cc[0], n = cc[1];
            if (flip_apply(m, h, n, uint32_t(round))) {
                int f = agg_inc(&n_flip);     // at most T/2 <= flips.cap()
                int32_t* q = flips.slot(f);
                q[0] = h / 3; q[1] = n;
            }
        }
        for (int c = me; c < nc_prev; c += nt) {
            const int32_t* cc = cand_nxt.slot(c);
            lock_nxt[cc[0] / 3] = LOCK_FREE;
            lock_nxt[cc[1]] = LOCK_FREE;
        }
        for (int i = me; i < LOC_MARK; i += nt) mark_nxt[i] = 0u;
        sync();
        const int nf = n_flip;
        auto add_next = [&](int hh, int nn, uint32_t p) {
            atomicMin(lock_nxt + hh / 3, p);
            atomicMin(lock_nxt + nn, p);
            int idx = agg_inc(&n_cand[nxt]);
            if (idx < cand_nxt.cap()) { int32_t* c = cand_nxt.slot(idx); c[0] = hh; c[1] = nn; }
        };
        // C1: resolve the outer neighbours (read only); propose the outer edges.
        // The four edges of a pair go through each step together (claims,
        // tests, one list reservation per warp), so their latencies overlap.
        for (int f = me; f < nf; f += nt) {
            int32_t* q = flips.slot(f);
            const int t = q[0], n = q[1];
            int r[4], c[4], tw[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                r[k] = flip_resolve_slot(m, outer_slot(t, n, k), uint32_t(round), T);
                if (r[k] == -2) { set_err(err, ERRF_BOUNDS); r[k] = -1; }
            }
#pragma unroll
            for (int k = 0; k < 4; ++k) q[2 + k] = r[k];
            uint32_t old[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const int x = outer_slot(t, n, k);
                // a hull edge (r < 0) tests against its own triangle, is never claimed, and is masked out
                c[k] = r[k] >= 0 ? min(x, r[k]) : x;
                tw[k] = r[k] >= 0 ? (c[k] == x ? r[k] : x) : x;
                old[k] = r[k] >= 0 ? atomicOr(mark_nxt + (c[k] >> 5), 1u << (c[k] & 31)) : ~0u;
            }
            // the four tests are independent (no branch between them), so their loads overlap
            bool flippable[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) flippable[k] = edge_flippable(m, c[k], tw[k]);
            unsigned want = 0;
#pragma unroll
            for (int k = 0; k < 4; ++k)
                if (!(old[k] & (1u << (c[k] & 31))) && flippable[k]) want |= 1u << k;
            // reserve popc(want) entries per lane with one atomic per warp
            const unsigned act = __activemask();
            const int lane = tid & 31, cnt = __popc(want);
            const unsigned b0 = __ballot_sync(act, cnt & 1), b1 = __ballot_sync(act, cnt & 2),
                           b2 = __ballot_sync(act, cnt & 4);
            const unsigned lt = (1u << lane) - 1u;
            const int before = __popc(b0 & lt) + 2 * __popc(b1 & lt) + 4 * __popc(b2 & lt);
            const int total = __popc(b0) + 2 * __popc(b1) + 4 * __popc(b2);
            const int leader = __ffs(act) - 1;
            int base = 0;
            if (lane == leader && total > 0) base = atomicAdd(&n_cand[nxt], total);
            base = __shfl_sync(act, base, leader) + before;
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                if (!(want & (1u << k))) continue;
                const uint32_t p = prio(uint32_t(c[k]), uint32_t(round + 1));
                atomicMin(lock_nxt + c[k] / 3, p);
                atomicMin(lock_nxt + tw[k] / 3, p);
                if (base < cand_nxt.cap()) { int32_t* e = cand_nxt.slot(base); e[0] = c[k]; e[1] = tw[k] / 3; }
                ++base;
            }
        }
        sync();
        // C2: relink; re-propose the lost proposals (their edges are no outer
        // edge of a flipped pair, so the bitset need not see them)
        if (me == 0) { n_flip = 0; n_cand[cur] = 0; }   // both were read before the last barrier
        for (int f = me; f < nf; f += nt) {
            int32_t* q = flips.slot(f);
            flip_relink(m, q[0], q[1], q + 2);
        }
        for (int c = me; c < nc; c += nt) {
            const int32_t* cc = cand_cur.slot(c);
            const int h = cc[0], n = cc[1], t = h / 3;
            if (m.fround(t) != round && m.fround(n) != round) add_next(h, n, prio(uint32_t(h), uint32_t(round + 1)));
        }
        flips_total += nf;
        nc_prev = nc;
        sync();
        return 0;
    };
    // The whole CTA runs the rounds while they are large; once a round
    // starts with at most FLIP_TAIL proposals, warp 0 runs every remaining
    // round alone with warp barriers (the same rounds: the phases only lose
    // the cost of block-wide barriers), and the other warps wait at the end.
    int state = 0;
    for (; round < max_rounds; ++round) {
        const int nc_top = n_cand[round & 1];   // uniform: read after a block barrier
        if (nc_top > 0 && nc_top <= FLIP_TAIL) break;
        state = flip_round(tid, NT, [] { __syncthreads(); });
        if (state) break;
    }
    if (state == 0 && round < max_rounds && tid < 32) {
        for (; round < max_rounds; ++round) {
            state = flip_round(tid, 32, [] { __syncwarp(); });
            if (state) break;
        }
    }
    __syncthreads();
    for (int t = tid; t < T; t += NT) {
        int32_t v[3] = {m.lv[3 * t], m.lv[3 * t + 1], m.lv[3 * t + 2]};
        normalise(v);
        for (int k = 0; k < 3; ++k) D.tri[3 * t + k] = v[k];
    }
    if (tid == 0) {
        D.ctr[8] = 1;
        D.ctr[4] = round + 1;
        D.ctr[5] = flips_total;
        if (!converged) set_err(err, ERRF_FLIP_LIMIT);
    }
}

struct ClusterSync {
    __device__ void operator()() const { cg::this_cluster().sync(); }
    template <class X>
    __device__ X* remote(X* p, int r) const { return cg::this_cluster().map_shared_rank(p, unsigned(r)); }
    __device__ int rank() const { return int(cg::this_cluster().block_rank()); }
};

// Flip rounds in distributed shared memory: a cluster of csize CTAs, each
// holding a slice of at most SLICE_MAX triangles.  A problem already handled
// (ctr[8] set by the one-SM kernel) or larger than csize * SLICE_MAX is
// skipped; the kernel that handles a problem sets ctr[8].
//
// The rounds are those of k_flip_local (three phases between cluster
// barriers: B flip, C1 resolve + propose the outer edges, C2 relink +
// re-propose the lost proposals; two lock arrays by round parity).  A
// proposal is queued at the CTA that owns its lower half-edge, so a CTA
// flips at most its own triangles in a round (f < FLIP_PER_CTA), and that
// CTA releases the proposal's locks in the next round.
//
// Latency bounds it: some twenty rounds, most of them with a few hundred
// proposals or fewer, of three chains of remote accesses (about 300 cycles
// each, a barrier 750).  So the lists' heads lie in shared memory, the four
// edges of a pair go through each step of C1 together, on the pair's own
// four vertices, and a warp's lanes read the CTAs' counts once: 367 -> 271 us
// at 2880x1988.
__global__ void __launch_bounds__(CL_THREADS) k_flip_smem(DelDev d0, DelDev d1, int csize, int max_rounds,
                                                          unsigned* err) {
    grid_dep_wait();
    using Sync = ClusterSync;
    extern __shared__ __align__(16) uint8_t csm[];
    __shared__ int n_cand[2], n_flip, s_flips;
    Sync sync;
    const int rank = sync.rank();
    const int prob = blockIdx.x / csize;
    const DelDev& D = prob ? d1 : d0;
    const int T = D.ctr[0];
    // uniform over the CTAs of a problem: no barrier has been passed yet
    if (D.ctr[8] != 0 || T > csize * SLICE_MAX) return;
    int shift = 6;
    while ((csize << shift) < T) ++shift;
    ClusterTri m;
    // the own slice
    int32_t* const lv = reinterpret_cast<int32_t*>(csm);
    uint32_t* const lxy = reinterpret_cast<uint32_t*>(lv + 3 * SLICE_MAX);
    int32_t* const lopp = reinterpret_cast<int32_t*>(lxy + 3 * SLICE_MAX);
    uint32_t* const lock0 = reinterpret_cast<uint32_t*>(lopp + 3 * SLICE_MAX);
    uint32_t* const lock1 = lock0 + SLICE_MAX;
    int32_t* const lround = reinterpret_cast<int32_t*>(lock1 + SLICE_MAX);
    uint32_t* const mark0 = reinterpret_cast<uint32_t*>(lround + SLICE_MAX);
    m.lv = smem_u32(lv);
    m.lxy = smem_u32(lxy);
    m.lopp = smem_u32(lopp);
    m.lround = smem_u32(lround);
    uint32_t* const mark1 = mark0 + CL_MARK;
    int32_t* const heads = reinterpret_cast<int32_t*>(mark1 + CL_MARK);
    m.shift = shift;
    m.mask = (1 << shift) - 1;
    const int t0 = rank << shift, t1 = min(T, (rank + 1) << shift);
    const int tid = threadIdx.x;
    for (int t = t0 + tid; t < t1; t += CL_THREADS) {
        const int l = t - t0;
        int v[3], o[3];
        uint32_t xy[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) { v[k] = D.tri[3 * t + k]; o[k] = D.opp[3 * t + k]; }
#pragma unroll
        for (int k = 0; k < 3; ++k) xy[k] = pack_xy(D.x[v[k]], D.y[v[k]]);
#pragma unroll
        for (int k = 0; k < 3; ++k) { lv[3 * l + k] = v[k]; lxy[3 * l + k] = xy[k]; lopp[3 * l + k] = o[k]; }
        lock0[l] = LOCK_FREE;
        lock1[l] = LOCK_FREE;
        lround[l] = -1;
    }
    if (tid == 0) { n_cand[0] = 0; n_cand[1] = 0; n_flip = 0; }
    // the proposal lists of CTA r, by round parity, and the own flip list
    auto cand_list = [&](int parity, int r) -> List2 {
        int32_t* g = parity ? D.cwl + size_t(r) * 2 * WL_PER_CTA : D.ccand + size_t(r) * 2 * CAND_PER_CTA;
        return List2{sync.remote(heads + parity * 2 * CL_CAND, r), g, CL_CAND, CAND_PER_CTA - CL_CAND, 2};
    };
    const List2 flips{heads + 4 * CL_CAND, D.cflips + size_t(rank) * 6 * FLIP_PER_CTA, CL_FLIP, FLIP_PER_CTA - CL_FLIP,
                      6};
    sync();
    // round 0's proposals: every interior edge of the own slice once
    m.llock = smem_u32(lock0);
    {
        const List2 c0 = cand_list(0, rank);
        auto add0 = [&](int hh, int nn) {
            int idx = agg_inc(&n_cand[0]);
            if (idx < CAND_PER_CTA) { int32_t* c = c0.slot(idx); c[0] = hh; c[1] = nn; }
        };
        propose_owned(3 * t0, 3 * t1, flips.s + 64 * (tid >> 5), [&](int h) { return m.opp(h); }, [&](int h) {
            if (!flip_propose(m, h, T, 0u, false, add0)) set_err(err, ERRF_BOUNDS);
        });
    }
    sync();
    int round = 0, flips_total = 0, nc_prev = 0;
    bool converged = false;
    for (; round < max_rounds; ++round) {
        const int cur = round & 1, nxt = cur ^ 1;
        const List2 cand_cur = cand_list(cur, rank);
        const List2 cand_old = cand_list(nxt, rank);   // the previous round's list, until C1 refills it
        const uint32_t lock_nxt = smem_u32(cur ? lock0 : lock1);
        uint32_t* const mark_nxt = cur ? mark0 : mark1;
        // every CTA's count is final since the last barrier, so all CTAs take the same decision
        // (each warp's lanes read one count each)
        const int lane = tid & 31, theirs = lane < csize ? *sync.remote(&n_cand[cur], lane) : 0;
        const int total = __reduce_add_sync(0xffffffffu, theirs);
        const bool over = __any_sync(0xffffffffu, theirs > CAND_PER_CTA);
        if (over) {
            if (tid == 0) set_err(err, ERRF_BOUNDS);
            break;
        }
        if (total == 0) { converged = true; break; }
        const int nc = n_cand[cur];
        // B: flip the winners (own triangles); release the previous round's locks; clear the next bitset
        m.llock = smem_u32(cur ? lock1 : lock0);
        for (int c = tid; c < nc; c += CL_THREADS) {
            const int32_t* cc = cand_cur.slot(c);
            const int h = cc[0], n = cc[1];
            if (flip_apply(m, h, n, uint32_t(round))) {
                const int f = agg_inc(&n_flip);
                if (f < FLIP_PER_CTA) { int32_t* q = flips.slot(f); q[0] = h / 3; q[1] = n; }
            }
        }
        for (int c = tid; c < nc_prev; c += CL_THREADS) {
            const int32_t* cc = cand_old.slot(c);
            const int t = cc[0] / 3, n = cc[1];
            cl_st(m.at1(lock_nxt, t), LOCK_FREE);
            cl_st(m.at1(lock_nxt, n), LOCK_FREE);
        }
        for (int i = tid; i < CL_MARK; i += CL_THREADS) mark_nxt[i] = 0u;
        sync();
        const int nf = min(n_flip, FLIP_PER_CTA);
        // a proposal for the next round, queued at the CTA owning its lower half-edge h
        auto add_next = [&](int h, int n, uint32_t p) {
            cl_min(m.at1(lock_nxt, h / 3), p);
            cl_min(m.at1(lock_nxt, n), p);
            const int owner = (h / 3) >> shift;
            int idx = agg_inc_keyed(sync.remote(&n_cand[nxt], owner));
            if (idx < CAND_PER_CTA) {
                int32_t* e = cand_list(nxt, owner).slot(idx);
                e[0] = h;
                e[1] = n;
            }
        };
        // C1: resolve the outer neighbours (read only); propose the outer edges
        for (int f = tid; f < nf; f += CL_THREADS) {
            int32_t* q = flips.slot(f);
            const int t = q[0], n = q[1];
            // the pair's vertices in the order of its outer edges: c, a, d, b
            const int32_t id[4] = {m.v(t, 0), m.v(t, 1), m.v(t, 2), m.v(n, 1)};
            const uint32_t xy[4] = {m.xy(t, 0), m.xy(t, 1), m.xy(t, 2), m.xy(n, 1)};
            int32_t r[4];
            flip_resolve4(m, t, n, id, uint32_t(round), T, r);
            int c[4], tw[4], vd[4];
            uint32_t xd[4];
            unsigned claimed = 0;
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                if (r[k] == -2) { set_err(err, ERRF_BOUNDS); r[k] = -1; }
                q[2 + k] = r[k];
                const int x = outer_slot(t, n, k);
                // a hull edge (r < 0) is never claimed
                c[k] = r[k] >= 0 ? min(x, r[k]) : x;
                tw[k] = r[k] >= 0 ? max(x, r[k]) : x;
                // the vertex beyond the edge
                const int o = r[k] >= 0 ? r[k] : x, to = o / 3, so = o % 3;
                vd[k] = m.v(to, so == 0 ? 2 : so - 1);
                xd[k] = m.xy(to, so == 0 ? 2 : so - 1);
            }
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                // the edge's bit lives at the CTA that owns its lower half-edge
                const int owner = (c[k] / 3) >> shift;
                const int lb = c[k] - 3 * (owner << shift);
                const uint32_t bit = 1u << (lb & 31);
                if (r[k] >= 0 && !(cl_or(cl_map(smem_u32(mark_nxt) + 4u * uint32_t(lb >> 5), owner), bit) & bit)) claimed |= 1u << k;
            }
            // edge_flippable from the pair's side (the determinant and the
            // perturbation are the same from either side)
            unsigned want = 0;
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const int k1 = (k + 1) & 3, kc = k == 0 || k == 3 ? 2 : 0;
                if (inside_sos_p(id[k], xy[k], id[k1], xy[k1], id[kc], xy[kc], vd[k], xd[k])) want |= 1u << k;
            }
            want &= claimed;
            // add_next for the four edges, step by step
            const unsigned act = __activemask();
            int base[4], lead[4], before[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const int owner = (c[k] / 3) >> shift;
                const bool w = want >> k & 1u;
                const unsigned peers = __match_any_sync(act, w ? owner : -1);
                lead[k] = __ffs(peers) - 1;
                before[k] = __popc(peers & ((1u << lane) - 1u));
                base[k] = 0;
                if (w && lane == lead[k]) base[k] = cl_add(cl_map(smem_u32(&n_cand[nxt]), owner), __popc(peers));
            }
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                if (!(want >> k & 1u)) continue;
                const uint32_t p = prio(uint32_t(c[k]), uint32_t(round + 1));
                cl_min(m.at1(lock_nxt, c[k] / 3), p);
                cl_min(m.at1(lock_nxt, tw[k] / 3), p);
            }
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const int idx = __shfl_sync(act, base[k], lead[k]) + before[k];
                if ((want >> k & 1u) && idx < CAND_PER_CTA) {
                    int32_t* e = cand_list(nxt, (c[k] / 3) >> shift).slot(idx);
                    e[0] = c[k];
                    e[1] = tw[k] / 3;
                }
            }
        }
        sync();
        // C2: relink; re-propose the own proposals that lost (no outer edge of a flipped pair)
        if (tid == 0) { n_flip = 0; n_cand[cur] = 0; }   // both were read before the last barrier
        for (int f = tid; f < nf; f += CL_THREADS) {
            const int32_t* q = flips.slot(f);
            flip_relink(m, q[0], q[1], q + 2);
        }
        for (int c = tid; c < nc; c += CL_THREADS) {
            const int32_t* cc = cand_cur.slot(c);
            const int h = cc[0], n = cc[1], t = h / 3;
            const int rt = m.fround(t), rn = m.fround(n);
            if (rt != round && rn != round) add_next(h, n, prio(uint32_t(h), uint32_t(round + 1)));
        }
        flips_total += nf;
        nc_prev = nc;
        sync();
    }
    // write back this CTA's slice
    for (int t = t0 + tid; t < t1; t += CL_THREADS) {
        const int l = t - t0;
        int32_t v[3] = {lv[3 * l], lv[3 * l + 1], lv[3 * l + 2]};
        normalise(v);
        for (int k = 0; k < 3; ++k) D.tri[3 * t + k] = v[k];
    }
    if (tid == 0) s_flips = flips_total;
    sync();
    if (rank == 0 && tid == 0) {
        int total = 0;
        for (int r = 0; r < csize; ++r) total += *sync.remote(&s_flips, r);
        D.ctr[8] = 1;
        D.ctr[4] = round + 1;
        D.ctr[5] = total;
        if (!converged) set_err(err, ERRF_FLIP_LIMIT);
    }
    sync();   // keep every CTA's shared memory alive until remote readers are done
}

}  // namespace

int cluster_size_for_flip() {
    int sizes[2] = {16, 8};
    size_t smem = CL_SMEM;
    allow_smem(k_flip_smem);
    cudaFuncSetAttribute(k_flip_smem, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    for (int cs : sizes) {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(2 * cs);
        cfg.blockDim = dim3(CL_THREADS);
        cfg.dynamicSmemBytes = smem;
        cudaLaunchAttribute attr;
        attr.id = cudaLaunchAttributeClusterDimension;
        attr.val.clusterDim.x = cs;
        attr.val.clusterDim.y = 1;
        attr.val.clusterDim.z = 1;
        cfg.attrs = &attr;
        cfg.numAttrs = 1;
        int n = 0;
        if (cudaOccupancyMaxActiveClusters(&n, k_flip_smem, &cfg) == cudaSuccess && n >= 2) return cs;
        cudaGetLastError();
    }
    return 0;
}

cudaError_t launch_delaunay(DelDev& d0, DelDev& d1, const int32_t* row_off, int nrows, int nmax, int W, int H,
                            int step, int crow, int num_sms, int csize, unsigned* err, cudaStream_t st,
                            int* nlaunch, bool flips, bool force_global, int round_limit) {
    const int xbs = flips ? 0 : (W + 7) / 8 + 1;
    launch_k(k_rowsort, dim3(nrows, 2), ROW_THREADS, 0, st, d0, d1, row_off, nrows, xbs, err);
    const size_t plan_smem = size_t(PLAN_ARRAYS) * sizeof(int32_t) * nrows;
    const RowGeom rg{step, crow, H, 1.0f / float(step)};
    allow_smem(k_plan);
    launch_k(k_plan, 2, 1024, plan_smem, st, d0, d1, row_off, nrows, rg, flips ? 1 : 0, err);
    if (!flips) {
        launch_k(k_star, dim3(2, imax(1, imin((nmax + STAR_WARPS - 1) / STAR_WARPS, 6 * num_sms))), STAR_WARPS * 32,
                 0, st, d0, d1, nrows, rg, xbs, err);
        launch_k(k_star_far, dim3(2, imax(1, imin(nmax, 2 * num_sms))), FAR_THREADS, 0, st, d0, d1, err);
        launch_k(k_star_emit, dim3(imax(1, (nmax + EMIT_THREADS - 1) / EMIT_THREADS), 2), EMIT_THREADS, 0, st, d0, d1,
                 err);
        if (nlaunch) *nlaunch += 5;
        return cudaGetLastError();
    }
    // shared memory: two rows' coordinates, or the pockets' rows
    const size_t smem = std::max(size_t(2) * nrows, size_t(2) * SORT_CAP) * sizeof(int32_t);
    const int blocks = 4 * num_sms;
    auto pockets = [&](int threads) { return (2 * nrows * POCKET_LANES + threads - 1) / threads; };
    allow_smem(k_strips);
    launch_k(k_strips, dim3(nrows + pockets(STRIP_THREADS), 2), STRIP_THREADS, smem, st, d0, d1, row_off, nrows);
    launch_k(k_hash_clear, dim3(blocks + pockets(CLEAR_THREADS), 2), CLEAR_THREADS, size_t(2) * nrows * sizeof(int32_t),
             st, d0, d1, nrows, pockets(CLEAR_THREADS));
    launch_k(k_hash_insert, dim3(blocks, 2), 256, 0, st, d0, d1, err);
    launch_k(k_link, dim3(blocks, 2), 256, 0, st, d0, d1, err);
    int launched = 6;
    const int max_rounds = round_limit > 0 ? round_limit : 100000;
    if (!force_global) {
        allow_smem(k_flip_local);
        launch_k(k_flip_local, 2, 1024, LOC_SMEM, st, d0, d1, max_rounds, err);
        ++launched;
    }
    if (csize > 0 && !force_global) {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(2 * csize);
        cfg.blockDim = dim3(CL_THREADS);
        cfg.dynamicSmemBytes = CL_SMEM;
        cfg.stream = st;
        cudaLaunchAttribute attr;
        attr.id = cudaLaunchAttributeClusterDimension;
        attr.val.clusterDim.x = csize;
        attr.val.clusterDim.y = 1;
        attr.val.clusterDim.z = 1;
        cfg.attrs = &attr;
        cfg.numAttrs = 1;
        cudaError_t e = cudaLaunchKernelEx(&cfg, k_flip_smem, d0, d1, csize, max_rounds, err);
        if (e != cudaSuccess) return e;
        ++launched;
    }
    // The fallback, for triangulations larger than a cluster holds; not
    // launched when none can be (at most 2 * nmax + 16 triangles).  It packs
    // the corner coordinates itself; every flip kernel writes its triangles
    // rotated to start at their smallest vertex index.
    if (force_global || csize == 0 || 2LL * nmax + 16 > (long long)csize * SLICE_MAX) {
        launch_k(k_flip_global, 2, FLIP_THREADS, 0, st, d0, d1, max_rounds, err);
        ++launched;
    }
    if (nlaunch) *nlaunch += launched;
    return cudaGetLastError();
}

}  // namespace elas
