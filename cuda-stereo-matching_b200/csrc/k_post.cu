// Post-filters: speckle removal, gap interpolation, adaptive mean, median.
//
// The reference declares these only as parameters (src/Elas.h:31-36,
// KernelsCommon.h:19-21) and its process() stops after the left/right check
// (src/Elas.cu:107-119).  The semantics are the project's own and are
// written out in the CPU oracle (oracle/elas_oracle.cpp, orc_postprocess):
//   speckle   4-connected segments (|d_p - d_q| <= speckle_sim_threshold);
//             segments smaller than speckle_size become invalid.  Union-find
//             with atomic hooking of the larger root under the smaller.
//   gap       rows, then columns: a run of <= ipol_gap_width invalid pixels
//             between valid a and b becomes (a+b)/2 if |a-b| <= 3 else
//             min(a,b).  Widths up to 8 run inside the fused tile kernel,
//             wider gaps as a row pass and a column pass.
//   mean      5x5 weighted mean of valid pixels, w = 1/(1+(d_q-d_p)^2).
//   median    lower median of the valid pixels of the 3x3 window.
#include <cuda_runtime.h>
#include <mutex>
#include <type_traits>
#include "../../include/elas_b200.h"
#include "common.cuh"
#include "launch.cuh"
#include "kernels.h"

namespace elas {

namespace {

constexpr int UF_LIMIT = 1 << 22;   // bound on any union-find walk / retry loop

// Root of x with path halving (labels only ever move to a smaller index, so
// concurrent halving keeps every node in its tree).
__device__ __forceinline__ int uf_find(int32_t* lab, int x, unsigned* err) {
    for (int it = 0; it < UF_LIMIT; ++it) {
        int p = lab[x];
        if (p == x) return x;
        int gp = lab[p];
        if (gp != p) lab[x] = gp;
        x = p;
    }
    atomicOr(err, ERRF_BOUNDS);
    return x;
}

// Labels start at the left neighbour when it is connected (the most common
// union), else at the pixel itself.  One thread per pixel on a 1-D grid (a
// map of any height fits).
__global__ void k_uf_init(const float* __restrict__ D, int32_t* __restrict__ lab, int32_t* __restrict__ sz, int W,
                          int H, float thr) {
    grid_dep_wait();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= W * H) return;
    const int u = i % W;
    float d = D[i];
    int l = -1;
    if (d >= 0) {
        l = i;
        if (u > 0) {
            float q = D[i - 1];
            if (q >= 0 && fabsf(q - d) <= thr) l = i - 1;
        }
    }
    lab[i] = l;
    sz[i] = 0;
}

__device__ void uf_union(int32_t* lab, int a, int b, unsigned* err) {
    for (int it = 0; it < UF_LIMIT; ++it) {
        int ra = uf_find(lab, a, err), rb = uf_find(lab, b, err);
        if (ra == rb) return;
        if (ra < rb) {   // keep (a, ra) and (b, rb) paired: hook the larger root
            int t = ra; ra = rb; rb = t;
            t = a; a = b; b = t;
        }
        int old = atomicCAS(&lab[ra], ra, rb);
        if (old == ra) return;
        a = old;         // ra gained a parent meanwhile: continue from it
    }
    atomicOr(err, ERRF_BOUNDS);
}

__global__ void k_uf_union(const float* __restrict__ D, int32_t* lab, int W, int H, float thr, unsigned* err) {
    grid_dep_wait();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= W * H) return;
    const int u = i % W, v = i / W;
    float d = D[i];
    if (d < 0) return;
    if (u + 1 < W) {
        float q = D[i + 1];
        if (q >= 0 && fabsf(q - d) <= thr) uf_union(lab, i, i + 1, err);
    }
    if (v + 1 < H) {
        float q = D[i + W];
        if (q >= 0 && fabsf(q - d) <= thr) uf_union(lab, i, i + W, err);
    }
}

// Root of every pixel into `root` (written only by its own thread: `lab`
// itself may still receive path-halving writes from other threads) and
// segment sizes; lanes of a warp that share a root add once (segments are
// large, so this removes most of the contention on the root counters).
__global__ void k_uf_count(int32_t* lab, int32_t* __restrict__ root, int32_t* sz, int n, unsigned* err) {
    grid_dep_wait();
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    int r = -1;
    if (i < n && lab[i] >= 0) r = uf_find(lab, i, err);
    if (i < n) root[i] = r;
    unsigned peers = __match_any_sync(0xffffffffu, r);
    int leader = __ffs(peers) - 1;
    if (r >= 0 && (threadIdx.x & 31) == leader) atomicAdd(&sz[r], __popc(peers));
}

// ---------------------------------------------------------------------------
// Speckle segmentation in tiles.  The segments (4-connected valid pixels,
// |d_p - d_q| <= thr) are labelled first inside every 32x32 tile with a
// union-find in shared memory; only links across tile borders then go
// through the global union-find, and sizes are counted once per tile-local
// component.  The segments, hence the result, are those of a whole-image
// union-find.
//   lab[i]  the global index of i's tile-local root (-1 invalid); the local
//           roots are the nodes of the global forest (a local root's entry is
//           its parent there, itself until the border pass hooks it)
//   sz[r]   at a local root r only: the pixel count of its tile component;
//           after the count, -(global root + 1)
//   acc[g]  the segment size at global root g (zeroed at every local root by
//           the tile kernel; global roots are local roots)
//   roots   [0] the number of local roots, then their global indices
// Only lab is written per pixel.  A pixel j's segment size is then
// acc[-sz[lab[j]] - 1]: lab[j] is j's local root or, for a local root that
// was hooked, another local root of the same segment.
constexpr int SPK_T = 32;

__device__ __forceinline__ int lfind(int* L, int x) {
    for (int it = 0; it < SPK_T * SPK_T; ++it) {
        const int p = L[x];
        if (p == x) return x;
        const int gp = L[p];
        if (gp != p) L[x] = gp;
        x = p;
    }
    return x;
}
__device__ __forceinline__ void lunion(int* L, int a, int b) {
    for (int it = 0; it < SPK_T * SPK_T; ++it) {
        int ra = lfind(L, a), rb = lfind(L, b);
        if (ra == rb) return;
        if (ra < rb) { int t = ra; ra = rb; rb = t; t = a; a = b; b = t; }
        const int old = atomicCAS(&L[ra], ra, rb);
        if (old == ra) return;
        a = old;
    }
}

// uf_find and uf_union on labels that other CTAs of the same launch wrote or
// still link: loads go to L2 (a line in L1 may hold another tile's labels
// from before).
__device__ __forceinline__ int uf_find_l2(int32_t* lab, int x, unsigned* err) {
    for (int it = 0; it < UF_LIMIT; ++it) {
        const int p = __ldcg(lab + x);
        if (p == x) return x;
        const int gp = __ldcg(lab + p);
        if (gp != p) __stcg(lab + x, gp);
        x = p;
    }
    atomicOr(err, ERRF_BOUNDS);
    return x;
}
__device__ void uf_union_l2(int32_t* lab, int a, int b, unsigned* err) {
    for (int it = 0; it < UF_LIMIT; ++it) {
        int ra = uf_find_l2(lab, a, err), rb = uf_find_l2(lab, b, err);
        if (ra == rb) return;
        if (ra < rb) { int t = ra; ra = rb; rb = t; t = a; a = b; b = t; }
        const int old = atomicCAS(&lab[ra], ra, rb);
        if (old == ra) return;
        a = old;
    }
    atomicOr(err, ERRF_BOUNDS);
}

// The left/right check of one pixel (k_lr in k_dense.cu) with the other
// view's map: the pixel it points at must hold the same disparity within
// thr.  dir: -1 for the left view, +1 for the right one.
__device__ __forceinline__ float lr_checked(float d, const float* __restrict__ other_row, int u, int W, float dir,
                                            float scale, float thr) {
    const float uw = float(u) + dir * (d * scale);
    if (!(d >= 0 && uw >= 0 && uw < float(W))) return -1.0f;
    return fabsf(other_row[int(uw)] - d) > thr ? -1.0f : d;
}

// A CTA of 32 x ROWS threads per 32x32 tile, each thread taking the tile rows
// ty, ty + ROWS, .. (a warp holds one tile row at a time).  Bound
// by instruction issue and, on small images, by its chain of barriers, so
// the nodes of the tile's forest are runs (connected pixels of one row, named
// by their first pixel) and every decision about runs is made on ballots:
// where runs start, which pixels continue one, which vertical links repeat
// the one to their left.  Only run heads find roots and add their length;
// the other pixels get their head's label by a shuffle.
// LR: the input is the dense result of both views and the tile also makes
// the left/right check, writing the checked map (cur) that the rest of the
// chain reads, so no pass of its own runs.
// Links across a tile's borders are made by whichever of the two tiles ends
// last, found by a ticket per border (zeroed by an earlier kernel of the
// pair): its four border warps each link one border, so no second pass over
// the borders runs either.  Neighbouring lanes hold neighbouring pixel pairs,
// and a segment crossing a border over many pixels makes the same union many
// times: a lane skips its union when the lane before it holds the same
// connected pair.
// Check, tiles and borders as three kernels with a node per pixel: 3.7 + 15.6
// + 9.0 us at 1242x375, 32 + 113 + 31 at 2880x1988; this kernel 21 and 136
// (eight CTAs per SM; five: 25 and 182).  While all tiles fit the SMs at once,
// taller CTAs shorten the chain, as a warp does not go through four rows'
// unions and finds one after the other: a row per warp (ROWS = 32) up to two
// tiles per SM (160x120: 16.1 -> 12.4 us), two rows up to four (450x375: 18.3
// -> 15.7).
template <bool LR, int SPK_ROWS>
__global__ void __launch_bounds__(SPK_T * SPK_ROWS, 64 / SPK_ROWS)
    k_spk_tile(PostViews pv, LrInput lr, int W, int H, float thr, unsigned* err) {
    grid_dep_wait();
    constexpr int SPK_RPT = SPK_T / SPK_ROWS;
    __shared__ float S[SPK_T][SPK_T];
    __shared__ int L[SPK_T * SPK_T];            // forest, at run heads only
    __shared__ int C[SPK_T * SPK_T];            // pixel counts, at tile-local roots
    __shared__ uint32_t starts[SPK_T], conts[SPK_T];    // per row: run heads; pixels connected to their left
    __shared__ int n_roots, base;
    const bool second = blockIdx.z != 0;
    float* D = second ? pv.cur[1] : pv.cur[0];
    int32_t* lab = second ? pv.lab[1] : pv.lab[0];
    int32_t* tick = second ? pv.tick[1] : pv.tick[0];
    const int tx = threadIdx.x, warp = threadIdx.y, tid = warp * SPK_T + tx;
    const int x = blockIdx.x * SPK_T + tx, y0 = blockIdx.y * SPK_T;
    const uint32_t upto = 0xffffffffu >> (31 - tx);     // this lane and the ones before it
    float d[SPK_RPT];
    uint32_t st[SPK_RPT], ct[SPK_RPT];
#pragma unroll
    for (int j = 0; j < SPK_RPT; ++j) {
        const int y = y0 + warp + SPK_ROWS * j;
        const bool in = x < W && y < H;
        const size_t at = size_t(y) * W + x;
        if (LR) {
            d[j] = in ? (second ? lr.d1 : lr.d0)[at] : -1.0f;
            if (in) {
                d[j] = lr_checked(d[j], (second ? lr.d0 : lr.d1) + size_t(y) * W, x, W, second ? 1.0f : -1.0f,
                                  lr.scale, lr.thr);
                D[at] = d[j];
            }
        } else {
            d[j] = in ? D[at] : -1.0f;
        }
    }
    if (tid == 0) n_roots = 0;
#pragma unroll
    for (int j = 0; j < SPK_RPT; ++j) {
        const int ty = warp + SPK_ROWS * j, t = ty * SPK_T + tx;
        const float dl = __shfl_up_sync(0xffffffffu, d[j], 1);
        const bool valid = d[j] >= 0, cont = valid && tx > 0 && dl >= 0 && fabsf(d[j] - dl) <= thr;
        st[j] = __ballot_sync(0xffffffffu, valid && !cont);
        ct[j] = __ballot_sync(0xffffffffu, cont);
        S[ty][tx] = d[j];
        if (valid && !cont) {
            L[t] = t;
            C[t] = 0;
        }
        if (tx == 0) {
            starts[ty] = st[j];
            conts[ty] = ct[j];
        }
    }
    __syncthreads();
    // vertical links; one is implied when the left neighbours make the same
#pragma unroll
    for (int j = 0; j < SPK_RPT; ++j) {
        const int ty = warp + SPK_ROWS * j;
        if (ty + 1 == SPK_T) continue;
        const float q = S[ty + 1][tx];
        const uint32_t v = __ballot_sync(0xffffffffu, d[j] >= 0 && q >= 0 && fabsf(q - d[j]) <= thr);
        const uint32_t first = v & ~((v << 1) & ct[j] & conts[ty + 1]);
        if ((first >> tx) & 1u)
            lunion(L, ty * SPK_T + 31 - __clz(st[j] & upto), (ty + 1) * SPK_T + 31 - __clz(starts[ty + 1] & upto));
    }
    __syncthreads();
    // run heads find their root and add their run's length; the local roots
    // take consecutive list slots
    int r[SPK_RPT], slot[SPK_RPT];
#pragma unroll
    for (int j = 0; j < SPK_RPT; ++j) {
        const int t = (warp + SPK_ROWS * j) * SPK_T + tx;
        const bool head = (st[j] >> tx) & 1u;
        r[j] = -1;
        if (head) {
            r[j] = lfind(L, t);
            atomicAdd(&C[r[j]], __ffs(~((ct[j] >> tx) >> 1)));      // 1 + the pixels that continue it
        }
        const uint32_t roots = __ballot_sync(0xffffffffu, head && r[j] == t);
        int b = 0;
        if (tx == 0 && roots) b = atomicAdd(&n_roots, __popc(roots));
        b = __shfl_sync(0xffffffffu, b, 0);
        slot[j] = (roots >> tx) & 1u ? b + __popc(roots & (upto >> 1)) : -1;
    }
    __syncthreads();
    if (tid == 0) base = n_roots > 0 ? atomicAdd(second ? pv.roots[1] : pv.roots[0], n_roots) : 0;
    __syncthreads();
#pragma unroll
    for (int j = 0; j < SPK_RPT; ++j) {
        const int ty = warp + SPK_ROWS * j, y = y0 + ty;
        const uint32_t mine = st[j] & upto;
        const int root = __shfl_sync(0xffffffffu, r[j], mine ? 31 - __clz(mine) : 0);
        if (x < W && y < H) {
            const size_t i = size_t(y) * W + x;
            const int rx = blockIdx.x * SPK_T + (root & (SPK_T - 1)), ry = y0 + (root / SPK_T);
            lab[i] = d[j] >= 0 ? int(size_t(ry) * W + rx) : -1;
            if (slot[j] >= 0) {         // a local root: its count, its segment-size slot, its list entry
                (second ? pv.sz[1] : pv.sz[0])[i] = C[ty * SPK_T + tx];
                (second ? pv.root[1] : pv.root[0])[i] = 0;
                (second ? pv.roots[1] : pv.roots[0])[1 + base + slot[j]] = int(i);
            }
        }
    }
    __syncthreads();
    // borders: warps 0 and 1 the ones to the right and left, 2 and 3 those below and above
    if (warp >= 4) return;
    const int txn = gridDim.x, tyn = gridDim.y;
    const bool vertical = warp < 2;
    const int bx = blockIdx.x - (warp == 1), by = blockIdx.y - (warp == 3);     // the tile left of or above the border
    if (bx < 0 || by < 0 || (vertical ? bx + 1 >= txn : by + 1 >= tyn)) return;
    int before = 0;
    if (tx == 0) {
        __threadfence();                // this tile's labels before its ticket
        before = atomicAdd(&tick[(vertical ? 0 : txn * tyn) + by * txn + bx], 1);
        __threadfence();                // the other tile's labels after it
    }
    before = __shfl_sync(0xffffffffu, before, 0);
    __syncwarp();                       // ... in every lane (the shuffle orders no memory)
    if (before == 0) return;            // the other tile is yet to end
    const int xa = vertical ? bx * SPK_T + SPK_T - 1 : bx * SPK_T + tx;
    const int ya = vertical ? by * SPK_T + tx : by * SPK_T + SPK_T - 1;
    int a = -1, b = -1;
    if (xa < W && ya < H) {
        const size_t i = size_t(ya) * W + xa, k = i + (vertical ? 1 : W);
        const float p = __ldcg(D + i), q = __ldcg(D + k);
        if (p >= 0 && q >= 0 && fabsf(q - p) <= thr) {
            a = __ldcg(lab + i);
            b = __ldcg(lab + k);
        }
    }
    const int pa = __shfl_up_sync(0xffffffffu, a, 1), pb = __shfl_up_sync(0xffffffffu, b, 1);
    if (a >= 0 && !(tx > 0 && pa == a && pb == b)) uf_union_l2(lab, a, b, err);
}

// Sizes: every tile-local root (from the roots list) adds its count at its
// global root g and keeps -(g + 1) in its size slot (only this thread reads
// that slot).
__global__ void k_spk_count(PostViews pv, int n, unsigned* err) {
    grid_dep_wait();
    const int view = blockIdx.z;
    int32_t* lab = pv.lab[view];
    int32_t* sz = pv.sz[view];
    int32_t* acc = pv.root[view];
    const int32_t* roots = pv.roots[view];
    const int nr = min(roots[0], n);
    const int lane = threadIdx.x & 31;
    // warp-uniform trips; lanes with the same global root add their counts
    // with one atomic (neighbouring list entries often share a segment)
    for (int k0 = blockIdx.x * blockDim.x + (threadIdx.x & ~31); k0 < nr; k0 += gridDim.x * blockDim.x) {
        const int k = k0 + lane;
        int i = -1, c = 0, g = -1;
        if (k < nr) {
            i = roots[1 + k];
            c = sz[i];
            g = uf_find(lab, i, err);
        }
        const unsigned peers = __match_any_sync(0xffffffffu, g);
        const int total = __reduce_add_sync(peers, c);
        if (g >= 0 && lane == __ffs(peers) - 1) atomicAdd(&acc[g], total);
        if (i >= 0) sz[i] = -(g + 1);
    }
}

// out = in with the pixels of segments smaller than min_size set invalid:
// a pixel's tile-local root (itself, or lab[i]) holds -(global root + 1).
__global__ void k_spk_apply(PostViews pv, int n, int min_size) {
    grid_dep_wait();
    const int view = blockIdx.z;
    const float* __restrict__ D = pv.cur[view];
    float* __restrict__ O = pv.nxt[view];
    const int32_t* __restrict__ lab = pv.lab[view];
    const int32_t* __restrict__ sz = pv.sz[view];
    const int32_t* __restrict__ acc = pv.root[view];
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const float d = D[i];
        float o = d;
        if (d >= 0 && acc[-sz[lab[i]] - 1] < min_size) o = -1.0f;
        O[i] = o;
    }
}

__global__ void k_uf_apply(float* D, const int32_t* __restrict__ root, const int32_t* sz, int n, int min_size) {
    grid_dep_wait();
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    int r = root[i];
    if (r >= 0 && sz[r] < min_size) D[i] = -1.0f;
}

// Gaps wider than the tile filter's halo, rows then columns.  A run of
// invalid pixels between valid a and b is filled from a and b alone, which
// no fill changes, so every pixel can look for its two ends by itself: in a
// bit mask of the line's valid pixels kept in shared memory (32 pixels a
// word, empty words skipped).  Bound by latency (a handful of dependent
// loads a pixel); one thread walking a whole line in order took 1089 us for
// the rows (and 16 for the speckle pass before them) and 348 us for the
// columns of a 1242x375 pair, this pair of kernels 13 us each.
__device__ __forceinline__ float gap_value(float a, float b) {
    return fabsf(a - b) <= 3.0f ? __fmul_rn(0.5f, __fadd_rn(a, b)) : fminf(a, b);
}

// One CTA per row: cur -> nxt, applying the speckle decision of k_spk_apply
// on the way in when spk_min > 0 (no separate pass).
constexpr int GAP_THREADS = 256;
__global__ void __launch_bounds__(GAP_THREADS) k_gap_rows(PostViews pv, int W, int gap, int spk_min) {
    grid_dep_wait();
    extern __shared__ uint32_t mask[];          // (W + 31) / 32 words
    const int view = blockIdx.z, lane = threadIdx.x & 31;
    const size_t base = size_t(blockIdx.x) * W;
    const float* __restrict__ src = pv.cur[view] + base;
    float* __restrict__ dst = pv.nxt[view] + base;
    const int32_t* __restrict__ lab = pv.lab[view] + base;
    const int32_t* __restrict__ sz = pv.sz[view];
    const int32_t* __restrict__ acc = pv.root[view];
    const int nw = (W + 31) / 32;
    for (int x0 = threadIdx.x & ~31; x0 < W; x0 += GAP_THREADS) {
        const int x = x0 + lane;
        float d = x < W ? src[x] : -1.0f;
        if (spk_min > 0 && x < W) {
            const int l = lab[x];
            if (d >= 0 && acc[-sz[l] - 1] < spk_min) d = -1.0f;
        }
        const unsigned m = __ballot_sync(0xffffffffu, d >= 0);
        if (lane == 0) mask[x0 >> 5] = m;
        if (d >= 0) dst[x] = d;
    }
    __syncthreads();
    for (int x0 = threadIdx.x & ~31; x0 < W; x0 += GAP_THREADS) {
        const int x = x0 + lane;
        const unsigned m = mask[x0 >> 5];
        if (x >= W || ((m >> lane) & 1u)) continue;
        unsigned below = m & ((1u << lane) - 1u), above = m & ~((2u << lane) - 1u);
        int wl = x0 >> 5, wh = wl;
        while (!below && wl > 0) below = mask[--wl];
        while (!above && wh + 1 < nw) above = mask[++wh];
        float f = -1.0f;
        if (below && above) {
            const int lo = 32 * wl + 31 - __clz(below), hi = 32 * wh + __ffs(above) - 1;
            if (hi - lo - 1 <= gap) f = gap_value(src[lo], src[hi]);
        }
        dst[x] = f;
    }
}

// One CTA per 32 columns, a warp per 32 rows at a time (lane = column):
// src -> dst, in place when they are the same.
constexpr int GAP_COL_WARPS = 16;
__global__ void __launch_bounds__(32 * GAP_COL_WARPS) k_gap_cols(PostViews pv, int W, int H, int gap) {
    grid_dep_wait();
    extern __shared__ uint32_t mask[];          // [(H + 31) / 32][32]
    const int view = blockIdx.z, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int x = blockIdx.x * 32 + lane, nb = (H + 31) / 32;
    const float* src = pv.cur[view] + x;
    float* dst = pv.nxt[view] + x;
    const bool in = x < W, copy = src != dst;
    for (int b = warp; b < nb; b += GAP_COL_WARPS) {
        const int n = min(32, H - 32 * b);
        uint32_t bits = 0;
#pragma unroll 8
        for (int r = 0; r < n; ++r) {
            const float d = in ? src[size_t(32 * b + r) * W] : -1.0f;
            bits |= d >= 0 ? 1u << r : 0u;
        }
        mask[32 * b + lane] = bits;
    }
    __syncthreads();
    if (!in) return;
    for (int b = warp; b < nb; b += GAP_COL_WARPS) {
        const int n = min(32, H - 32 * b);
        const uint32_t bits = mask[32 * b + lane];
        int lo = -1;                            // the last valid row before the current one
        for (int w = b - 1; w >= 0 && lo < 0; --w)
            if (const uint32_t m = mask[32 * w + lane]) lo = 32 * w + 31 - __clz(m);
        bool open = false;                      // inside a run whose fill value f is known
        float f = -1.0f;
        for (int r = 0; r < n; ++r) {
            const size_t at = size_t(32 * b + r) * W;
            if ((bits >> r) & 1u) {
                lo = 32 * b + r;
                open = false;
                if (copy) dst[at] = src[at];
                continue;
            }
            if (!open) {
                open = true;
                f = -1.0f;
                int hi = -1;
                if (const uint32_t m = bits >> r) hi = 32 * b + r + __ffs(m) - 1;
                for (int w = b + 1; w < nb && hi < 0; ++w)
                    if (const uint32_t m = mask[32 * w + lane]) hi = 32 * w + __ffs(m) - 1;
                if (lo >= 0 && hi >= 0 && hi - lo - 1 <= gap) f = gap_value(src[size_t(lo) * W], src[size_t(hi) * W]);
            }
            if (copy || f >= 0) dst[at] = f;
        }
    }
}

// 3-value and 9-value medians.  A column of three sorted rows of three gives
// the median of nine: the middle one of the largest low, the middle middle
// and the smallest high.
__device__ __forceinline__ float med3(float a, float b, float c) {
    return fmaxf(fminf(a, b), fminf(fmaxf(a, b), c));
}
struct Tri { float lo, mid, hi; };
__device__ __forceinline__ Tri sort3(float a, float b, float c) {
    const float l = fminf(a, b), h = fmaxf(a, b);
    return {fminf(l, c), fmaxf(l, fminf(h, c)), fmaxf(h, c)};
}
__device__ __forceinline__ float med9(const Tri& p, const Tri& q, const Tri& r) {
    return med3(fmaxf(fmaxf(p.lo, q.lo), r.lo), med3(p.mid, q.mid, r.mid), fminf(fminf(p.hi, q.hi), r.hi));
}

// Speckle decision, gap interpolation (rows, then columns), adaptive mean
// and median in one pass over a tile of PT_OW x (4 R - 2) output pixels, every
// intermediate in shared memory.  The input region carries a halo of G + 3
// for gaps up to G (the column pass needs the row pass G rows away, the mean
// 2 more, the median 1 more).  Eight warps: two side by side over 64
// columns, four strips of R rows (the mean's region is 64 x 4 R: whole
// warps).
//
// Bound by latency and instruction issue (56 % of the issue slots with three
// CTAs per SM; the first stall is the load stage's chain of map and label,
// size slot and segment size), so each stage keeps what neighbouring pixels
// share in registers:
//   load    a warp loads whole rows and, as it knows their valid pixels from
//           ballots, fills the row gaps at once: run lengths come from the
//           bits on either side.  Fills are written in place (only invalid
//           pixels are written, only valid ones read).  The column pass
//           does the same with the rows' bit masks.
//   mean    a thread walks down a column with the 5 x 5 window in registers
//           (five loads a pixel instead of 25).  Every value is a multiple
//           of 1/4 (integer disparities, halves from the row gaps, quarters
//           from the column gaps) in [0, disp_max], so v * 16 + 2^23 is exact
//           and the difference of two such floats' bits is the byte offset
//           of the pair's weight 1 / (1 + (d_q - d_p)^2), made once by the
//           same correctly rounded operations as the direct formula: an add
//           and a load a weight.  The table covers differences of either
//           sign; invalid pixels get bits so far up that they meet the
//           zeros behind it, and a weight of 0 leaves both sums as they are.
//   median  a thread walks down a column with three sorted rows of three;
//           only a window with invalid pixels sorts for itself.
// A thread per pixel for each stage took 314 us at 2880x1988 (D 0-511) and 37
// at 1242x375; this form 207 and 25.
constexpr int PGMAX = 8, PT_OW = 62, POST_THREADS = 256;
constexpr uint32_t MAGIC_F32 = 0x4b000000u;     // bits of 2^23
// weights of the mean: entries -4 D .. 8 D + 1 of the difference in quarters
inline size_t post_weights(int D) { return 12 * size_t(D) + 2; }
__device__ __forceinline__ float lds_f32(uint32_t addr) {
    float v;
    asm("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(addr));
    return v;
}

template <int G, bool GAP, bool MEAN, bool MEDIAN, int R>
__global__ void __launch_bounds__(POST_THREADS, MEAN ? 3 : 4) k_post_tile(PostViews pv, int W, int H, int gap,
                                                                          int spk_min, int D, int nviews) {
    grid_dep_wait();
    constexpr int OW = PT_OW, OH = 4 * R - 2, HALO = G + 3, SW = OW + 2 * HALO, SH = OH + 2 * HALO;
    constexpr int NSEG = (SW + 31) / 32, NWARP = POST_THREADS / 32;
    static_assert(NSEG == 3 && OW + 2 == 64, "three ballots a row, two warps over the mean's columns");
    extern __shared__ float WT[];               // weights when MEAN
    __shared__ float S[SH][SW];                 // the input region, gaps filled in place
    __shared__ uint32_t msk[SH][NSEG];          // its valid pixels after the row pass
    __shared__ float M[MEAN && MEDIAN ? OH + 2 : 1][OW + 2];    // after the mean: [-1, OW + 1) x [-1, OH + 1)
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const float OUT = -2.0f;                    // outside the image (never valid, never filled)
    if (MEAN)
        for (int j = tid; j < 12 * D + 2; j += POST_THREADS) {
            const float q = float(j - 4 * D) * 0.25f;
            WT[j] = j <= 8 * D ? __frcp_rn(__fmaf_rn(q, q, 1.0f)) : 0.0f;
        }
    const uint32_t wt0 = MEAN ? smem_u32(WT) + 16u * uint32_t(D) : 0u;      // the weight of difference 0
    const uint32_t kinv = MAGIC_F32 + 4u * uint32_t(8 * D + 1);             // bits of an invalid pixel
    const int tiles_x = (W + OW - 1) / OW, tiles_y = (H + OH - 1) / OH, per_view = tiles_x * tiles_y;
    for (int tile = blockIdx.x; tile < nviews * per_view; tile += gridDim.x) {
        const bool second = tile >= per_view;
        const int tv = second ? tile - per_view : tile;
        const float* __restrict__ src = second ? pv.cur[1] : pv.cur[0];
        float* __restrict__ dst = second ? pv.nxt[1] : pv.nxt[0];
        const int32_t* __restrict__ lab = second ? pv.lab[1] : pv.lab[0];
        const int32_t* __restrict__ sz = second ? pv.sz[1] : pv.sz[0];
        const int32_t* __restrict__ acc = second ? pv.root[1] : pv.root[0];
        const int u0 = (tv % tiles_x) * OW, v0 = (tv / tiles_x) * OH;
        if (!(MEAN && MEDIAN)) __syncthreads();     // the previous tile's last stage read S
        // Load, speckle decision and row gaps.  The decision is k_spk_apply's:
        // the local root lab[j] holds -(global root + 1) in its size slot,
        // whose segment size is acc[global root]; the value and the label are
        // loaded together and two rows' chains overlap (four: no faster).
        const int x0 = u0 - HALO + lane;
        uint32_t cols = 0;                      // bit k: column x0 + 32 k is in the region and the image
#pragma unroll
        for (int k = 0; k < NSEG; ++k)
            cols |= 32 * k + lane < SW && x0 + 32 * k >= 0 && x0 + 32 * k < W ? 1u << k : 0u;
#pragma unroll 2
        for (int r = warp; r < SH; r += NWARP) {
            const int y = v0 - HALO + r;
            const bool row = y >= 0 && y < H;
            const ptrdiff_t at = ptrdiff_t(row ? y : 0) * W + x0;
            float d[NSEG];
            int l[NSEG];
            uint32_t m[NSEG + 2];
#pragma unroll
            for (int k = 0; k < NSEG; ++k) {
                d[k] = row && ((cols >> k) & 1u) ? src[at + 32 * k] : OUT;
                l[k] = spk_min > 0 && row && ((cols >> k) & 1u) ? lab[at + 32 * k] : -1;
            }
            if (spk_min > 0) {
#pragma unroll
                for (int k = 0; k < NSEG; ++k) l[k] = d[k] >= 0 ? sz[l[k]] : 0;     // a valid pixel has a label
#pragma unroll
                for (int k = 0; k < NSEG; ++k)
                    if (d[k] >= 0 && acc[-l[k] - 1] < spk_min) d[k] = -1.0f;
            }
            m[0] = m[NSEG + 1] = 0;
#pragma unroll
            for (int k = 0; k < NSEG; ++k) {
                m[k + 1] = __ballot_sync(0xffffffffu, d[k] >= 0);
                if (32 * k + lane < SW) S[r][32 * k + lane] = d[k];
            }
            if (GAP) {
                __syncwarp();
                uint32_t after[NSEG];
#pragma unroll
                for (int k = 0; k < NSEG; ++k) {
                    after[k] = m[k + 1];
                    // nothing to fill in a full word, nor (gaps up to 8) in an empty one
                    if (m[k + 1] != 0u && m[k + 1] != 0xffffffffu) {
                        const int c = 32 * k + lane;
                        // bit 31: the pixel to the left; bit 0: the one to the right
                        const uint32_t lf = __funnelshift_r(m[k], m[k + 1], lane);
                        const uint32_t rt = __funnelshift_rc(m[k + 1], m[k + 2], lane + 1);
                        const int dl = __clz(lf) + 1, dr = rt ? __ffs(rt) : 33;     // 33: none within 32
                        const bool fill = d[k] < 0 && dl <= gap && dr <= gap && dl + dr - 1 <= gap;
                        if (fill) S[r][c] = gap_value(S[r][c - dl], S[r][c + dr]);
                        after[k] = __ballot_sync(0xffffffffu, d[k] >= 0 || fill);
                    }
                }
                if (lane < NSEG) msk[r][lane] = lane == 0 ? after[0] : (lane == 1 ? after[1] : after[2]);
            }
        }
        __syncthreads();
        if (GAP) {
            // column gaps of [-3, OW + 3) x [-3, OH + 3)
            for (int r = HALO - 3 + warp; r < HALO + OH + 3; r += NWARP) {
                const int y = v0 - HALO + r;
                if (y < 0 || y >= H) continue;
#pragma unroll
                for (int k = 0; k < NSEG; ++k) {
                    const int c = 32 * k + lane, x = u0 - HALO + c;
                    const bool wanted = c >= HALO - 3 && c < HALO + OW + 3 && x >= 0 && x < W;
                    const bool inv = wanted && !((msk[r][k] >> lane) & 1u);
                    if (!__any_sync(0xffffffffu, inv)) continue;
                    int dl = 0, dr = 0;
#pragma unroll
                    for (int j = G; j >= 1; --j) {
                        if ((msk[r - j][k] >> lane) & 1u) dl = j;
                        if ((msk[r + j][k] >> lane) & 1u) dr = j;
                    }
                    if (inv && dl && dr && dl + dr - 1 <= gap) S[r][c] = gap_value(S[r - dl][c], S[r + dr][c]);
                }
            }
            __syncthreads();
        }
        const int col = 32 * (warp & 1) + lane, row0 = R * (warp >> 1);
        if (MEAN) {
            // mean at column col - 1, rows row0 - 1 .., in the oracle's (dy, dx)
            // order: num by fma, den by add
            float v[5][5];
            uint32_t q[5][5];
            auto load = [&](int slot, int r) {
#pragma unroll
                for (int c = 0; c < 5; ++c) {
                    v[slot][c] = S[HALO - 3 + r][HALO - 3 + col + c];
                    q[slot][c] = v[slot][c] >= 0 ? __float_as_uint(fmaf(v[slot][c], 16.0f, 8388608.0f)) : kinv;
                }
            };
#pragma unroll
            for (int r = 0; r < 4; ++r) load(r, row0 + r);
#pragma unroll
            for (int i = 0; i < R; ++i) {
                load((i + 4) % 5, row0 + i + 4);
                const float vp = v[(i + 2) % 5][2];
                float out = vp;
                if (__any_sync(0xffffffffu, vp >= 0)) {
                    const uint32_t base = wt0 - (vp >= 0 ? q[(i + 2) % 5][2] : MAGIC_F32);
                    float num = 0.0f, den = 0.0f;
#pragma unroll
                    for (int dy = 0; dy < 5; ++dy)
#pragma unroll
                        for (int dx = 0; dx < 5; ++dx) {
                            const int s = (i + dy) % 5;
                            const float w = dy == 2 && dx == 2 ? 1.0f : lds_f32(base + q[s][dx]);
                            num = __fmaf_rn(w, v[s][dx], num);
                            den = __fadd_rn(den, w);
                        }
                    if (vp >= 0) out = __fdiv_rn(num, den);
                }
                if (MEDIAN) {
                    M[row0 + i][col] = out;
                } else {
                    const int u = u0 + col - 1, y = v0 + row0 + i - 1;
                    if (col >= 1 && col <= OW && u < W && row0 + i >= 1 && row0 + i <= OH && y < H)
                        dst[size_t(y) * W + u] = out;
                }
            }
            if (MEDIAN) __syncthreads();
        }
        if (MEDIAN || !MEAN) {
            // output column col, rows row0 ..; row r of the window's column
            auto at = [&](int r, int c) { return MEAN ? M[r][c] : S[HALO - 1 + r][HALO - 1 + c]; };
            const int u = u0 + col;
            if (col < OW && u < W) {
                Tri t[3];
                float mid[3];                   // the window's middle column
                auto load = [&](int slot, int r) {
                    mid[slot] = at(r, col + 1);
                    if (MEDIAN) t[slot] = sort3(at(r, col), mid[slot], at(r, col + 2));
                };
                load(0, row0);
                load(1, row0 + 1);
#pragma unroll
                for (int i = 0; i < R; ++i) {
                    const int y = v0 + row0 + i;
                    if (row0 + i >= OH || y >= H) break;
                    load((i + 2) % 3, row0 + i + 2);
                    const float c = mid[(i + 1) % 3];
                    float out = c;
                    if (MEDIAN && c >= 0) {
                        if (fminf(fminf(t[0].lo, t[1].lo), t[2].lo) >= 0) {
                            out = med9(t[0], t[1], t[2]);
                        } else {
                            // n < 9 valid values: their lower median is the median of
                            // nine when the invalid ones count as the lowest and the
                            // highest value in turn
                            float a[9];
                            bool low = true;
#pragma unroll
                            for (int k = 0; k < 9; ++k) {
                                const float w = at(row0 + i + k / 3, col + k % 3);
                                a[k] = w >= 0 ? w : (low ? -INFINITY : INFINITY);
                                low = low != (w < 0);
                            }
                            out = med9(sort3(a[0], a[1], a[2]), sort3(a[3], a[4], a[5]), sort3(a[6], a[7], a[8]));
                        }
                    }
                    dst[size_t(y) * W + u] = out;
                }
            }
        }
    }
}

}  // namespace

bool post_any(const DevParams& p, bool median, bool adaptive_mean) {
    return p.speckle_size > 0 || p.ipol_gap_width > 0 || median || adaptive_mean;
}

size_t post_tickets(int W, int H) { return size_t(2) * ((W + SPK_T - 1) / SPK_T) * ((H + SPK_T - 1) / SPK_T); }

cudaError_t launch_post(PostViews pv, const LrInput& lr, int nviews, const Geom& g, const DevParams& p, bool median,
                        bool adaptive_mean, unsigned* err, cudaStream_t st, int* nlaunch, int num_sms, int* last_args) {
    const int W = g.W, H = g.H, n = W * H;
    int launched = 0;
    auto flip = [&]() {
        for (int k = 0; k < 2; ++k) { float* t = pv.cur[k]; pv.cur[k] = pv.nxt[k]; pv.nxt[k] = t; }
    };
    // every chain's first pass works out of place, so the L/R map it starts
    // from stays as it is; the tile filter, always the last pass, writes the
    // final buffers
    // with the tile filter following, speckle removal is applied as it loads
    const bool fuse = p.ipol_gap_width <= PGMAX && (p.ipol_gap_width > 0 || adaptive_mean || median);
    if (p.speckle_size > 0) {
        const dim3 tiles((W + SPK_T - 1) / SPK_T, (H + SPK_T - 1) / SPK_T, nviews);
        const int per_sm = (int(tiles.x * tiles.y * tiles.z) + num_sms - 1) / num_sms;
        const int rows = per_sm <= 2 ? 32 : (per_sm <= 4 ? 16 : 8);
        const dim3 threads(SPK_T, rows);
        auto kern = rows == 32 ? (lr.d0 ? k_spk_tile<true, 32> : k_spk_tile<false, 32>)
                  : rows == 16 ? (lr.d0 ? k_spk_tile<true, 16> : k_spk_tile<false, 16>)
                               : (lr.d0 ? k_spk_tile<true, 8> : k_spk_tile<false, 8>);
        launch_k(kern, tiles, threads, 0, st, pv, lr, W, H, p.speckle_sim_threshold, err);
        const int gn = imax(1, imin(8 * 1024, (n + 255) / 256));
        // the roots list is far shorter than the image: a grid of one CTA per
        // SM walks it (idle CTAs cost their launch; measured against four)
        launch_k(k_spk_count, dim3(imin(gn, num_sms), 1, nviews), 256, 0, st, pv, n, err);
        launched += 2;
        if (!fuse && p.ipol_gap_width <= PGMAX) {
            // the chain's only pass: straight into the final buffers
            for (int k = 0; k < nviews; ++k) pv.nxt[k] = pv.out[k];
            launch_k(k_spk_apply, dim3(gn, 1, nviews), 256, 0, st, pv, n, p.speckle_size);
            *last_args = 3;
            flip();
            launched += 1;
        }
    }
    const int gap = p.ipol_gap_width;
    const int spk = fuse ? p.speckle_size : 0;
    const bool tile_gap = gap > 0 && gap <= PGMAX;
    if (gap > PGMAX) {   // wide gaps: cur -> nxt by rows, then by columns
        launch_k(k_gap_rows, dim3(H, 1, nviews), GAP_THREADS, size_t((W + 31) / 32) * sizeof(uint32_t), st, pv, W, gap,
                 p.speckle_size);
        flip();
        // in place before the tile filter; as the chain's last pass straight
        // into the final buffers
        PostViews pc = pv;
        const bool last = !adaptive_mean && !median;
        for (int k = 0; k < 2; ++k) pc.nxt[k] = last ? pv.out[k] : pv.cur[k];
        allow_smem(k_gap_cols);
        launch_k(k_gap_cols, dim3((W + 31) / 32, 1, nviews), 32 * GAP_COL_WARPS,
                 size_t((H + 31) / 32) * 32 * sizeof(uint32_t), st, pc, W, H, gap);
        *last_args = 4;
        if (last)
            for (int k = 0; k < nviews; ++k) pv.cur[k] = pv.out[k];
        launched += 2;
    }
    if (tile_gap || adaptive_mean || median) {
        for (int k = 0; k < nviews; ++k) pv.nxt[k] = pv.out[k];
        const size_t smem = adaptive_mean ? post_weights(g.D) * sizeof(float) : 0;
        const int key = (tile_gap ? 4 : 0) | (adaptive_mean ? 2 : 0) | (median ? 1 : 0);
        const int ctas = (adaptive_mean ? 3 : 4) * num_sms;     // resident at once
        auto tiles_of = [&](int oh) { return ((W + PT_OW - 1) / PT_OW) * ((H + oh - 1) / oh) * nviews; };
        auto go = [&](auto kern, int oh) {
            if (smem) allow_smem(kern);
            launch_k(kern, imax(1, imin(tiles_of(oh), ctas)), POST_THREADS, smem, st, pv, W, H, gap, spk, g.D, nviews);
            *last_args = 7;
        };
        // R rows a strip (see k_post_tile): the height for which the rounds of
        // resident CTAs take the least, a round costing about 24 rows more
        // than the 4 R it computes (halo, table, latency: 10, 12.5 and 14 us
        // for R = 4, 5 and 8).  1242x375: two rounds of R = 8 28 us, two of
        // R = 5 25; 960x540: three of R = 4 30, two of R = 8 27.6.
        auto pick = [&](auto r) {
            constexpr int R = decltype(r)::value, OH = 4 * R - 2;
            if (!tile_gap || gap <= 3) {   // halo 6
                switch (key) {
                case 1: go(k_post_tile<3, false, false, true, R>, OH); break;
                case 2: go(k_post_tile<3, false, true, false, R>, OH); break;
                case 3: go(k_post_tile<3, false, true, true, R>, OH); break;
                case 4: go(k_post_tile<3, true, false, false, R>, OH); break;
                case 5: go(k_post_tile<3, true, false, true, R>, OH); break;
                case 6: go(k_post_tile<3, true, true, false, R>, OH); break;
                default: go(k_post_tile<3, true, true, true, R>, OH); break;
                }
            } else {                       // gaps 4..8: halo 11
                switch (key) {
                case 4: go(k_post_tile<PGMAX, true, false, false, R>, OH); break;
                case 5: go(k_post_tile<PGMAX, true, false, true, R>, OH); break;
                case 6: go(k_post_tile<PGMAX, true, true, false, R>, OH); break;
                default: go(k_post_tile<PGMAX, true, true, true, R>, OH); break;
                }
            }
        };
        auto cost = [&](int r) { return (tiles_of(4 * r - 2) + ctas - 1) / ctas * (4 * r + 24); };
        int best = 8;
        for (int r : {5, 4})
            if (cost(r) < cost(best)) best = r;
        if (best == 8) pick(std::integral_constant<int, 8>{});
        else if (best == 5) pick(std::integral_constant<int, 5>{});
        else pick(std::integral_constant<int, 4>{});
        flip();
        launched += 1;
    }
    if (nlaunch) *nlaunch += launched;
    return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// Allocation-free speckle removal (elas_b200_speckle_noalloc).
//
// For callers that must not allocate device memory -- code inside a CUDA
// stream capture (cudaMalloc cannot be captured), plugin hosts and real-time
// loops that forbid allocation after start-up.  Its scratch (labels, roots,
// segment sizes and an error word) is this one file-scope array, resident on
// every GPU that loads the library until the process exits.  In host code
// the array's name is only a host-side stand-in, so its device address is
// looked up with cudaGetSymbolAddress once per device and CUDA context (the
// first call on a device, and the first after a cudaDeviceReset, which
// should therefore happen outside any stream capture) and cached.  Every
// call reuses the array; the kernels initialise all of it that must start
// at zero, and calls that overlap on the GPU race.
//
// The error word receives the bounds flag of the union-find walks, which
// valid inputs cannot raise: labels only ever decrease, so a find walks at
// most width*height <= 2^19 nodes, and a union retries only after another
// thread's hook succeeded, at most 2^19 times -- both below UF_LIMIT.  The
// call does not read it back (that would synchronise the caller's stream).
static __device__ __align__(256) int32_t g_noalloc_scratch[3 * ELAS_NOALLOC_MAX_PIXELS + 64];

namespace {
constexpr int kNoallocMaxDevices = 64;
struct NoallocSlot {
    void* ctx = nullptr;        // CUcontext the address was looked up in
    int32_t* base = nullptr;
};
NoallocSlot g_noalloc_slot[kNoallocMaxDevices];
std::mutex g_noalloc_mutex;

// The current CUDA context through the runtime's driver entry point (no
// link against libcuda); null if the entry point is unavailable.
void* current_context() {
    using GetCtx = int (*)(void**);
    static GetCtx fn = [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuCtxGetCurrent", &p, cudaEnableDefault, &q) != cudaSuccess ||
            q != cudaDriverEntryPointSuccess)
            p = nullptr;
        return reinterpret_cast<GetCtx>(p);
    }();
    void* ctx = nullptr;
    if (!fn || fn(&ctx) != 0) return nullptr;
    return ctx;
}
}  // namespace

}  // namespace elas

extern "C" int elas_b200_speckle_noalloc(const float* d_in, float* d_out, int32_t width, int32_t height,
                                         float sim_threshold, int32_t min_size, void* stream) {
    using namespace elas;
    if (!d_in || !d_out || width <= 0 || height <= 0 || min_size < 0) return ELAS_ERR_INVALID_ARG;
    if (int64_t(width) * height > ELAS_NOALLOC_MAX_PIXELS) return ELAS_ERR_TOO_LARGE;
    int dev = -1;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kNoallocMaxDevices) return ELAS_ERR_NO_DEVICE;
    int32_t* base = nullptr;
    {
        std::lock_guard<std::mutex> lock(g_noalloc_mutex);
        NoallocSlot& slot = g_noalloc_slot[dev];
        void* ctx = current_context();
        if (!slot.base || ctx != slot.ctx) {
            void* p = nullptr;
            if (cudaGetSymbolAddress(&p, g_noalloc_scratch) != cudaSuccess || !p) return ELAS_ERR_CUDA;
            slot.base = static_cast<int32_t*>(p);
            slot.ctx = ctx;
        }
        base = slot.base;
    }
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const int W = width, H = height, n = W * H, tb = 256;
    int32_t* lab = base;
    int32_t* root = base + ELAS_NOALLOC_MAX_PIXELS;
    int32_t* sz = base + 2 * ELAS_NOALLOC_MAX_PIXELS;
    unsigned* err = reinterpret_cast<unsigned*>(base + 3 * ELAS_NOALLOC_MAX_PIXELS);
    // each call's own status: an earlier, unrelated launch error is not this call's
    if (d_out != d_in &&
        cudaMemcpyAsync(d_out, d_in, size_t(n) * sizeof(float), cudaMemcpyDeviceToDevice, st) != cudaSuccess)
        return ELAS_ERR_CUDA;
    if (cudaMemsetAsync(err, 0, sizeof(unsigned), st) != cudaSuccess) return ELAS_ERR_CUDA;
    if (min_size > 0) {
        const int blocks = (n + tb - 1) / tb;
        if (launch_k(k_uf_init, blocks, tb, 0, st, d_out, lab, sz, W, H, sim_threshold) != cudaSuccess ||
            launch_k(k_uf_union, blocks, tb, 0, st, d_out, lab, W, H, sim_threshold, err) != cudaSuccess ||
            launch_k(k_uf_count, blocks, tb, 0, st, lab, root, sz, n, err) != cudaSuccess ||
            launch_k(k_uf_apply, blocks, tb, 0, st, d_out, root, sz, n, min_size) != cudaSuccess)
            return ELAS_ERR_CUDA;
    }
    return ELAS_OK;
}
