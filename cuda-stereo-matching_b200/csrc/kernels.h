// Launchers of the ELAS B200 kernels (internal interface of the library).
#pragma once

#include <cuda_runtime.h>
#include <cstdint>
#include "common.cuh"

namespace elas {

// Device view of one triangulation problem (see delaunay_core.h).
struct DelDev {
    const int32_t* x;      // [Nmax] point x (u for the left view, u-d for the right)
    const int32_t* y;      // [Nmax] point y (v)
    int32_t* srt;          // [Nmax] per-row sorted unique point indices (at row_off offsets)
    int32_t* rcnt;         // [rows] unique points per row
    int32_t* ne;           // [rows] non-empty rows
    int32_t* soff;         // [rows] strip triangle offsets
    int32_t* chain;        // [6*rows] hull pockets: key, predecessor and point of each row, both sides
    int32_t* tri;          // [3*Tmax]
    int32_t* opp;          // [3*Tmax]
    uint32_t* txy;         // [3*Tmax] packed corner coordinates (global flip kernel)
    uint32_t* lock;        // [Tmax]
    int32_t* fround;       // [Tmax]
    int32_t* cand;         // [6*Tmax]
    int32_t* flips;        // [3*Tmax]
    int32_t* wl0;          // [6*Tmax]
    int32_t* wl1;          // [6*Tmax]
    int32_t* cwl;          // cluster kernel: per-CTA worklists  [16 * 2 * 6 * 4096]
    int32_t* ccand;        // cluster kernel: per-CTA proposals  [16 * 2 * 6 * 4096]
    int32_t* cflips;       // cluster kernel: per-CTA flips      [16 * 6 * 4096]
    int32_t* ctr;          // [16]: 0 triangles, 1 strip and 2, 3 pocket triangles, 4 flip rounds, 5 flips,
                           //       6 non-empty rows, 8 handled by the cluster kernel, 9 points,
                           //       10 points of far, 11 star pool cursor, 12 unused (0),
                           //       13 window doublings that prove the stars
    uint32_t* pxy;         // [Nmax] packed coordinates by point (PXY_NONE: dropped duplicate)
    uint32_t* sxy;         // [Nmax] packed coordinates beside srt
    int32_t* xb;           // [rows][(W + 7) / 8 + 1] first sorted position at or right of each 8-pixel column
    int32_t* far;          // [Nmax][FAR_REC] points whose star the window does not prove, with what it found
    int32_t* tcnt;         // [Nmax] triangles owned by each point (star construction)
    int32_t* toff;         // [Nmax] their offsets in tri
    int32_t* sown;         // [24*Nmax] owned triangles' vertex pairs, per point
    int32_t* spool;        // [2*Tmax] pairs of points owning more than the slot holds
    int32_t* hnext;        // [Nmax] successor on the hull boundary (-1: interior point)
    int32_t* hprev;        // [Nmax] predecessor on the hull boundary
    int32_t* box;          // [8] x0, y0, x1, y1 of all points, [4] star window half-size
    unsigned long long* hkey;  // [Hmax]
    int32_t* hcnt;         // [Hmax]
    int32_t* hval;         // [2*Hmax]
    int32_t* hslot;        // [3*Tmax]
    static constexpr int FAR_REC = 32;
    int Tmax;
    uint32_t Hmax;         // power of two
};

// Also zeroes the words that later kernels of the pair only add to (memset
// nodes of their own would cost 3-5 us each on a pair's critical path).
struct PairZero {
    unsigned* err;         // the error word
    int32_t* stats;        // four proposal counters (nullable)
    int32_t* roots[2];     // lengths of the speckle filter's roots lists
    int32_t* tick;         // ntick border tickets of the speckle filter
    int ntick;
};
constexpr int DESCRIPTOR_ARGS = 7;     // of its kernel: the images come first
cudaError_t launch_descriptor(const uint8_t* img0, const uint8_t* img1, uint4* desc0, uint4* desc1,
                              int W, int H, const PairZero& z, cudaStream_t st);

// Rows of the candidate lattice that the column filter and the row plan of
// the triangulations hold in one CTA's shared memory (40 and 36 bytes a
// row); taller lattices are refused before anything is launched.
constexpr int LATTICE_ROWS_MAX = 5796;
constexpr size_t SMEM_PER_CTA = 227 * 1024;

// bins (nullable): packed learned search sets per candidate; then stats[0]
// counts candidates the proposal settled and stats[1] those that fell back
// to the full sweep.
// row_cnt (ch entries) receives the number of support points per lattice
// row, which launch_compact consumes.
cudaError_t launch_support(const uint4* desc0, const uint4* desc1, int32_t* can_lr, int32_t* can_tmp,
                           int32_t* can, int32_t* row_cnt, const Geom& g, const DevParams& p, int num_sms,
                           unsigned* err, cudaStream_t st, const uint32_t* bins = nullptr, int32_t* stats = nullptr);

cudaError_t launch_compact(const int32_t* can, const int32_t* row_cnt, int32_t* row_off, int32_t* uvd, int32_t* x0,
                           int32_t* x1, int32_t* y, const Geom& g, cudaStream_t st, int corners, int* nlaunch);

// A grid cell's candidate list for the dense step: CELL_LIST 16-bit slots (a
// multiple of 16 bytes, for the bulk copies), the first CELL_LIST_MAX for
// the disparities, the last one for their number, which is larger than
// CELL_LIST_MAX where the list does not hold the cell (its bitset does).
constexpr int CELL_LIST = 48, CELL_LIST_MAX = CELL_LIST - 2;
cudaError_t launch_grid(const int32_t* can, uint32_t* tmp0, uint32_t* tmp1, uint32_t* grid0, uint32_t* grid1,
                        int16_t* list0, int16_t* list1, const Geom& g, cudaStream_t st, int* nlaunch);

// Default: every point's star found directly (k_star).  flips: row strips
// and Lawson edge flips instead; then force_global flips every problem with
// the global-memory kernel (tests) and round_limit > 0 caps the flip rounds
// (ERRF_FLIP_LIMIT when hit).  Both give the same triangles (the unique
// triangulation under the perturbation), in different list orders.  Lattice
// row r lies at y = r * step, the corners' row crow (-1: none) at y = H - 1.
cudaError_t launch_delaunay(DelDev& d0, DelDev& d1, const int32_t* row_off, int nrows, int nmax, int W, int H,
                            int step, int crow, int num_sms, int cluster_size, unsigned* err, cudaStream_t st,
                            int* nlaunch, bool flips = false, bool force_global = false, int round_limit = 0);
// Largest cluster (16 or 8 CTAs) with two co-resident copies for the flip
// kernel, or 0 if none fits.
int cluster_size_for_flip();

// Triangles binned by 64x32 prior tile, both views: a bin of PT_BIN
// entries per tile, the rest of a full bin's triangles in an overflow list.
constexpr int PT_BIN = 128;
struct PriorTiles {
    int32_t* cnt;      // [2][tiles + 1] triangles per tile; [tiles]: overflow pairs
    int32_t* bins;     // [2][tiles][PT_BIN] triangle indices
    int32_t* ovf;      // [2][ovf_cap][2] (tile, triangle) beyond full bins
    int ovf_cap;       // pairs per view (more raise ERRF_BOUNDS)
};
size_t prior_tile_count(const Geom& g);
size_t prior_overflow_capacity(const Geom& g, int Tmax);

// Plane prior of both views: prior[v*W+u] = (triangle+1) << pshift | d,
// d = d_plane clamped to [0, dcap] (dcap = disp_max + plane_radius + 1),
// 0 where no triangle covers the pixel.  Every pixel is written.
// rast: scratch of 2 * Tmax * raster_bytes() for the per-triangle set-up.
// tiled: paint tile by tile in shared memory (tl used) instead of with
// global atomics into the zeroed prior; the same bytes either way.
// zeroed: the caller has zeroed what the paint adds to already (direct:
// both priors; tiled: the tile counts).
// bin_cap: (tiled paint) entries used of each tile's bin (tests lower it so
// that the overflow list is used).
cudaError_t launch_prior(const int32_t* tri0, const int32_t* tri1, const int32_t* ctr0, const int32_t* ctr1,
                         int Tmax, const int32_t* can, const int32_t* uvd, void* rast, const PriorTiles& tl,
                         uint32_t* prior0, uint32_t* prior1, const Geom& g, int pshift, int dcap, int num_sms,
                         unsigned* err, cudaStream_t st, int* nlaunch, bool tiled, bool zeroed = false,
                         int bin_cap = PT_BIN);
// Images from this many pixels up take the tiled prior paint, whose cost
// grows more slowly with the number of triangles (prior stage, direct and
// tiled: 33 and 39 us at 1920x1080; at 2400x1500 49 and 57 or, on a scene
// with more support points, 84 and 60; 119 and 82 at 2880x1988).
constexpr long long PRIOR_TILED_MIN_PIXELS = 3LL << 20;
// Images up to this many pixels take the star construction of the
// Delaunay triangulations, larger ones the strips and flips.  The line was
// drawn at the crossover of earlier constructions (now the stars are faster
// on both sides: a pair of the synthetic scene 3 takes 158 against 256 us at
// 1242x375, 1265 against 1448 at 2880x1988), and stays: the list orders
// differ, and a pixel that two triangles cover keeps the last one.
constexpr long long DELAUNAY_STARS_MAX_PIXELS = 1LL << 21;
size_t raster_bytes();

size_t dense_smem_bytes(const Geom& g);
cudaError_t launch_dense(const uint4* desc0, const uint4* desc1, const uint32_t* prior0, const uint32_t* prior1,
                         const uint32_t* grid0, const uint32_t* grid1, const int16_t* list0, const int16_t* list1,
                         float* disp0, float* disp1, const Geom& g, const DevParams& p, int pshift, unsigned* err,
                         cudaStream_t st, int threads, int sub = 0,
                         bool force_bitset = false);

// L/R check into o0/o1 and, where given, also into c0 and c1 (arguments
// LR_ARG_C0 and the next of its kernel's LR_ARGS).
constexpr int LR_ARGS = 10, LR_ARG_C0 = 4;
cudaError_t launch_lr(const float* d0, const float* d1, float* o0, float* o1, float* c0, float* c1, const Geom& g,
                      int lr_threshold, cudaStream_t st, int sub);

// Buffers of the post-filter chain, per view: it starts from the L/R map cur
// (left as it is), keeps intermediate maps in nxt and ends in out (which
// may be mapped host memory: it is only written, once).  lab/root/sz are
// union-find scratch (W*H int32 each), roots the list of tile-local roots
// (W*H + 1 int32; its length, the first entry, starts at 0), tick a ticket
// per tile border (post_tickets int32, all 0 at the start).
struct PostViews {
    float* cur[2];
    float* nxt[2];
    float* out[2];
    int32_t* lab[2];
    int32_t* root[2];
    int32_t* sz[2];
    int32_t* roots[2];
    int32_t* tick[2];
};
// The dense maps, for a chain whose first kernel (the speckle tiles) also
// makes the L/R check into cur; d0 null: cur holds the checked maps already.
struct LrInput {
    const float* d0;
    const float* d1;
    float thr, scale;
};

// Whether the parameters ask for any post-filter.
bool post_any(const DevParams& p, bool median, bool adaptive_mean);
size_t post_tickets(int W, int H);

// Post-filters on nviews (1 or 2) disparity images.  last_args: the number
// of arguments of the last kernel launched; its first one is a PostViews
// whose nxt are the final buffers.
cudaError_t launch_post(PostViews pv, const LrInput& lr, int nviews, const Geom& g, const DevParams& p, bool median,
                        bool adaptive_mean, unsigned* err, cudaStream_t st, int* nlaunch, int num_sms, int* last_args);

}  // namespace elas
