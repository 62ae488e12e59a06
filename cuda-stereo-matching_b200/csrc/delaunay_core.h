// Delaunay triangulation of the support points with exact int64 predicates.
//
// Replaces the reference's CPU round trip through Shewchuk's Triangle
// (Elas::computeDelaunyTrianguation, src/Elas.cu:282-328).
//
// Two constructions of the same triangulation: stars (below, PXY_NONE on),
// and strips with edge flips, all steps data-parallel:
//  1. Per candidate row, sort the row's points by x and drop duplicated
//     coordinates (the lowest support index of a group is kept; Triangle
//     keeps the first of its randomised sort, src/triangle.cpp divconqdelaunay).
//  2. Insert the points row by row: the strip between two consecutive
//     non-empty rows is triangulated by merging the two rows by x; every
//     point finds its own triangle by a binary search in the other row
//     (merge path), so the strips are built fully in parallel.
//  3. Fill the pockets between the rows' first (last) points and the convex
//     hull with the triangles of the monotone-chain stack walk, each point
//     finding its own.
//  4. Build edge adjacency with an open-addressing hash of undirected edges.
//  5. Lawson edge flipping in rounds driven by a worklist: round 0 tests
//     every interior edge; later rounds test only the four outer edges of
//     each quad flipped in the previous round and the proposals that lost
//     their lock.  An edge flips when it holds the minimum priority on both
//     of its triangles; neighbour links are repaired through a forwarding
//     table in two phases (resolve, then write).  Converges to the unique
//     Delaunay triangulation under the symbolic perturbation below.
//
// Predicates: orientation and incircle on integer coordinates, exact in
// int32 / int64 arithmetic for the library's image limits (pack_xy below).
// Ties (four
// co-circular points) are broken by simulation of simplicity: point i is
// lifted to x^2+y^2 - eps^(i+1); then d is inside circle(a,b,c) iff the
// lowest index m of {a,b,c,d} is d, or d's barycentric coordinate for m is
// negative.  That makes the triangulation unique, and equal to Triangle's
// wherever no four points are co-circular.
//
// Everything here is __host__ __device__ so the same code runs in a
// sequential host emulation used by the CPU tests, which adds sequential
// forms of its own of the parallel steps.
#pragma once

#include <cmath>
#include <cstdint>
#include "common.cuh"

namespace elas {
namespace del {

HD uint32_t hash64(uint64_t k) {
    k ^= k >> 33;
    k *= 0xff51afd7ed558ccdull;
    k ^= k >> 33;
    k *= 0xc4ceb9fe1a85ec53ull;
    k ^= k >> 33;
    return uint32_t(k);
}

HD uint64_t edge_key(int a, int b) {
    return a < b ? (uint64_t(uint32_t(a)) << 32 | uint32_t(b)) : (uint64_t(uint32_t(b)) << 32 | uint32_t(a));
}

// Bijective 32-bit mix: unique flip priorities per edge within a round.
HD uint32_t prio(uint32_t e, uint32_t round) {
    uint32_t x = e + round * 0x9E3779B9u;
    x ^= x >> 16; x *= 0x7feb352du;
    x ^= x >> 15; x *= 0x846ca68bu;
    x ^= x >> 16;
    return x;
}

constexpr int32_t FINAL = 1 << 30;          // opp entry already refers to the new slot
constexpr uint32_t LOCK_FREE = 0xFFFFFFFFu;
constexpr unsigned long long HASH_EMPTY = ~0ull;

// Packed point coordinates, 16 bits each with a bias of 2^15 (coordinates
// in [-32768, 32767]; the predicates are translation invariant): every
// triangle record carries its vertices' coordinates, so the predicates
// never chase the point arrays.
HD uint32_t pack_xy(int32_t x, int32_t y) {
    return (uint32_t(x + 32768) & 0xffffu) | ((uint32_t(y + 32768) & 0xffffu) << 16);
}
HD int32_t px_of(uint32_t p) { return int32_t(p & 0xffffu) - 32768; }
HD int32_t py_of(uint32_t p) { return int32_t(p >> 16) - 32768; }

// Coordinate differences of packed points (the bias cancels).
HD int32_t dx_p(uint32_t a, uint32_t b) { return int32_t(a & 0xffffu) - int32_t(b & 0xffffu); }
HD int32_t dy_p(uint32_t a, uint32_t b) { return int32_t(a >> 16) - int32_t(b >> 16); }

// Narrow exact predicates.  The library accepts width <= 14000,
// height <= 16384 and disp_max <= 4095, so point x lies in [-4095, 13999]
// (right view: u - d) and y in [0, 16383]: |dx| <= 18094, |dy| <= 16383.
// Then every square sum and every 2x2 orientation term is below 2^30 in
// magnitude (int32), and the lifted determinant is a sum of three 32x32-bit
// products below 2^59 each (int64).  Both are exact.
HD int64_t orient_p(uint32_t a, uint32_t b, uint32_t c) {
    return int64_t(dx_p(b, a) * dy_p(c, a) - dy_p(b, a) * dx_p(c, a));
}

// > 0 iff d lies inside the circumcircle of the counter-clockwise (a,b,c):
// the 3x3 lifted determinant expanded along its lifted column,
// |a-d|^2 * orient(b,c) + |b-d|^2 * orient(c,a) + |c-d|^2 * orient(a,b)
// with every orientation taken relative to d.
HD int64_t incircle_p(uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
    const int32_t adx = dx_p(a, d), ady = dy_p(a, d);
    const int32_t bdx = dx_p(b, d), bdy = dy_p(b, d);
    const int32_t cdx = dx_p(c, d), cdy = dy_p(c, d);
    const int32_t al = adx * adx + ady * ady, bl = bdx * bdx + bdy * bdy, cl = cdx * cdx + cdy * cdy;
    const int32_t obc = bdx * cdy - bdy * cdx, oca = cdx * ady - cdy * adx, oab = adx * bdy - ady * bdx;
    return int64_t(al) * obc + int64_t(bl) * oca + int64_t(cl) * oab;
}

// inside_sos on packed coordinates; ia..id are the point indices that order
// the symbolic perturbation.
HD bool inside_sos_p(int ia, uint32_t a, int ib, uint32_t b, int ic, uint32_t c, int id, uint32_t d) {
    int64_t det = incircle_p(a, b, c, d);
    if (det != 0) return det > 0;
    int m = imin(imin(ia, ib), imin(ic, id));
    if (m == id) return true;
    if (m == ia) return orient_p(d, b, c) < 0;
    if (m == ib) return orient_p(a, d, c) < 0;
    return orient_p(a, b, d) < 0;
}

// Flip rounds are written against an accessor M that stores, per triangle t:
// v(t,k) vertex indices, xy(t,k) packed coordinates, opp(3t+k) neighbour
// half-edges, a lock word and the last round t was flipped in.  The flat
// accessor (global memory, host emulation) and the cluster accessor
// (distributed shared memory) share this code.
//
// Is the edge of half-edge h (twin tw) not locally Delaunay?  Tested from
// h's side: h's triangle (a, b, c) against the vertex of tw's triangle
// opposite the edge.
template <class M>
HD bool edge_flippable(const M& m, int h, int tw) {
    const int t = h / 3, s = h % 3, n = tw / 3, sn = tw % 3;
    const int s1 = s == 2 ? 0 : s + 1, s2 = s1 == 2 ? 0 : s1 + 1, sd = sn == 0 ? 2 : sn - 1;
    return inside_sos_p(m.v(t, s), m.xy(t, s), m.v(t, s1), m.xy(t, s1), m.v(t, s2), m.xy(t, s2), m.v(n, sd),
                        m.xy(n, sd));
}

// Phase A: test half-edge h; propose it if its edge is not locally Delaunay.
// `owner`: only the triangle with the smaller index tests a shared edge.
template <class M, class Append>
HD bool flip_propose(M& m, int h, int T, uint32_t round, bool owner, Append append_cand) {
    int t = h / 3;
    int o = m.opp(h);
    if (o < 0) return true;
    int n = o / 3;
    if (n >= T || t >= T) return false;
    if (owner && n <= t) return true;
    if (edge_flippable(m, h, o)) {
        uint32_t p = prio(uint32_t(h), round);
        m.lock_min(t, p);
        m.lock_min(n, p);
        append_cand(h, n);
    }
    return true;
}

// Phase B: flip the proposal (h, n) if it won both locks.
template <class M>
HD bool flip_apply(M& m, int h, int n, uint32_t round) {
    int t = h / 3, s = h % 3;
    uint32_t p = prio(uint32_t(h), round);
    if (m.lock(t) != p || m.lock(n) != p) return false;
    int sn = m.opp(h) % 3;
    int s1 = s == 2 ? 0 : s + 1, s2 = s1 == 2 ? 0 : s1 + 1;
    int sn1 = sn == 2 ? 0 : sn + 1, sn2 = sn1 == 2 ? 0 : sn1 + 1;
    int a = m.v(t, s), b = m.v(t, s1), c = m.v(t, s2), d = m.v(n, sn2);
    uint32_t pa = m.xy(t, s), pb = m.xy(t, s1), pc = m.xy(t, s2), pd = m.xy(n, sn2);
    int O_bc = m.opp(3 * t + s1), O_ca = m.opp(3 * t + s2);
    int O_ad = m.opp(3 * n + sn1), O_db = m.opp(3 * n + sn2);
    // t' = (c, a, d), n' = (d, b, c); the new diagonal is slot 2 of both
    m.set_v(t, c, a, d, pc, pa, pd);
    m.set_v(n, d, b, c, pd, pb, pc);
    m.set_opp(3 * t, O_ca); m.set_opp(3 * t + 1, O_ad); m.set_opp(3 * t + 2, FINAL | (3 * n + 2));
    m.set_opp(3 * n, O_db); m.set_opp(3 * n + 1, O_bc); m.set_opp(3 * n + 2, FINAL | (3 * t + 2));
    m.set_fround(t, int32_t(round));
    m.set_fround(n, int32_t(round));
    return true;
}

// The four outer half-edges of a flipped pair (t, n): t' slots 0,1 and n' slots 0,1.
HD int outer_slot(int t, int n, int k) { return k < 2 ? 3 * t + k : 3 * n + (k - 2); }

// Phase C1 (read only): where does the neighbour across outer slot x of a
// flipped pair live now?  Its old reference o still holds if o's triangle
// did not flip this round; otherwise the edge is one of the outer slots of
// that triangle's new pair, found by matching the reversed edge.  Returns
// the half-edge, -1 for the hull, or -2 if nothing matched or an index left
// [0, T) (corrupt state).
template <class M>
HD int flip_resolve_slot(M& m, int x, uint32_t round, int T) {
    int o = m.opp(x);
    if (o < 0) return -1;
    int mt = o / 3;
    if (mt >= T) return -2;
    if (m.fround(mt) != int32_t(round)) return o;
    int xt = x / 3, xk = x % 3;
    int a = m.v(xt, xk), b = m.v(xt, xk == 2 ? 0 : xk + 1);
    const int o2 = m.opp(3 * mt + 2);
    if (o2 < 0) return -2;
    int mt2 = (o2 & ~FINAL) / 3;
    if (mt2 >= T) return -2;
    const int cand_t[2] = {mt, mt2};
    for (int i = 0; i < 2; ++i)
        for (int k = 0; k < 2; ++k) {
            int tt = cand_t[i];
            if (m.v(tt, k) == b && m.v(tt, k + 1) == a) return 3 * tt + k;
        }
    return -2;
}

// Phase C2: write the links both ways and clear the FINAL marks.
template <class M>
HD void flip_relink(M& m, int t, int n, const int32_t* res) {
    for (int k = 0; k < 4; ++k) {
        int x = outer_slot(t, n, k);
        int r = res[k];
        m.set_opp(x, r);
        if (r >= 0) m.set_opp(r, x);
    }
    m.set_opp(3 * t + 2, 3 * n + 2);
    m.set_opp(3 * n + 2, 3 * t + 2);
}

// flip_resolve_slot for the four outer slots of a flipped pair, step by
// step, so that the four chains of loads overlap.  q: the pair's vertices
// c, a, d, b (t' = (c, a, d), n' = (d, b, c)), whose order is that of the
// outer edges: slot k runs from q[k] to q[k + 1].
template <class M>
HD void flip_resolve4(const M& m, int t, int n, const int32_t (&q)[4], uint32_t round, int T, int32_t (&r)[4]) {
    int mt[4];
    bool moved[4];
    for (int k = 0; k < 4; ++k) r[k] = m.opp(outer_slot(t, n, k));
    for (int k = 0; k < 4; ++k) {
        mt[k] = r[k] < 0 ? t : r[k] / 3;
        r[k] = r[k] < 0 ? -1 : (mt[k] >= T ? -2 : r[k]);
        moved[k] = false;
        if (r[k] >= 0) moved[k] = m.fround(mt[k]) == int32_t(round);
    }
    if (!(moved[0] || moved[1] || moved[2] || moved[3])) return;
    int mt2[4];
    for (int k = 0; k < 4; ++k) mt2[k] = moved[k] ? m.opp(3 * mt[k] + 2) : -1;
    for (int k = 0; k < 4; ++k) {
        mt2[k] = mt2[k] < 0 ? T : (mt2[k] & ~FINAL) / 3;
        if (!moved[k]) continue;
        r[k] = -2;
        if (mt2[k] >= T) continue;
        const int a = q[k], b = q[(k + 1) & 3];
        const int u0 = m.v(mt[k], 0), u1 = m.v(mt[k], 1), u2 = m.v(mt[k], 2);
        const int w0 = m.v(mt2[k], 0), w1 = m.v(mt2[k], 1), w2 = m.v(mt2[k], 2);
        if (w1 == b && w2 == a) r[k] = 3 * mt2[k] + 1;
        if (w0 == b && w1 == a) r[k] = 3 * mt2[k];
        if (u1 == b && u2 == a) r[k] = 3 * mt[k] + 1;
        if (u0 == b && u1 == a) r[k] = 3 * mt[k];
    }
}

// Flat storage: plain arrays (global memory on the device, host memory in
// the emulation).  AMin performs the lock's atomic minimum.
template <class AMin>
struct FlatTri {
    int32_t* tv;      // [3T] vertex indices
    uint32_t* txy;    // [3T] packed coordinates
    int32_t* topp;    // [3T]
    uint32_t* tlock;  // [T]
    int32_t* tround;  // [T]
    AMin amin;
    HD int v(int t, int k) const { return tv[3 * t + k]; }
    HD uint32_t xy(int t, int k) const { return txy[3 * t + k]; }
    HD int opp(int h) const { return topp[h]; }
    HD uint32_t lock(int t) const { return tlock[t]; }
    HD int32_t fround(int t) const { return tround[t]; }
    HD void lock_min(int t, uint32_t p) { amin(&tlock[t], p); }
    HD void set_v(int t, int a, int b, int c, uint32_t pa, uint32_t pb, uint32_t pc) {
        tv[3 * t] = a; tv[3 * t + 1] = b; tv[3 * t + 2] = c;
        txy[3 * t] = pa; txy[3 * t + 1] = pb; txy[3 * t + 2] = pc;
    }
    HD void set_opp(int h, int o) { topp[h] = o; }
    HD void set_fround(int t, int32_t r) { tround[t] = r; }
};

// ---------------------------------------------------------------------------
// Stars: the Delaunay neighbours of one point, found directly.
//
// Under the perturbation the triangulation is unique, so each point's star
// (its neighbours in counter-clockwise order) can be computed on its own and
// the stars of all points agree.  The walk around p starts at p's nearest
// neighbour q0 (the disc with diameter p q0 holds no other point, so p q0 is
// an edge of every Delaunay triangulation).  From an edge p->q the next
// neighbour on a side is, among the points strictly on that side, the one
// whose circle through p and q holds no other of them: the circles through
// p and q form a pencil, and "b lies inside the circle through p, q, a" is a
// strict total order on the points of one side (the perturbed incircle
// determinant is antisymmetric in a and b).  The minimum of that order is the
// next neighbour; a side with no point marks a hull edge.  The walk goes
// counter-clockwise until it returns to q0.  A point of the hull boundary
// starts at its successor on the boundary (counter-clockwise, the interior
// on the left) instead and walks until it reaches its predecessor.

constexpr uint32_t PXY_NONE = 0xFFFFFFFFu;   // a dropped duplicate point

// That order for a and b known to lie strictly left of p->q: is b the better
// next neighbour (inside_sos_p(p, q, a, b))?  By the centres of their circles on the bisector of p and q: with u = q - p
// a point s (relative to p) has its centre at t = (|s|^2 - u.s) / cross(u, s)
// (up to a common scale), and b is inside a's circle when its t is smaller.
// Numerators stay below 2^31 and denominators below 2^30 at the coordinate
// limits of orient_p, so the cross products are exact in int64.  Equal
// centres (four co-circular points) go by the perturbation: the lowest
// index decides as in inside_sos_p, where d = b, and a's own barycentric
// coordinate is positive as b lies left of p->q.
HD bool star_better_left(int ip, uint32_t pp, int iq, uint32_t pq, int ia, uint32_t pa, int ib, uint32_t pb) {
    const int32_t ux = dx_p(pq, pp), uy = dy_p(pq, pp);
    const int32_t ax = dx_p(pa, pp), ay = dy_p(pa, pp), bx = dx_p(pb, pp), by = dy_p(pb, pp);
    const int32_t ca = ux * ay - uy * ax, cb = ux * by - uy * bx;
    const int32_t na = ax * ax + ay * ay - (ux * ax + uy * ay), nb = bx * bx + by * by - (ux * bx + uy * by);
    const int64_t l = int64_t(nb) * ca, r = int64_t(na) * cb;
    if (l != r) return l < r;
    const int m = imin(imin(ip, iq), imin(ia, ib));
    if (m == ib) return true;
    if (m == ia) return false;
    return (m == ip ? orient_p(pb, pq, pa) : orient_p(pp, pb, pa)) < 0;
}

// Does every point inside the circle through p, q and r lie in the square
// |x - px|, |y - py| <= R?  Points exist only in the box [bx0, bx1] x
// [by0, by1] (all points of the problem), so only the part of the circle
// inside the box counts: its extent is bounded through the circle's chords
// at the box edges nearest the centre.  By comparisons only: every quantity
// is scaled by D = |2 cross(q - p, r - p)| (the centre's numerators, the box,
// R), so no division and no square root.  The centre numerators and the
// scaled box are exact integers in double; the squared terms (below 2^93)
// carry a relative rounding of 2^-53, and every point outside the square is
// at least R + 1 away from p in x or in y, a pixel of margin.
HD bool circle_inside(uint32_t pp, uint32_t pq, uint32_t pr, int R, const int32_t* box) {
    const double qx = dx_p(pq, pp), qy = dy_p(pq, pp), rx = dx_p(pr, pp), ry = dy_p(pr, pp);
    const double d2x = 2.0 * (qx * ry - qy * rx);
    const double q2 = qx * qx + qy * qy, r2 = rx * rx + ry * ry;
    const double sg = d2x < 0.0 ? -1.0 : 1.0, D = fabs(d2x);
    const double CX = sg * (ry * q2 - qy * r2), CY = sg * (qx * r2 - rx * q2);   // centre * D
    const double RHO2 = CX * CX + CY * CY;                                       // radius^2 * D^2
    const double BX0 = (box[0] - px_of(pp)) * D, BY0 = (box[1] - py_of(pp)) * D;
    const double BX1 = (box[2] - px_of(pp)) * D, BY1 = (box[3] - py_of(pp)) * D;
    const double EY = fmin(fmax(CY, BY0), BY1) - CY, EX = fmin(fmax(CX, BX0), BX1) - CX;
    if (EY * EY >= RHO2 || EX * EX >= RHO2) return true;     // the circle misses the box
    const double RD = double(R) * D, H2 = RHO2 - EY * EY, V2 = RHO2 - EX * EX;
    // each side of the clipped extent: the box edge itself, or the chord end
    auto side_ok = [](double edge, double c, double rd, double h2) {
        // max(c - h, edge) >= -rd  (edge, c scaled), i.e. edge >= -rd or h <= c + rd
        return edge >= -rd || (c + rd >= 0.0 && h2 <= (c + rd) * (c + rd));
    };
    return side_ok(BX0, CX, RD, H2) && side_ok(-BX1, -CX, RD, H2) && side_ok(BY0, CY, RD, V2) &&
           side_ok(-BY1, -CY, RD, V2);
}

// When a star is proven.  With every point of the square of half-size R
// around p at hand, the nearest neighbour at distance d is certain once
// d <= R and the next neighbour r after q once circle_inside(R) holds for p,
// q, r: monotone in R, and certain in any case once the square covers the
// box of all points (which also proves a hull edge).  A search over growing
// squares starts at half-size R0 and doubles it until its answer is
// certain; the number of doublings a star needs is therefore a property of
// the star, whatever points were looked at to find it.  The tests' sequential
// emulation searches that way; the device finds the star from fewer points
// and counts the same doublings.

// The window's half-size R0 of a problem: 3.5 mean point spacings (the
// square root of the box area per point), within [16, 128] pixels: the
// largest such r with 4 r^2 n <= 49 area.  Most stars are then proven by
// the window (a smaller one proves fewer, a larger one holds more points
// than a step should look at).
HD int star_r0(const int32_t* box, int n) {
    const int64_t area = int64_t(box[2] - box[0] + 1) * (box[3] - box[1] + 1);
    int r = 16;
    for (int st = 64; st > 0; st >>= 1)
        if (r + st <= 128 && 4LL * (r + st) * (r + st) * (n > 0 ? n : 1) <= 49 * area) r += st;
    return r;
}
constexpr int STAR_NB = 256;      // neighbours of one point

// The hull boundary, counter-clockwise (the interior on the left of each
// step), from the rows' extreme points: the top row left to right, the
// right chain down, the bottom row right to left, the left chain up.  The
// chains are the rows' last (first) points, top to bottom, without the
// concave ones; collinear points stay, as every point on the boundary is a
// vertex of the triangulation.  Position j of that cycle: top row (tl
// points) left to right, right chain rows 1..nr-1, bottom row (bl points)
// right to left from its second last, left chain rows nl-2..1.  Returns
// (row position, index within that row); the cycle has
// tl + (nr - 1) + (bl - 1) + (nl - 2) points when the top and bottom rows
// differ.
HD int hull_cycle_len(int tl, int bl, int nl, int nr) { return tl + (nr - 1) + (bl - 1) + (nl - 2); }
HD void hull_cycle_at(int j, int R, int tl, int bl, const int32_t* lstk, int nl, const int32_t* rstk, int nr,
                      int* row, int* pos, bool* last) {
    *last = false;
    if (j < tl) { *row = 0; *pos = j; return; }
    j -= tl;
    if (j < nr - 1) { *row = rstk[j + 1]; *pos = 0; *last = true; return; }
    j -= nr - 1;
    if (j < bl - 1) { *row = R - 1; *pos = bl - 2 - j; return; }
    j -= bl - 1;
    *row = lstk[nl - 2 - j];
    *pos = 0;
}

// Triangles of a star of deg neighbours: (p, nb(i), nb(i+1)), wrapping when
// closed.  Triangle i is emitted by p when p is its smallest vertex, which
// makes it come out normalised (see normalise below).
HD int star_tris(int deg, bool closed) { return closed ? deg : (deg > 0 ? deg - 1 : 0); }

// Rotate a triangle so its smallest vertex index comes first.
HD void normalise(int32_t* v) {
    int a = v[0], b = v[1], c = v[2];
    while (a > b || a > c) { int x = a; a = b; b = c; c = x; }
    v[0] = a; v[1] = b; v[2] = c;
}

}  // namespace del
}  // namespace elas
