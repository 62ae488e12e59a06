// Test helper: sequential host emulation of the CUDA Delaunay pipeline
// (cuda-stereo-matching_b200/csrc/k_delaunay.cu).  Every data-parallel
// phase of the device code runs here as a loop over its items and calls the
// same __host__ __device__ functions (delaunay_core.h), so the algorithm can
// be checked on the CPU against the exact checker and Triangle.
#include <algorithm>
#include <cstdlib>
#include <cstdint>
#include <cstring>
#include <unordered_map>
#include <vector>

#include "../../cuda-stereo-matching_b200/csrc/delaunay_core.h"

// Sequential forms of steps that the device's kernels make in parallel.
namespace elas {
namespace del {

struct Pts {
    const int32_t* x;
    const int32_t* y;
};

// Strip between an upper row A[0..m) and a lower row B[0..n), both sorted
// by strictly increasing x: walking the merge of A[1..m) and B[1..n) by x
// (A first on equal x), each element advances its row by one point and
// creates one counter-clockwise triangle.  These two functions give the
// triangle of one element and its position in the strip, so every point
// can emit its triangles independently.
//
// Number of elements of the sorted X[0..n) with x < v (strict) or x <= v.
HD int count_below(Pts P, const int32_t* X, int n, int32_t v, bool inclusive) {
    int lo = 0, hi = n;
    while (lo < hi) {
        int mid = (lo + hi) >> 1;
        int32_t x = P.x[X[mid]];
        if (inclusive ? (x <= v) : (x < v)) lo = mid + 1;
        else hi = mid;
    }
    return lo;
}

// Element A[k], 1 <= k < m: triangle (A[k-1], A[k], B[j]); returns its position.
HD int strip_tri_upper(Pts P, const int32_t* A, const int32_t* B, int n, int k, int32_t* tri) {
    int cl = count_below(P, B, n, P.x[A[k]], false);
    int j = cl > 0 ? cl - 1 : 0;
    tri[0] = A[k - 1]; tri[1] = A[k]; tri[2] = B[j];
    return (k - 1) + j;
}

// Element B[k], 1 <= k < n: triangle (A[i], B[k], B[k-1]); returns its position.
HD int strip_tri_lower(Pts P, const int32_t* A, int m, const int32_t* B, int k, int32_t* tri) {
    int cl = count_below(P, A, m, P.x[B[k]], true);
    int i = cl > 0 ? cl - 1 : 0;
    tri[0] = A[i]; tri[1] = B[k]; tri[2] = B[k - 1];
    return i + (k - 1);
}

// Fill the pocket between a boundary chain (one point per non-empty row,
// top to bottom: point index ci[k] at (cx[k], cy[k])) and its convex hull.
// side = +1 for the left chain (first points), -1 for the right chain
// (last points).  `stack` has room for 4 * len ints: an entry is the
// record (point index, x, y, -) of a chain point, so a pop reads one
// 16-byte record.  The next chain point is loaded one step ahead.  Returns
// the number of counter-clockwise triangles written.
HD int fill_pockets(const int32_t* ci, const int32_t* cx, const int32_t* cy, int len, int side, int32_t* stack,
                    int32_t* tri) {
    // the two top stack entries are kept in registers: (a, b) = stack[sp-2], stack[sp-1]
    int sp = 0, k = 0;
    // orientations are exact in int32 within the library's coordinate range
    // (|dx| <= 18094, |dy| <= 16383, see orient_p)
    int32_t ia = 0, ib = 0;
    int32_t ax = 0, ay = 0, bx = 0, by = 0;
    int32_t nx = len > 0 ? cx[0] : 0, ny = len > 0 ? cy[0] : 0, ni = len > 0 ? ci[0] : 0;
    for (int i = 0; i < len; ++i) {
        const int32_t x = nx, y = ny;
        const int32_t ii = ni;
        if (i + 1 < len) { nx = cx[i + 1]; ny = cy[i + 1]; ni = ci[i + 1]; }
        while (sp >= 2) {
            const int32_t o = (bx - ax) * (y - ay) - (by - ay) * (x - ax);
            if (side > 0 ? (o > 0) : (o < 0)) {
                tri[3 * k] = ia;
                tri[3 * k + 1] = side > 0 ? ib : ii;
                tri[3 * k + 2] = side > 0 ? ii : ib;
                ++k;
                --sp;
                ib = ia; bx = ax; by = ay;
                if (sp >= 2) {
                    const int32_t* q = stack + 4 * (sp - 2);
                    ia = q[0]; ax = q[1]; ay = q[2];
                }
            } else {
                break;
            }
        }
        int32_t* e = stack + 4 * sp;
        e[0] = ii; e[1] = x; e[2] = y; e[3] = 0;
        ++sp;
        ia = ib; ax = bx; ay = by;
        ib = ii; bx = x; by = y;
    }
    return k;
}

// For the edge p->q and two points a, b on the walk's side, is b the better
// next neighbour (inside the circle through p, q and a)?  side > 0: left of
// p->q, triangle (p, q, a) counter-clockwise; side < 0: right, triangle
// (p, a, q).
HD bool star_better(int ip, uint32_t pp, int iq, uint32_t pq, int ia, uint32_t pa, int ib, uint32_t pb, int side) {
    return side > 0 ? inside_sos_p(ip, pp, iq, pq, ia, pa, ib, pb) : inside_sos_p(ip, pp, ia, pa, iq, pq, ib, pb);
}

// Is b strictly on the walk's side of p->q?
HD bool star_side(uint32_t pp, uint32_t pq, uint32_t pb, int side) {
    const int64_t o = orient_p(pp, pq, pb);
    return side > 0 ? o > 0 : o < 0;
}

// Walk the star.  An interior point (hn < 0) starts at nearest(), p's
// nearest neighbour, and walks counter-clockwise until it is back there.  A
// point of the hull boundary starts at hn, its successor on the boundary
// (counter-clockwise, the interior on the left), and walks until it reaches
// hp, its predecessor.  next(q, side) returns the next neighbour after q on
// that side (-1: none, so p->q is a hull edge; -2: the search failed).
// The neighbours are appended to ccw (counter-clockwise) and, should an
// interior point meet the hull (all points collinear), to cw (clockwise from
// the start); star_at gives them in counter-clockwise order.  Returns false
// if a search failed or a list would pass cap.
template <class Nearest, class Next>
HD bool star_walk(int hn, int hp, Nearest nearest, Next next, int32_t* ccw, int32_t* cw, int cap, int* m, int* k,
                  bool* closed) {
    *m = 0;
    *k = 0;
    *closed = false;
    const int q0 = hn >= 0 ? hn : nearest();
    if (q0 < 0) return q0 == -1;
    ccw[(*m)++] = q0;
    int q = q0;
    for (;;) {
        const int r = next(q, +1);
        if (r == -2) return false;
        if (r < 0) break;
        if (r == q0) {
            *closed = hn < 0;
            return hn < 0;
        }
        if (*m >= cap) return false;
        ccw[(*m)++] = r;
        if (r == hp) return true;
        q = r;
    }
    if (hn >= 0) return true;
    q = q0;
    for (;;) {
        const int r = next(q, -1);
        if (r == -2) return false;
        if (r < 0) break;
        if (*k >= cap) return false;
        cw[(*k)++] = r;
        q = r;
    }
    return true;
}

// The hull boundary, counter-clockwise (the interior on the left of each
// step), from the rows' extreme points: the top row left to right, the
// right chain down, the bottom row right to left, the left chain up.  The
// chains are the rows' last (first) points with the concave ones removed by
// the monotone stack walk; collinear points stay, as every point on the
// boundary is a vertex of the triangulation.  xy[s] holds the packed
// coordinates of the leftmost (side 0) or rightmost (side 1) point of
// non-empty row s (of R, top to bottom).  Writes the chain as row positions
// (top to bottom; room for R) and its length.
HD void hull_chain(int side, int R, const uint32_t* xy, int32_t* st, int* len) {
    int sp = 0;
    uint32_t a = 0, b = 0;     // the stack's top two points
    for (int s = 0; s < R; ++s) {
        const uint32_t x = xy[s];
        while (sp >= 2) {
            const int64_t o = orient_p(a, b, x);
            if (side ? o < 0 : o > 0) {
                --sp;
                b = a;
                if (sp >= 2) a = xy[st[sp - 2]];
            } else {
                break;
            }
        }
        st[sp++] = s;
        a = b;
        b = x;
    }
    *len = sp;
}

// The same chain, decided point by point (for a parallel build): row i's
// point is dropped by the stack walk exactly when it lies strictly inside
// the segment of two other chain points j < i < k (strictly right of L_j ->
// L_k for the left chain, left of it for the right chain).  With
// coordinates relative to point i and x mirrored for the right chain, that
// holds iff min_{j<i} x_j / -y_j + min_{k>i} x_k / y_k < 0 (the rows above
// have y < 0, those below y > 0); both minima and their sum are compared
// as exact fractions.  |x| <= 18094 and 0 < y <= 16383 (the coordinate
// limits of orient_p), so every cross product is below 2^29 and the final
// sum below 2^30: exact in int32.
HD bool hull_on_chain(int side, int R, const uint32_t* xy, int i) {
    if (i == 0 || i == R - 1) return true;
    const uint32_t c = xy[i];
    const int sg = side ? -1 : 1;
    // each minimum over four interleaved partial minima (independent chains)
    int32_t n[2][4], d[2][4];
    for (int h = 0; h < 2; ++h)
        for (int u = 0; u < 4; ++u) {
            n[h][u] = 1;
            d[h][u] = 0;     // +infinity: 1/0 compares above every fraction below
        }
    auto fold = [&](int h, int u, uint32_t v, int dsign) {
        const int32_t x = sg * dx_p(v, c), dd = dsign * dy_p(v, c);
        if (d[h][u] == 0 || x * d[h][u] < n[h][u] * dd) {
            n[h][u] = x;
            d[h][u] = dd;
        }
    };
    int j = 0;
    for (; j + 4 <= i; j += 4)
        for (int u = 0; u < 4; ++u) fold(0, u, xy[j + u], -1);
    for (; j < i; ++j) fold(0, 0, xy[j], -1);
    int k = i + 1;
    for (; k + 4 <= R; k += 4)
        for (int u = 0; u < 4; ++u) fold(1, u, xy[k + u], 1);
    for (; k < R; ++k) fold(1, 0, xy[k], 1);
    int32_t sn = n[0][0], sd = d[0][0], tn = n[1][0], td = d[1][0];
    for (int u = 1; u < 4; ++u) {
        if (d[0][u] != 0 && n[0][u] * sd < sn * d[0][u]) { sn = n[0][u]; sd = d[0][u]; }
        if (d[1][u] != 0 && n[1][u] * td < tn * d[1][u]) { tn = n[1][u]; td = d[1][u]; }
    }
    return sn * td + tn * sd >= 0;
}

// Neighbour i in counter-clockwise order: the clockwise part reversed, then
// the counter-clockwise part.
HD int32_t star_at(const int32_t* ccw, int m, const int32_t* cw, int k, int i) {
    (void)m;
    return i < k ? cw[k - 1 - i] : ccw[i - k];
}

}  // namespace del
}  // namespace elas

using namespace elas::del;

// px, py: n points; row_off: nrows+1 offsets of the points of each lattice
// row (points of a row share y).  tris_out: room for cap triangles.  Returns
// the triangle count, or -1 on an internal error.  stats (nullable):
// [0] flip rounds, [1] flips.
// phased = 0: rounds in the propose / flip / resolve / relink formulation
// with worklists (k_flip_global).  phased = 1: rounds in the three-phase
// formulation of k_flip_local and k_flip_smem (flip; resolve and propose
// the outer edges; relink and re-propose the lost proposals; two lock
// arrays by round parity).  Both must give the same triangles, in the same
// slots, after the same rounds and flips.
static int emu_core(const int32_t* px, const int32_t* py, int n, const int32_t* row_off, int nrows,
                    int32_t* tris_out, int cap, long long* stats, int phased) {
    Pts P{px, py};
    // 1. per-row sort + dedup (k_rowsort)
    std::vector<int32_t> srt(std::max(n, 1)), rcnt(nrows, 0);
    for (int r = 0; r < nrows; ++r) {
        std::vector<int32_t> v;
        for (int i = row_off[r]; i < row_off[r + 1]; ++i) v.push_back(i);
        std::sort(v.begin(), v.end(), [&](int a, int b) { return px[a] != px[b] ? px[a] < px[b] : a < b; });
        int m = 0;
        for (size_t k = 0; k < v.size(); ++k)
            if (k == 0 || px[v[k]] != px[v[k - 1]]) srt[row_off[r] + m++] = v[k];
        rcnt[r] = m;
    }
    // 2. plan (k_plan)
    std::vector<int> ne, soff;
    for (int r = 0; r < nrows; ++r)
        if (rcnt[r] > 0) ne.push_back(r);
    const int R = int(ne.size());
    int off = 0;
    for (int s = 0; s + 1 < R; ++s) { soff.push_back(off); off += rcnt[ne[s]] + rcnt[ne[s + 1]] - 2; }
    const int Tmax = 2 * n + 16;
    std::vector<int32_t> tri(3 * size_t(Tmax), -1);
    int T = 0;
    if (R >= 2) {
        if (off + 2 * R > Tmax) return -1;
        std::vector<int32_t> ci(R), cx(R), cy(R), stk(4 * size_t(R));
        int pockets = 0;
        for (int side = 0; side < 2; ++side) {
            for (int s = 0; s < R; ++s) {
                int r = ne[s];
                int i = srt[row_off[r] + (side ? rcnt[r] - 1 : 0)];
                ci[s] = i; cx[s] = px[i]; cy[s] = py[i];
            }
            pockets += fill_pockets(ci.data(), cx.data(), cy.data(), R, side ? -1 : +1, stk.data(),
                                    &tri[3 * size_t(off + pockets)]);
        }
        T = off + pockets;
        // 3. strips (k_strips), every point of every non-empty row
        for (int lo = 0; lo < R; ++lo) {
            int r = ne[lo];
            const int32_t* A = &srt[row_off[r]];
            for (int k = 1; k < rcnt[r]; ++k) {
                int32_t t3[3];
                if (lo + 1 < R) {
                    int rb = ne[lo + 1];
                    int pos = strip_tri_upper(P, A, &srt[row_off[rb]], rcnt[rb], k, t3);
                    std::memcpy(&tri[3 * size_t(soff[lo] + pos)], t3, 12);
                }
                if (lo >= 1) {
                    int ra = ne[lo - 1];
                    int pos = strip_tri_lower(P, &srt[row_off[ra]], rcnt[ra], A, k, t3);
                    std::memcpy(&tri[3 * size_t(soff[lo - 1] + pos)], t3, 12);
                }
            }
        }
    }
    for (int i = 0; i < 3 * T; ++i)
        if (tri[i] < 0) return -1;   // a strip slot nobody wrote
    // 4. adjacency (k_hash_insert + k_link)
    std::vector<int32_t> opp(3 * size_t(Tmax), -1);
    std::unordered_map<uint64_t, std::vector<int>> edges;
    for (int h = 0; h < 3 * T; ++h) {
        int t = h / 3, s = h % 3;
        edges[edge_key(tri[3 * t + s], tri[3 * t + (s + 1) % 3])].push_back(h);
    }
    for (auto& kv : edges) {
        if (kv.second.size() == 2) { opp[kv.second[0]] = kv.second[1]; opp[kv.second[1]] = kv.second[0]; }
        else if (kv.second.size() != 1) return -1;
    }
    // 5. flips (k_flip_local / k_flip_smem / k_flip_global)
    std::vector<uint32_t> txy(3 * size_t(Tmax)), lock(Tmax, LOCK_FREE);
    std::vector<int32_t> fround(Tmax, -1), cand(6 * size_t(Tmax)), flips(6 * size_t(Tmax)), wl[2];
    wl[0].resize(6 * size_t(Tmax));
    wl[1].resize(6 * size_t(Tmax));
    for (int i = 0; i < 3 * T; ++i) txy[i] = pack_xy(px[tri[i]], py[tri[i]]);
    auto amin = [](uint32_t* p, uint32_t v) { if (v < *p) *p = v; };
    FlatTri<decltype(amin)> m{tri.data(), txy.data(), opp.data(), lock.data(), fround.data(), amin};
    std::vector<char> mark(3 * size_t(T), 0);
    int n_cur = 3 * T;
    long long rounds = 0, nflips = 0;
    if (phased) {
        std::vector<uint32_t> lock1(Tmax, LOCK_FREE);
        std::vector<int32_t> cl[2];
        // round 0's proposals: every interior edge once (owner rule), with lock array 0
        m.tlock = lock.data();
        for (int h = 0; h < 3 * T; ++h)
            if (!flip_propose(m, h, T, 0u, true, [&](int hh, int nn) { cl[0].push_back(hh); cl[0].push_back(nn); }))
                return -1;
        for (int round = 0; round < 100000; ++round) {
            const int cur = round & 1, nxt = cur ^ 1;
            std::vector<int32_t>& cc = cl[cur];
            std::vector<int32_t>& cn = cl[nxt];
            uint32_t* lock_cur = cur ? lock1.data() : lock.data();
            uint32_t* lock_nxt = cur ? lock.data() : lock1.data();
            rounds = round + 1;
            if (cc.empty()) break;
            // B: flip the winners; release the previous round's locks (list cn); clear the bitset
            m.tlock = lock_cur;
            int nf = 0;
            for (size_t c = 0; c < cc.size(); c += 2)
                if (flip_apply(m, cc[c], cc[c + 1], uint32_t(round))) {
                    flips[6 * nf] = cc[c] / 3;
                    flips[6 * nf + 1] = cc[c + 1];
                    ++nf;
                }
            for (size_t c = 0; c < cn.size(); c += 2) {
                lock_nxt[cn[c] / 3] = LOCK_FREE;
                lock_nxt[cn[c + 1]] = LOCK_FREE;
            }
            cn.clear();
            std::fill(mark.begin(), mark.end(), 0);
            auto propose_next = [&](int h, int nn) {
                const uint32_t p = prio(uint32_t(h), uint32_t(round + 1));
                if (p < lock_nxt[h / 3]) lock_nxt[h / 3] = p;
                if (p < lock_nxt[nn]) lock_nxt[nn] = p;
                cn.push_back(h);
                cn.push_back(nn);
            };
            // C1: resolve every flipped pair's outer neighbours, then test and
            // propose the outer edges (vertices are final after B)
            for (int f = 0; f < nf; ++f)
                for (int k = 0; k < 4; ++k) {
                    int r = flip_resolve_slot(m, outer_slot(flips[6 * f], flips[6 * f + 1], k), uint32_t(round), T);
                    if (r == -2) return -1;
                    flips[6 * f + 2 + k] = r;
                }
            for (int f = 0; f < nf; ++f)
                for (int k = 0; k < 4; ++k) {
                    const int x = outer_slot(flips[6 * f], flips[6 * f + 1], k), r = flips[6 * f + 2 + k];
                    if (r < 0) continue;
                    const int c = std::min(x, r), tw = c == x ? r : x;
                    if (mark[c]) continue;
                    mark[c] = 1;
                    if (edge_flippable(m, c, tw)) propose_next(c, tw / 3);
                }
            // C2: relink; re-propose the lost proposals without a new test
            for (int f = 0; f < nf; ++f) flip_relink(m, flips[6 * f], flips[6 * f + 1], &flips[6 * f + 2]);
            for (size_t c = 0; c < cc.size(); c += 2) {
                const int h = cc[c], n2 = cc[c + 1], t = h / 3;
                if (fround[t] != round && fround[n2] != round) propose_next(h, n2);
            }
            nflips += nf;
        }
        n_cur = 0;
    }
    for (int round = 0; !phased && round < 100000; ++round) {
        const std::vector<int32_t>& cur = wl[round & 1];
        std::vector<int32_t>& nxt = wl[(round + 1) & 1];
        int nc = 0;
        for (int k = 0; k < n_cur; ++k) {
            int h = round == 0 ? k : cur[k];
            if (!flip_propose(m, h, T, uint32_t(round), round == 0, [&](int hh, int nn) {
                    cand[2 * nc] = hh; cand[2 * nc + 1] = nn; ++nc;
                }))
                return -1;
        }
        ++rounds;
        if (nc == 0) break;
        int nf = 0;
        for (int c = 0; c < nc; ++c)
            if (flip_apply(m, cand[2 * c], cand[2 * c + 1], uint32_t(round))) {
                flips[6 * nf] = cand[2 * c] / 3;
                flips[6 * nf + 1] = cand[2 * c + 1];
                ++nf;
            }
        for (int f = 0; f < nf; ++f)
            for (int k = 0; k < 4; ++k) {
                int r = flip_resolve_slot(m, outer_slot(flips[6 * f], flips[6 * f + 1], k), uint32_t(round), T);
                if (r == -2) return -1;
                flips[6 * f + 2 + k] = r;
            }
        // the next worklist holds each interior edge once, as its lower half-edge
        int nn = 0;
        std::fill(mark.begin(), mark.end(), 0);
        auto push = [&](int x, int r) {
            if (r < 0) return;
            const int c = std::min(x, r);
            if (mark[c]) return;
            mark[c] = 1;
            nxt[nn++] = c;
        };
        for (int f = 0; f < nf; ++f) {
            int t = flips[6 * f], n2 = flips[6 * f + 1];
            flip_relink(m, t, n2, &flips[6 * f + 2]);
            for (int k = 0; k < 4; ++k) push(outer_slot(t, n2, k), flips[6 * f + 2 + k]);
        }
        for (int c = 0; c < nc; ++c) {
            int h = cand[2 * c], n2 = cand[2 * c + 1], t = h / 3;
            lock[t] = LOCK_FREE;
            lock[n2] = LOCK_FREE;
            if (fround[t] != round && fround[n2] != round) push(h, opp[h]);
        }
        nflips += nf;
        n_cur = nn;
    }
    for (int t = 0; t < T; ++t) normalise(&tri[3 * size_t(t)]);
    if (T <= cap) std::memcpy(tris_out, tri.data(), sizeof(int32_t) * 3 * size_t(T));
    if (stats) { stats[0] = rounds; stats[1] = nflips; }
    return T;
}

extern "C" int emu_delaunay(const int32_t* px, const int32_t* py, int n, const int32_t* row_off, int nrows,
                            int32_t* tris_out, int cap, long long* stats) {
    return emu_core(px, py, n, row_off, nrows, tris_out, cap, stats, 0);
}

extern "C" int emu_delaunay_phased(const int32_t* px, const int32_t* py, int n, const int32_t* row_off, int nrows,
                                   int32_t* tris_out, int cap, long long* stats) {
    return emu_core(px, py, n, row_off, nrows, tris_out, cap, stats, 1);
}

// Star construction (k_plan, k_star, k_star_far, k_star_emit), sequentially:
// the same rows, hull boundary, star order and owner rule, one point after
// another, each search over squares that grow until its answer is certain.
// Triangles come out in point order, as on the device.  stats (nullable): [0]
// 0, [1] squares grown, [2] candidates examined.  Returns the triangle count,
// or -1.
extern "C" int emu_delaunay_star(const int32_t* px, const int32_t* py, int n, const int32_t* row_off, int nrows,
                                 int32_t* tris_out, int cap, long long* stats) {
    // rows sorted by (x, index), repeated x dropped (k_rowsort)
    std::vector<int32_t> srt(std::max(n, 1)), rcnt(nrows, 0);
    std::vector<uint32_t> pxy(std::max(n, 1), PXY_NONE), sxy(std::max(n, 1), 0);
    for (int r = 0; r < nrows; ++r) {
        std::vector<int32_t> v;
        for (int i = row_off[r]; i < row_off[r + 1]; ++i) v.push_back(i);
        std::sort(v.begin(), v.end(), [&](int a, int b) { return px[a] != px[b] ? px[a] < px[b] : a < b; });
        int m = 0;
        for (size_t k = 0; k < v.size(); ++k)
            if (k == 0 || px[v[k]] != px[v[k - 1]]) {
                srt[row_off[r] + m] = v[k];
                sxy[row_off[r] + m] = pxy[v[k]] = pack_xy(px[v[k]], py[v[k]]);
                ++m;
            }
        rcnt[r] = m;
    }
    std::vector<int> ne;
    for (int r = 0; r < nrows; ++r)
        if (rcnt[r] > 0) ne.push_back(r);
    // hull boundary and the box of all points (k_plan)
    std::vector<int32_t> hnext(std::max(n, 1), -1), hprev(std::max(n, 1), -1);
    int32_t box[4] = {0, 0, 0, 0};
    const int R = int(ne.size());
    if (R >= 1) {
        box[0] = px[srt[row_off[ne[0]]]];
        box[2] = px[srt[row_off[ne[0]] + rcnt[ne[0]] - 1]];
        for (int s2 = 0; s2 < R; ++s2) {
            box[0] = std::min(box[0], px[srt[row_off[ne[s2]]]]);
            box[2] = std::max(box[2], px[srt[row_off[ne[s2]] + rcnt[ne[s2]] - 1]]);
        }
        box[1] = py[row_off[ne[0]]];
        box[3] = py[row_off[ne[R - 1]]];
    }
    if (R >= 2) {
        std::vector<int32_t> lst(R), rst(R);
        int nl = 0, nr = 0;
        auto first = [&](int s2) { return srt[row_off[ne[s2]]]; };
        auto last = [&](int s2) { return srt[row_off[ne[s2]] + rcnt[ne[s2]] - 1]; };
        std::vector<uint32_t> xyf(R), xyl(R);
        for (int s2 = 0; s2 < R; ++s2) {
            xyf[s2] = pxy[first(s2)];
            xyl[s2] = pxy[last(s2)];
        }
        hull_chain(0, R, xyf.data(), lst.data(), &nl);
        hull_chain(1, R, xyl.data(), rst.data(), &nr);
        const int tl = rcnt[ne[0]], bl = rcnt[ne[R - 1]];
        const int C = hull_cycle_len(tl, bl, nl, nr);
        auto at = [&](int j) {
            int row, pos;
            bool lastp;
            hull_cycle_at(j, R, tl, bl, lst.data(), nl, rst.data(), nr, &row, &pos, &lastp);
            return lastp ? last(row) : srt[row_off[ne[row]] + pos];
        };
        for (int j = 0; j < C; ++j) {
            hnext[at(j)] = at(j + 1 == C ? 0 : j + 1);
            hprev[at(j)] = at(j == 0 ? C - 1 : j - 1);
        }
    }
    long long squares = 0, evals = 0;
    const int R0 = star_r0(box, n);
    std::vector<int32_t> tri, ccw(STAR_NB), cw(STAR_NB);
    std::vector<std::pair<int32_t, uint32_t>> win;
    for (int p = 0; p < n; ++p) {
        const uint32_t pp = pxy[p];
        if (pp == PXY_NONE) continue;
        const int32_t x0 = px_of(pp), y0 = py_of(pp);
        auto covers = [&](int Rs) {
            return x0 - Rs <= box[0] && x0 + Rs >= box[2] && y0 - Rs <= box[1] && y0 + Rs >= box[3];
        };
        // the points of the square of half-size Rs around p that are not in the one of half-size hole
        auto each_in = [&](int Rs, int hole, auto&& take) {
            for (int r : ne) {
                const int dy = std::abs(py[row_off[r]] - y0);
                if (dy > Rs) continue;
                for (int j = row_off[r]; j < row_off[r] + rcnt[r]; ++j) {
                    const int dx = std::abs(px_of(sxy[j]) - x0);
                    if (dx <= Rs && (dx > hole || dy > hole)) {
                        ++evals;
                        take(srt[j], sxy[j]);
                    }
                }
            }
        };
        // the window, which grows for the point's later searches
        win.clear();
        int Rw = R0;
        each_in(Rw, -1, [&](int32_t s2, uint32_t sx) { win.push_back({s2, sx}); });
        auto grow = [&](auto&& take) {
            ++squares;
            each_in(2 * Rw, Rw, [&](int32_t s2, uint32_t sx) {
                take(s2, sx);
                win.push_back({s2, sx});
            });
            Rw *= 2;
        };
        auto nearest = [&]() -> int {
            unsigned long long best = ~0ull;
            auto take = [&](int s2, uint32_t sx) {
                if (s2 == p) return;
                const int32_t dx = dx_p(sx, pp), dy = dy_p(sx, pp);
                best = std::min<unsigned long long>(best, uint64_t(uint32_t(dx * dx + dy * dy)) << 32 | uint32_t(s2));
            };
            for (auto& c : win) take(c.first, c.second);
            for (;; grow(take)) {
                if (best != ~0ull && (best >> 32) <= uint64_t(Rw) * uint64_t(Rw)) return int(uint32_t(best));
                if (covers(Rw)) return best == ~0ull ? -1 : int(uint32_t(best));
            }
        };
        auto next = [&](int q, int side) -> int {
            const uint32_t pq = pxy[q];
            int bi = -1;
            uint32_t bxy = 0;
            auto take = [&](int s2, uint32_t sx) {
                if (!star_side(pp, pq, sx, side)) return;
                if (bi < 0 || star_better(p, pp, q, pq, bi, bxy, s2, sx, side)) {
                    bi = s2;
                    bxy = sx;
                }
            };
            for (auto& c : win) take(c.first, c.second);
            for (;; grow(take))
                if ((bi >= 0 && circle_inside(pp, pq, bxy, Rw, box)) || covers(Rw)) return bi;
        };
        int m = 0, k = 0;
        bool closed = false;
        if (!star_walk(hnext[p], hprev[p], nearest, next, ccw.data(), cw.data(), STAR_NB, &m, &k, &closed))
            return -1;
        const int deg = m + k, nt = star_tris(deg, closed);
        for (int i = 0; i < nt; ++i) {
            const int a = star_at(ccw.data(), m, cw.data(), k, i);
            const int b = star_at(ccw.data(), m, cw.data(), k, i + 1 == deg ? 0 : i + 1);
            if (p < a && p < b) {
                tri.push_back(p);
                tri.push_back(a);
                tri.push_back(b);
            }
        }
    }
    const int T = int(tri.size() / 3);
    if (T <= cap) std::memcpy(tris_out, tri.data(), sizeof(int32_t) * tri.size());
    if (stats) { stats[0] = 0; stats[1] = squares; stats[2] = evals; }
    return T;
}

// hull_chain (the stack walk) and hull_on_chain (the test that the device
// makes in two levels, rows of a group and then what they leave) on one chain: returns 1 if they keep the same points.
extern "C" int emu_hull_agree(const int32_t* xs, const int32_t* ys, int R, int side) {
    std::vector<uint32_t> xy(std::max(R, 1));
    for (int i = 0; i < R; ++i) xy[i] = pack_xy(xs[i], ys[i]);
    std::vector<int32_t> st(std::max(R, 1));
    int n = 0;
    hull_chain(side, R, xy.data(), st.data(), &n);
    std::vector<char> keep(std::max(R, 1), 0);
    for (int j = 0; j < n; ++j) keep[st[j]] = 1;
    for (int i = 0; i < R; ++i)
        if (bool(keep[i]) != hull_on_chain(side, R, xy.data(), i)) return 0;
    return 1;
}

// The flip predicates on packed coordinates, for checks against exact
// integer arithmetic.  xy: (x, y) of a, b, c[, d].
extern "C" long long emu_orient_p(const int32_t* xy) {
    return orient_p(pack_xy(xy[0], xy[1]), pack_xy(xy[2], xy[3]), pack_xy(xy[4], xy[5]));
}
extern "C" long long emu_incircle_p(const int32_t* xy) {
    return incircle_p(pack_xy(xy[0], xy[1]), pack_xy(xy[2], xy[3]), pack_xy(xy[4], xy[5]), pack_xy(xy[6], xy[7]));
}

// star_better and star_better_left on one edge p->q and two points a, b
// (xy: x, y of p, q, a, b; id: their indices): -1 where a or b is not
// strictly left of the edge, else whether the two agree.
extern "C" int emu_star_better_agree(const int32_t* xy, const int32_t* id) {
    uint32_t c[4];
    for (int k = 0; k < 4; ++k) c[k] = pack_xy(xy[2 * k], xy[2 * k + 1]);
    if (!star_side(c[0], c[1], c[2], 1) || !star_side(c[0], c[1], c[3], 1)) return -1;
    return star_better(id[0], c[0], id[1], c[1], id[2], c[2], id[3], c[3], 1) ==
           star_better_left(id[0], c[0], id[1], c[1], id[2], c[2], id[3], c[3]);
}
