// The common 3D cells of the device remesher, eight threads a cell: voronoi_cell.h's build_cell_dual over the first
// search shell in two kernels, the same operations in the same order a value, so a cell has the bits that one thread
// gives it. A cell that they do not finish (it reaches past the shell, outgrows the storage below or is degenerate) goes on
// a list for the one-thread kernel, which builds it from the start or says why it cannot.
//
//   k_search  a warp a cell: the offsets of the shell over the lanes, the images found ranked by (distance, index, offset),
//             each as the bisector plane the clip needs;
//   k_clip    eight lanes a cell, the cell in shared memory: the candidates' planes against eight vertices at a time, a
//             cut's survivors, edges and new vertices over the lanes, then a face a lane.
//
// One thread a cell keeps 5 KB of it in local memory, which 1,024 threads an SM spill through L2 to HBM, and waits for
// it; here a cell is 2.7 KB of shared memory and the lanes share the long steps (a vertex: 9 products of three, three
// divisions). The four cells of a warp go from cut to cut together: every loop's trip count is the warp's, so all its votes
// and shuffles are over the full warp.
#pragma once

#include <cuda_runtime.h>

#include "voronoi_cell.h"
#include "voronoi_grid.h"

namespace luna_voronoi {

constexpr int kLanes = 8;         // threads a cell in k_clip
constexpr int kFound = 96;        // images a search holds (a lattice cell's first ball has 39); a denser ball is searched
                                  // again at 0.6 of its radius squared
constexpr int kKept = 48;         // the nearest of them, kept for the clip (a lattice cell asks for 25)
constexpr int kLanePlanes = 34;   // planes of a cell, the box's six among them (a lattice cell: 22)
constexpr int kLaneVerts = 48;    // vertices of a cell (a lattice cell: 28)
constexpr int kLaneDrop = 20;     // vertices that one cut drops
constexpr int kLaneFaces = kLanePlanes - 6;
constexpr int kSearchWarps = 4;   // cells of a block in k_search
constexpr int kClipThreads = 64;
static_assert(kLaneVerts <= 64 && kLaneVerts % kLanes == 0 && kLanePlanes <= 64 && 3 * kLaneVerts < 256, "masks and bytes of k_clip");

// The sorted candidates of a chunk of cells.
struct Shell {
    double4* plane;  // [cells][kKept]: unit normal towards the image, distance of the bisector
    double* d2;      // [cells][kKept]: squared distance of the image
    int32_t* j;      // [cells][kKept]: the generator
    int32_t* n;      // [cells]: candidates kept, -1: more in the smallest ball tried than a search holds
    double* cover;   // [cells]: every image within this squared distance is among them (0 if some were left out)
};

constexpr int kSpan = 2 * GridShape::kReach + 1;  // bucket offsets an axis

// Of a cell's search, by axis and offset: the squared distance to the bucket's slab (bucket_reaches' near), the bucket's
// part of the flat index, its images' shift.
struct SearchBlock {
    double near2[kSearchWarps][3][kSpan], shift[kSearchWarps][3][kSpan];
    int part[kSearchWarps][3][kSpan];
    double d[kSearchWarps][3][kFound], d2[kSearchWarps][kFound];
    int32_t j[kSearchWarps][kFound], at[kSearchWarps][kFound];
    int n[kSearchWarps];
};

// Bound by the instructions of the bucket tests (179 offsets a cell) and of the ranking (every image against every other).
__global__ void __launch_bounds__(32 * kSearchWarps) k_search(int64_t base, int64_t cells, const double* __restrict__ pos, const double3 box,
                                                               Grid g, Shell out) {
    __shared__ SearchBlock sh;
    const int w = threadIdx.x / 32, lane = threadIdx.x % 32;
    const int64_t s = static_cast<int64_t>(blockIdx.x) * kSearchWarps + w;
    if (s >= cells) return;
    const double* xi = pos + 3 * (base + s);
    const double x[3] = {xi[0], xi[1], xi[2]};
    int bi[3];
    double wmax = 0, wmin = 1e300;
    for (int a = 0; a < 3; ++a) {
        bi[a] = bucket_of(g, x, a);
        wmax = g.w[a] > wmax ? g.w[a] : wmax;
        wmin = g.w[a] < wmin ? g.w[a] : wmin;
    }
    const double reach = static_cast<double>(g.reach - 1) * wmin;
    double hi2 = 4.41 * wmax * wmax;
    hi2 = hi2 < reach * reach ? hi2 : reach * reach;
    for (int t = lane; t < 3 * kSpan; t += 32) {
        const int a = t / kSpan, o = t % kSpan - GridShape::kReach;
        const double wa = a == 0 ? g.w[0] : a == 1 ? g.w[1] : g.w[2], xa = a == 0 ? x[0] : a == 1 ? x[1] : x[2];
        const double lo = static_cast<double>((a == 0 ? bi[0] : a == 1 ? bi[1] : bi[2]) + o) * wa - xa, hi = lo + wa, margin = 1e-6 * wa;
        double near = lo > 0 ? lo - margin : hi < 0 ? -hi - margin : 0;
        near = near > 0 ? near : 0;
        const int nb = a == 0 ? g.nb[0] : a == 1 ? g.nb[1] : g.nb[2];
        int c = (a == 0 ? bi[0] : a == 1 ? bi[1] : bi[2]) + o, wraps = 0;
        for (; c < 0; c += nb) --wraps;
        for (; c >= nb; c -= nb) ++wraps;
        sh.near2[w][a][o + GridShape::kReach] = near * near;
        sh.shift[w][a][o + GridShape::kReach] = static_cast<double>(wraps) * (a == 0 ? box.x : a == 1 ? box.y : box.z);
        sh.part[w][a][o + GridShape::kReach] = a == 0 ? c * g.nb[1] * g.nb[2] : a == 1 ? c * g.nb[2] : c;
    }
    int m = 0;
    for (int attempt = 0;; ++attempt) {
        if (lane == 0) sh.n[w] = 0;
        __syncwarp();
        for (int k0 = 0; k0 < g.n_offsets && g.bound2[k0] <= hi2; k0 += 32) {
            const int k = k0 + lane;
            if (k >= g.n_offsets || g.bound2[k] > hi2) continue;
            int o[3];
            for (int a = 0; a < 3; ++a) o[a] = g.offsets[3 * k + a] + GridShape::kReach;
            if (!(sh.near2[w][0][o[0]] + sh.near2[w][1][o[1]] + sh.near2[w][2][o[2]] <= hi2)) continue;
            const int b = sh.part[w][0][o[0]] + sh.part[w][1][o[1]] + sh.part[w][2][o[2]];
            const double shift[3] = {sh.shift[w][0][o[0]], sh.shift[w][1][o[1]], sh.shift[w][2][o[2]]};
            const int64_t end = g.start[b + 1];
            for (int64_t q = g.start[b]; q < end; ++q) {
                const int32_t j = g.items[q];
                double d[3], d2 = 0;
                for (int a = 0; a < 3; ++a) {
                    d[a] = pos[3 * static_cast<int64_t>(j) + a] + shift[a] - x[a];
                    d2 += d[a] * d[a];
                }
                if (!(d2 > 0 && d2 <= hi2)) continue;
                const int e = atomicAdd(&sh.n[w], 1);
                if (e >= kFound) break;
                for (int a = 0; a < 3; ++a) sh.d[w][a][e] = d[a];
                sh.d2[w][e] = d2;
                sh.j[w][e] = j;
                sh.at[w][e] = k;
            }
        }
        __syncwarp();
        m = sh.n[w];
        if (m <= kFound || attempt == 4) break;
        hi2 *= 0.6;
        __syncwarp();
    }
    if (m > kFound) {
        if (lane == 0) out.n[s] = -1;
        return;
    }
    const int64_t row = s * kKept;
    for (int e0 = lane; e0 < m; e0 += 64) {  // two images a lane against all
        const double lower = sh.d2[w][e0], upper = e0 + 32 < m ? sh.d2[w][e0 + 32] : 0;
        int less[2] = {0, 0}, equal[2] = {0, 0};
        for (int f = 0; f < m; ++f) {
            const double d2f = sh.d2[w][f];
            less[0] += d2f < lower;
            equal[0] += d2f == lower;
            less[1] += d2f < upper;
            equal[1] += d2f == upper;
        }
#pragma unroll 1
        for (int e = e0; e < m && e <= e0 + 32; e += 32) {
            const double d2 = e == e0 ? lower : upper;
            const int32_t j = sh.j[w][e];
            int rank = e == e0 ? less[0] : less[1];
            if ((e == e0 ? equal[0] : equal[1]) > 1)
                for (int f = 0; f < m; ++f)
                    rank += sh.d2[w][f] == d2 && (sh.j[w][f] < j || (sh.j[w][f] == j && sh.at[w][f] < sh.at[w][e]));
            if (rank >= kKept) continue;
            const double inv = 1.0 / sqrt(d2);
            out.plane[row + rank] = make_double4(sh.d[w][0][e] * inv, sh.d[w][1][e] * inv, sh.d[w][2][e] * inv, 0.5 * d2 * inv);
            out.d2[row + rank] = d2;
            out.j[row + rank] = j;
        }
    }
    if (lane == 0) {
        out.n[s] = m < kKept ? m : kKept;
        out.cover[s] = m <= kKept ? hi2 : 0.0;
    }
}

// A cell of k_clip. An odd number of 64-B pieces, so that two of a half-warp's cells are 16 banks apart.
struct LaneCell {
    double pn[kLanePlanes][4];   // planes n.x <= c
    double tv[3][kLaneVerts];    // vertices
    uint32_t tri[kLaneVerts];    // each vertex's three planes, a byte each, in its cyclic order, and its age (a cut's
                                 // vertices are numbered on); after the walk the faces' neighbours
    uint8_t from[kLanePlanes];   // the plane's candidate
    union {
        struct {
            uint16_t ek[3 * kLaneDrop];  // the dropped vertices' edges by age
            union {
                uint32_t tri[kLaneDrop];     // the dropped vertices' planes
                uint16_t eb[3 * kLaneDrop];  // the boundary's edges
            };
            uint8_t slot[kLaneDrop];  // the dropped vertices' slots
        } cut;
        struct {
            uint8_t loop[3 * kLaneVerts];  // the faces' vertices in order
            uint8_t plane[kLaneFaces], first[kLaneFaces], size[kLaneFaces], rank[kLaneFaces];
        } faces;
    } u;
};
constexpr int kLaneCellBytes = (sizeof(LaneCell) + 63) / 64 * 64;
constexpr int kLaneCellStride = kLaneCellBytes / 64 % 2 ? kLaneCellBytes : kLaneCellBytes + 64;

struct LaneOut {
    double* volume;
    double* centroid;
    int64_t* first;
    int32_t* count;
    int32_t* fj;
    double* fa;
    double* fc;
    unsigned long long capacity;
    unsigned long long* faces;  // the cursor of the face records
    int32_t* left;              // the cells left for the one-thread kernel, and how many
    unsigned int* n_left;
};

__device__ __forceinline__ double group_max(double r) {
    for (int o = 1; o < kLanes; o <<= 1) {
        const double x = __shfl_xor_sync(0xffffffffu, r, o);
        r = x > r ? x : r;
    }
    return r;
}

// Bound by instruction issue and the latency of the serial steps (a cut waits for the test before it): 20 warps an SM by
// shared memory and registers, 0.60 of the issue slots, 7,470 warp instructions a cell, 0.24 GB of DRAM traffic for 131,072
// cells (one thread a cell: 6,730, 0.25 and 7.6 GB). Cells of the 128^3 jittered mesh: 28.4 ms with the search's 5.4,
// against 47 with a thread a cell; 64^3 3.6 against 6.4. Moving a cut's survivors down in order (31.4 ms) in place of
// numbering the vertices by age cost 8 ms with the code it needed, a third of the warps' time waiting for instructions:
// the loops that hold a division are kept rolled.
__global__ void __launch_bounds__(kClipThreads, 10) k_clip(int64_t base, int64_t cells, const double3 box, Shell in, LaneOut out) {
    constexpr unsigned full = 0xffffffffu;
    __shared__ __align__(64) unsigned char shared[kClipThreads / kLanes * kLaneCellStride];
    LaneCell& S = *reinterpret_cast<LaneCell*>(shared + threadIdx.x / kLanes * kLaneCellStride);
    const int l = threadIdx.x % kLanes, shift = threadIdx.x % 32 / kLanes * kLanes;
    const int64_t s = (static_cast<int64_t>(blockIdx.x) * kClipThreads + threadIdx.x) / kLanes, i = base + s, row = s * kKept;
    const bool mine = s < cells;
    const int n = mine ? in.n[s] : -1;
    const double cover = n >= 0 ? in.cover[s] : 0;
    const auto votes = [&](bool x) { return __ballot_sync(full, x) >> shift & 0xffu; };  // of the cell's lanes
    const auto rounds = [&](int x) { return (__reduce_max_sync(full, x) + kLanes - 1) / kLanes; };

    // the starting box: plane a's low side 2 a, its high side 2 a + 1; vertex l at the corner of l's bits
    const double side[3] = {box.x, box.y, box.z};
    double scale = 0;
    for (int a = 0; a < 3; ++a) scale = side[a] > scale ? side[a] : scale;
    const double eps = 1e-13 * scale;
    if (l < 6) {
        for (int a = 0; a < 3; ++a) S.pn[l][a] = a == l / 2 ? ((l & 1) ? 1.0 : -1.0) : 0.0;
        S.pn[l][3] = 0.5 * side[l / 2];
    }
    __syncwarp();
    const auto vertex = [&](int t, const double* a, const double* b, const double* c) {  // DualT::vertex; its squared radius
        double bc[3], ca[3], ab[3], v[3];
        cross3(b, c, bc);
        cross3(c, a, ca);
        cross3(a, b, ab);
        const double det = dot3(a, bc);
        for (int k = 0; k < 3; ++k) {
            v[k] = (a[3] * bc[k] + b[3] * ca[k] + c[3] * ab[k]) / det;
            S.tv[k][t] = v[k];
        }
        return dot3(v, v);
    };
    double rmax2 = 0;
    {
        const bool high[3] = {(l & 4) != 0, (l & 2) != 0, (l & 1) != 0};
        const int p0 = high[0], p1 = 2 + high[1], p2 = 4 + high[2];
        const bool odd = (high[0] + high[1] + high[2]) % 2 == 0;  // an odd number of low sides: the other way round
        S.tri[l] = static_cast<uint32_t>(p0 | (odd ? p2 : p1) << 8 | (odd ? p1 : p2) << 16 | l << 24);
        double v[3];
        for (int a = 0; a < 3; ++a) S.tv[a][l] = v[a] = high[a] ? 0.5 * side[a] : -(0.5 * side[a]);
        rmax2 = group_max(dot3(v, v));
    }
    __syncwarp();

    int nt = 8, np = 6, born = 8, k = 0;
    bool active = n >= 0, closed = false;
    double next[4] = {0, 0, 0, 0}, next_d2 = 0;
    const auto fetch = [&]() {
        if (k < n) {
            const double4 p = in.plane[row + k];
            next[0] = p.x;
            next[1] = p.y;
            next[2] = p.z;
            next[3] = p.w;
            next_d2 = in.d2[row + k];
        }
    };
    fetch();
    while (__any_sync(full, active)) {
        // each cell to its next cut
        bool look = active, hit = false;
        double plane[4] = {0, 0, 0, 0};
        uint64_t out_mask = 0;
        while (__any_sync(full, look)) {
            if (look && (k >= n || next_d2 > 4.0 * rmax2)) {  // past twice the reach, or no candidate left
                closed = k < n || 4.0 * rmax2 <= cover;
                look = active = false;
            }
            if (look) {
                for (int a = 0; a < 4; ++a) plane[a] = next[a];
                ++k;
                fetch();
            }
            uint64_t mask = 0;
            const int R = rounds(look ? nt : 0);
#pragma unroll 1
            for (int r = 0; r < R; ++r) {
                const int t = l + kLanes * r;
                bool o = false;
                if (look && t < nt) {
                    const double v[3] = {S.tv[0][t], S.tv[1][t], S.tv[2][t]};
                    o = dot3(plane, v) - plane[3] > eps;
                }
                mask |= static_cast<uint64_t>(votes(o)) << (kLanes * r);
            }
            if (look && mask) {
                hit = true;
                look = false;
                out_mask = mask;
            }
        }
        if (!__any_sync(full, hit)) continue;
        // the cut
        const int nd = __popcll(out_mask);
        if (hit && (np >= kLanePlanes || nd > kLaneDrop)) hit = active = false;
        const int q = np, ne = hit ? 3 * nd : 0;
        if (hit) {
            if (l < 4) S.pn[q][l] = plane[l];
            if (l == 4) S.from[q] = static_cast<uint8_t>(k - 1);
            ++np;
        }
        double r2 = 0;
        for (int t = l; hit && t < nt; t += kLanes) {
            if (out_mask >> t & 1) {
                const int x = __popcll(out_mask & ((1ull << t) - 1));
                S.u.cut.tri[x] = S.tri[t];
                S.u.cut.slot[x] = static_cast<uint8_t>(t);
            } else {
                const double v[3] = {S.tv[0][t], S.tv[1][t], S.tv[2][t]}, d = dot3(v, v);
                r2 = d > r2 ? d : r2;
            }
        }
        __syncwarp();
#pragma unroll 1
        for (int x = l; x < nd && hit; x += kLanes) {
            const uint32_t tr = S.u.cut.tri[x], a = tr & 0xff, b = tr >> 8 & 0xff, c = tr >> 16 & 0xff;
            int e = 0;
            for (int y = 0; y < nd; ++y) e += 3 * (S.u.cut.tri[y] >> 24 < tr >> 24);
            S.u.cut.ek[e] = static_cast<uint16_t>(a << 8 | b);
            S.u.cut.ek[e + 1] = static_cast<uint16_t>(b << 8 | c);
            S.u.cut.ek[e + 2] = static_cast<uint16_t>(c << 8 | a);
        }
        __syncwarp();
        int nb = 0;  // the boundary edges, in order
        const int RE = rounds(ne);
#pragma unroll 1
        for (int r = 0; r < RE; ++r) {
            const int e = l + kLanes * r;
            bool boundary = false;
            uint16_t x = 0;
            if (e < ne) {
                x = S.u.cut.ek[e];
                const uint16_t rev = static_cast<uint16_t>((x & 0xff) << 8 | x >> 8);
                boundary = true;
                for (int f = 0; f < ne; f += 3) boundary = boundary && S.u.cut.ek[f] != rev && S.u.cut.ek[f + 1] != rev && S.u.cut.ek[f + 2] != rev;
            }
            const unsigned b = votes(boundary);
            if (boundary) S.u.cut.eb[nb + __popc(b & ((1u << l) - 1))] = x;
            nb += __popc(b);
        }
        // the new vertices: in the dropped ones' slots, then at the end; slots left over are filled from the end
        const int end = nt - nd + nb;
        if (hit && (end > kLaneVerts || born + nb > 256)) hit = active = false;
        __syncwarp();
#pragma unroll 1
        for (int e = l; hit && e < nb; e += kLanes) {
            const int a = S.u.cut.eb[e] >> 8, b = S.u.cut.eb[e] & 0xff, t = e < nd ? S.u.cut.slot[e] : nt + e - nd;
            S.tri[t] = static_cast<uint32_t>(a | b << 8 | q << 16) | static_cast<uint32_t>(born + e) << 24;
            const double d = vertex(t, S.pn[a], S.pn[b], plane);
            r2 = d > r2 ? d : r2;
        }
        if (hit && nb < nd) {
            const uint64_t from = ~out_mask & ((1ull << nt) - 1) >> end << end;  // as many as slots left over below end
            for (int x = nb + l; x < nd; x += kLanes) {
                const int t = S.u.cut.slot[x];
                if (t >= end) break;
                uint64_t u = from;
                for (int y = nb; y < x; ++y) u &= u - 1;
                const int v = __ffsll(static_cast<long long>(u)) - 1;
                for (int a = 0; a < 3; ++a) S.tv[a][t] = S.tv[a][v];
                S.tri[t] = S.tri[v];
            }
        }
        __syncwarp();
        r2 = group_max(r2);
        if (hit) {
            rmax2 = r2;
            nt = end;
            born += nb;
        }
    }

    // The faces: one per plane still holding vertices, in plane order.
    bool ok = closed;
    uint64_t alive = 0;
    for (int t = l; ok && t < nt; t += kLanes) {
        const uint32_t tr = S.tri[t];
        alive |= 1ull << (tr & 0xff) | 1ull << (tr >> 8 & 0xff) | 1ull << (tr >> 16 & 0xff);
    }
    for (int o = 1; o < kLanes; o <<= 1) alive |= __shfl_xor_sync(full, alive, o);
    if (alive & 0x3f) ok = false;  // the box
    const int nf = ok ? __popcll(alive) : 0;
    const int RF = rounds(nf);
    int at = 0;
    bool bad = false;
#pragma unroll 1
    for (int r = 0; r < RF; ++r) {  // each face's vertices in order, from its oldest
                                     // (DualT::finish: from its lowest, in an order that a cut keeps by age)
        const int f = l + kLanes * r;
        int p = 0, m = 0, t0 = 0;
        uint64_t has = 0;
        if (f < nf) {
            uint64_t a = alive;
#pragma unroll 1
            for (int e = 0; e < f; ++e) a &= a - 1;
            p = __ffsll(static_cast<long long>(a)) - 1;
            uint32_t oldest = 256;
            for (int t = 0; t < nt; ++t) {
                const uint32_t tr = S.tri[t], x = tr ^ static_cast<uint32_t>(p) * 0x010101u;
                if ((x - 0x010101u) & ~x & 0x808080u) {  // one of its three bytes is p
                    has |= 1ull << t;
                    if (tr >> 24 < oldest) {
                        oldest = tr >> 24;
                        t0 = t;
                    }
                }
            }
            m = __popcll(has);
        }
        int first = m;  // an exclusive sum over the cell's lanes
        for (int o = 1; o < kLanes; o <<= 1) {
            const int x = __shfl_up_sync(full, first, o, kLanes);
            if (l >= o) first += x;
        }
        const int total = __shfl_sync(full, first, kLanes - 1, kLanes);
        first += at - m;
        at += total;
        if (f < nf) {
            S.u.faces.plane[f] = static_cast<uint8_t>(p);
            S.u.faces.first[f] = static_cast<uint8_t>(first);
            S.u.faces.size[f] = static_cast<uint8_t>(m);
            bad = bad || m < 3;
            const uint32_t tr0 = S.tri[t0];
            uint32_t b = (tr0 & 0xff) == p ? tr0 >> 16 & 0xff : (tr0 >> 8 & 0xff) == p ? tr0 & 0xff : tr0 >> 8 & 0xff;
            S.u.faces.loop[first] = static_cast<uint8_t>(t0);
#pragma unroll 1
            for (int e = 1; e <= m; ++e) {  // the vertex with p followed by b
                int next_t = -1;
                uint32_t next_b = 0;
#pragma unroll 1
                for (uint64_t c = has; c && next_t < 0; c &= c - 1) {
                    const int t = __ffsll(static_cast<long long>(c)) - 1;
                    const uint32_t tr = S.tri[t], x = tr & 0xff, y = tr >> 8 & 0xff, z = tr >> 16 & 0xff;
                    if (x == p && y == b) {
                        next_t = t;
                        next_b = z;
                    } else if (y == p && z == b) {
                        next_t = t;
                        next_b = x;
                    } else if (z == p && x == b) {
                        next_t = t;
                        next_b = y;
                    }
                }
                if (next_t < 0 || (next_t == t0) != (e == m)) {  // a walk that is not once around
                    bad = true;
                    break;
                }
                if (e < m) S.u.faces.loop[first + e] = static_cast<uint8_t>(next_t);
                b = next_b;
            }
        }
    }
    __syncwarp();  // (the walk has read S.tri)
    for (int f = l; f < nf; f += kLanes) S.tri[f] = static_cast<uint32_t>(in.j[row + S.from[S.u.faces.plane[f]]]);
    __syncwarp();
    for (int f = l; f < nf; f += kLanes) {
        const int32_t j = static_cast<int32_t>(S.tri[f]);
        bad = bad || j == i;
        int rank = 0;
        for (int e = 0; e < nf; ++e) {
            const int32_t x = static_cast<int32_t>(S.tri[e]);
            rank += x < j;
            bad = bad || (x == j && e != f);
        }
        S.u.faces.rank[f] = static_cast<uint8_t>(rank);
    }
    if (votes(bad)) ok = false;
    __syncwarp();
    // the records of the warp's cells
    const int records = ok ? nf : 0;
    int before = 0, all = 0;
    for (int c = 0; c < 32 / kLanes; ++c) {
        const int x = __shfl_sync(full, records, c * kLanes);
        if (c * kLanes < shift) before += x;
        all += x;
    }
    unsigned long long cursor = 0;
    if (threadIdx.x % 32 == 0 && all > 0) cursor = atomicAdd(out.faces, static_cast<unsigned long long>(all));
    cursor = __shfl_sync(full, cursor, 0) + before;
    const bool room = ok && cursor + nf <= out.capacity;  // (the host grows the buffer and runs the cells again)
    const int RO = rounds(records);
#pragma unroll 1
    for (int r = 0; r < RO; ++r) {  // cell_faces3's area and centroid
        const int f = l + kLanes * r;
        if (ok && f < nf) {
            uint8_t* loop = S.u.faces.loop + S.u.faces.first[f];
            const int m = S.u.faces.size[f], p = S.u.faces.plane[f];
            const auto load = [&](int e, double* v) {
                const int t = loop[e];
                for (int a = 0; a < 3; ++a) v[a] = S.tv[a][t];
            };
            double p0[3], A[3];
            load(0, p0);
#pragma unroll 1
            for (int turn = 0; turn < 2; ++turn) {
                double p1[3], p2[3];
                load(1, p1);
                for (int a = 0; a < 3; ++a) A[a] = 0;
#pragma unroll 1
                for (int e = 1; e + 1 < m; ++e) {
                    load(e + 1, p2);
                    const double e1[3] = {p1[0] - p0[0], p1[1] - p0[1], p1[2] - p0[2]};
                    const double e2[3] = {p2[0] - p0[0], p2[1] - p0[1], p2[2] - p0[2]};
                    double t[3];
                    cross3(e1, e2, t);
                    for (int a = 0; a < 3; ++a) A[a] += 0.5 * t[a];
                    for (int a = 0; a < 3; ++a) p1[a] = p2[a];
                }
                if (turn == 1 || !(dot3(A, S.pn[p]) < 0)) break;
#pragma unroll 1
                for (int x = 1, y = m - 1; x < y; ++x, --y) {  // the other way round
                    const uint8_t sw = loop[x];
                    loop[x] = loop[y];
                    loop[y] = sw;
                }
            }
            const double amag = sqrt(dot3(A, A));
            double C[3] = {0, 0, 0}, wsum = 0;
            double p1[3], p2[3];
            load(1, p1);
#pragma unroll 1
            for (int e = 1; e + 1 < m; ++e) {
                load(e + 1, p2);
                const double e1[3] = {p1[0] - p0[0], p1[1] - p0[1], p1[2] - p0[2]};
                const double e2[3] = {p2[0] - p0[0], p2[1] - p0[1], p2[2] - p0[2]};
                double t[3];
                cross3(e1, e2, t);
                const double wgt = amag > 0 ? dot3(t, A) / amag : 0.0;
                for (int a = 0; a < 3; ++a) C[a] += wgt * ((p0[a] + p1[a] + p2[a]) / 3.0);
                wsum += wgt;
                for (int a = 0; a < 3; ++a) p1[a] = p2[a];
            }
            if (wsum > 0)
                for (int a = 0; a < 3; ++a) C[a] /= wsum;
            else
                for (int a = 0; a < 3; ++a) C[a] = p0[a];
            if (room) {
                const unsigned long long rec = cursor + S.u.faces.rank[f];
                out.fj[rec] = static_cast<int32_t>(S.tri[f]);
                for (int a = 0; a < 3; ++a) {
                    out.fa[3 * rec + a] = A[a];
                    out.fc[3 * rec + a] = C[a];
                }
            }
        }
    }
    // cell_faces3's volume and first moment: a triangle a lane, the terms added in the faces' and triangles' order
    __syncwarp();
    struct Triangles {  // (in the planes' room: they are done with)
        uint16_t at[3 * kLaneVerts];  // the face's first vertex and the triangle's second, in u.faces.loop
        double term[kLanes][4];
    };
    static_assert(sizeof(Triangles) <= sizeof(S.pn), "Triangles");
    Triangles& tris = *reinterpret_cast<Triangles*>(S.pn);
    for (int f = l; ok && f < nf; f += kLanes) {
        const int first = S.u.faces.first[f], m = S.u.faces.size[f];
        for (int e = 1; e + 1 < m; ++e) tris.at[first - 2 * f + e - 1] = static_cast<uint16_t>(first << 8 | (first + e));
    }
    __syncwarp();
    const int n_tris = ok ? at - 2 * nf : 0;
    double sum = 0;  // of lane 0: the volume, of lanes 1 to 3: the moment
    const int RT = rounds(n_tris);
#pragma unroll 1
    for (int r = 0; r < RT; ++r) {
        const int t = l + kLanes * r;
        double term[4] = {0, 0, 0, 0};
        if (t < n_tris) {
            const int x = tris.at[t], c0 = S.u.faces.loop[x >> 8], c1 = S.u.faces.loop[x & 0xff], c2 = S.u.faces.loop[(x & 0xff) + 1];
            const double p0[3] = {S.tv[0][c0], S.tv[1][c0], S.tv[2][c0]}, p1[3] = {S.tv[0][c1], S.tv[1][c1], S.tv[2][c1]},
                         p2[3] = {S.tv[0][c2], S.tv[1][c2], S.tv[2][c2]};
            double x12[3];
            cross3(p1, p2, x12);
            const double v6 = dot3(p0, x12);
            term[0] = v6 / 6.0;
            for (int a = 0; a < 3; ++a) term[a + 1] = v6 / 6.0 * (p0[a] + p1[a] + p2[a]) / 4.0;
        }
        for (int a = 0; a < 4; ++a) tris.term[l][a] = term[a];
        __syncwarp();
        if (l < 4)
            for (int e = 0; e < kLanes; ++e) sum += tris.term[e][l];
        __syncwarp();
    }
    const double volume = __shfl_sync(full, sum, 0, kLanes);
    if (!mine) return;
    if (ok && l >= 1 && l < 4) out.centroid[3 * i + l - 1] = sum / volume;
    if (l != 0) return;
    out.first[i] = ok ? static_cast<int64_t>(cursor) : 0;
    out.count[i] = records;
    if (ok)
        out.volume[i] = volume;
    else
        out.left[atomicAdd(out.n_left, 1u)] = static_cast<int32_t>(i);
}

}  // namespace luna_voronoi
