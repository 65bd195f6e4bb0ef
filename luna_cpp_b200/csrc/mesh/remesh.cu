// The moving mesh's remesh on the device (include/luna_remesh.h).
//
// The cells are clipped with the host builder's operations in its order (voronoi_cell.h; this file is compiled with
// -fmad=false), so they have the host builder's bits. The rest is assembly in the host builder's order, done with scans and
// per-segment sorts instead of its serial passes:
//   buckets   counts (atomics), an exclusive scan, a fill (atomics), then each bucket's items sorted by index;
//   cells     (3D: cell_lanes.cuh, eight threads a cell; the cells it leaves, and 2D, one thread a cell) each cell's faces,
//             by neighbour, appended to one face buffer at an atomic cursor (a cell's faces stay together; where they
//             land does not matter, every later pass addresses them through the cell);
//   faces     per owner (the lower-numbered cell): its faces towards higher cells, numbered by a scan, and
//   lists     per cell, every face it is a side of (f, or ~f where it is not the owner), by neighbour: a cell's records as
//             they are (k_emit_lists). Where a higher cell sees a face that the lower one misses (degenerate vertices),
//             the general passes (assemble_general): such faces flipped into the owner's frame, a segment with them
//             re-sorted by neighbour, the lists filled and sorted.
#include <cuda_runtime.h>

#include <cub/device/device_scan.cuh>
#include <string>
#include <type_traits>

#include "luna_b200.h"
#include "luna_remesh.h"
#include "cell_lanes.cuh"
#include "voronoi_cell.h"
#include "voronoi_grid.h"

#ifndef LUNA_REMESH_DUAL
#define LUNA_REMESH_DUAL 1  // 3D cells kept as triangles of plane triples (DualT), as the host builder's default; 0: face
                            // loops (Poly3T), as the host builder with LUNA_MESH_DUAL=0
#endif

namespace luna {
luna_status report_error(luna_status s, const std::string& what);
}  // namespace luna

namespace {

using namespace luna_voronoi;

luna_status fail(luna_status s, const std::string& what) { return luna::report_error(s, what); }

#define RM_CUDA(call)                                                                                                 \
    do {                                                                                                              \
        cudaError_t e_ = (call);                                                                                      \
        if (e_ != cudaSuccess) return fail(LUNA_ECUDA, std::string(#call) + ": " + cudaGetErrorString(e_));          \
    } while (0)
#define RM_TRY(call)                     \
    do {                                 \
        luna_status s_ = (call);         \
        if (s_ != LUNA_OK) return s_;    \
    } while (0)

// A device buffer that only grows.
template <class T>
struct Buf {
    T* ptr = nullptr;
    size_t count = 0;
    Buf() = default;
    Buf(const Buf&) = delete;
    Buf& operator=(const Buf&) = delete;
    ~Buf() {
        if (ptr) cudaFree(ptr);
    }
    luna_status reserve(size_t n, const char* what) {
        if (n == 0) n = 1;
        if (ptr && n <= count) return LUNA_OK;
        if (ptr) cudaFree(ptr);
        ptr = nullptr;
        count = 0;
        const cudaError_t e = cudaMalloc(&ptr, n * sizeof(T));
        if (e != cudaSuccess) {
            ptr = nullptr;
            cudaGetLastError();
            return fail(e == cudaErrorMemoryAllocation ? LUNA_ENOMEM : LUNA_ECUDA,
                        std::string("cudaMalloc(") + what + "): " + cudaGetErrorString(e));
        }
        count = n;
        return LUNA_OK;
    }
    size_t bytes() const { return count * sizeof(T); }
};

struct Counters {
    unsigned long long faces;         // face records the cells appended
    unsigned long long inconsistent;  // faces seen from one side only
    int error;                        // the first cell error (voronoi_cell.h), 0: none
    int error_cell;
    int nonfinite;                    // a generator coordinate was not finite
    unsigned int left;                // cells that the eight-lane kernels left for one thread
    unsigned int boxes, close;        // of the sampled generators: in a rectangular lattice; with a neighbour close by (k_sample)
    unsigned int retry;               // cells the fast path handed to the far search
};

struct Box {
    double s[3];
};

constexpr bool kEightLanes = LUNA_REMESH_DUAL;  // 3D cells by cell_lanes.cuh first
constexpr int64_t kChunk = 1 << 17;             // cells whose candidates are held at a time (277 MB)

// Which meshes past kSampleFrom cells have one thread a cell from the start (k_sample), all measured as whole builds in ms by
// one thread / by lanes:
// - a rectangular lattice: 48^3 0.71 / 0.88, 64^3 1.24 / 1.92 (32^3 0.46 / 0.36: hence the limit). One thread builds such a cell
//   of 6 planes and 26 candidates without touching most of its local memory, while the lanes' search and clip cost what
//   they always cost (with a tenth of the spacing as jitter: 48^3 3.4 / 1.7, 64^3 7.0 / 3.8);
// - points as irregular as random ones, of which the lanes leave half and more, while one thread a cell is one wave
//   (1,024 an SM): 65,000 points 6.95 / 7.19, 100,000 8.5 / 8.9, 131,072 9.7 / 10.3; past that 160,000 13.6 / 11.8, 262,144
//   18.5 / 16.1. What tells them is the share of generators with another within 0.4 of the mean spacing: 0.24 of random
//   points, more where the density varies, 0.22 of a lattice jittered by 0.7 (48^3 7.0 / 6.85) and 0.11 by 0.5 (5.7 / 5.1).
constexpr int64_t kSampleFrom = 64000, kOneWave = 148 * 1024;
constexpr int kSamples = 256, kLatticeSamples = 240, kIrregularSamples = 42;
// Few cells with a thread each are given more warps: 2^s threads a cell, of which one works, while the threads stay within
// this many (not half of what is resident). A warp of 32 hard cells walks each one's branches in turn; a warp of one walks one.
// Measured, a build of 512, 4,096, 16,384 and 32,768 random points, of a 20^3 lattice jittered by half its spacing and of
// 2^18 points with a gradient of density: 3.29, 3.66, 4.26, 5.39, 2.94 and 32.0 ms with all warps full, 1.38, 2.15, 4.12, 5.27,
// 1.30 and 24.7 with this limit; 1.37, 2.09, 3.93, 5.49, 1.29 and 24.9 with about twice as many, but then
// 7.9 for 65,536 random points by lanes (7.2 with full warps), 10 and 13 with four and eight times as many.
constexpr int64_t kSpreadThreads = 1 << 16;
int spread_of(int64_t cells) {
    int s = 0;
    while (s < 5 && cells << (s + 1) <= kSpreadThreads) ++s;
    return s;
}

int grid_blocks(int64_t n, int per) { return static_cast<int>((n + per - 1) / per); }

template <int D>
__global__ void k_wrap(int64_t n, const double* __restrict__ in, double* __restrict__ pos, Box box, Counters* c) {
    const int64_t k = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
    if (k >= n * D) return;
    double x = in[k];
    if (!isfinite(x)) {
        atomicOr(&c->nonfinite, 1);
        x = 0;
    }
    pos[k] = wrap_coordinate(x, box.s[k % D]);
}

template <int D>
__global__ void k_bucket_count(int64_t n, const double* __restrict__ pos, Grid g, int64_t* __restrict__ bucket,
                               unsigned long long* __restrict__ count) {
    const int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
    if (i >= n) return;
    int64_t b = 0;
    for (int a = 0; a < D; ++a) b = b * g.nb[a] + bucket_of(g, pos + D * i, a);
    bucket[i] = b;
    atomicAdd(count + b, 1ull);
}

__global__ void k_bucket_fill(int64_t n, const int64_t* __restrict__ bucket, const int64_t* __restrict__ start,
                              unsigned int* __restrict__ cursor, int32_t* __restrict__ items) {
    const int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
    if (i >= n) return;
    const int64_t b = bucket[i];
    items[start[b] + atomicAdd(cursor + b, 1u)] = static_cast<int32_t>(i);
}

// Each bucket's items by index, as the host fills them.
__global__ void k_bucket_sort(int64_t buckets, const int64_t* __restrict__ start, int32_t* __restrict__ items) {
    const int64_t b = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
    if (b >= buckets) return;
    const int64_t s0 = start[b], s1 = start[b + 1];
    for (int64_t k = s0 + 1; k < s1; ++k) {
        const int32_t x = items[k];
        int64_t j = k - 1;
        while (j >= s0 && items[j] > x) {
            items[j + 1] = items[j];
            --j;
        }
        items[j + 1] = x;
    }
}

struct CellOut {
    double* volume;       // [n]
    double* centroid;     // [n][D]
    int64_t* first;       // [n]: the cell's first record in the face buffer
    int32_t* count;       // [n]
    int32_t* fj;          // [capacity]: neighbour
    double* fa;           // [capacity][D]: area vector out of the cell
    double* fc;           // [capacity][D]: centroid relative to the cell's generator
    unsigned long long capacity;
};

// Counts, of kSamples generators spread over the mesh, those whose cell is the box between their six nearest images along
// the axes (no other image of the 5^3 buckets around them cuts the box's corners, by the clip's own tolerance), and those
// with another generator within 0.4 of the mean spacing. A block a generator, a thread a bucket: about 10 us, with its read.
__global__ void __launch_bounds__(128) k_sample(int64_t n, const double* __restrict__ pos, Box box, Grid g, Counters* c) {
    __shared__ unsigned long long nearest[7];  // of the images along each axis, on its low side and its high side; of all, squared
    constexpr unsigned long long kNone = 0x7fefffffffffffffull;
    const int64_t i = n * blockIdx.x / gridDim.x;
    const int o = static_cast<int>(threadIdx.x) < 125 ? static_cast<int>(threadIdx.x) : 62;  // (the last three: the middle again)
    const int off[3] = {o / 25 - 2, o / 5 % 5 - 2, o % 5 - 2};
    double x[3], shift[3], scale = 0, share = 1.0 / n;  // share: the volume of a generator
    int64_t b = 0;
    for (int a = 0; a < 3; ++a) {
        x[a] = pos[3 * i + a];
        share *= box.s[a];
        scale = box.s[a] > scale ? box.s[a] : scale;
        int t = bucket_of(g, pos + 3 * i, a) + off[a], wraps = 0;
        for (; t < 0; t += g.nb[a]) --wraps;
        for (; t >= g.nb[a]; t -= g.nb[a]) ++wraps;
        shift[a] = wraps * box.s[a];
        b = b * g.nb[a] + t;
    }
    const double eps = 1e-13 * scale;
    const int64_t q0 = g.start[b], q1 = g.start[b + 1];
    const auto image = [&](int64_t q, double* d) {
        double d2 = 0;
        for (int a = 0; a < 3; ++a) {
            d[a] = pos[3 * static_cast<int64_t>(g.items[q]) + a] + shift[a] - x[a];
            d2 += d[a] * d[a];
        }
        return d2;
    };
    if (threadIdx.x < 7) nearest[threadIdx.x] = kNone;
    __syncthreads();
    for (int64_t q = q0; q < q1; ++q) {
        double d[3];
        const double d2 = image(q, d);
        if (!(d2 > 0)) continue;
        atomicMin(&nearest[6], static_cast<unsigned long long>(__double_as_longlong(d2)));
        for (int a = 0; a < 3; ++a)
            if (fabs(d[(a + 1) % 3]) <= eps && fabs(d[(a + 2) % 3]) <= eps)
                atomicMin(&nearest[2 * a + (d[a] > 0)], static_cast<unsigned long long>(__double_as_longlong(fabs(d[a]))));
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        const double d2 = __longlong_as_double(static_cast<long long>(nearest[6]));
        if (d2 * sqrt(d2) < 0.4 * 0.4 * 0.4 * share) atomicAdd(&c->close, 1u);
    }
    bool cut = false;
    for (int f = 0; f < 6; ++f) cut = cut || nearest[f] == kNone;
    if (cut) return;  // (the whole block)
    for (int64_t q = q0; q < q1; ++q) {
        double d[3];
        const double d2 = image(q, d);
        double corner = 0;
        for (int a = 0; a < 3; ++a) corner += fabs(d[a]) * __longlong_as_double(static_cast<long long>(nearest[2 * a + (d[a] > 0)]));
        cut = cut || !(corner - d2 <= 2 * eps * sqrt(d2));
    }
    if (!__syncthreads_or(cut) && threadIdx.x == 0) atomicAdd(&c->boxes, 1u);
}

// The cells (all of them, or those of the list), each built by one thread, 2^spread threads a cell (spread_of): 2D cells, a
// lattice's, and the 3D cells that cell_lanes.cuh leaves (uniform random points: 54 to 65 % of them; a lattice jittered by
// 0.1: none). Without Far, a cell whose search would
// pass the grid's sorted offsets or fill the candidate store is put on the retry list for the Far pass (the same cell
// either way, voronoi_cell.h), which keeps the common cell's code small. 1,024 threads an SM (64 registers, a few
// spilled): 57.5 ms for the 128^3 jittered remesh against 62 ms at 80 registers, 58.6 ms at 896 threads and 58 ms at
// 1,280; in 64-thread blocks (16 an SM) about 1 % faster than in 128-thread blocks, and no faster with the L1 carveout
// preferred.
template <int D, bool Far>
__global__ void __launch_bounds__(64, 16) k_cells(int64_t n, int spread, const int32_t* __restrict__ list, const double* __restrict__ pos, Box box,
                                               Grid g, CellOut out, Counters* c, int32_t* __restrict__ retry) {
    const int64_t t = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x, k = t >> spread;
    if (k >= n || (t & ((1 << spread) - 1))) return;
    const int64_t i = list ? list[k] : k;
#if LUNA_REMESH_DUAL
    using Poly = std::conditional_t<D == 3, Dual, Poly2>;
#else
    using Poly = std::conditional_t<D == 3, Poly3, Poly2>;
#endif
    Poly poly;
    CellFaces faces;
    Candidates cand;
    double volume = 0, centroid[3] = {0, 0, 0};
#if LUNA_REMESH_DUAL
    int code;
    if constexpr (D == 3)
        code = build_cell_dual<Far>(i, pos, box.s, g, poly, faces, cand, volume, centroid);
    else
        code = build_cell<D, Far>(i, pos, box.s, g, poly, faces, cand, volume, centroid);
#else
    const int code = build_cell<D, Far>(i, pos, box.s, g, poly, faces, cand, volume, centroid);
#endif
    if (code != kCellOk) {
        out.first[i] = 0;
        out.count[i] = 0;
        if (!Far && (code == kOutOfOffsets || code == kCandidates))
            retry[atomicAdd(&c->retry, 1u)] = static_cast<int32_t>(i);
        else if (atomicCAS(&c->error, 0, code) == 0)
            c->error_cell = static_cast<int>(i);
        return;
    }
    out.volume[i] = volume;
    for (int a = 0; a < D; ++a) out.centroid[D * i + a] = centroid[a];
    const unsigned long long base = atomicAdd(&c->faces, static_cast<unsigned long long>(faces.n));
    out.first[i] = static_cast<int64_t>(base);
    out.count[i] = faces.n;
    if (base + faces.n > out.capacity) return;  // the host grows the buffer and runs the cells again
    for (int e = 0; e < faces.n; ++e) {
        const int f = faces.order[e];
        const int64_t r = static_cast<int64_t>(base) + e;
        out.fj[r] = faces.j[f];
        for (int a = 0; a < D; ++a) {
            out.fa[D * r + a] = faces.a[f][a];
            out.fc[D * r + a] = faces.c[f][a];
        }
    }
}

// Whether cell c has a face towards j (its records are sorted by neighbour).
__device__ __forceinline__ bool has_face(const int64_t* first, const int32_t* count, const int32_t* fj, int32_t c, int32_t j) {
    int64_t lo = first[c], hi = lo + count[c];
    while (lo < hi) {
        const int64_t mid = (lo + hi) >> 1;
        if (fj[mid] < j)
            lo = mid + 1;
        else
            hi = mid;
    }
    return lo < first[c] + count[c] && fj[lo] == j;
}

struct FaceOut {
    int32_t* owner;
    int32_t* neighbour;
    double* area;
    double* fcen;
};

// ---- The assembly of a mesh whose cells agree on their faces (every face seen from both its cells: all but meshes with
// degenerate vertices): a cell's records, by neighbour, are its list, the ones towards higher cells its owned faces in
// order, and the number of one that a lower cell owns is found in that cell's records. No atomics and no sorts; bound by
// the records copied. 128^3: 0.7 ms (k_forward, the scans and k_emit_lists' 0.63) where the general passes take 4.6.

// Each cell's owned faces (records towards higher cells) and its list's length.
__global__ void k_forward(int64_t n, const int64_t* __restrict__ first, const int32_t* __restrict__ count, const int32_t* __restrict__ fj,
                          int64_t* __restrict__ owned, int32_t* __restrict__ degree) {
    const int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
    if (i > n) return;
    if (i == n) {
        owned[n] = 0;
        degree[n] = 0;
        return;
    }
    const int64_t f0 = first[i], end = f0 + count[i];
    int64_t lo = f0, hi = end;
    while (lo < hi) {  // the first record past i
        const int64_t mid = (lo + hi) >> 1;
        if (fj[mid] <= i)
            lo = mid + 1;
        else
            hi = mid;
    }
    owned[i] = end - lo;
    degree[i] = count[i];
}

// Faces and lists, kEmitLanes threads a cell (neighbouring lanes copy neighbouring records). *missing counts the faces
// that a higher cell sees and the lower one does not (the mesh is then assembled by the general passes).
constexpr int kEmitLanes = 8;
template <int D>
__global__ void k_emit_lists(int64_t n, const int64_t* __restrict__ first, const int32_t* __restrict__ count, const int32_t* __restrict__ fj,
                             const double* __restrict__ fa, const double* __restrict__ fc, const int64_t* __restrict__ face_start,
                             const int32_t* __restrict__ start, FaceOut out, int32_t* __restrict__ list, unsigned int* __restrict__ missing) {
    const int64_t t = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x, i = t / kEmitLanes;
    if (i >= n) return;
    const int64_t f0 = first[i], own0 = face_start[i];
    const int m = count[i], back = m - static_cast<int>(face_start[i + 1] - own0), s0 = start[i];
    for (int k = static_cast<int>(t % kEmitLanes); k < m; k += kEmitLanes) {
        const int64_t r = f0 + k;
        const int32_t j = fj[r];
        if (k >= back) {
            const int64_t f = own0 + k - back;
            out.owner[f] = static_cast<int32_t>(i);
            out.neighbour[f] = j;
            for (int a = 0; a < D; ++a) {
                out.area[D * f + a] = fa[D * r + a];
                out.fcen[D * f + a] = fc[D * r + a];
            }
            list[s0 + k] = static_cast<int32_t>(f);
        } else {
            const int64_t end = first[j] + count[j], begin = end - (face_start[j + 1] - face_start[j]);
            int64_t lo = begin, hi = end;
            while (lo < hi) {
                const int64_t mid = (lo + hi) >> 1;
                if (fj[mid] < i)
                    lo = mid + 1;
                else
                    hi = mid;
            }
            if (lo < end && fj[lo] == i)
                list[s0 + k] = ~static_cast<int32_t>(face_start[j] + (lo - begin));
            else
                atomicAdd(missing, 1u);
        }
    }
}

// Per owner: its faces towards higher cells (fwd), and (flips) the faces higher cells saw that it missed.
__global__ void k_count_owned(int64_t n, const int64_t* __restrict__ first, const int32_t* __restrict__ count,
                              const int32_t* __restrict__ fj, int32_t* __restrict__ fwd, int32_t* __restrict__ flips,
                              Counters* c) {
    const int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
    if (i >= n) return;
    int own = 0;
    unsigned long long inconsistent = 0;
    const int64_t f0 = first[i];
    for (int k = 0; k < count[i]; ++k) {
        const int32_t j = fj[f0 + k];
        const bool seen = has_face(first, count, fj, j, static_cast<int32_t>(i));
        if (j > i) {
            ++own;
            if (!seen) ++inconsistent;
        } else if (!seen) {
            ++inconsistent;
            atomicAdd(flips + j, 1);
        }
    }
    fwd[i] = own;
    if (inconsistent) atomicAdd(&c->inconsistent, inconsistent);
}

__global__ void k_segment_lengths(int64_t n, const int32_t* __restrict__ fwd, const int32_t* __restrict__ flips,
                                  int64_t* __restrict__ length) {
    const int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
    if (i > n) return;
    length[i] = i < n ? static_cast<int64_t>(fwd[i]) + flips[i] : 0;
}


template <int D>
__global__ void k_emit(int64_t n, const int64_t* __restrict__ first, const int32_t* __restrict__ count,
                       const int32_t* __restrict__ fj, const double* __restrict__ fa, const double* __restrict__ fc,
                       const double* __restrict__ pos, Box box, const int64_t* __restrict__ face_start,
                       const int32_t* __restrict__ fwd, unsigned int* __restrict__ flip_cursor, FaceOut out) {
    const int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
    if (i >= n) return;
    const int64_t f0 = first[i];
    int64_t next = face_start[i];
    for (int k = 0; k < count[i]; ++k) {
        const int64_t r = f0 + k;
        const int32_t j = fj[r];
        if (j > i) {
            const int64_t f = next++;
            out.owner[f] = static_cast<int32_t>(i);
            out.neighbour[f] = j;
            for (int a = 0; a < D; ++a) {
                out.area[D * f + a] = fa[D * r + a];
                out.fcen[D * f + a] = fc[D * r + a];
            }
        } else if (!has_face(first, count, fj, j, static_cast<int32_t>(i))) {
            // owner j missed it: the area flips; the centroid, relative to j's generator, is this cell's centroid plus
            // the nearest image of x_i - x_j
            const int64_t f = face_start[j] + fwd[j] + atomicAdd(flip_cursor + j, 1u);
            out.owner[f] = j;
            out.neighbour[f] = static_cast<int32_t>(i);
            for (int a = 0; a < D; ++a) {
                double d = pos[D * i + a] - pos[D * j + a];
                d -= box.s[a] * nearbyint(d / box.s[a]);
                out.area[D * f + a] = -fa[D * r + a];
                out.fcen[D * f + a] = fc[D * r + a] + d;
            }
        }
    }
}

// An owner's segment holding flipped faces, sorted by neighbour.
template <int D>
__global__ void k_sort_segments(int64_t n, const int64_t* __restrict__ face_start, const int32_t* __restrict__ flips,
                                FaceOut out) {
    const int64_t o = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
    if (o >= n || flips[o] == 0) return;
    const int64_t s0 = face_start[o], s1 = face_start[o + 1];
    for (int64_t k = s0 + 1; k < s1; ++k) {
        const int32_t key = out.neighbour[k];
        double a[D], c[D];
        for (int x = 0; x < D; ++x) {
            a[x] = out.area[D * k + x];
            c[x] = out.fcen[D * k + x];
        }
        int64_t j = k - 1;
        while (j >= s0 && out.neighbour[j] > key) {
            out.neighbour[j + 1] = out.neighbour[j];
            for (int x = 0; x < D; ++x) {
                out.area[D * (j + 1) + x] = out.area[D * j + x];
                out.fcen[D * (j + 1) + x] = out.fcen[D * j + x];
            }
            --j;
        }
        out.neighbour[j + 1] = key;
        for (int x = 0; x < D; ++x) {
            out.area[D * (j + 1) + x] = a[x];
            out.fcen[D * (j + 1) + x] = c[x];
        }
    }
}

__global__ void k_degree(int64_t F, const int32_t* __restrict__ owner, const int32_t* __restrict__ neighbour,
                         int32_t* __restrict__ degree) {
    const int64_t f = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
    if (f >= F) return;
    atomicAdd(degree + owner[f], 1);
    atomicAdd(degree + neighbour[f], 1);
}

__global__ void k_list_fill(int64_t F, const int32_t* __restrict__ owner, const int32_t* __restrict__ neighbour,
                            const int32_t* __restrict__ start, unsigned int* __restrict__ cursor, int32_t* __restrict__ list,
                            int32_t* __restrict__ key) {
    const int64_t f = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
    if (f >= F) return;
    const int32_t o = owner[f], j = neighbour[f];
    int32_t s = start[o] + static_cast<int32_t>(atomicAdd(cursor + o, 1u));
    list[s] = static_cast<int32_t>(f);
    key[s] = j;
    s = start[j] + static_cast<int32_t>(atomicAdd(cursor + j, 1u));
    list[s] = ~static_cast<int32_t>(f);
    key[s] = o;
}

// Each cell's list by neighbour.
__global__ void k_list_sort(int64_t n, const int32_t* __restrict__ start, int32_t* __restrict__ list, int32_t* __restrict__ key) {
    const int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
    if (i >= n) return;
    const int32_t s0 = start[i], s1 = start[i + 1];
    for (int32_t k = s0 + 1; k < s1; ++k) {
        const int32_t x = key[k], e = list[k];
        int32_t j = k - 1;
        while (j >= s0 && key[j] > x) {
            key[j + 1] = key[j];
            list[j + 1] = list[j];
            --j;
        }
        key[j + 1] = x;
        list[j + 1] = e;
    }
}

const char* cell_error(int code) {
    switch (code) {
        case kOutOfOffsets: return "a cell reaches farther than a box side from its generator (too few points for the box)";
        case kReachesBox: return "a cell reaches the box (box too small for the points)";
        case kTouchesSelf: return "a cell touches its own periodic image (box too small for the points)";
        case kDuplicatePair: return "two faces between the same pair of cells (box too small for unique nearest images)";
        case kCapacity: return "a cell has more vertices or faces than the remesher holds";
        case kCandidates: return "more generators at one distance from a cell than the remesher holds";
        default: return "unknown cell error";
    }
}

}  // namespace

struct luna_remesh {
    int dim = 3;
    Box box{};
    cudaStream_t stream = nullptr;
    int64_t shape_n = -1;
    GridShape shape;
    Buf<int32_t> offsets;
    Buf<double> bound2;
    Buf<double> input, pos;
    Buf<int64_t> bucket, bucket_start;
    Buf<unsigned long long> bucket_count;
    Buf<unsigned int> cursor;
    Buf<int32_t> items;
    Buf<double> volume, centroid;
    Buf<int64_t> first;
    Buf<int32_t> left;   // cells that the eight-lane kernels left for one thread
    int64_t one_thread = 0;  // cells of the last build with a thread each
    Buf<int32_t> retry;  // cells the fast path handed to the far search
    Buf<double4> shell_plane;  // a chunk's candidates (Shell)
    Buf<double> shell_d2, shell_cover;
    Buf<int32_t> shell_j, shell_n;
    Buf<int32_t> count, fj;
    Buf<double> fa, fc;
    Buf<int32_t> fwd, flips;
    Buf<int64_t> seg_length, face_start;
    Buf<int32_t> owner, neighbour, degree, start, list, key;
    Buf<double> area, fcen;
    Buf<Counters> counters;
    Buf<unsigned char> scan_temp;
    unsigned long long capacity = 0;

    template <class T>
    luna_status exclusive_scan(const T* in, T* out, int64_t items) {
        size_t bytes = 0;
        RM_CUDA(cub::DeviceScan::ExclusiveSum(nullptr, bytes, in, out, items, stream));
        RM_TRY(scan_temp.reserve(bytes, "scan scratch"));
        RM_CUDA(cub::DeviceScan::ExclusiveSum(scan_temp.ptr, bytes, in, out, items, stream));
        return LUNA_OK;
    }

    template <int D>
    luna_status build(int64_t n, const double* points, bool on_device, luna_mesh_desc* mesh, int64_t* inconsistent);
    template <int D>
    luna_status assemble_general(int64_t n, int64_t* faces_out, Counters* h_out);
    template <int D>
    luna_status reserve_faces(int64_t F) {
        RM_TRY(owner.reserve(F, "owner"));
        RM_TRY(neighbour.reserve(F, "neighbour"));
        RM_TRY(area.reserve(F * D, "area"));
        RM_TRY(fcen.reserve(F * D, "face_centroid"));
        return list.reserve(2 * F, "cell_face");
    }
};

// Faces and lists where some face is seen from one of its cells only: the lower cell owns it all the same.
template <int D>
luna_status luna_remesh::assemble_general(int64_t n, int64_t* faces_out, Counters* h_out) {
    const int T = 256;
    int64_t F = 0;
    Counters h{};
    RM_CUDA(cudaMemsetAsync(flips.ptr, 0, n * sizeof(int32_t), stream));
    k_count_owned<<<grid_blocks(n, T), T, 0, stream>>>(n, first.ptr, count.ptr, fj.ptr, fwd.ptr, flips.ptr, counters.ptr);
    k_segment_lengths<<<grid_blocks(n + 1, T), T, 0, stream>>>(n, fwd.ptr, flips.ptr, seg_length.ptr);
    RM_CUDA(cudaGetLastError());
    RM_TRY(exclusive_scan(static_cast<const int64_t*>(seg_length.ptr), face_start.ptr, n + 1));
    RM_CUDA(cudaMemcpyAsync(&F, face_start.ptr + n, sizeof(int64_t), cudaMemcpyDeviceToHost, stream));
    RM_CUDA(cudaMemcpyAsync(&h, counters.ptr, sizeof(Counters), cudaMemcpyDeviceToHost, stream));
    RM_CUDA(cudaStreamSynchronize(stream));
    if (2 * F >= (int64_t(1) << 31) - 1) return fail(LUNA_EINVAL, "luna_remesh_build: too many faces for int32 lists");
    RM_TRY(reserve_faces<D>(F));
    RM_TRY(key.reserve(2 * F, "list keys"));
    const FaceOut faces{owner.ptr, neighbour.ptr, area.ptr, fcen.ptr};
    RM_CUDA(cudaMemsetAsync(cursor.ptr, 0, n * sizeof(unsigned int), stream));
    k_emit<D><<<grid_blocks(n, T), T, 0, stream>>>(n, first.ptr, count.ptr, fj.ptr, fa.ptr, fc.ptr, pos.ptr, box, face_start.ptr,
                                                    fwd.ptr, cursor.ptr, faces);
    k_sort_segments<D><<<grid_blocks(n, T), T, 0, stream>>>(n, face_start.ptr, flips.ptr, faces);
    RM_CUDA(cudaGetLastError());

    // lists, by neighbour
    RM_CUDA(cudaMemsetAsync(degree.ptr, 0, (n + 1) * sizeof(int32_t), stream));
    if (F > 0) k_degree<<<grid_blocks(F, T), T, 0, stream>>>(F, owner.ptr, neighbour.ptr, degree.ptr);
    RM_CUDA(cudaGetLastError());
    RM_TRY(exclusive_scan(static_cast<const int32_t*>(degree.ptr), start.ptr, n + 1));
    RM_CUDA(cudaMemsetAsync(cursor.ptr, 0, n * sizeof(unsigned int), stream));
    if (F > 0) k_list_fill<<<grid_blocks(F, T), T, 0, stream>>>(F, owner.ptr, neighbour.ptr, start.ptr, cursor.ptr, list.ptr, key.ptr);
    k_list_sort<<<grid_blocks(n, T), T, 0, stream>>>(n, start.ptr, list.ptr, key.ptr);
    RM_CUDA(cudaGetLastError());
    RM_CUDA(cudaStreamSynchronize(stream));
    *faces_out = F;
    *h_out = h;
    return LUNA_OK;
}

template <int D>
luna_status luna_remesh::build(int64_t n, const double* points, bool on_device, luna_mesh_desc* mesh, int64_t* inconsistent) {
    const int T = 256;
    if (shape_n != n) {  // the grid's shape depends on n and the box only
        shape.build(D, n, box.s);
        RM_TRY(offsets.reserve(shape.offsets.size(), "bucket offsets"));
        RM_TRY(bound2.reserve(shape.bound2.size(), "bucket bounds"));
        RM_CUDA(cudaMemcpy(offsets.ptr, shape.offsets.data(), shape.offsets.size() * sizeof(int32_t), cudaMemcpyHostToDevice));
        RM_CUDA(cudaMemcpy(bound2.ptr, shape.bound2.data(), shape.bound2.size() * sizeof(double), cudaMemcpyHostToDevice));
        shape_n = n;
    }
    const int64_t B = shape.buckets;
    RM_TRY(counters.reserve(1, "remesh counters"));
    RM_TRY(pos.reserve(n * D, "generators"));
    RM_TRY(bucket.reserve(n, "buckets"));
    RM_TRY(bucket_count.reserve(B + 1, "bucket counts"));
    RM_TRY(bucket_start.reserve(B + 1, "bucket starts"));
    RM_TRY(cursor.reserve(B > n + 1 ? B : n + 1, "cursors"));
    RM_TRY(items.reserve(n, "bucket items"));
    RM_TRY(volume.reserve(n, "volumes"));
    RM_TRY(centroid.reserve(n * D, "centroids"));
    RM_TRY(first.reserve(n, "cell records"));
    RM_TRY(retry.reserve(n, "far cells"));
    RM_TRY(count.reserve(n, "cell records"));
    RM_TRY(fwd.reserve(n, "owned faces"));
    RM_TRY(flips.reserve(n, "flipped faces"));
    RM_TRY(seg_length.reserve(n + 1, "segments"));
    RM_TRY(face_start.reserve(n + 1, "segments"));
    RM_TRY(degree.reserve(n + 1, "degrees"));
    RM_TRY(start.reserve(n + 1, "cell_face_start"));

    const double* src = points;
    if (!on_device) {
        RM_TRY(input.reserve(n * D, "generators"));
        RM_CUDA(cudaMemcpyAsync(input.ptr, points, n * D * sizeof(double), cudaMemcpyHostToDevice, stream));
        src = input.ptr;
    }
    RM_CUDA(cudaMemsetAsync(counters.ptr, 0, sizeof(Counters), stream));
    k_wrap<D><<<grid_blocks(n * D, T), T, 0, stream>>>(n, src, pos.ptr, box, counters.ptr);
    RM_CUDA(cudaGetLastError());

    // buckets
    const Grid g = shape.view(bucket_start.ptr, items.ptr, offsets.ptr, bound2.ptr);
    RM_CUDA(cudaMemsetAsync(bucket_count.ptr, 0, (B + 1) * sizeof(unsigned long long), stream));
    k_bucket_count<D><<<grid_blocks(n, T), T, 0, stream>>>(n, pos.ptr, g, bucket.ptr, bucket_count.ptr);
    RM_CUDA(cudaGetLastError());
    RM_TRY(exclusive_scan(reinterpret_cast<const int64_t*>(bucket_count.ptr), bucket_start.ptr, B + 1));
    RM_CUDA(cudaMemsetAsync(cursor.ptr, 0, B * sizeof(unsigned int), stream));
    k_bucket_fill<<<grid_blocks(n, T), T, 0, stream>>>(n, bucket.ptr, bucket_start.ptr, cursor.ptr, items.ptr);
    k_bucket_sort<<<grid_blocks(B, T), T, 0, stream>>>(B, bucket_start.ptr, items.ptr);
    RM_CUDA(cudaGetLastError());

    // cells: a first guess of the face records (16 a cell in 3D, 6 in 2D on a jittered lattice), grown once if short
    if (capacity == 0) capacity = static_cast<unsigned long long>(n) * (D == 3 ? 18 : 7);
    Counters h{};
    const auto read_counters = [&]() -> luna_status {
        RM_CUDA(cudaMemcpyAsync(&h, counters.ptr, sizeof(Counters), cudaMemcpyDeviceToHost, stream));
        RM_CUDA(cudaStreamSynchronize(stream));
        return LUNA_OK;
    };
    bool by_lanes = D == 3 && kEightLanes;
    if (by_lanes && n >= kSampleFrom) {
        k_sample<<<kSamples, 128, 0, stream>>>(n, pos.ptr, box, g, counters.ptr);
        RM_CUDA(cudaGetLastError());
        RM_TRY(read_counters());
        by_lanes = h.boxes < kLatticeSamples && (h.close < kIrregularSamples || n > kOneWave);
    }
    if (by_lanes) {
        const int64_t chunk = n < kChunk ? n : kChunk;
        RM_TRY(left.reserve(n, "cells left"));
        RM_TRY(shell_plane.reserve(chunk * kKept, "candidates"));
        RM_TRY(shell_d2.reserve(chunk * kKept, "candidates"));
        RM_TRY(shell_j.reserve(chunk * kKept, "candidates"));
        RM_TRY(shell_n.reserve(chunk, "candidates"));
        RM_TRY(shell_cover.reserve(chunk, "candidates"));
    }
    for (int attempt = 0; attempt < 2; ++attempt) {
        RM_TRY(fj.reserve(capacity, "face records"));
        RM_TRY(fa.reserve(capacity * D, "face records"));
        RM_TRY(fc.reserve(capacity * D, "face records"));
        if (attempt > 0) RM_CUDA(cudaMemsetAsync(counters.ptr, 0, sizeof(Counters), stream));
        const CellOut out{volume.ptr, centroid.ptr, first.ptr, count.ptr, fj.ptr, fa.ptr, fc.ptr, capacity};
        one_thread = n;
        if constexpr (D == 3 && kEightLanes)
            if (by_lanes) {
                const LaneOut lanes{out.volume, out.centroid, out.first, out.count, out.fj, out.fa, out.fc, out.capacity,
                                    &counters.ptr->faces, left.ptr, &counters.ptr->left};
                const Shell shell{shell_plane.ptr, shell_d2.ptr, shell_j.ptr, shell_n.ptr, shell_cover.ptr};
                const double3 sides = make_double3(box.s[0], box.s[1], box.s[2]);
                for (int64_t base = 0; base < n; base += kChunk) {
                    const int64_t cells = n - base < kChunk ? n - base : kChunk;
                    k_search<<<grid_blocks(cells, kSearchWarps), 32 * kSearchWarps, 0, stream>>>(base, cells, pos.ptr, sides, g, shell);
                    k_clip<<<grid_blocks(cells * kLanes, kClipThreads), kClipThreads, 0, stream>>>(base, cells, sides, shell, lanes);
                }
                RM_CUDA(cudaGetLastError());
                RM_TRY(read_counters());
                one_thread = h.nonfinite ? 0 : h.left;
            }
        if (one_thread > 0) {
            const int spread = D == 3 && by_lanes ? spread_of(one_thread) : 0;
            k_cells<D, false><<<grid_blocks(one_thread << spread, 64), 64, 0, stream>>>(one_thread, spread, by_lanes ? left.ptr : nullptr, pos.ptr,
                                                                                       box, g, out, counters.ptr, retry.ptr);
            RM_CUDA(cudaGetLastError());
            RM_TRY(read_counters());
        }
        if (h.retry > 0 && !h.error && !h.nonfinite) {  // the far search for the cells the fast path handed on
            const int spread = D == 3 ? spread_of(h.retry) : 0;
            k_cells<D, true><<<grid_blocks(static_cast<int64_t>(h.retry) << spread, 64), 64, 0, stream>>>(h.retry, spread, retry.ptr, pos.ptr, box, g,
                                                                                                         out, counters.ptr, nullptr);
            RM_CUDA(cudaGetLastError());
            RM_TRY(read_counters());
        }
        if (h.nonfinite) return fail(LUNA_EINVAL, "luna_remesh_build: non-finite point");
        if (h.error) return fail(LUNA_EINVAL, std::string("luna_remesh_build: cell ") + std::to_string(h.error_cell) + ": " + cell_error(h.error));
        if (h.faces <= capacity) break;
        capacity = h.faces + h.faces / 16;
    }

    // faces, by owner then neighbour, and lists, by neighbour
    k_forward<<<grid_blocks(n + 1, T), T, 0, stream>>>(n, first.ptr, count.ptr, fj.ptr, seg_length.ptr, degree.ptr);
    RM_CUDA(cudaGetLastError());
    RM_TRY(exclusive_scan(static_cast<const int64_t*>(seg_length.ptr), face_start.ptr, n + 1));
    RM_TRY(exclusive_scan(static_cast<const int32_t*>(degree.ptr), start.ptr, n + 1));
    int64_t F = 0;
    RM_CUDA(cudaMemcpyAsync(&F, face_start.ptr + n, sizeof(int64_t), cudaMemcpyDeviceToHost, stream));
    RM_CUDA(cudaStreamSynchronize(stream));
    bool agreed = static_cast<unsigned long long>(2 * F) == h.faces && 2 * F < (int64_t(1) << 31) - 1;
    if (agreed) {
        RM_TRY(reserve_faces<D>(F));
        RM_CUDA(cudaMemsetAsync(cursor.ptr, 0, sizeof(unsigned int), stream));
        k_emit_lists<D><<<grid_blocks(n * kEmitLanes, T), T, 0, stream>>>(n, first.ptr, count.ptr, fj.ptr, fa.ptr, fc.ptr, face_start.ptr, start.ptr,
                                                                          FaceOut{owner.ptr, neighbour.ptr, area.ptr, fcen.ptr}, list.ptr, cursor.ptr);
        RM_CUDA(cudaGetLastError());
        unsigned int missing = 0;
        RM_CUDA(cudaMemcpyAsync(&missing, cursor.ptr, sizeof(missing), cudaMemcpyDeviceToHost, stream));
        RM_CUDA(cudaStreamSynchronize(stream));
        agreed = missing == 0;
    }
    if (!agreed) RM_TRY(assemble_general<D>(n, &F, &h));

    *mesh = luna_mesh_desc{};
    mesh->dim = D;
    mesh->n_cells = n;
    mesh->n_faces = F;
    mesh->owner = owner.ptr;
    mesh->neighbour = neighbour.ptr;
    mesh->cell_face_start = start.ptr;
    mesh->cell_face = list.ptr;
    mesh->area = area.ptr;
    mesh->face_centroid = fcen.ptr;
    mesh->centroid = centroid.ptr;
    mesh->volume = volume.ptr;
    mesh->positions = pos.ptr;
    for (int a = 0; a < 3; ++a) mesh->box[a] = a < D ? box.s[a] : 0.0;
    mesh->on_device = 1;
    if (inconsistent) *inconsistent = static_cast<int64_t>(h.inconsistent);
    return LUNA_OK;
}

extern "C" {

LUNA_API luna_status luna_remesh_create(int dim, const double* box, luna_remesh** out) {
    if (!out || !box) return fail(LUNA_EINVAL, "luna_remesh_create: null argument");
    *out = nullptr;
    if (dim != 2 && dim != 3) return fail(LUNA_EINVAL, "luna_remesh_create: dim must be 2 or 3");
    for (int a = 0; a < dim; ++a)
        if (!(box[a] > 0) || !std::isfinite(box[a])) return fail(LUNA_EINVAL, "luna_remesh_create: box sides must be positive");
    auto* r = new luna_remesh();
    r->dim = dim;
    for (int a = 0; a < 3; ++a) r->box.s[a] = a < dim ? box[a] : 1.0;
    *out = r;
    return LUNA_OK;
}

LUNA_API luna_status luna_remesh_destroy(luna_remesh* r) {
    delete r;
    return LUNA_OK;
}

LUNA_API luna_status luna_remesh_set_stream(luna_remesh* r, void* stream) {
    if (!r) return fail(LUNA_EINVAL, "luna_remesh_set_stream: null remesher");
    r->stream = static_cast<cudaStream_t>(stream);
    return LUNA_OK;
}

LUNA_API luna_status luna_remesh_build(luna_remesh* r, int64_t n, const double* points, int on_device, luna_mesh_desc* mesh,
                                       int64_t* inconsistent) {
    if (!r || !points || !mesh) return fail(LUNA_EINVAL, "luna_remesh_build: null argument");
    if (n < 2 || n >= (int64_t(1) << 30)) return fail(LUNA_EINVAL, "luna_remesh_build: n out of range");
    return r->dim == 3 ? r->build<3>(n, points, on_device != 0, mesh, inconsistent) : r->build<2>(n, points, on_device != 0, mesh, inconsistent);
}

LUNA_API luna_status luna_remesh_points(luna_remesh* r, int64_t n, double** points) {
    if (!r || !points) return fail(LUNA_EINVAL, "luna_remesh_points: null argument");
    if (n < 2 || n >= (int64_t(1) << 30)) return fail(LUNA_EINVAL, "luna_remesh_points: n out of range");
    RM_TRY(r->input.reserve(static_cast<size_t>(n) * r->dim, "generators"));
    *points = r->input.ptr;
    return LUNA_OK;
}

LUNA_API luna_status luna_remesh_one_thread(const luna_remesh* r, int64_t* out) {
    if (!r || !out) return fail(LUNA_EINVAL, "luna_remesh_one_thread: null argument");
    *out = r->one_thread;
    return LUNA_OK;
}

LUNA_API luna_status luna_remesh_device_bytes(const luna_remesh* r, int64_t* out) {
    if (!r || !out) return fail(LUNA_EINVAL, "luna_remesh_device_bytes: null argument");
    const size_t b = r->offsets.bytes() + r->bound2.bytes() + r->input.bytes() + r->pos.bytes() + r->bucket.bytes() +
                     r->bucket_start.bytes() + r->bucket_count.bytes() + r->cursor.bytes() + r->items.bytes() + r->volume.bytes() +
                     r->centroid.bytes() + r->first.bytes() + r->retry.bytes() + r->left.bytes() + r->shell_plane.bytes() + r->shell_d2.bytes() +
                     r->shell_cover.bytes() + r->shell_j.bytes() + r->shell_n.bytes() + r->count.bytes() + r->fj.bytes() + r->fa.bytes() + r->fc.bytes() +
                     r->fwd.bytes() + r->flips.bytes() + r->seg_length.bytes() + r->face_start.bytes() + r->owner.bytes() +
                     r->neighbour.bytes() + r->degree.bytes() + r->start.bytes() + r->list.bytes() + r->key.bytes() + r->area.bytes() +
                     r->fcen.bytes() + r->counters.bytes() + r->scan_temp.bytes();
    *out = static_cast<int64_t>(b);
    return LUNA_OK;
}

}  // extern "C"
