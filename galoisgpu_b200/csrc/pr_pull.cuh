// pr_pull.cuh -- PageRank by pulled sweeps, for graphs whose edges are
// symmetric (every u->v has as many v->u): device code of gft_pr's pull path.
//
// The ranks the residual pushes of pr.cu converge to solve
//     x = (1 - a) + a * A D^-1 x         (A: adjacency, D: out-degrees).
// On a symmetric graph A D^-1 is similar to a symmetric matrix, so its
// spectrum is real and lies in [-1, 1], and the Chebyshev semi-iterative
// method (Golub and Varga, "Chebyshev semi-iterative methods, successive
// overrelaxation iterative methods, and second order Richardson iterative
// methods", Numer. Math. 3, 1961) applies:
//     x(k+1) = x(k-1) + w(k+1) * (x'(k) - x(k-1)),   x'(k) = (1-a) + a A D^-1 x(k),
//     w(1) = 1, w(2) = 2 / (2 - a^2), w(k+1) = 4 / (4 - a^2 w(k)).
// It gains a factor (1 - sqrt(1 - a^2)) / a = 0.56 a sweep where a round of
// pushes gains 0.85: about 25 sweeps over the edges instead of 104 rounds
// (RMAT-22, 127 M edges: 67.0 -> 14.2 ms, and 7e-8 instead of 7e-5 from the
// 64-bit solution, as a hub's sum no longer swallows small addends).
// The sweeps end once, at every vertex, the residual x'(k) - x(k) and the move
// x(k+1) - x(k) are both at most EPSILON * max(1, rank).  The residual is what
// the pushes stop on too, and it bounds the error: |x(k) - x| <= |residual| /
// (1 - a) in the 2-norm weighted by 1/sqrt(degree), where A D^-1 is symmetric;
// the move carries the bound over to x(k+1).  The move alone says nothing: an
// error mode of eigenvalue l is T_k(l) / T_k(1/a) of what it was, which two
// sweeps can leave equal (l = -a/2 after the second sweep: the complete graph
// of 24 vertices with 17 leaves on each stopped there, 1.5e-2 off).
// A sweep reads a vertex's terms instead of adding to its neighbours'
// residuals: no atomics, and a sum's order does not depend on the schedule.
//
// What bounds a sweep is the gather of y = D^-1 x, one 4-byte value per edge.
// L1 looks up one line a cycle for lanes on different lines, an L2 gather
// moves a 32-byte sector per value, and every edge costs the instructions of
// its gather, so vertices are renumbered by degree,
// largest first: the first kPullHub values of y, which on a skewed graph
// stand behind most edges, are copied into shared memory at the start of
// each sweep, where 32 lanes on different banks are served together.  The
// renumbered rows are stored in 16-byte quads of edges; an edge is the byte
// offset of its value, and rows are padded with the offset of a zero that lies
// between the values in shared memory and the rest.  Rows of one class (8 classes per octave of quads) are padded
// to the class's largest, so a row's place follows from its number and the
// lanes of a warp run the same trip count; the padding is at most 1/8.
//
// Launches, on the caller's stream, none of which the host waits for:
//   pr_sample   looks for the reverse of a few hundred edges; a directed
//               graph is given up at once (the host then runs the pushes)
//   pr_classes  counts the rows of each class, and refuses a graph whose rows
//               do not lie in its edges (a wrapped one can): the buffers are
//               sized by its number of edges
//   pr_place    numbers the vertices, class by class
//   pr_relabel  writes the renumbered rows, and sums over all edges u->v a
//               64-bit hash of {u, v}, added for u < v and subtracted for
//               u > v: zero for a symmetric graph, and for another one only
//               by a 2^-64 chance
//   pr_sweeps   persistent, one CTA per SM: the sweeps, and the ranks back in
//               the caller's order
#pragma once
#include <stdint.h>

#include "gft_internal.h"
#include "traverse.cuh"

namespace gft {
namespace dev {

constexpr int kPullClasses = 256;
constexpr int kPullBlock = 1024;
constexpr uint32_t kPullHub = 49152;  // y values in shared memory: 192 KB, one CTA per SM
constexpr uint32_t kPullTile = 4096;  // vertices numbered together by one CTA
constexpr unsigned kPullMaxSweeps = 64;  // 0.56^64 = 5e-17: rounding ends the progress long before
constexpr double kPullAlpha = 0.85f;     // apps/pr/kernel.cu:19, the 32-bit constant
constexpr float kPullEpsilon = 0.000001f;  // apps/pr/kernel.cu:20

struct PullState {
    unsigned long long hash;  // pr_relabel's sum: 0 for a symmetric graph
    unsigned asymmetric;      // pr_sample found an edge without its reverse; pr_sweeps: the pushes have to run
    unsigned outside;         // pr_classes found a row, or pr_relabel an edge, leaving the graph
    unsigned moved[3];        // per sweep, triple buffered: some residual or move was above EPSILON
    unsigned unit[3];         // per sweep, triple buffered: units claimed beyond every warp's first
    unsigned rows[kPullClasses];    // rows of each class
    unsigned cursor[kPullClasses];  // rows of each class numbered so far
};

struct PullParams {
    const uint32_t *__restrict__ row_start;
    const uint32_t *__restrict__ edge_dst;
    uint32_t nnodes, nedges;
    float *rank;         // the caller's output
    uint32_t *perm;      // number -> vertex
    uint32_t *number;    // vertex -> number (vertices without edges: not set)
    float *inv_deg;      // by number
    float *x[2];         // by number
    float *y[2];         // by place (pull_place)
    uint4 *quads;
    PullState *st;
    TraversalCtl *ctl;
    unsigned long long timeout_ns;
};

// Class of a row of q quads: exact below 8, then 8 per octave; class 0 has no edges.
__host__ __device__ __forceinline__ unsigned pull_class(uint32_t q)
{
    if (q < 8) return q;
#ifdef __CUDA_ARCH__
    const unsigned lg = 31u - __clz(q);
#else
    const unsigned lg = 31u - (unsigned)__builtin_clz(q);
#endif
    return 8u * (lg - 2u) + ((q >> (lg - 3u)) & 7u);
}
// Quads that rows of class c are stored with: the largest of the class.
__host__ __device__ __forceinline__ uint32_t pull_class_quads(unsigned c)
{
    if (c < 8) return c;
    const unsigned lg = c / 8u + 2u;
    return ((9u + (c & 7u)) << (lg - 3u)) - 1u;
}

__device__ __forceinline__ uint32_t pull_quads_of(uint32_t deg) { return deg / 4u + (deg % 4u != 0u); }

// Numbers below this one have their y in shared memory.
__device__ __forceinline__ unsigned pull_hubs(unsigned active) { return min(active, kPullHub); }
// Place of a numbered vertex's value in y: place nhub is the padding's zero.
__device__ __forceinline__ uint32_t pull_place(uint32_t i, unsigned nhub) { return i + (i >= nhub); }

// 64-bit mix of an unordered pair (SplitMix64's finaliser, Steele, Lea and
// Flood, OOPSLA 2014, over the packed pair).
__device__ __forceinline__ unsigned long long pull_pair_hash(uint32_t a, uint32_t b)
{
    unsigned long long z = ((unsigned long long)min(a, b) << 32 | max(a, b)) + 0x9E3779B97F4A7C15ull;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}

// A warp per sampled edge u->v looks for u among v's edges (lists of more
// than kPullSampleScan edges are taken on trust: pr_relabel's hash decides).
constexpr unsigned kPullSamples = 256, kPullSampleScan = 1024;

__global__ void __launch_bounds__(256) pr_sample(PullParams p)
{
    const unsigned lane = threadIdx.x & 31, w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (w >= kPullSamples || p.nedges == 0) return;
    const uint32_t e = (uint32_t)(((unsigned long long)(w * 2654435761u + 12345u) * p.nedges) >> 32);
    // The row of edge e: the last one that starts at or before it.
    uint32_t lo = 0, hi = p.nnodes;
    while (hi - lo > 1) {
        const uint32_t mid = lo + (hi - lo) / 2;
        if (p.row_start[mid] <= e) lo = mid;
        else hi = mid;
    }
    const uint32_t v = p.edge_dst[e];
    bool found = false;
    if (v < p.nnodes) {
        const uint32_t s = p.row_start[v], d = p.row_start[v + 1] - s;
        found = d > kPullSampleScan || s > p.nedges || d > p.nedges - s;
        for (uint32_t i = lane; i < d && !found; i += 32) found = p.edge_dst[s + i] == lo;
    }
    if (!__any_sync(kFull, found) && lane == 0) p.st->asymmetric = 1;
}

__global__ void __launch_bounds__(1024) pr_classes(PullParams p)
{
    __shared__ unsigned s_rows[kPullClasses];
    if (__ldcg(&p.st->asymmetric)) return;
    for (unsigned c = threadIdx.x; c < kPullClasses; c += blockDim.x) s_rows[c] = 0;
    __syncthreads();
    const unsigned lane = threadIdx.x & 31;
    const uint32_t step = gridDim.x * blockDim.x;
    bool outside = false;
    for (uint32_t v0 = blockIdx.x * blockDim.x + threadIdx.x - lane; v0 < p.nnodes; v0 += step) {  // warp uniform
        const uint32_t v = v0 + lane;
        unsigned c = kPullClasses;
        if (v < p.nnodes) {
            const uint32_t s = p.row_start[v], e = p.row_start[v + 1];
            outside |= e < s || e > p.nedges;
            c = pull_class(pull_quads_of(e - s));
        }
        const unsigned peers = __match_any_sync(kFull, c);
        if (c < kPullClasses && lane == __ffs(peers) - 1) atomicAdd(&s_rows[c], __popc(peers));
    }
    __syncthreads();
    for (unsigned c = threadIdx.x; c < kPullClasses; c += blockDim.x)
        if (s_rows[c]) atomicAdd(&p.st->rows[c], s_rows[c]);
    if (outside) p.st->outside = 1;
}

// First number of each class, largest rows first (class 0 stays unnumbered):
// s_first[c], by 256 threads or more.
__device__ __forceinline__ void pull_class_firsts(const PullState *st, unsigned *s_first)
{
    __shared__ unsigned s_warp[kPullClasses / 32];
    const unsigned t = threadIdx.x, lane = t & 31, c = kPullClasses - 1 - t;
    unsigned rows = 0, incl = 0;
    if (t < kPullClasses) {
        rows = c ? __ldcg(&st->rows[c]) : 0u;
        incl = warp_incl_sum(rows, lane);
        if (lane == 31) s_warp[t >> 5] = incl;
    }
    __syncthreads();
    if (t < kPullClasses) {
        unsigned before = 0;
        for (unsigned i = 0; i < (t >> 5); i++) before += s_warp[i];
        s_first[c] = before + incl - rows;
    }
    __syncthreads();
}

// Numbers the vertices: a CTA takes tiles of kPullTile vertices and reserves
// the numbers of a tile's rows class by class, so vertices that are near
// each other keep near numbers within a class.
__global__ void __launch_bounds__(1024) pr_place(PullParams p)
{
    __shared__ unsigned s_first[kPullClasses], s_rows[kPullClasses], s_base[kPullClasses];
    if (__ldcg(&p.st->asymmetric) | __ldcg(&p.st->outside)) return;
    pull_class_firsts(p.st, s_first);
    constexpr int kPer = kPullTile / 1024;
    const unsigned lane = threadIdx.x & 31, lt = lanemask_lt();
    const uint32_t tiles = (p.nnodes + kPullTile - 1) / kPullTile;
    for (uint32_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        for (unsigned c = threadIdx.x; c < kPullClasses; c += blockDim.x) s_rows[c] = 0;
        __syncthreads();
        unsigned cls[kPer], at[kPer];
        uint32_t deg[kPer];
#pragma unroll
        for (int k = 0; k < kPer; k++) {
            const uint32_t v = tile * kPullTile + k * 1024 + threadIdx.x;
            deg[k] = v < p.nnodes ? p.row_start[v + 1] - p.row_start[v] : 0u;
            cls[k] = v < p.nnodes ? pull_class(pull_quads_of(deg[k])) : kPullClasses;
        }
#pragma unroll
        for (int k = 0; k < kPer; k++) {
            const unsigned peers = __match_any_sync(kFull, cls[k]);
            const int lead = __ffs(peers) - 1;
            unsigned base = 0;
            if ((int)lane == lead && cls[k] < kPullClasses) base = atomicAdd(&s_rows[cls[k]], __popc(peers));
            at[k] = __shfl_sync(kFull, base, lead) + __popc(peers & lt);
        }
        __syncthreads();
        for (unsigned c = threadIdx.x + 1; c < kPullClasses; c += blockDim.x)
            if (s_rows[c]) s_base[c] = s_first[c] + atomicAdd(&p.st->cursor[c], s_rows[c]);
        __syncthreads();
#pragma unroll
        for (int k = 0; k < kPer; k++) {
            const uint32_t v = tile * kPullTile + k * 1024 + threadIdx.x;
            if (v >= p.nnodes) continue;
            if (cls[k] == 0) {
                p.number[v] = 0;  // no row names it, or the graph is not symmetric
                p.rank[v] = (float)(1.0 - kPullAlpha);
            } else {
                const uint32_t i = s_base[cls[k]] + at[k];
                p.number[v] = i;
                p.perm[i] = v;
                p.inv_deg[i] = (float)(1.0 / deg[k]);
            }
        }
        __syncthreads();
    }
}

// The non-empty classes, largest rows first, in shared memory.
struct PullTable {
    unsigned n;                      // classes
    unsigned active;                 // numbered rows
    unsigned first[kPullClasses];    // first number
    unsigned rows[kPullClasses];
    unsigned quads[kPullClasses];    // quads per row
    unsigned quad0[kPullClasses];    // first quad
};

__device__ __forceinline__ void pull_table(const PullState *st, PullTable &t)
{
    __shared__ unsigned s_first[kPullClasses];
    pull_class_firsts(st, s_first);
    if (threadIdx.x < 32) {  // 32 classes at a time, in order
        unsigned n = 0, quad = 0, active = 0;
        for (int c0 = kPullClasses - 1; c0 > 0; c0 -= 32) {
            const int c = c0 - (int)threadIdx.x;
            const unsigned rows = c > 0 ? __ldcg(&st->rows[c]) : 0u;
            const unsigned q = c > 0 ? pull_class_quads(c) : 0u;
            const unsigned have = __ballot_sync(kFull, rows != 0);
            const unsigned incl = warp_incl_sum(rows * q, threadIdx.x);
            if (rows) {
                const unsigned i = n + __popc(have & lanemask_lt());
                t.first[i] = s_first[c];
                t.rows[i] = rows;
                t.quads[i] = q;
                t.quad0[i] = quad + incl - rows * q;
            }
            n += __popc(have);
            quad += __shfl_sync(kFull, incl, 31);
            active += __reduce_add_sync(kFull, rows);
        }
        if (threadIdx.x == 0) {
            t.n = n;
            t.active = active;
        }
    }
    __syncthreads();
}

// Lanes that share a row of q quads: a quad per lane up to 4, then two to four
// quads per lane, so that few of them are padding.
__device__ __forceinline__ unsigned pull_lanes(uint32_t q)
{
    return q <= 2 ? q : q <= 16 ? 4u : q <= 32 ? 8u : q <= 64 ? 16u : 32u;
}

// Calls f(class, row, first quad, end, lane of the row, lanes per row) for the
// rows of every class, a long row in segments of kPullSegment quads, dealt to
// the grid's warps in turn: rows are sorted by size, so every warp gets about
// the same number of edges.
constexpr uint32_t kPullSegment = 512;

template <class F>
__device__ __forceinline__ void pull_segments(const PullTable &t, unsigned gwarp, unsigned nwarps, unsigned lane, F &&f)
{
    unsigned dealt = 0;
    for (unsigned c = 0; c < t.n; c++) {
        const uint32_t q = t.quads[c], segs = (q + kPullSegment - 1) / kPullSegment;
        const unsigned s = pull_lanes(q), per = 32 / s;
        const unsigned chunks = segs > 1 ? t.rows[c] * segs : (t.rows[c] + per - 1) / per;
        for (unsigned k = (gwarp + nwarps - dealt) % nwarps; k < chunks; k += nwarps) {
            const unsigned r = segs > 1 ? k / segs : k * per + lane / s;
            const uint32_t j = segs > 1 ? k % segs * kPullSegment : 0;
            if (r < t.rows[c]) f(c, r, j, min(q, j + kPullSegment), lane % s, s);
        }
        dealt = (dealt + chunks) % nwarps;
    }
}

__global__ void __launch_bounds__(512, 3) pr_relabel(PullParams p)
{
    __shared__ PullTable s_t;
    // pr_classes' finding; one of this launch may already be seen, and ends it.
    if (__syncthreads_or(__ldcg(&p.st->asymmetric) | __ldcg(&p.st->outside))) return;
    pull_table(p.st, s_t);
    const unsigned lane = threadIdx.x & 31;
    const unsigned gwarp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nwarps = (gridDim.x * blockDim.x) >> 5;
    const unsigned nhub = pull_hubs(s_t.active);
    unsigned long long hash = 0;
    bool outside = false;
    pull_segments(s_t, gwarp, nwarps, lane, [&](unsigned c, unsigned r, uint32_t j0, uint32_t j1, unsigned l,
                                                unsigned s) {
        const uint32_t q = s_t.quads[c];
        const uint32_t u = __ldg(p.perm + s_t.first[c] + r);
        const uint32_t start = __ldg(p.row_start + u), deg = __ldg(p.row_start + u + 1) - start;
        uint4 *out = p.quads + s_t.quad0[c] + (size_t)r * q;
        for (uint32_t j = j0 + l; j < j1; j += s) {
            uint32_t d[4], e[4];
#pragma unroll
            for (int k = 0; k < 4; k++) d[k] = 4 * j + k < deg ? __ldcs(p.edge_dst + start + 4 * j + k) : 0xFFFFFFFFu;
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const bool in = d[k] < p.nnodes;
                e[k] = 4u * (in ? pull_place(__ldg(p.number + d[k]), nhub) : nhub);
                if (4 * j + k < deg) {
                    outside |= !in;
                    if (d[k] != u) hash += u < d[k] ? pull_pair_hash(u, d[k]) : 0ull - pull_pair_hash(u, d[k]);
                }
            }
            __stcs(out + j, make_uint4(e[0], e[1], e[2], e[3]));
        }
    });
    if (outside) p.st->outside = 1;
    warp_add_u64(&p.st->hash, hash, lane);
}

// ---------------------------------------------------------------------------
// Sweeps
// ---------------------------------------------------------------------------
struct PullSweep {
    const char *hub;   // shared memory: y[0, nhub], the last one 0
    unsigned hub_end;  // byte offset of that zero
    const char *y;     // this sweep's values
    float *yn, *xo;    // next values; x(k-1), replaced by x(k+1)
    const float *xc, *inv_deg;
    unsigned nhub;
    float omega;
    bool moved;

    // One of the two terms is the value and the other 0: no branch, so all
    // of a lane's gathers are in flight together.  y changes between sweeps
    // (the grid barrier's acquire drops the SM's L1 lines), never within one.
    __device__ __forceinline__ float at(uint32_t off) const
    {
        float g = 0.f;
        asm volatile("{\n\t.reg .pred p;\n\tsetp.gt.u32 p, %1, %2;\n\t@p ld.global.ca.f32 %0, [%3];\n\t}"
                     : "+f"(g)
                     : "r"(off), "r"(hub_end), "l"(y + off));
        return *reinterpret_cast<const float *>(hub + min(off, hub_end)) + g;
    }
    __device__ __forceinline__ float sum(const uint4 &e) const
    {
        const float a = at(e.x), b = at(e.y), c = at(e.z), d = at(e.w);
        return (a + b) + (c + d);
    }
    __device__ __forceinline__ void finish(uint32_t i, float s, float old, float cur, float inv)
    {
        const float xr = (float)(1.0 - kPullAlpha) + (float)kPullAlpha * s;
        const float xn = old + omega * (xr - old);
        xo[i] = xn;
        yn[pull_place(i, nhub)] = xn * inv;
        moved |= fmaxf(fabsf(xr - cur), fabsf(xn - cur)) > kPullEpsilon * fmaxf(1.f, xn);
    }
};

// Chunks k0, k0 + step, ... below k1, of 32 / S rows of one class of q <= 4 * S
// quads: S lanes per row, U rows per group of lanes at once, up to four
// quads per lane.  A lane's sum has at most 16 terms and a row's 256: 32-bit
// sums in a tree.
template <int S, int U>
__device__ __forceinline__ void pull_rows(PullSweep &sw, unsigned first, unsigned rows, uint32_t q, const uint4 *quads,
                                          unsigned k0, unsigned k1, unsigned step, unsigned lane)
{
    constexpr unsigned per = 32 / S;
    const unsigned l = lane % S;
    const uint4 pad = make_uint4(sw.hub_end, sw.hub_end, sw.hub_end, sw.hub_end);
    for (unsigned k = k0; k < k1; k += step * U) {
        unsigned r[U];
        uint4 e[U];
        float acc[U], old[U], cur[U], inv[U];
#pragma unroll
        for (int u = 0; u < U; u++) {
            r[u] = (k + u * step) * per + lane / S;
            const bool has = k + u * step < k1 && r[u] < rows;
            if (!has) r[u] = rows;
            e[u] = has && l < q ? __ldcs(quads + (size_t)r[u] * q + l) : pad;
            old[u] = cur[u] = inv[u] = 0.f;
            if (l == 0 && has) {
                old[u] = __ldcg(sw.xo + first + r[u]);
                cur[u] = __ldcg(sw.xc + first + r[u]);
                inv[u] = __ldcs(sw.inv_deg + first + r[u]);
            }
        }
        if (S < 4) {  // a quad per lane
#pragma unroll
            for (int u = 0; u < U; u++) acc[u] = sw.sum(e[u]);
        } else {
            uint4 e1[U], e2[U], e3[U];
            const bool two = q > S, three = q > 2 * S, four = q > 3 * S;  // the same for the class
#pragma unroll
            for (int u = 0; u < U; u++) {
                const uint4 *row = quads + (size_t)r[u] * q;
                const bool has = r[u] < rows;
                e1[u] = two && has && l + S < q ? __ldcs(row + l + S) : pad;
                e2[u] = three && has && l + 2 * S < q ? __ldcs(row + l + 2 * S) : pad;
                e3[u] = four && has && l + 3 * S < q ? __ldcs(row + l + 3 * S) : pad;
            }
#pragma unroll
            for (int u = 0; u < U; u++) acc[u] = sw.sum(e[u]);
            if (two) {
#pragma unroll
                for (int u = 0; u < U; u++) acc[u] += sw.sum(e1[u]);
            }
            if (three) {
#pragma unroll
                for (int u = 0; u < U; u++) acc[u] += sw.sum(e2[u]);
            }
            if (four) {
#pragma unroll
                for (int u = 0; u < U; u++) acc[u] += sw.sum(e3[u]);
            }
        }
#pragma unroll
        for (int u = 0; u < U; u++) {
#pragma unroll
            for (int o = S / 2; o > 0; o >>= 1) acc[u] += __shfl_xor_sync(kFull, acc[u], o);
            if (l == 0 && r[u] < rows) sw.finish(first + r[u], acc[u], old[u], cur[u], inv[u]);
        }
    }
}

// Rows r0, r0 + step, ... below r1 of more quads, a warp per row, four quads per lane at once
// (fewer in the last turn); the turns' sums are added in 64 bits.
__device__ __forceinline__ void pull_long_rows(PullSweep &sw, unsigned first, unsigned r0, unsigned r1, unsigned step,
                                               uint32_t q, const uint4 *quads, unsigned lane)
{
    const uint4 pad = make_uint4(sw.hub_end, sw.hub_end, sw.hub_end, sw.hub_end);
    for (unsigned r = r0; r < r1; r += step) {
        const uint4 *row = quads + (size_t)r * q;
        float old = 0.f, cur = 0.f, inv = 0.f;
        if (lane == 0) {
            old = __ldcg(sw.xo + first + r);
            cur = __ldcg(sw.xc + first + r);
            inv = __ldcs(sw.inv_deg + first + r);
        }
        double acc = 0;
        for (uint32_t j = 0; j < q; j += 128) {
            uint4 e[4];
#pragma unroll
            for (int v = 0; v < 4; v++) e[v] = j + 32 * v + lane < q ? __ldcs(row + j + 32 * v + lane) : pad;
            float s = sw.sum(e[0]);
#pragma unroll
            for (int v = 1; v < 4; v++)
                if (j + 32 * v < q) s += sw.sum(e[v]);
            acc += s;
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(kFull, acc, o);
        if (lane == 0) sw.finish(first + r, (float)acc, old, cur, inv);
    }
}

// The sweeps' work list: the rows of the classes from c0 on, cut into units of
// about `target` quads, a warp's claim.  Rows of one size do not cost the
// same (their values are in shared memory, in L2 or in between), and warps
// that were dealt equal shares waited for the slowest at each sweep's
// barrier (22% of the warps' time, RMAT-21).
struct PullUnits {
    unsigned total;
    unsigned first[kPullClasses];  // first unit of each class
    unsigned chunks[kPullClasses];  // chunks (see pull_rows; a long row) per unit
};

__device__ __forceinline__ unsigned pull_chunks(uint32_t q, unsigned rows)
{
    const unsigned per = q > 64 ? 1u : 32 / pull_lanes(q);
    return (rows + per - 1) / per;
}

__device__ __forceinline__ void pull_units(const PullTable &t, unsigned c0, uint32_t target, PullUnits &u)
{
    if (threadIdx.x < 32) {  // 32 classes at a time, in order
        unsigned total = 0;
        for (unsigned b = c0; b < t.n; b += 32) {
            const unsigned c = b + threadIdx.x;
            unsigned units = 0;
            if (c < t.n) {
                const uint32_t q = t.quads[c];
                const unsigned size = max(1u, target / (q > 64 ? q : q * (32 / pull_lanes(q))));
                u.chunks[c] = size;
                units = (pull_chunks(q, t.rows[c]) + size - 1) / size;
            }
            const unsigned incl = warp_incl_sum(units, threadIdx.x);
            if (c < t.n) u.first[c] = total + incl - units;
            total += __shfl_sync(kFull, incl, 31);
        }
        if (threadIdx.x == 0) u.total = total;
    }
    __syncthreads();
}

__global__ void __launch_bounds__(kPullBlock, 1) pr_sweeps(PullParams p)
{
    extern __shared__ __align__(16) float s_hub[];
    __shared__ PullTable s_t;
    __shared__ PullUnits s_u;
    __shared__ double s_red[2][32];
    TraversalCtl *ctl = p.ctl;
    const unsigned lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned tid = blockIdx.x * kPullBlock + threadIdx.x, nthreads = gridDim.x * kPullBlock;
    const unsigned gwarp = warp * gridDim.x + blockIdx.x, nwarps = nthreads / 32;  // neighbours on different SMs
    GridSync gs{&ctl->barrier.v, u32_of(ctl->release), &ctl->error, &ctl->error_where, gridDim.x, 0, p.timeout_ns};
    // The launches before this one decided: every thread sees the same words
    // (a CTA that starts after tid 0's store still finds the cause).
    if ((__ldcg(&p.st->asymmetric) | __ldcg(&p.st->outside)) || __ldcg(&p.st->hash) != 0) {
        if (tid == 0) p.st->asymmetric = 1;
        return;
    }
    pull_table(p.st, s_t);
    const uint32_t n = s_t.active;
    const unsigned nhub = pull_hubs(n), zero = 4 * nhub;
    unsigned long long quads_total = 0;
    if (s_t.n) quads_total = (unsigned long long)s_t.quad0[s_t.n - 1] + (unsigned long long)s_t.rows[s_t.n - 1] * s_t.quads[s_t.n - 1];
    // A row of more than a quarter of a warp's share of the quads (at least
    // 512 quads, four steps of a warp) is summed by a whole CTA.
    const uint32_t giant = max(512u, (uint32_t)(quads_total / (4ull * nwarps)));
    // Units are claimed where rows differ.  On a graph of at most 32 edges a
    // vertex the chunks are dealt in turn: they cost the same, and units of a
    // few short rows would cost a claim each (1000^2 road grid: 0.48 ms
    // dealt, 0.97 ms claimed; RMAT-22: 16.2 ms dealt, 14.1 ms claimed; RMAT-11:
    // 0.65 and 0.23 ms).
    const bool skewed = s_t.n && s_t.quads[0] > kUniformDegree / 4;
    unsigned c0 = 0;
    while (c0 < s_t.n && s_t.quads[c0] >= giant) c0++;
    pull_units(s_t, c0, min(512u, max(32u, (uint32_t)(quads_total / (8ull * nwarps)))), s_u);

    // x(0): the share of a's flow that a vertex of its degree gets when every
    // vertex has the mean rank 1, a good guess for all that the
    // iteration then has to correct.
    const float per_edge = p.nedges ? (float)(kPullAlpha * (double)n / (double)p.nedges) : 0.f;
    for (uint32_t i = tid; i < n; i += nthreads) {
        const float inv = __ldcg(p.inv_deg + i);
        const float x = (float)(1.0 - kPullAlpha) + per_edge / inv;
        p.x[0][i] = x;
        p.x[1][i] = x;
        p.y[0][pull_place(i, nhub)] = x * inv;
    }
    if (threadIdx.x == 0) s_hub[nhub] = 0.f;  // the copies below end before it
    if (!gs.sync()) return;

    unsigned k = 0;
    double omega = 1.0;
    while (n && k < kPullMaxSweeps) {
        const unsigned cur = k & 1;
        const float *y = cur ? p.y[1] : p.y[0];
        PullSweep sw{reinterpret_cast<const char *>(s_hub), zero, reinterpret_cast<const char *>(y),
                     cur ? p.y[0] : p.y[1], cur ? p.x[0] : p.x[1], cur ? p.x[1] : p.x[0], p.inv_deg, nhub,
                     (float)omega, false};
        if (tid == 0) {
            p.st->moved[(k + 1) % 3] = 0;
            p.st->unit[(k + 1) % 3] = 0;
        }
        for (unsigned i = threadIdx.x * 4; i < nhub; i += kPullBlock * 4) {
            const float4 v = __ldcg(reinterpret_cast<const float4 *>(y + i));  // y holds a multiple of 4
            if (i + 4 <= nhub) {
                *reinterpret_cast<float4 *>(s_hub + i) = v;
            } else {
                s_hub[i] = v.x;
                if (i + 1 < nhub) s_hub[i + 1] = v.y;
                if (i + 2 < nhub) s_hub[i + 2] = v.z;
            }
        }
        __syncthreads();
        unsigned c = 0, dealt = 0, buf = 0;
        for (; c < s_t.n && s_t.quads[c] >= giant; c++) {  // a CTA per row
            const uint32_t q = s_t.quads[c];
            for (unsigned r = (blockIdx.x + gridDim.x - dealt) % gridDim.x; r < s_t.rows[c]; r += gridDim.x) {
                const uint4 *e = p.quads + s_t.quad0[c] + (size_t)r * q;
                double acc = 0;
                for (uint32_t j = threadIdx.x; j < q; j += 2 * kPullBlock) {
                    const uint4 a = __ldcs(e + j);
                    const uint4 b = j + kPullBlock < q ? __ldcs(e + j + kPullBlock) : make_uint4(zero, zero, zero, zero);
                    acc += sw.sum(a) + sw.sum(b);
                }
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(kFull, acc, o);
                if (lane == 0) s_red[buf][warp] = acc;
                __syncthreads();
                if (warp == 0) {
                    double s = s_red[buf][lane];
#pragma unroll
                    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(kFull, s, o);
                    const uint32_t i = s_t.first[c] + r;
                    if (lane == 0) sw.finish(i, (float)s, __ldcg(sw.xo + i), __ldcg(sw.xc + i), __ldcg(sw.inv_deg + i));
                }
                buf ^= 1;  // the other buffer's readers passed this row's barrier
            }
            dealt = (dealt + s_t.rows[c]) % gridDim.x;
        }
        const auto rows_of = [&](unsigned k0, unsigned k1, unsigned step) {  // chunks of class c
            const uint32_t q = s_t.quads[c], rows = s_t.rows[c], first = s_t.first[c];
            const uint4 *e = p.quads + s_t.quad0[c];
            const unsigned s = pull_lanes(q);
            if (q > 64) pull_long_rows(sw, first, k0, k1, step, q, e, lane);
            else if (s == 16) pull_rows<16, 1>(sw, first, rows, q, e, k0, k1, step, lane);
            else if (s == 8) pull_rows<8, 1>(sw, first, rows, q, e, k0, k1, step, lane);
            else if (s == 4) pull_rows<4, 2>(sw, first, rows, q, e, k0, k1, step, lane);
            else if (s == 2) pull_rows<2, 4>(sw, first, rows, q, e, k0, k1, step, lane);
            else pull_rows<1, 4>(sw, first, rows, q, e, k0, k1, step, lane);
        };
        if (skewed) {
            for (unsigned unit = gwarp; unit < s_u.total;) {
                while (c + 1 < s_t.n && unit >= s_u.first[c + 1]) c++;
                const unsigned size = s_u.chunks[c], k0 = (unit - s_u.first[c]) * size;
                rows_of(k0, min(pull_chunks(s_t.quads[c], s_t.rows[c]), k0 + size), 1);
                if (s_u.total <= nwarps) break;
                unsigned next = 0;
                if (lane == 0) next = nwarps + atomicAdd(&p.st->unit[k % 3], 1u);
                unit = __shfl_sync(kFull, next, 0);
            }
        } else {
            dealt = 0;
            for (; c < s_t.n; c++) {
                const unsigned chunks = pull_chunks(s_t.quads[c], s_t.rows[c]);
                rows_of((gwarp + nwarps - dealt) % nwarps, chunks, nwarps);
                dealt = (dealt + chunks) % nwarps;
            }
        }
        if (__any_sync(kFull, sw.moved) && lane == 0) *(volatile unsigned *)&p.st->moved[k % 3] = 1;
        if (!gs.sync()) return;
        const bool more = ld_relaxed_u32(&p.st->moved[k % 3]) != 0;
        k++;
        omega = k == 1 ? 2.0 / (2.0 - kPullAlpha * kPullAlpha) : 4.0 / (4.0 - kPullAlpha * kPullAlpha * omega);
        if (!more) break;
    }
    const float *x = (k & 1) ? p.x[1] : p.x[0];  // the first sweep wrote x[1], the second x[0], ...
    for (uint32_t i = tid; i < n; i += nthreads) p.rank[__ldg(p.perm + i)] = __ldcg(x + i);
    if (tid == 0) {
        ctl->levels = k;
        ctl->iterations = gs.epoch;
        ctl->edges = (unsigned long long)k * p.nedges;
        ctl->pushes = (unsigned long long)k * n;
    }
}

}  // namespace dev
}  // namespace gft
