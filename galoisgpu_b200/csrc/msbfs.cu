// msbfs.cu -- multi-source BFS (gft_msbfs): up to 256 BFS queries on one
// graph in one persistent, cooperative launch.  No counterpart in the
// reference, which runs one source per process.
//
// Every vertex carries a row of WP words of bits, one bit per source (WP =
// ceil(k / 32) rounded up to 1, 2, 4 or 8, so a row is one aligned vector
// load): `seen` (sources that reached it) and, per level L, the frontier
// plane F_L (sources that reached it exactly at level L).  The planes are the
// result: level(source i, v) is the L whose plane has bit i set at v, so
// recording levels costs no writes beyond the frontier itself, and
// gft_msbfs_levels turns one source's planes into the int32 level array
// gft_bfs would produce.
//
// Each level runs in one of two directions, chosen from the edges leaving
// the frontier (m_f) against the graph's edges (Beamer, Asanovic,
// Patterson, "Direction-Optimizing Breadth-First Search", SC 2012):
//   top-down  (m_f small): a warp per frontier vertex u ORs F_L[u] & ~seen[v]
//             into next[v] for each neighbour v, then a commit pass over
//             the touched vertices moves next -> F_{L+1} and seen;
//   bottom-up (m_f large): each vertex v ORs F_L[u] over its neighbours u,
//             restricted to the sources v still lacks, and stops once it has
//             them all.  A thread takes a vertex of at most kThreadDegree
//             edges (checking four edges at a time); the warp takes larger
//             ones together.  Uses v's out-edges as its in-edges, so it
//             requires a symmetric graph (flag GFT_MSBFS_SYMMETRIC); without
//             the flag every level runs top-down.
// A vertex of kHubDegree edges or more is a hub, whose edges all warps of the
// grid take in kHubEdges-edge chunks: with one warp per vertex most of a level
// was the grid waiting for the largest ones (256 sources on RMAT-20, levels
// of eight sources read back: 4.79 -> 1.50 ms, with the frontier rows reduced
// by one instruction per word instead of five shuffles, and the source set-up
// by a CTA instead of a thread).  Top-down, a hub stands on a list from the
// moment it joins the frontier, so its chunks are expanded beside the other
// vertices.  Bottom-up, the level itself finds the hubs that lack sources and
// scans them after one more barrier.
#include <string.h>

#include <algorithm>

#include "gft_internal.h"
#include "traverse.cuh"

namespace gft {
namespace dev {

constexpr uint32_t kThreadDegree = 32;  // bottom-up: larger vertices are scanned by the whole warp
constexpr uint32_t kHubDegree = 1024;   // either direction: larger vertices are scanned by the whole grid
constexpr uint32_t kHubEdges = 512;     // edges of a hub per warp step
// Bottom-up levels split hubs from this many sources on.  A hub that lacks few
// sources finds them among its first edges, and the split costs a barrier per
// level (RMAT-12, 14, 16, 18, 20 split / not, us: 8 sources 131/118, 157/134,
// 170/170, 218/231, 312/261; 32 sources 137/122, 159/146, 186/190, 236/303,
// 547/1001).
constexpr uint32_t kSplitSources = 16;

// A row of WP words of source bits.
template <int WP>
struct Bits {
    uint32_t w[WP];
    __device__ __forceinline__ void clear()
    {
#pragma unroll
        for (int i = 0; i < WP; i++) w[i] = 0;
    }
    __device__ __forceinline__ bool any() const
    {
        uint32_t a = 0;
#pragma unroll
        for (int i = 0; i < WP; i++) a |= w[i];
        return a != 0;
    }
    __device__ __forceinline__ bool covers(const Bits &need) const
    {
        bool c = true;
#pragma unroll
        for (int i = 0; i < WP; i++) c &= (w[i] & need.w[i]) == need.w[i];
        return c;
    }
};

// Row loads and stores as aligned vectors (the row of v starts at v * WP
// words; the arrays are 16-byte aligned).
template <int WP>
__device__ __forceinline__ Bits<WP> ld_row(const uint32_t *base, uint32_t v)
{
    Bits<WP> b;
    const uint32_t *p = base + (size_t)v * WP;
    if constexpr (WP == 8) {
        const uint4 a = __ldcg(reinterpret_cast<const uint4 *>(p)), c = __ldcg(reinterpret_cast<const uint4 *>(p) + 1);
        b.w[0] = a.x, b.w[1] = a.y, b.w[2] = a.z, b.w[3] = a.w, b.w[4] = c.x, b.w[5] = c.y, b.w[6] = c.z, b.w[7] = c.w;
    } else if constexpr (WP == 4) {
        const uint4 a = __ldcg(reinterpret_cast<const uint4 *>(p));
        b.w[0] = a.x, b.w[1] = a.y, b.w[2] = a.z, b.w[3] = a.w;
    } else if constexpr (WP == 2) {
        const uint2 a = __ldcg(reinterpret_cast<const uint2 *>(p));
        b.w[0] = a.x, b.w[1] = a.y;
    } else {
        b.w[0] = __ldcg(p);
    }
    return b;
}

template <int WP>
__device__ __forceinline__ void st_row(uint32_t *base, uint32_t v, const Bits<WP> &b)
{
    uint32_t *p = base + (size_t)v * WP;
    if constexpr (WP == 8) {
        reinterpret_cast<uint4 *>(p)[0] = make_uint4(b.w[0], b.w[1], b.w[2], b.w[3]);
        reinterpret_cast<uint4 *>(p)[1] = make_uint4(b.w[4], b.w[5], b.w[6], b.w[7]);
    } else if constexpr (WP == 4) {
        reinterpret_cast<uint4 *>(p)[0] = make_uint4(b.w[0], b.w[1], b.w[2], b.w[3]);
    } else if constexpr (WP == 2) {
        reinterpret_cast<uint2 *>(p)[0] = make_uint2(b.w[0], b.w[1]);
    } else {
        p[0] = b.w[0];
    }
}

struct MsParams {
    const uint32_t *__restrict__ row_start;
    const uint32_t *__restrict__ edge_dst;
    uint32_t nnodes, nedges;
    uint32_t k;                // sources
    const uint32_t *sources;   // device copy, k entries
    uint32_t *planes;          // (max_levels) x nnodes x WP words
    uint32_t max_levels;
    uint32_t *seen, *next;     // nnodes x WP words each (next zeroed)
    uint32_t *queue[2];        // frontier vertices per level
    uint32_t *touched;         // top-down: vertices given new bits
    uint32_t *tstamp;          // top-down: level + 1 at which v was last touched
    uint2 *hubs;               // bottom-up: (vertex, first chunk) of the level's hubs
    uint2 *fhubs[2];           // the same of the frontier's hubs, by level
    uint32_t hub_cap;
    uint32_t split_hubs;       // bottom-up: hubs are scanned by the whole grid
    uint32_t max_share;        // top-down: warps that at most share a frontier vertex
    uint32_t symmetric;
    uint32_t alpha;            // bottom-up when m_f * alpha > nedges
    TraversalCtl *ctl;
    unsigned long long timeout_ns;
};

// Bits of all k sources.
template <int WP>
__device__ __forceinline__ Bits<WP> all_sources(uint32_t k)
{
    Bits<WP> b;
#pragma unroll
    for (int i = 0; i < WP; i++)
        b.w[i] = 32u * (i + 1) <= k ? ~0u : (32u * i >= k ? 0u : (1u << (k % 32)) - 1u);
    return b;
}

// The sources that `need` lacks and that stand in frontier rows of the edges
// [s, e), gathered by the whole warp; ends once all of them are found.  The
// same result in every lane.
template <int WP>
__device__ __forceinline__ Bits<WP> warp_gather(const MsParams &p, const uint32_t *F, uint32_t s, uint32_t e,
                                                const Bits<WP> &need, unsigned lane)
{
    constexpr int kFly = WP >= 8 ? 2 : 4;  // rows a lane has in flight
    Bits<WP> a;
    a.clear();
    for (uint32_t b = s; b < e; b += 32 * kFly) {
        uint32_t u[kFly];
#pragma unroll
        for (int k = 0; k < kFly; k++) {
            const uint32_t i = b + 32 * k + lane;
            u[k] = i < e ? __ldcs(p.edge_dst + i) : 0xFFFFFFFFu;
        }
        Bits<WP> f[kFly];
#pragma unroll
        for (int k = 0; k < kFly; k++) {
            f[k].clear();
            if (u[k] != 0xFFFFFFFFu) f[k] = ld_row<WP>(F, u[k]);
        }
#pragma unroll
        for (int w = 0; w < WP; w++) {
            uint32_t x = 0;
#pragma unroll
            for (int k = 0; k < kFly; k++) x |= f[k].w[w];
            a.w[w] |= __reduce_or_sync(kFull, x & need.w[w]);
        }
        if (a.covers(need)) break;  // warp uniform after the reduction
    }
    return a;
}

// Top-down: ORs the frontier row of u into next[v] for the edges [s, e),
// `step` edges apart per turn of the warp.
template <int WP>
__device__ __forceinline__ void warp_scatter(const MsParams &p, const Bits<WP> &fu, uint32_t s, uint32_t e,
                                             uint32_t step, uint32_t stamp, WarpQueue &tq, unsigned lane)
{
    for (uint32_t eb = s; eb < e; eb += step) {  // warp-uniform trip count
        const uint32_t ei = eb + lane;
        bool touched = false;
        uint32_t v = 0;
        if (ei < e) {
            v = __ldcs(p.edge_dst + ei);
            const Bits<WP> sv = ld_row<WP>(p.seen, v);
#pragma unroll
            for (int w = 0; w < WP; w++) {
                const uint32_t b = fu.w[w] & ~sv.w[w];
                if (b) {
                    atomicOr(p.next + (size_t)v * WP + w, b);
                    touched = true;
                }
            }
            touched = touched && atomicExch(p.tstamp + v, stamp) != stamp;
        }
        tq.push(touched, v, lane);
    }
}

// Puts the v of the lanes with `is` on a hub list, with one reservation per
// warp: a level of a skewed graph can list thousands.  Not inlined: its
// registers would cost the levels spills.
static __device__ __noinline__ void append_hubs(uint2 *hubs, uint32_t hub_cap, TraversalCtl *ctl,
                                                unsigned long long *hub_ctr, bool is, uint32_t v, uint32_t deg,
                                                unsigned lane)
{
    const unsigned mask = __ballot_sync(kFull, is);
    const unsigned nch = is ? (deg + kHubEdges - 1) / kHubEdges : 0u;
    const unsigned incl = warp_incl_sum(nch, lane);
    unsigned long long old = 0;
    if (lane == 31) old = atomicAdd(hub_ctr, ((unsigned long long)__popc(mask) << 32) | incl);
    old = __shfl_sync(kFull, old, 31);
    const unsigned h = (unsigned)(old >> 32) + __popc(mask & lanemask_lt());
    if (!is) return;
    if (h < hub_cap) hubs[h] = make_uint2(v, (unsigned)old + incl - nch);
    else raise_error(&ctl->error, &ctl->error_where, GFT_ERR_OVERFLOW, h);
}

__device__ __forceinline__ void list_hubs(const MsParams &p, uint2 *hubs, unsigned long long *hub_ctr, bool is,
                                          uint32_t v, uint32_t deg, unsigned lane)
{
    if (__any_sync(kFull, is)) append_hubs(hubs, p.hub_cap, p.ctl, hub_ctr, is, v, deg, lane);
}

// The grid's warps dealt to n items: `share` of them to each (at most
// max_share) while the items are fewer than the warps.
struct WarpShare {
    unsigned share = 1, first, step, part = 0;
    __device__ __forceinline__ WarpShare(unsigned max_share, unsigned n, unsigned gwarp, unsigned nwarps)
        : first(gwarp), step(nwarps)
    {
        if (max_share == 1 || 2 * n > nwarps || n == 0) return;
        share = min(max_share, nwarps / n);
        first = gwarp / share;
        step = nwarps / share;  // at least n: the warps left over have nothing
        part = gwarp % share;
    }
};

// Calls f(vertex, first edge, end, ws) for the chunks of a hub list that
// `ws` deals to this warp.
template <class F>
__device__ __forceinline__ void for_hub_chunks(const MsParams &p, const uint2 *hubs, unsigned long long hv,
                                               const WarpShare &ws, F &&f)
{
    const unsigned nh = (unsigned)(hv >> 32), nc = (unsigned)hv;
    for (unsigned c = ws.first; c < nc; c += ws.step) {
        unsigned lo = 0, hi = nh;
        while (hi - lo > 1) {
            const unsigned mid = (lo + hi) >> 1;
            if (__ldcg(&hubs[mid].y) <= c) lo = mid;
            else hi = mid;
        }
        const uint2 hb = __ldcg(hubs + lo);
        const uint32_t s = __ldg(p.row_start + hb.x), e = __ldg(p.row_start + hb.x + 1);
        const uint32_t at = s + (c - hb.y) * kHubEdges;
        f(hb.x, at, min(e, at + kHubEdges), ws);
    }
}

// kHubs: some vertex has kHubDegree edges or more.  Without, a level has no
// hub step: with one in every level, road 512^2 took 1.62 ms instead of 1.20
// and grid 256^2 5.32 instead of 3.89 (one source; part of it frontiers of a
// few vertices shared by every warp of the grid, see max_share).
template <int WP, bool kHubs>
__global__ void __launch_bounds__(512, 2) msbfs_kernel(MsParams p)
{
    constexpr int BLOCK = 512;
    constexpr int kStep = WP >= 8 ? 2 : 4;  // edges a thread checks at once in bottom-up levels
    TraversalCtl *ctl = p.ctl;
    const unsigned lane = threadIdx.x & 31;
    const unsigned tid = blockIdx.x * BLOCK + threadIdx.x, nthreads = gridDim.x * BLOCK;
    const unsigned gwarp = tid / 32, nwarps = nthreads / 32;
    GridSync gs{&ctl->barrier.v, u32_of(ctl->release), &ctl->error, &ctl->error_where, gridDim.x, 0, p.timeout_ns};
    const uint32_t n = p.nnodes;
    const size_t plane_words = (size_t)n * WP;
    // Warp-aggregated appends (one reservation per flush) for the next
    // frontier and the top-down touched list.
    __shared__ uint32_t s_next[BLOCK / 32][kQueueBuf];
    __shared__ uint32_t s_touch[BLOCK / 32][kQueueBuf];
    WarpQueue nq{s_next[threadIdx.x >> 5], 0, nullptr, nullptr, n, &ctl->error, &ctl->error_where};
    WarpQueue tq{s_touch[threadIdx.x >> 5], 0, p.touched, nullptr, n, &ctl->error, &ctl->error_where};
    const Bits<WP> all = all_sources<WP>(p.k);
    // counters: qlen[slot] frontier size, claim[slot] touched count,
    // hub[slot].v frontier edge count m_f.

    // Level 0: the sources themselves.
    for (size_t i = tid; i < plane_words; i += nthreads) {
        p.seen[i] = 0;
        p.planes[i] = 0;
    }
    if (!gs.sync()) return;
    if (blockIdx.x == 0) {  // a thread per source; k <= 256
        __shared__ uint32_t s_src[256];
        __shared__ unsigned s_n;
        const uint32_t i = threadIdx.x;
        if (i < p.k) s_src[i] = p.sources[i];
        if (i == 0) s_n = 0;
        __syncthreads();
        unsigned long long mf = 0;
        if (i < p.k) {
            const uint32_t s = s_src[i];
            atomicOr(p.seen + (size_t)s * WP + i / 32, 1u << (i % 32));
            atomicOr(p.planes + (size_t)s * WP + i / 32, 1u << (i % 32));
            bool dup = false;
            for (uint32_t j = 0; j < i; j++) dup |= s_src[j] == s;
            if (!dup) {
                p.queue[0][atomicAdd(&s_n, 1u)] = s;
                mf = p.row_start[s + 1] - p.row_start[s];
            }
        }
        if (kHubs)
            list_hubs(p, p.fhubs[0], &ctl->hub_claim[0].v, mf >= kHubDegree, s_src[i % 256], (uint32_t)mf, lane);
        warp_add_u64(&ctl->hub[0].v, mf, lane);
        __syncthreads();
        if (i == 0) *u32_of(ctl->qlen[0]) = s_n;
    }
    if (!gs.sync()) return;

    uint32_t L = 0;
    for (;;) {
        const unsigned slot = L % 3, nslot = (L + 1) % 3, rslot = (L + 2) % 3;
        const uint32_t nf = ld_relaxed_u32(u32_of(ctl->qlen[slot]));
        if (nf == 0) break;
        if (L + 1 >= p.max_levels) {
            if (tid == 0) raise_error(&ctl->error, &ctl->error_where, GFT_ERR_OVERFLOW, L + 1);
            gs.sync();
            return;
        }
        const unsigned long long mf = ld_relaxed_u64(&ctl->hub[slot].v);
        if (tid == 0) {
            *u32_of(ctl->qlen[rslot]) = 0;
            *u32_of(ctl->claim[rslot]) = 0;
            ctl->hub[rslot].v = 0;
            ctl->handoff[rslot].v = 0;
            ctl->hub_claim[rslot].v = 0;
        }
        // (hubs << 32) | chunks: those a bottom-up level finds, and those of
        // the next frontier.
        unsigned long long *hub_ctr = &ctl->handoff[slot].v, *fhub_next = &ctl->hub_claim[nslot].v;
        uint2 *fhubs_next = (L & 1) ? p.fhubs[0] : p.fhubs[1];
        const uint32_t *F = p.planes + (size_t)L * plane_words;
        uint32_t *Fn = p.planes + (size_t)(L + 1) * plane_words;
        nq.queue = ((L + 1) & 1) ? p.queue[1] : p.queue[0];  // no dynamic index: keeps p out of local memory
        nq.len = u32_of(ctl->qlen[nslot]);
        tq.len = u32_of(ctl->claim[slot]);
        unsigned long long my_mf = 0;
        const bool bottom_up = p.symmetric && mf * p.alpha > p.nedges;
        if (bottom_up) {
            // Dense pass over 32-vertex blocks: every vertex's next plane row
            // is written (0 when nothing new), so the plane needs no clearing.
            for (uint32_t b0 = gwarp * 32; b0 < n; b0 += nwarps * 32) {  // warp-uniform trip count
                const uint32_t v = b0 + lane;
                Bits<WP> need, acc;
                need.clear();
                acc.clear();
                uint32_t s = 0, e = 0;
                if (v < n) {
                    const Bits<WP> sv = ld_row<WP>(p.seen, v);
#pragma unroll
                    for (int i = 0; i < WP; i++) need.w[i] = all.w[i] & ~sv.w[i];
                    if (need.any()) {
                        s = __ldg(p.row_start + v);
                        e = __ldg(p.row_start + v + 1);
                    }
                }
                bool hub = false;
                if (kHubs && p.split_hubs) {  // a hub's row is written after the hub phase
                    hub = e - s >= kHubDegree;
                    list_hubs(p, p.hubs, hub_ctr, hub, v, e - s, lane);
                    if (hub) e = s;
                }
                const bool heavy = e - s > kThreadDegree;
                if (!heavy) {  // this thread's own vertex, kStep edges at a time
                    for (uint32_t i = s; i < e; i += kStep) {
                        uint32_t u[kStep];
#pragma unroll
                        for (int k = 0; k < kStep; k++) u[k] = i + k < e ? __ldcs(p.edge_dst + i + k) : 0xFFFFFFFFu;
#pragma unroll
                        for (int k = 0; k < kStep; k++)
                            if (u[k] != 0xFFFFFFFFu) {
                                const Bits<WP> f = ld_row<WP>(F, u[k]);
#pragma unroll
                                for (int w = 0; w < WP; w++) acc.w[w] |= f.w[w] & need.w[w];
                            }
                        if (acc.covers(need)) break;
                    }
                }
                // The whole warp scans each heavy vertex of the block in turn.
                unsigned hm = __ballot_sync(kFull, heavy);
                while (hm) {
                    const int j = __ffs(hm) - 1;
                    hm &= hm - 1;
                    const uint32_t sj = __shfl_sync(kFull, s, j), ej = __shfl_sync(kFull, e, j);
                    Bits<WP> nj;
#pragma unroll
                    for (int w = 0; w < WP; w++) nj.w[w] = __shfl_sync(kFull, need.w[w], j);
                    const Bits<WP> a = warp_gather<WP>(p, F, sj, ej, nj, lane);
                    if ((int)lane == j) acc = a;
                }
                const bool got = acc.any();
                if (v < n && !hub) {
                    st_row<WP>(Fn, v, acc);
                    if (got) {
                        Bits<WP> s2;
#pragma unroll
                        for (int i = 0; i < WP; i++) s2.w[i] = (all.w[i] & ~need.w[i]) | acc.w[i];
                        st_row<WP>(p.seen, v, s2);
                        my_mf += e - s;
                    }
                }
                if (kHubs && !p.split_hubs)
                    list_hubs(p, fhubs_next, fhub_next, got && e - s >= kHubDegree, v, e - s, lane);
                nq.push(got, v, lane);
            }
            unsigned long long hv = 0;
            if (kHubs && p.split_hubs) {
                if (!gs.sync()) return;
                hv = ld_relaxed_u64(hub_ctr);
            }
            if (hv) {
                const WarpShare ws(1, (unsigned)hv, gwarp, nwarps);
                for_hub_chunks(p, p.hubs, hv, ws, [&](uint32_t v, uint32_t s, uint32_t e, const WarpShare &) {
                    const Bits<WP> sv = ld_row<WP>(p.seen, v);
                    Bits<WP> need;
#pragma unroll
                    for (int i = 0; i < WP; i++) need.w[i] = all.w[i] & ~sv.w[i];
                    const Bits<WP> a = warp_gather<WP>(p, F, s, e, need, lane);
#pragma unroll
                    for (int i = 0; i < WP; i++)
                        if (lane == i && a.w[i]) atomicOr(p.next + (size_t)v * WP + i, a.w[i]);
                });
                if (!gs.sync()) return;
                const unsigned nh = (unsigned)(hv >> 32);
                for (unsigned b = gwarp * 32; b < nh; b += nwarps * 32) {  // warp-uniform trip count
                    bool got = false;
                    uint32_t v = 0, deg = 0;
                    if (b + lane < nh) {
                        v = __ldcg(&p.hubs[b + lane].x);
                        const Bits<WP> nb = ld_row<WP>(p.next, v);  // the sources it lacked
                        got = nb.any();
                        st_row<WP>(Fn, v, nb);
                        if (got) {
                            Bits<WP> z, sv = ld_row<WP>(p.seen, v);
                            z.clear();
                            st_row<WP>(p.next, v, z);
#pragma unroll
                            for (int i = 0; i < WP; i++) sv.w[i] |= nb.w[i];
                            st_row<WP>(p.seen, v, sv);
                            deg = __ldg(p.row_start + v + 1) - __ldg(p.row_start + v);
                            my_mf += deg;
                        }
                    }
                    list_hubs(p, fhubs_next, fhub_next, got, v, deg, lane);
                    nq.push(got, v, lane);
                }
            }
        } else {
            // Top-down: clear the next plane, expand, commit.
            for (size_t i = tid; i < plane_words; i += nthreads) Fn[i] = 0;
            if (!gs.sync()) return;
            const uint32_t *q = (L & 1) ? p.queue[1] : p.queue[0];
            // A frontier of fewer vertices than warps gives each vertex
            // several warps, up to one per 32 edges.
            const WarpShare ws(p.max_share, nf, gwarp, nwarps);
            for (uint32_t qi = ws.first; qi < nf; qi += ws.step) {
                const uint32_t u = __ldcg(q + qi);
                const uint32_t s = __ldg(p.row_start + u), e = __ldg(p.row_start + u + 1);
                if (kHubs && e - s >= kHubDegree) continue;  // on the list
                warp_scatter<WP>(p, ld_row<WP>(F, u), s + ws.part * 32, e, 32 * ws.share, L + 1, tq, lane);
            }
            if (kHubs) {
                const unsigned long long hv = ld_relaxed_u64(&ctl->hub_claim[slot].v);
                for_hub_chunks(p, (L & 1) ? p.fhubs[1] : p.fhubs[0], hv,
                               WarpShare(kHubEdges / 32, (unsigned)hv, nwarps - 1 - gwarp, nwarps),
                               [&](uint32_t u, uint32_t s, uint32_t e, const WarpShare &w) {
                                   warp_scatter<WP>(p, ld_row<WP>(F, u), s + w.part * 32, e, 32 * w.share, L + 1, tq,
                                                    lane);
                               });
            }
            tq.flush(lane);
            if (!gs.sync()) return;
            const uint32_t nt = ld_relaxed_u32(u32_of(ctl->claim[slot]));
            for (uint32_t b = gwarp * 32; b < nt; b += nwarps * 32) {  // warp-uniform trip count
                const uint32_t ti = b + lane;
                bool got = false;
                uint32_t v = 0, deg = 0;
                if (ti < nt) {
                    v = __ldcg(p.touched + ti);
                    Bits<WP> nb = ld_row<WP>(p.next, v);
                    const Bits<WP> sv = ld_row<WP>(p.seen, v);
#pragma unroll
                    for (int w = 0; w < WP; w++) nb.w[w] &= ~sv.w[w];
                    Bits<WP> z;
                    z.clear();
                    st_row<WP>(p.next, v, z);
                    if (nb.any()) {
                        st_row<WP>(Fn, v, nb);
                        Bits<WP> s2;
#pragma unroll
                        for (int w = 0; w < WP; w++) s2.w[w] = sv.w[w] | nb.w[w];
                        st_row<WP>(p.seen, v, s2);
                        got = true;
                        deg = p.row_start[v + 1] - p.row_start[v];
                        my_mf += deg;
                    }
                }
                if (kHubs) list_hubs(p, fhubs_next, fhub_next, got && deg >= kHubDegree, v, deg, lane);
                nq.push(got, v, lane);
            }
        }
        nq.flush(lane);
        warp_add_u64(&ctl->hub[nslot].v, my_mf, lane);
        if (!gs.sync()) return;
        L++;
    }
    if (tid == 0) {
        ctl->levels = L;  // planes 0..L-1 hold the levels
        ctl->iterations = gs.epoch;
    }
}

// Level of source i at every vertex, from the planes (rows of wp words).
__global__ void msbfs_levels_kernel(const uint32_t *__restrict__ planes, uint32_t nnodes, uint32_t wp,
                                    uint32_t levels, uint32_t i, int32_t *out)
{
    const uint32_t w = i / 32, bit = 1u << (i % 32);
    const size_t plane_words = (size_t)nnodes * wp;
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < nnodes; v += gridDim.x * blockDim.x) {
        int32_t lv = 0x7FFFFFFF;
        for (uint32_t L = 0; L < levels; L++)
            if (planes[(size_t)L * plane_words + (size_t)v * wp + w] & bit) {
                lv = (int32_t)L;
                break;
            }
        out[v] = lv;
    }
}

}  // namespace dev
}  // namespace gft

using namespace gft;

namespace {

// Words per vertex row for k sources: ceil(k / 32) rounded up to a power of
// two, so every row is one aligned vector.
uint32_t row_words(uint32_t k)
{
    const uint32_t w = (k + 31) / 32;
    return w <= 1 ? 1 : w <= 2 ? 2 : w <= 4 ? 4 : 8;
}

template <bool kHubs>
const void *msbfs_kernel_for(uint32_t wp)
{
    switch (wp) {
    case 1: return (const void *)dev::msbfs_kernel<1, kHubs>;
    case 2: return (const void *)dev::msbfs_kernel<2, kHubs>;
    case 4: return (const void *)dev::msbfs_kernel<4, kHubs>;
    case 8: return (const void *)dev::msbfs_kernel<8, kHubs>;
    }
    return nullptr;
}

}  // namespace

extern "C" {

size_t gft_msbfs_plane_bytes(uint32_t nnodes, uint32_t k)
{
    return (size_t)nnodes * row_words(k) * 4;
}

gft_status gft_msbfs(gft_engine *e, const gft_graph *g, const uint32_t *h_sources, uint32_t k, uint32_t *d_planes,
                     uint32_t max_levels, uint32_t flags, void *stream_, gft_stats *stats)
{
    if (!e || !g || !h_sources || !d_planes) return fail(GFT_ERR_INVALID_ARG, "gft_msbfs: null argument");
    if (k == 0 || k > 256) return fail(GFT_ERR_INVALID_ARG, "gft_msbfs: k must be 1..256 (got %u)", k);
    if (max_levels < 2) return fail(GFT_ERR_INVALID_ARG, "gft_msbfs: max_levels must be >= 2");
    if ((uintptr_t)d_planes % 16 != 0) return fail(GFT_ERR_INVALID_ARG, "gft_msbfs: d_planes must be 16-byte aligned");
    std::lock_guard<std::mutex> lk(e->mu);
    GFT_TRY(check_engine_graph(e, g));
    const DeviceGraph &G = g->g;
    for (uint32_t i = 0; i < k; i++)
        if (h_sources[i] >= G.nnodes) return fail(GFT_ERR_INVALID_ARG, "gft_msbfs: source %u out of range", i);
    cudaStream_t stream = (cudaStream_t)stream_;
    DeviceScope device_scope(e->device);
    GFT_CUDA_TRY(device_scope.err);
    const uint32_t WP = row_words(k);
    const size_t vwords = (size_t)G.nnodes * WP;
    auto a256 = [](size_t x) { return (x + 255) & ~(size_t)255; };
    size_t off = 0;
    auto take = [&](size_t bytes) {
        size_t o = off;
        off += a256(bytes);
        return o;
    };
    const size_t o_seen = take(vwords * 4), o_next = take(vwords * 4), o_q0 = take((size_t)G.nnodes * 4),
                 o_q1 = take((size_t)G.nnodes * 4), o_t = take((size_t)G.nnodes * 4),
                 o_ts = take((size_t)G.nnodes * 4), o_src = take((size_t)k * 4);
    const uint32_t hub_cap = G.nedges / dev::kHubDegree + 1;
    const size_t o_hubs = take((size_t)hub_cap * sizeof(uint2)), o_fhubs0 = take((size_t)hub_cap * sizeof(uint2)),
                 o_fhubs1 = take((size_t)hub_cap * sizeof(uint2));
    GFT_TRY(e->scratch.ensure(off));
    char *base = static_cast<char *>(e->scratch.ptr);
    const bool hubs = G.max_degree >= dev::kHubDegree;
    const void *kern = hubs ? msbfs_kernel_for<true>(WP) : msbfs_kernel_for<false>(WP);
    LaunchShape shape;
    GFT_TRY(resolve_shape(e, kern, 512, 2, 0, &shape));
    dev::MsParams p{};
    p.row_start = G.row_start;
    p.edge_dst = G.edge_dst;
    p.nnodes = G.nnodes;
    p.nedges = G.nedges;
    p.k = k;
    p.sources = reinterpret_cast<uint32_t *>(base + o_src);
    p.planes = d_planes;
    p.max_levels = max_levels;
    p.seen = reinterpret_cast<uint32_t *>(base + o_seen);
    p.next = reinterpret_cast<uint32_t *>(base + o_next);
    p.queue[0] = reinterpret_cast<uint32_t *>(base + o_q0);
    p.queue[1] = reinterpret_cast<uint32_t *>(base + o_q1);
    p.touched = reinterpret_cast<uint32_t *>(base + o_t);
    p.tstamp = reinterpret_cast<uint32_t *>(base + o_ts);
    p.hubs = reinterpret_cast<uint2 *>(base + o_hubs);
    p.fhubs[0] = reinterpret_cast<uint2 *>(base + o_fhubs0);
    p.fhubs[1] = reinterpret_cast<uint2 *>(base + o_fhubs1);
    p.hub_cap = hub_cap;
    p.split_hubs = k >= dev::kSplitSources;
    // More warps than a vertex has 32-edge steps would all read its queue
    // entry, row and plane row from L2 for nothing.
    p.max_share = std::max(1u, (std::min(G.max_degree, dev::kHubDegree) + 31) / 32);
    p.symmetric = (flags & GFT_MSBFS_SYMMETRIC) ? 1u : 0u;
    // Bottom-up once the frontier's edges exceed 1/64 of the graph's: a
    // bottom-up level checks a vertex's rows only until its sources are
    // covered, a top-down one pays atomics per edge for every source row.
    // 256 sources: RMAT-24 44.3 -> 42.8 ms and road 512^2 2.47 -> 2.28 ms
    // against 1/16 (Beamer et al.'s single-source value).
    p.alpha = 64;
    p.ctl = reinterpret_cast<TraversalCtl *>(e->ctl.ptr);
    p.timeout_ns = 20000ull * 1000000ull;
    GFT_CUDA_TRY(cudaMemcpyAsync(base + o_src, h_sources, (size_t)k * 4, cudaMemcpyHostToDevice, stream));
    GFT_CUDA_TRY(cudaMemsetAsync(base + o_next, 0, vwords * 4, stream));
    GFT_CUDA_TRY(cudaMemsetAsync(base + o_ts, 0, (size_t)G.nnodes * 4, stream));
    GFT_CUDA_TRY(cudaMemsetAsync(e->ctl.ptr, 0, sizeof(TraversalCtl), stream));
    void *args[] = {&p};
    GFT_CUDA_TRY(cudaEventRecord(e->ev0, stream));
    GFT_CUDA_TRY(cudaLaunchCooperativeKernel(kern, dim3(shape.blocks), dim3(512), args, 0, stream));
    GFT_CUDA_TRY(cudaEventRecord(e->ev1, stream));
    TraversalCtl *h = reinterpret_cast<TraversalCtl *>(e->host_ctl);
    const size_t cold = offsetof(TraversalCtl, error);
    GFT_CUDA_TRY(cudaMemcpyAsync(reinterpret_cast<char *>(h) + cold, reinterpret_cast<char *>(e->ctl.ptr) + cold,
                                 sizeof(TraversalCtl) - cold, cudaMemcpyDeviceToHost, stream));
    GFT_CUDA_TRY(cudaStreamSynchronize(stream));
    if (h->error)
        return fail((gft_status)h->error, "gft_msbfs: device reported %s (site %u)",
                    gft_status_string((gft_status)h->error), h->error_where);
    if (stats) {
        memset(stats, 0, sizeof *stats);
        float ms = 0;
        cudaEventElapsedTime(&ms, e->ev0, e->ev1);
        stats->levels = h->levels;
        stats->iterations = h->iterations;
        stats->kernel_ms = ms;
        stats->grid_blocks = shape.blocks;
        stats->block_threads = 512;
    }
    return GFT_OK;
}

gft_status gft_msbfs_levels(const uint32_t *d_planes, uint32_t nnodes, uint32_t k, uint32_t levels, uint32_t i,
                            int32_t *d_out, void *stream)
{
    if (!d_planes || !d_out || i >= k || k > 256) return fail(GFT_ERR_INVALID_ARG, "gft_msbfs_levels: bad argument");
    // Launch on the device that holds the planes, whatever device is current.
    cudaPointerAttributes attr;
    GFT_CUDA_TRY(cudaPointerGetAttributes(&attr, d_planes));
    if (attr.type != cudaMemoryTypeDevice && attr.type != cudaMemoryTypeManaged)
        return fail(GFT_ERR_INVALID_ARG, "gft_msbfs_levels: d_planes is not device memory");
    DeviceScope device_scope(attr.device);
    GFT_CUDA_TRY(device_scope.err);
    dev::msbfs_levels_kernel<<<1184, 256, 0, (cudaStream_t)stream>>>(d_planes, nnodes, row_words(k), levels, i, d_out);
    GFT_CUDA_TRY(cudaGetLastError());
    return GFT_OK;
}

}  // extern "C"
