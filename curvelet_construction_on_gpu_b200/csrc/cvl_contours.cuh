// cvl_contours.cuh -- downstream of the curvelet path: the edgel link graph and
// its contour fragments ("one-chains"), as the reference's original_code builds
// them from a curvelet map:
//   construct_the_link_graph / form_links_from_a_curvelet
//       (original_code/form_curvelet_process.cpp:453-520)
//   link_edgels / are_linked / edgel_is_legal_first_edgel / edgel_is_legal
//       (original_code/edgel_link_graph.hpp:207-265)
//   extract_one_chains_from_the_link_graph (form_curvelet_process.cpp:563-654)
//   curve_fragment_graph::insert_fragment / get_output_array (curve_fragment_graph.hpp)
//
// What decides the result:
//  * A link joins two edgels in either direction (are_linked looks both ways).
//    Its direction is the one of its first occurrence, in the order curvelets
//    are visited: anchors ascending, each anchor's curvelets in record order,
//    each chain's consecutive pairs in order. So every occurrence gets the index
//    occ = row * (W - 1) + k, and each edge's bucket of occurrences decides its
//    links locally: the entry with the smallest occ per neighbour gives the
//    direction; votes count every entry.
//  * Tracing only ever takes front() of a list of exactly one link, so the
//    in/out degree, the single parent and the single child of each edge are all
//    the tracer needs.
//  * "Legal" (in <= 1, out <= 1, not linked) has a static part. Edges that pass
//    it, joined by links between two of them, form disjoint simple paths and
//    cycles. A trace marks edges of its own component only, so components are
//    independent: one thread per component replays the reference's loop over
//    start edges in ascending id order, restricted to its component. Fragments
//    are then written in start-id order, which is the reference's order.
#pragma once

#include <cstdint>

namespace cvlc {

constexpr unsigned DIR_OUT = 0x80000000u;    // bucket entry: the link leaves this edge
constexpr unsigned FIRST_OCC = 0x40000000u;  // bucket entry: the first occurrence of its link
constexpr unsigned ID_MASK = 0x3fffffffu;    // edge ids below 2^30

enum : unsigned char { F_LEGAL = 1, F_FIRST = 2, F_SEEN = 4, F_NO_CHILD = 8, F_NO_PARENT = 16 };

constexpr unsigned ERR_ID = 1u;       // a chain id outside the map
constexpr unsigned ERR_SCRATCH = 2u;  // scratch sizing violated (never expected)

struct Graph {
    int n;
    const unsigned long long *occ_off;  // [n + 1]
    uint2 *bucket;                      // (other | DIR_OUT | FIRST_OCC, occ)
    int *outdeg, *indeg, *child, *parent;
    unsigned char *flags;
    struct Hop *hop;                    // [n] what a trace reads of an edge
};

// An edge as the trace visits it, one 32-byte sector: a trace is one chain of these loads.
struct __align__(16) Hop {
    int child, parent;  // of an edge with exactly one
    unsigned flags;     // F_*
    unsigned linked;    // marked by a trace (of the edge's own component only)
    double x, y;
};

// row length of a chain row (column 0 is the anchor)
__device__ __forceinline__ int chain_len(const unsigned *row, int W) {
    int len = 0;
    while (len < W - 1 && row[1 + len] != 0u) ++len;
    return len;
}

// ---- 1. occurrences per edge -----------------------------------------------------
__global__ void k_link_count(const unsigned *chains, long long C, int W, unsigned min_group, int n,
                             unsigned *occ_cnt, unsigned *err) {
    const long long r = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= C) return;
    const unsigned *row = chains + r * W;
    const int len = chain_len(row, W);
    for (int k = 0; k < len; ++k)  // every row's ids, linked or not
        if (row[1 + k] - 1u >= (unsigned)n) {
            atomicOr(err, ERR_ID);
            return;
        }
    if ((unsigned)len < min_group) return;
    for (int k = 0; k + 1 < len; ++k) {
        const unsigned u = row[1 + k] - 1u, v = row[2 + k] - 1u;
        atomicAdd(&occ_cnt[u], 1u);
        atomicAdd(&occ_cnt[v], 1u);
    }
}

__global__ void k_link_fill(const unsigned *chains, long long C, int W, unsigned min_group, int n,
                            const unsigned long long *occ_off, unsigned *cursor, uint2 *bucket) {
    const long long r = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= C) return;
    const unsigned *row = chains + r * W;
    const int len = chain_len(row, W);
    if ((unsigned)len < min_group) return;
    for (int k = 0; k < len; ++k)  // a row k_link_count rejected adds nothing, as there
        if (row[1 + k] - 1u >= (unsigned)n) return;
    for (int k = 0; k + 1 < len; ++k) {
        const unsigned u = row[1 + k] - 1u, v = row[2 + k] - 1u;
        const unsigned occ = (unsigned)(r * (W - 1) + k);
        const unsigned pu = atomicAdd(&cursor[u], 1u);
        bucket[occ_off[u] + pu] = make_uint2(v | DIR_OUT, occ);
        const unsigned pv = atomicAdd(&cursor[v], 1u);
        bucket[occ_off[v] + pv] = make_uint2(u, occ);
    }
}

// is entry i the first occurrence of its link within the bucket?
__device__ __forceinline__ bool first_of_link(const uint2 *b, unsigned m, unsigned i) {
    const unsigned w = b[i].x & ID_MASK, occ = b[i].y;
    for (unsigned j = 0; j < m; ++j)
        if ((b[j].x & ID_MASK) == w && b[j].y < occ) return false;
    return true;
}

// ---- 2. degrees, the single child / parent ----------------------------------------
// A warp per edge, a lane per entry of its bucket (about 12): the entries of one link find
// each other by a match, their first by a minimum over them. Buckets of more than 32 entries
// compare entry by entry. (With a thread per edge each comparison was a load from the
// bucket: 202 us on a 242k-edge map's 3.0M entries, and k_link_list 130 us.)
__global__ void __launch_bounds__(256) k_link_degrees(Graph g) {
    const int lane = threadIdx.x & 31;
    const int u = (int)(blockIdx.x * 8u + (threadIdx.x >> 5));
    if (u >= g.n) return;
    uint2 *b = g.bucket + g.occ_off[u];
    const unsigned m = (unsigned)(g.occ_off[u + 1] - g.occ_off[u]);
    int od = 0, id = 0, ch = -1, pa = -1;
    if (m <= 32) {
        const uint2 e = lane < (int)m ? b[lane] : make_uint2(0xffffffffu, 0u);
        // (lanes past the bucket match each other only: their id is above every edge's)
        const unsigned same = __match_any_sync(0xffffffffu, lane < (int)m ? e.x & ID_MASK : 0xffffffffu);
        const bool first = lane < (int)m && __reduce_min_sync(same, e.y) == e.y;
        if (first) b[lane].x = e.x | FIRST_OCC;  // only this warp touches edge u's bucket
        const unsigned outs = __ballot_sync(0xffffffffu, first && (e.x & DIR_OUT));
        const unsigned ins = __ballot_sync(0xffffffffu, first && !(e.x & DIR_OUT));
        od = __popc(outs);
        id = __popc(ins);
        const unsigned w = e.x & ID_MASK;
        if (outs) ch = (int)__shfl_sync(0xffffffffu, w, __ffs(outs) - 1);
        if (ins) pa = (int)__shfl_sync(0xffffffffu, w, __ffs(ins) - 1);
    } else {
        for (unsigned i = lane; i < m; i += 32) {
            if (!first_of_link(b, m, i)) continue;
            const unsigned x = b[i].x;
            if (x & DIR_OUT) {
                ++od;
                ch = (int)(x & ID_MASK);
            } else {
                ++id;
                pa = (int)(x & ID_MASK);
            }
        }
        __syncwarp();  // every lane has compared before an entry is marked
        for (unsigned i = lane; i < m; i += 32)
            if (first_of_link(b, m, i)) atomicOr(&b[i].x, FIRST_OCC);  // (marks leave ids and occurrences as they are)
        od = __reduce_add_sync(0xffffffffu, od);
        id = __reduce_add_sync(0xffffffffu, id);
        ch = __reduce_max_sync(0xffffffffu, ch);
        pa = __reduce_max_sync(0xffffffffu, pa);
    }
    if (lane != 0) return;
    // (child and parent are read where there is exactly one)
    g.outdeg[u] = od;
    g.indeg[u] = id;
    g.child[u] = ch;
    g.parent[u] = pa;
    unsigned char f = 0;
    if (od <= 1 && id <= 1) f |= F_LEGAL;                  // edgel_is_legal, static part
    if (od == 1 && id == 1 && pa != ch) f |= F_FIRST;      // edgel_is_legal_first_edgel, static part
    if (od == 0) f |= F_NO_CHILD;
    if (id == 0) f |= F_NO_PARENT;
    g.flags[u] = f;
}

// the links leaving each edge in creation order (_cLinks), with their votes; a warp per edge
__global__ void __launch_bounds__(256) k_link_list(Graph g, const unsigned long long *link_off, int *pe, int *ce,
                                                   int *votes) {
    const int lane = threadIdx.x & 31;
    const int u = (int)(blockIdx.x * 8u + (threadIdx.x >> 5));
    if (u >= g.n) return;
    const uint2 *b = g.bucket + g.occ_off[u];
    const unsigned m = (unsigned)(g.occ_off[u + 1] - g.occ_off[u]);
    const unsigned long long base = link_off[u];
    constexpr unsigned OUT_FIRST = DIR_OUT | FIRST_OCC;
    if (m <= 32) {
        const uint2 e = lane < (int)m ? b[lane] : make_uint2(0u, 0u);
        const unsigned same = __match_any_sync(0xffffffffu, lane < (int)m ? e.x & ID_MASK : 0xffffffffu);
        const bool mine = (e.x & OUT_FIRST) == OUT_FIRST;
        unsigned rank = 0;
        for (unsigned k = __ballot_sync(0xffffffffu, mine); k; k &= k - 1)
            rank += __shfl_sync(0xffffffffu, e.y, __ffs(k) - 1) < e.y;
        if (mine) {
            pe[base + rank] = u;
            ce[base + rank] = (int)(e.x & ID_MASK);
            votes[base + rank] = __popc(same);
        }
        return;
    }
    for (unsigned i = lane; i < m; i += 32) {
        if ((b[i].x & OUT_FIRST) != OUT_FIRST) continue;
        const unsigned w = b[i].x & ID_MASK;
        unsigned rank = 0, vote = 0;
        for (unsigned j = 0; j < m; ++j) {
            const unsigned wj = b[j].x & ID_MASK;
            if (wj == w) ++vote;
            else if ((b[j].x & OUT_FIRST) == OUT_FIRST && b[j].y < b[i].y) ++rank;
        }
        pe[base + rank] = u;
        ce[base + rank] = (int)w;
        votes[base + rank] = (int)vote;
    }
}

// ---- 3. component structure --------------------------------------------------------
__global__ void k_link_hops(Graph g, const double *edges, int sz) {
    const int u = blockIdx.x * blockDim.x + threadIdx.x;
    if (u >= g.n) return;
    const double *E = edges + (size_t)u * sz;
    Hop h;
    h.child = g.child[u];
    h.parent = g.parent[u];
    h.flags = g.flags[u];
    h.linked = 0u;
    h.x = E[0];
    h.y = E[1];
    g.hop[u] = h;
}

// the next legal edge of a legal edge's component, forward or backward; -1: none
__device__ __forceinline__ int succ_of(const Graph &g, const Hop &h) {
    return !(h.flags & F_NO_CHILD) && (g.hop[h.child].flags & F_LEGAL) ? h.child : -1;
}
__device__ __forceinline__ int pred_of(const Graph &g, const Hop &h) {
    return !(h.flags & F_NO_PARENT) && (g.hop[h.parent].flags & F_LEGAL) ? h.parent : -1;
}

struct FragOut {
    double thres;         // gap * gap
    unsigned *first_ids;  // scratch for each component's start edges
    unsigned long long *first_ctr;
    int *region;          // fragment ids beyond the start edge: forward part, then backward part
    unsigned long long *region_ctr;
    unsigned long long region_cap, first_cap;
    unsigned long long *frag_src;  // per start edge: offset into region
    int *frag_nf, *frag_nb;        // per start edge: forward / backward counts (frag_nf = -1: no fragment)
    unsigned *err;
};

// sq_distance (original_code/curvelet_utils.hpp:17-20); the library builds with -fmad=false
__device__ __forceinline__ double pt_sqd(const Hop &A, const Hop &B) {
    return (A.x - B.x) * (A.x - B.x) + (A.y - B.y) * (A.y - B.y);
}

__device__ void heap_sift(unsigned *a, long long i, long long n) {
    for (;;) {
        long long c = 2 * i + 1;
        if (c >= n) return;
        if (c + 1 < n && a[c + 1] > a[c]) ++c;
        if (a[i] >= a[c]) return;
        const unsigned t = a[i];
        a[i] = a[c];
        a[c] = t;
        i = c;
    }
}

__device__ void heap_sort(unsigned *a, long long n) {
    for (long long i = n / 2 - 1; i >= 0; --i) heap_sift(a, i, n);
    for (long long e = n - 1; e > 0; --e) {
        const unsigned t = a[0];
        a[0] = a[e];
        a[e] = t;
        heap_sift(a, 0, e);
    }
}

// Replays extract_one_chains_from_the_link_graph over one component (entered at
// `start`: a path's head, or a cycle's smallest id), start edges ascending.
// Region bound: a trace pushes, on each side, at most one edge it does not mark
// (the step that ends it) besides the edges it marks; every edge of the component
// is marked at most once and the start edge is not stored. So a component of m
// edges and f start edges stores at most m + f ids; m + 2f are reserved.
// Both its walks are one chain of loads (a hop's child gives the next hop), which bounds
// the kernel: the longest path of a 242k-edge map took 224 us with the edge's fields in
// arrays of their own, three loads one after the other to a step, and all start edges sorted.
// The least start edge's trace usually marks the whole component, so the others are
// collected and sorted only when it does not.
__device__ void trace_component(const Graph &g, const FragOut &o, int start) {
    // (the walk marks the component as seen: k_trace_cycles takes what no path's head reached)
    long long m = 0, f = 0;
    int v = start, least = 0x7fffffff;
    Hop h = g.hop[v];
    for (;;) {
        ++m;
        if (h.flags & F_FIRST) {
            ++f;
            least = min(least, v);
        }
        g.flags[v] = (unsigned char)(h.flags | F_SEEN);
        if (h.flags & F_NO_CHILD) break;
        v = h.child;
        if (v == start) break;
        h = g.hop[v];
        if (!(h.flags & F_LEGAL)) break;
    }
    if (f == 0) return;
    const unsigned long long fb = atomicAdd(o.first_ctr, (unsigned long long)f);
    const unsigned long long rb = atomicAdd(o.region_ctr, (unsigned long long)(m + 2 * f));
    if (fb + f > o.first_cap || rb + m + 2 * f > o.region_cap) {
        atomicOr(o.err, ERR_SCRATCH);
        return;
    }
    int *out = o.region + rb;
    long long cur = 0, marked = 0;  // ids stored, start edges marked
    const long long cap = m + 2 * f;
    auto put = [&](int e) {
        if (cur < cap) out[cur] = e;
        ++cur;  // (past cap: ERR_SCRATCH below)
    };
    auto trace = [&](int s) {
        const long long src = cur;
        int nf = 0, nb = 0;
        const Hop S = g.hop[s];
        g.hop[s].linked = 1u;
        ++marked;
        int eA = S.child;
        Hop A = g.hop[eA];
        if (pt_sqd(S, A) < o.thres) {
            put(eA);
            ++nf;
        }
        while ((A.flags & F_LEGAL) && !A.linked) {
            g.hop[eA].linked = 1u;
            marked += (A.flags & F_FIRST) != 0;
            if (A.flags & F_NO_CHILD) break;
            const Hop B = A;
            eA = A.child;
            A = g.hop[eA];
            if (!(pt_sqd(B, A) < o.thres)) break;
            put(eA);
            ++nf;
        }
        if (eA != s) {
            eA = S.parent;
            A = g.hop[eA];
            if (pt_sqd(S, A) < o.thres) {
                put(eA);
                ++nb;
            }
            while ((A.flags & F_LEGAL) && !A.linked) {
                g.hop[eA].linked = 1u;
                marked += (A.flags & F_FIRST) != 0;
                if (A.flags & F_NO_PARENT) break;
                const Hop B = A;
                eA = A.parent;
                A = g.hop[eA];
                if (!(pt_sqd(B, A) < o.thres)) break;
                put(eA);
                ++nb;
            }
        }
        o.frag_src[s] = rb + src;
        o.frag_nf[s] = nf;
        o.frag_nb[s] = nb;
    };
    trace(least);
    if (marked < f) {
        unsigned *firsts = o.first_ids + fb;
        long long k = 0;
        v = start;
        do {
            h = g.hop[v];
            if ((h.flags & F_FIRST) && !h.linked) firsts[k++] = (unsigned)v;
            v = succ_of(g, h);
        } while (v >= 0 && v != start);
        heap_sort(firsts, k);
        for (long long q = 0; q < k && marked < f; ++q)
            if (!g.hop[firsts[q]].linked) trace((int)firsts[q]);
    }
    if (cur > cap) atomicOr(o.err, ERR_SCRATCH);
}

// components that are paths: entered at their head (no legal predecessor)
__global__ void k_trace_paths(Graph g, FragOut o) {
    const int u = blockIdx.x * blockDim.x + threadIdx.x;
    if (u >= g.n) return;
    const Hop h = g.hop[u];
    if (!(h.flags & F_LEGAL) || pred_of(g, h) >= 0) return;
    trace_component(g, o, u);
}

// components that are cycles (legal edges no head reached): entered at their
// smallest id, found by walking both ways until a smaller id shows up
__global__ void k_trace_cycles(Graph g, FragOut o) {
    const int u = blockIdx.x * blockDim.x + threadIdx.x;
    if (u >= g.n) return;
    if (!(g.flags[u] & F_LEGAL) || (g.flags[u] & F_SEEN)) return;
    int a = succ_of(g, g.hop[u]), b = pred_of(g, g.hop[u]);
    for (;;) {
        if (a < 0 || b < 0) return;  // not a cycle (cannot happen for an unseen legal edge)
        if (a == u) break;           // walked all the way round: u is the smallest
        if (a < u || b < u) return;
        if (a == b) break;           // the two walks met
        a = succ_of(g, g.hop[a]);
        if (a == u) break;
        if (a < u) return;
        if (a == b) break;
        b = pred_of(g, g.hop[b]);
    }
    trace_component(g, o, u);
}

// ---- 4. fragments in start order ------------------------------------------------------
__global__ void k_frag_sizes(int n, const int *frag_nf, const int *frag_nb, unsigned *is_frag,
                             unsigned long long *frag_len) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= n) return;
    const int nf = frag_nf[s];
    const long long len = nf < 0 ? 0 : 1LL + nf + frag_nb[s];
    const bool keep = len > 2;  // "prune out the short ones"
    is_frag[s] = keep ? 1u : 0u;
    frag_len[s] = keep ? (unsigned long long)len : 0ull;
}

__global__ void k_frag_write(int n, const int *frag_nf, const int *frag_nb, const unsigned long long *frag_src,
                             const int *region, const unsigned *frag_idx, const unsigned long long *id_off,
                             long long *frag_offsets, int *frag_ids) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= n) return;
    const long long len = frag_nf[s] < 0 ? 0 : 1LL + frag_nf[s] + frag_nb[s];
    if (s == n - 1) frag_offsets[frag_idx[n]] = (long long)id_off[n];
    if (len <= 2) return;
    const int nf = frag_nf[s], nb = frag_nb[s];
    const int *src = region + frag_src[s];
    int *dst = frag_ids + id_off[s];
    frag_offsets[frag_idx[s]] = (long long)id_off[s];
    for (int q = 0; q < nb; ++q) dst[q] = src[nf + nb - 1 - q];  // the backward part, pushed to the front
    dst[nb] = s;
    for (int q = 0; q < nf; ++q) dst[nb + 1 + q] = src[q];
}

}  // namespace cvlc
