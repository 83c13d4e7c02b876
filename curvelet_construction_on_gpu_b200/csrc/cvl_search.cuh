// cvl_search.cuh -- sm_100a kernels of the curvelet path: (b) the neighbour search in one
// pass, for the runs k_curvelets serves (cvl_curvelets.cuh).
//
// k_search: a warp per item, 32 or fewer anchors of a hash bucket, a lane per anchor. The
// anchors of one 8-pixel hash block share their candidates: the edges of the 3 x 3 blocks
// around it that lie within w pixels of it. The warp loads those once and keeps them in
// shared memory. Every lane tests them with the reference's predicate
// (preprocess.hpp:129-167), reading each at the same time as the others (a broadcast), and
// appends its neighbours to its column of a table. The rows of the anchors are allocated
// together and back to back, so the warp writes them as one coalesced run, a lane per pair,
// each with its rank by (distance, scan order) in its anchor's column and its classes.
//
// A run with a non-finite edge fails (ERR_NONFINITE, final since k_bin_keys), and nothing from
// here on may read what it left: k_bin_keys puts such an edge into bucket 0, whatever its
// cell, so an item that it heads would have another bucket's end, its neighbours' distances
// have no order, and rows would stay unwritten. k_bin_scatter lists no items of such a run, nor
// of one whose orientations k_curvelets cannot take, and k_curvelets and k_curvelets_exact
// leave at once. (On finite edges an item's head has its bucket's hash, and no item crosses it.)
//
// Rows are in no order, so the search needs no counting pass, no scan of the degrees and
// no host synchronisation before the pairs' buffers are sized: a run whose rows do not fit
// raises ERR_CAPACITY and goes again by the two passes (k_nb<COUNT>, k_nb<FILL>).
//
// Why: with a warp per anchor, both passes spent most of their issue slots on work done per
// warp for one anchor (the block ranges, a prefix sum, a five-step search per candidate,
// the rank sort), about 2,000 warp instructions per anchor on a dense map; here they are
// about 420 there. Measured: 7.06 -> 2.48 ms on a dense 3.65M-edge map (22 neighbours an edge),
// 0.84 -> 0.31 ms on a 735k-edge one (7). It is bound by latency at 24 warps an SM, which the
// table's size sets: with a single-precision distance and a 32-bit index per entry (12
// warps) it took 5.2 ms. A lane per anchor without the shared candidates took 5.6 ms.
// k_search_wide takes the anchors with more than SEARCH_CAP neighbours, whose list is cut
// at max_candidates, or whose block has more than SEARCH_TILE candidates, a warp each.
#pragma once

#include "cvl_kernels.cuh"

namespace cvl {

constexpr int SEARCH_CAP = 48;    // neighbours of a lane's anchor at most
constexpr int SEARCH_WARPS = 4;   // per block
constexpr int SEARCH_BLOCKS = 6;  // per SM: its 8,960 bytes a warp leave room for 24
constexpr int SEARCH_SBITS = 3;   // hash blocks of 8 pixels: windows of w <= 8 reach the 3 x 3 around
// Anchors of an item (a power of two): a whole warp's, or, on runs of up to 64 Ki edges, a
// quarter of that, as there are fewer blocks than warps and the heaviest one's chain is what the
// kernel takes (30k edges: 0.260 ms for a whole run with buckets dealt out, 0.232 with 32, 0.213
// with 8; a dense 3.65M-edge map's search takes 2.48 ms with 32, 3.10 with 16, 4.15 with 8).
inline unsigned search_item(long long n) { return n <= (64 << 10) ? 8u : 32u; }
constexpr int SEARCH_TILE = 160;  // candidates of a block at most (edges within w pixels of it)

// A row of the neighbour lists: its first pair's place, and its length above bit 48.
__device__ __forceinline__ unsigned long long pack_row(unsigned long long first, unsigned deg) {
    return first | ((unsigned long long)deg << 48);
}
constexpr unsigned long long NO_ROW = ~0ull;  // no room was left for the row (ERR_CAPACITY)

struct SearchArgs {
    Model md;
    EdgeRecords B;
    const FastEdge *e;                // [N]
    const double2 *cs2;               // [N]
    const int4 *at;                   // [N] pixel cell, input index, map
    const unsigned *bstart;
    unsigned long long *row;          // [N] pack_row
    unsigned long long *pair_ctr;     // pairs allocated
    unsigned long long pair_cap;
    int *csr_ids;
    unsigned char *pcls;              // run | close << 2 | branch1 << 3
    MapStats *stats;
    unsigned *err;
    unsigned *wide_cnt;               // anchors for k_search_wide
    int *wide_list;                   // [N]: an anchor is of one item, and is listed once
    const unsigned *items;            // each run of up to item_size anchors of a bucket, by its first (k_bin_scatter;
                                      // none where *unfit)
    const unsigned *item_cnt;
    float scale;                      // 65,000 over the longest pair's d2 (rounding and truncation keep d2's order)
    unsigned item_size;               // a power of two, at most 32
    unsigned *queue;                  // the next item (0 at start)
    unsigned pulls;                   // items a warp takes at most
};

struct SearchSmem {
    double2 cxy[SEARCH_TILE];              // the block's candidates
    double2 xy[32];                        // the anchors
    int cj[SEARCH_TILE];
    unsigned cat[SEARCH_TILE];             // pixel cell from the block's corner less w: x | y << 16
    unsigned short d2[SEARCH_CAP][32];     // columns: the anchors' neighbours, d2 on a scale of 2^16
    unsigned char id[SEARCH_CAP][32];      // and their candidates
};

__device__ __forceinline__ unsigned char pair_class(const Model &md, double ax, double ay, double lx, double ly,
                                                    double2 cs2) {
    const unsigned run = direction_class(ax, ay, lx, ly, cs2.x, cs2.y);  // (:454-462)
    const double DX = ax - lx, DY = ay - ly;
    const bool close = DX * DX + DY * DY < md.four_dx_dx;      // :682
    const bool branch1 = (DX * cs2.x + DY * cs2.y) < 0;        // :690
    return (unsigned char)(run | (close ? 4u : 0u) | (branch1 ? 8u : 0u));
}

// A warp's map statistics, flushed when the map changes.
struct SearchCounts {
    int map = -1;
    unsigned long long pairs = 0;
    unsigned deg = 0, cut = 0;
    __device__ __forceinline__ void flush(MapStats *stats, int lane) {
        if (lane != 0 || map < 0) return;
        if (pairs) atomicAdd(&stats[map].pairs, pairs);
        if (deg) atomicMax(&stats[map].max_deg, deg);
        if (cut) atomicAdd(&stats[map].truncated, cut);
    }
    __device__ __forceinline__ void add(MapStats *stats, int lane, int m, unsigned n, unsigned max_n, unsigned c) {
        if (m != map) {
            flush(stats, lane);
            map = m;
            pairs = 0;
            deg = cut = 0u;
        }
        pairs += n;
        deg = max(deg, max_n);
        cut += c;
    }
};

__global__ void __launch_bounds__(SEARCH_WARPS * 32, SEARCH_BLOCKS) k_search(const __grid_constant__ SearchArgs a) {
    extern __shared__ __align__(16) unsigned char se_smem[];
    SearchSmem &S = ((SearchSmem *)se_smem)[threadIdx.x >> 5];
    const Model &md = a.md;
    const int lane = threadIdx.x & 31;
    const unsigned lt_mask = (1u << lane) - 1u;
    const int cap = min(SEARCH_CAP, md.max_cand - 1);  // (a list of max_cand or more counts as cut)
    const int w = md.w;
    SearchCounts counts;
    // The heaviest block has 13 to 19 times the mean's work (anchors x candidates), so warps pull
    // items from a queue: a dense 3.65M-edge map's search 3.10 -> 2.48 ms, a 735k-edge one's
    // 0.39 -> 0.31, against listed buckets dealt out in turn.
    const unsigned n_items = *a.item_cnt;
    for (unsigned pull = 0; pull < a.pulls; ++pull) {
        unsigned it = 0;
        if (lane == 0) it = atomicAdd(a.queue, 1u);
        it = __shfl_sync(FULL, it, 0);
        if (it >= n_items) break;
        const unsigned c0 = a.items[it];
        const int4 head = a.at[c0];
        const unsigned bucket = cell_hash(head.w, head.x >> SEARCH_SBITS, head.y >> SEARCH_SBITS) & md.hash_mask;
        const unsigned c1 = min(a.bstart[bucket + 1], c0 + a.item_size);
        const int i = (int)(c0 + lane);
        const bool on = c0 + lane < c1;
        int4 ac = make_int4(0, 0, 0, -1);
        double ax = 0.0, ay = 0.0;
        __syncwarp();
        if (on) {
            ac = a.at[i];
            ax = a.e[i].x;
            ay = a.e[i].y;
            S.xy[lane] = make_double2(ax, ay);
        }
        // the anchors of one block (nearly always all of the bucket's) at a time
        for (unsigned todo = __ballot_sync(FULL, on); todo;) {
            const int lead = __ffs(todo) - 1;
            const int m = __shfl_sync(FULL, ac.w, lead);
            const int bx = __shfl_sync(FULL, ac.x >> SEARCH_SBITS, lead);
            const int by = __shfl_sync(FULL, ac.y >> SEARCH_SBITS, lead);
            const bool mine = on && ac.w == m && (ac.x >> SEARCH_SBITS) == bx && (ac.y >> SEARCH_SBITS) == by;
            todo &= ~__ballot_sync(FULL, mine);
            // the buckets of the 3 x 3 blocks, each once, and their prefix sums
            const unsigned hb = lane < 9 ? cell_hash(m, bx - 1 + lane % 3, by - 1 + lane / 3) & md.hash_mask
                                         : 0xffffffffu - (unsigned)lane;
            const unsigned same = __match_any_sync(FULL, hb);
            unsigned s = 0, len = 0;
            if (lane < 9 && __ffs(same) - 1 == lane) {
                s = a.bstart[hb];
                len = a.bstart[hb + 1] - s;
            }
            unsigned incl = len;
#pragma unroll
            for (int d = 1; d < 16; d <<= 1) {
                const unsigned o = __shfl_up_sync(FULL, incl, d);
                if (lane >= d) incl += o;
            }
            const unsigned span = __shfl_sync(FULL, incl, 8);
            const unsigned shift = s + len - incl;
            // the candidates: those within w pixels of the block
            const int x0 = (bx << SEARCH_SBITS) - w, y0 = (by << SEARCH_SBITS) - w;
            const unsigned side = (unsigned)((1 << SEARCH_SBITS) - 1 + 2 * w);
            int cnt = 0;
            for (unsigned e0 = 0; e0 < span; e0 += 32) {
                const unsigned e = e0 + lane;
                int q = 0;  // the bucket of edge e: the first whose prefix exceeds it
#pragma unroll
                for (int step = 8; step >= 1; step >>= 1) {
                    const unsigned v = __shfl_sync(FULL, incl, q + step - 1);
                    if (v <= e) q += step;
                }
                const int j = (int)(__shfl_sync(FULL, shift, q) + e);
                int4 c = make_int4(0, 0, 0, -1);
                if (e < span) c = a.at[j];
                const unsigned cx = (unsigned)(c.x - x0), cy = (unsigned)(c.y - y0);
                const bool in = e < span && c.w == m && cx <= side && cy <= side;
                const unsigned bal = __ballot_sync(FULL, in);
                const int at = cnt + __popc(bal & lt_mask);
                if (in && at < SEARCH_TILE) {
                    S.cat[at] = cx | cy << 16;
                    S.cj[at] = j;
                    S.cxy[at] = make_double2(a.e[j].x, a.e[j].y);
                }
                cnt += __popc(bal);
            }
            __syncwarp();
            int n = cnt > SEARCH_TILE ? cap + 1 : 0;
            if (cnt <= SEARCH_TILE) {
                const unsigned ox = (unsigned)(ac.x - x0 - w), oy = (unsigned)(ac.y - y0 - w), ww = 2u * (unsigned)w;
                for (int k = 0; k < cnt; ++k) {
                    const unsigned c = S.cat[k];
                    if (mine && (c & 0xffffu) - ox <= ww && (c >> 16) - oy <= ww) {
                        const double2 p = S.cxy[k];
                        const double d2 = sq_dist(ax, ay, p.x, p.y);  // preprocess.hpp:160
                        if (!(d2 > md.rad_sqr) && S.cj[k] != i) {     // :161-163
                            if (n < cap) {
                                S.d2[n][lane] = (unsigned short)((float)d2 * a.scale);
                                S.id[n][lane] = (unsigned char)k;
                            }
                            ++n;
                        }
                    }
                }
            }
            if (mine && n > cap) a.wide_list[atomicAdd(a.wide_cnt, 1u)] = i;
            const unsigned deg = !mine || n > cap ? 0u : (unsigned)n;
            // the rows of the anchors, back to back
            unsigned upto = deg;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const unsigned o = __shfl_up_sync(FULL, upto, d);
                if (lane >= d) upto += o;
            }
            const unsigned total = __shfl_sync(FULL, upto, 31);
            unsigned long long base = 0;
            if (lane == 0 && total) base = atomicAdd(a.pair_ctr, (unsigned long long)total);
            base = __shfl_sync(FULL, base, 0);
            const bool fits = base + total <= a.pair_cap;
            if (!fits && lane == 0) atomicOr(a.err, ERR_CAPACITY);
            if (mine && n <= cap) a.row[i] = fits ? pack_row(base + upto - deg, deg) : NO_ROW;
            counts.add(a.stats, lane, m, total, __reduce_max_sync(FULL, deg), 0u);
            __syncwarp();
            // a lane per pair: its anchor is the first lane whose inclusive prefix exceeds it
            for (unsigned p0 = 0; fits && p0 < total; p0 += 32) {
                const unsigned p = p0 + lane;
                int L = 0;
#pragma unroll
                for (int step = 16; step >= 1; step >>= 1) {
                    const unsigned v = __shfl_sync(FULL, upto, L + step - 1);
                    if (v <= p) L += step;
                }
                const unsigned first = __shfl_sync(FULL, upto, L) - __shfl_sync(FULL, deg, L);
                const unsigned num = __shfl_sync(FULL, deg, L);
                const int ocx = __shfl_sync(FULL, ac.x, L), ocy = __shfl_sync(FULL, ac.y, L);
                if (p >= total) continue;
                const unsigned k = p - first, d = S.d2[k][L];
                const int id = S.id[k][L];
                // rank by (d2, scan key) -- std::sort by distance, preprocess.hpp:172-176
                unsigned rank = 0, ties = 0;
                for (unsigned u = 0; u < num; ++u) {
                    const unsigned v = S.d2[u][L];
                    rank += v < d;
                    ties += v == d;
                }
                const double2 A = S.xy[L], P = S.cxy[id];
                const int nn = S.cj[id];
                if (ties > 1) {
                    const int4 c = a.at[nn];
                    const double de = sq_dist(A.x, A.y, P.x, P.y);
                    const unsigned long long key = scan_key(make_int2(c.x, c.y), ocx, ocy, w, c.z);
                    for (unsigned u = 0; u < num; ++u) {
                        if (u == k || S.d2[u][L] != d) continue;
                        const int o = S.id[u][L];
                        const double du = sq_dist(A.x, A.y, S.cxy[o].x, S.cxy[o].y);
                        if (du == de) {
                            const int4 co = a.at[S.cj[o]];
                            rank += scan_key(make_int2(co.x, co.y), ocx, ocy, w, co.z) < key;
                        } else {
                            rank += du < de;
                        }
                    }
                }
                const unsigned long long at = base + first + rank;
                a.csr_ids[at] = nn;
                a.pcls[at] = pair_class(md, A.x, A.y, P.x, P.y, a.cs2[c0 + L]);
            }
            __syncwarp();
        }
    }
    counts.flush(a.stats, lane);
}

// The anchors k_search left, a warp each: their candidates counted, then gathered and ranked
// as k_nb<FILL> does.
__global__ void __launch_bounds__(256) k_search_wide(const __grid_constant__ SearchArgs a) {
    extern __shared__ __align__(16) unsigned char sw_smem[];
    const Model &md = a.md;
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const unsigned lt_mask = (1u << lane) - 1u;
    const int n_wide = (int)*a.wide_cnt;
    NbrSmemT<double> S;
    {
        unsigned char *p = sw_smem + (size_t)wib * nbr_smem_per_warp(md.max_cand);
        S.d2 = (double *)p;
        S.key = (unsigned long long *)(p + (size_t)md.max_cand * 8);
        S.idx = (int *)(p + (size_t)md.max_cand * 16);
    }
    SearchCounts counts;
    for (int it = (int)blockIdx.x * 8 + wib; it < n_wide; it += (int)gridDim.x * 8) {
        const int i = a.wide_list[it];
        const int4 at = a.at[i];
        const int m = at.w;
        const int2 ac = make_int2(at.x, at.y);
        const double ax = a.e[i].x, ay = a.e[i].y;
        unsigned n = 0;
        __syncwarp();
        for_window_candidates(md, a.B, a.bstart, i, m, ac, ax, ay, lane,
                              [&](bool ok, int j, double d2, unsigned long long key) {
                                  const unsigned bal = __ballot_sync(FULL, ok);
                                  const unsigned p = n + __popc(bal & lt_mask);
                                  if (ok && p < (unsigned)md.max_cand) {
                                      S.d2[p] = d2;
                                      S.key[p] = key;
                                      S.idx[p] = j;
                                  }
                                  n += __popc(bal);
                              });
        const bool cut = n >= (unsigned)md.max_cand;
        if (n > (unsigned)md.max_cand) n = gather_truncated(md, a.B, a.bstart, i, m, ac, ax, ay, lane, S, a.err);
        __syncwarp();
        unsigned long long base = 0;
        if (lane == 0) base = atomicAdd(a.pair_ctr, (unsigned long long)n);
        base = __shfl_sync(FULL, base, 0);
        const bool fits = base + n <= a.pair_cap;
        if (lane == 0) {
            a.row[i] = fits ? pack_row(base, n) : NO_ROW;
            if (!fits) atomicOr(a.err, ERR_CAPACITY);
        }
        counts.add(a.stats, lane, m, n, n, cut ? 1u : 0u);
        const double2 cs2 = a.cs2[i];
        for (unsigned t = lane; fits && t < n; t += 32) {
            const double d = S.d2[t];
            const unsigned long long kt = S.key[t];
            unsigned rk = 0;
            for (unsigned u = 0; u < n; ++u) {
                const double du = S.d2[u];
                rk += (du < d) || (du == d && S.key[u] < kt);
            }
            const int nn = S.idx[t];
            a.csr_ids[base + rk] = nn;
            a.pcls[base + rk] = pair_class(md, ax, ay, a.e[nn].x, a.e[nn].y, cs2);
        }
    }
    counts.flush(a.stats, lane);
}

// Rows of a two-pass search (k_nb), for k_curvelets.
__global__ void k_pack_rows(int N, const unsigned long long *__restrict__ pair_off, unsigned long long *__restrict__ row) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < N; i += gridDim.x * blockDim.x)
        row[i] = pack_row(pair_off[i], (unsigned)(pair_off[i + 1] - pair_off[i]));
}

}  // namespace cvl
