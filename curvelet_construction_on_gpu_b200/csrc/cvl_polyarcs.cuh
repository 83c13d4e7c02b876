// cvl_polyarcs.cuh -- C^1 polyarcs along the contour fragments, as the reference's
// original_code fits them after the one-chains:
//   fit_polyarcs_to_all_edgel_chains / fit_polyarc_to_chain
//       (original_code/form_curvelet_process.cpp:661-796)
//   form_a_hypothesis (leading, forward: :388-444), CC_curve_model_3d's bundle,
//   intersection, compute_best_fit, update_best_fit (CC_curve_model_3d.cpp)
//   curvelet::compute_properties / update_length (curvelet.cpp:80-169)
//   polyarcmap::compute_best_fit_according_to_curvelets (polyarcmap.hpp:98-111)
//
// A warp per fragment, the bundle's cells across the lanes (CPL per lane), the
// fragment walked in order as fit_polyarc_to_chain walks it:
//   - from edge i, a polyarc starts when the next edge lies ahead of it (dot > 0)
//     and their bundle is valid; it grows over the following edges while each
//     one's bundle with the start edge is valid and the running intersection
//     stays valid; the next polyarc starts at its last edge;
//   - its best cell is the open cell of smallest rank (the rank table gives
//     compute_best_fit's order: nearest the grid centre, first in row-major order);
//   - the fit: a line or the circle through the start, middle and end edges, with the
//     reference's operand order (the library builds with -fmad=false), by a thread per
//     polyarc where they are packed (k_polyarcs_pack).
// compute_best_fit_according_to_curvelets runs at the end of every fragment over
// all polyarcs so far, so a polyarc fitted as an arc with |k| < k_th becomes a
// line at its next refit, keeping its centre, angle and length; every other fit
// repeats itself. A polyarc of any fragment but the last is refitted.
#pragma once

namespace cvl {

constexpr double POLY_K_TH = 1e-4;  // k_th, original_code/curvelet_utils.hpp:15

struct PolyArgs {
    Model md;                      // dx, dt, max_k; grid steps 0.1 px, 0.08 rad (CC_curve_model_3d.hpp:20-23)
    const double *edges;           // AoS [n][sz]
    int sz;
    int nfrags;
    const long long *frag_off;     // [nfrags + 1]
    const int *frag_ids;           // 0-based edge ids
    double rad, token_len;         // compute_properties' R and token_len
    long long *poly_start;         // [slots]: index into frag_ids of the polyarc's first edge
    int *poly_size;                // [slots]
    double *poly_fit;              // [slots][3]: the best cell's k_max, k_min, and the length along the edges
    unsigned *poly_count;          // [nfrags]
    unsigned *queue;               // the next fragment (0 at start)
};

// The polyarc slots of fragment f start at frag_off[f] - f: a fragment of N edges
// gives at most N - 1 polyarcs (each spans at least two edges and the next one
// starts no earlier than the last edge of the one before).
//
// A persistent grid whose warps pull fragments from a queue: the cell tables (a rank is a
// count over all cells) are made once per resident block, and a long fragment holds one
// warp, not a block. With a block per 4 fragments the tables were a third of the
// instructions. With the fits on lane 0 of the walking warp and a block per 4 fragments
// a 242k-edge map's 19k fragments took 325 us, now 253 and 14 in the packing.
template <int CPL>
__global__ void __launch_bounds__(128) k_polyarcs(PolyArgs a) {
    __shared__ double tab[4][4 * QMAX + 4];
    __shared__ double cell_dx2[CELLS_MAX];
    __shared__ unsigned char cell_j[CELLS_MAX];
    __shared__ unsigned short cell_rank[CELLS_MAX];
    const Model &md = a.md;
    cell_tables_init(md, cell_dx2, cell_j, cell_rank);
    __syncthreads();
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    double *sT = tab[wib], *cT = sT + QMAX, *sM = cT + QMAX, *sP = sM + QMAX, *own = sP + QMAX;
    bool on[CPL];
    int cj[CPL];
    double cdx2[CPL];
    unsigned rk[CPL];
#pragma unroll
    for (int u = 0; u < CPL; ++u) {
        const int c = lane + 32 * u;
        on[u] = c < md.cells;
        cj[u] = on[u] ? cell_j[c] : 0;
        cdx2[u] = on[u] ? cell_dx2[c] : 0.0;
        rk[u] = on[u] ? cell_rank[c] : 0xffffu;
    }
    for (;;) {
        unsigned q = 0;
        if (lane == 0) q = atomicAdd(a.queue, 1u);
        const int f = (int)__shfl_sync(FULL, q, 0);
        if (f >= a.nfrags) break;
        const int *ids = a.frag_ids + a.frag_off[f];
        const int N = (int)(a.frag_off[f + 1] - a.frag_off[f]);
        const long long slot0 = a.frag_off[f] - f;
        unsigned count = 0;
        int i = 0;
        while (i < N - 1) {
            const int iA = i, ia = ids[i];
            ++i;
            const double *A = a.edges + (size_t)ia * a.sz;
            const double ax = A[0], ay = A[1], T2 = A[2];
            double cosT2 = 0.0, sinT2 = 0.0;
            __syncwarp();  // the previous start's tables are read
            for (int j = lane; j <= md.Q; j += 32) {
                const double t = j < md.Q ? T2 + grid_offset(md.st, j, md.Q) : T2;  // T2t = T2 + Dt(j)
                double sv, cv;
                sincos(t, &sv, &cv);
                if (j < md.Q) {
                    sT[j] = sv;
                    cT[j] = cv;
                } else {
                    sinT2 = sv;
                    cosT2 = cv;
                }
            }
            cosT2 = __shfl_sync(FULL, cosT2, md.Q & 31);
            sinT2 = __shfl_sync(FULL, sinT2, md.Q & 31);
            // form_a_hypothesis(A, B) and its bundle: false when there is no model
            // (B not ahead of A) or the bundle is empty. The pair's sines and cosines come from
            // one sincos, a lane each: sin(T2t_j - T0 + dt) in lanes j < Q, sin(T2t_j - T0 - dt)
            // in the next Q, T0 + dt's and T0 - dt's in the two after them (sincos gives the
            // values of sin and cos: tests/probes/sincos_identity.cu). Made one call after the
            // other, they were most of a step, and a long fragment's steps are one chain.
            auto hypothesis = [&](double bx, double by, double T0, double *bmin, double *bmax) -> bool {
                // dot(vPointPoint(A, B), A's orientation) > 0: B ahead of A
                if (direction_class(ax, ay, bx, by, cosT2, sinT2) != 0u) return false;
                const double t_p = T0 + md.dt, t_m = T0 - md.dt;
                __syncwarp();  // the tables of the previous pair are read
                for (int j = lane; j < 2 * md.Q + 2; j += 32) {
                    const int jq = j < md.Q ? j : j - md.Q;
                    const double t = T2 + grid_offset(md.st, jq, md.Q);
                    const double arg = j < md.Q ? t - t_m : j < 2 * md.Q ? t - t_p : j == 2 * md.Q ? t_p : t_m;
                    double sv, cv;
                    sincos(arg, &sv, &cv);
                    if (j < md.Q) {
                        sM[j] = sv;
                    } else if (j < 2 * md.Q) {
                        sP[j - md.Q] = sv;
                    } else {
                        own[2 * (j - 2 * md.Q)] = sv;
                        own[2 * (j - 2 * md.Q) + 1] = cv;
                    }
                }
                __syncwarp();
                const PairGeom g = pair_geom(md, ax, ay, cosT2, sinT2, bx, by, own[0], own[1], own[2], own[3]);
                bool lv = false;
#pragma unroll
                for (int u = 0; u < CPL; ++u) {
                    bmin[u] = -md.max_k;
                    bmax[u] = md.max_k;
                    if (on[u] && !g.close) {
                        const double tt = sT[cj[u]] * g.DX - cT[cj[u]] * g.DY;
                        bundle_cell_tt(md, g.DX2, g.DY2, g.sin_p_DY, g.cos_p_DX, g.sin_m_DY, g.cos_m_DX, g.branch1,
                                       cdx2[u], tt, sM[cj[u]], sP[cj[u]], bmin[u], bmax[u]);
                    }
                    lv = lv || (on[u] && bmax[u] > bmin[u]);
                }
                return g.close || __any_sync(FULL, lv);
            };
            // the next edge's position and orientation, one step ahead of their use
            auto edge_at = [&](int q, double &x, double &y, double &th) {
                if (q < N) {
                    const double *B = a.edges + (size_t)ids[q] * a.sz;
                    x = B[0];
                    y = B[1];
                    th = B[2];
                }
            };
            double bx = 0.0, by = 0.0, bth = 0.0, nx = 0.0, ny = 0.0, nth = 0.0;
            edge_at(i, bx, by, bth);
            edge_at(i + 1, nx, ny, nth);
            double cmin[CPL], cmax[CPL];
            if (!hypothesis(bx, by, bth, cmin, cmax)) continue;
            // curvelet::compute_properties: every step counts (the anchor is the front)
            double L = sqrt((ax - bx) * (ax - bx) + (ay - by) * (ay - by));
            int j = i;
            while (j < N - 1) {
                const double px = bx, py = by;
                bx = nx;
                by = ny;
                bth = nth;
                edge_at(j + 2, nx, ny, nth);
                double rmin[CPL], rmax[CPL];
                if (!hypothesis(bx, by, bth, rmin, rmax)) break;
                // CC_curve_model_3d(cm1, cm2): Kmin = std::max, Kmax = std::min
                bool lv = false;
#pragma unroll
                for (int u = 0; u < CPL; ++u) {
                    rmin[u] = (cmin[u] < rmin[u]) ? rmin[u] : cmin[u];
                    rmax[u] = (rmax[u] < cmax[u]) ? rmax[u] : cmax[u];
                    lv = lv || (on[u] && rmax[u] > rmin[u]);
                }
                if (!__any_sync(FULL, lv)) break;
#pragma unroll
                for (int u = 0; u < CPL; ++u) {
                    cmin[u] = rmin[u];
                    cmax[u] = rmax[u];
                }
                L += sqrt((px - bx) * (px - bx) + (py - by) * (py - by));
                ++j;
            }
            // compute_best_fit: the open cell of smallest rank
            unsigned best = 0xffffu;
#pragma unroll
            for (int u = 0; u < CPL; ++u)
                if (on[u] && cmax[u] > cmin[u] && rk[u] < best) best = rk[u];
            best = __reduce_min_sync(FULL, best);
            double mymax = 0.0, mymin = 0.0;
            bool mine = false;
#pragma unroll
            for (int u = 0; u < CPL; ++u)
                if (on[u] && rk[u] == best && cmax[u] > cmin[u]) {
                    mine = true;
                    mymax = cmax[u];
                    mymin = cmin[u];
                }
            const unsigned who = __ballot_sync(FULL, mine);
            const int src = who ? __ffs(who) - 1 : 0;
            const double kmax = __shfl_sync(FULL, mymax, src);
            const double kmin = __shfl_sync(FULL, mymin, src);
            if (lane == 0) {
                const long long s = slot0 + count;
                a.poly_start[s] = a.frag_off[f] + iA;
                a.poly_size[s] = j - iA + 1;
                a.poly_fit[3 * s] = kmax;
                a.poly_fit[3 * s + 1] = kmin;
                a.poly_fit[3 * s + 2] = L;
            }
            ++count;
            i = j;
        }
        if (lane == 0) a.poly_count[f] = count;
    }
}

// polyarcs of all fragments packed in order (fragment, then start), and their fits; a
// thread per polyarc
__global__ void __launch_bounds__(128) k_polyarcs_pack(PolyArgs a, long long n_poly,
                                                       const unsigned long long *__restrict__ poly_off,
                                                       long long *__restrict__ start_out, int *__restrict__ size_out,
                                                       double *__restrict__ info_out) {
    const long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (p >= n_poly) return;
    int f = 0;  // the last fragment with poly_off[f] <= p (it has polyarcs: the next one's are past p)
    for (int lo = 0, hi = a.nfrags; hi - lo > 1;) {
        const int mid = (lo + hi) >> 1;
        if ((long long)poly_off[mid] <= p) lo = mid; else hi = mid;
        f = lo;
    }
    const long long s = a.frag_off[f] - f + (p - (long long)poly_off[f]);
    const long long start = a.poly_start[s];
    const int size = a.poly_size[s];
    const double kmax = a.poly_fit[3 * s], kmin = a.poly_fit[3 * s + 1];
    double L = a.poly_fit[3 * s + 2];
    start_out[p] = start;
    size_out[p] = size;
    const int *ids = a.frag_ids + start;
    const double *A = a.edges + (size_t)ids[0] * a.sz;
    const double ax = A[0], ay = A[1], T2 = A[2];
    double k = (kmax + kmin) / 2;  // set_best_fit's _k
    const double quality = 2 / (1.0 * a.rad / L + 1.0 * L / a.token_len / size);
    // update_best_fit(middle, end) with _pt = the start edge
    const double *P1 = a.edges + (size_t)ids[size / 2] * a.sz;
    const double *P2 = a.edges + (size_t)ids[size - 1] * a.sz;
    double theta, angle = 0.0, cx = 0.0, cy = 0.0;
    bool arc = false;
    if (fabs(k) < POLY_K_TH) {
        k = 0.0;
        theta = cvl_atan2(P2[1] - ay, P2[0] - ax);
    } else {
        const double d1 = ax * ax + ay * ay, d2 = P1[0] * P1[0] + P1[1] * P1[1], d3 = P2[0] * P2[0] + P2[1] * P2[1];
        const double a11 = 2.0 * (ax - P1[0]), a12 = 2.0 * (ay - P1[1]), a21 = 2.0 * (P2[0] - P1[0]),
                     a22 = 2.0 * (P2[1] - P1[1]);
        const double b1 = d1 - d2, b2 = d3 - d2;
        const double det = a11 * a22 - a21 * a12;
        if (fabs(det) < POLY_K_TH) {
            k = 0.0;
            theta = cvl_atan2(P2[1] - ay, P2[0] - ax);
        } else {
            cx = (b1 * a22 - b2 * a12) / det;
            cy = (b2 * a11 - b1 * a21) / det;
            const double v1x = ax - cx, v1y = ay - cy, v2x = P2[0] - cx, v2y = P2[1] - cy;
            const double c = v1x * v2y - v1y * v2x, d = v1x * v2x + v1y * v2y;
            angle = cvl_atan2(fabs(c), d);
            theta = cvl_atan2(c * v1x, -c * v1y);
            k = 1.0 / sqrt(v2x * v2x + v2y * v2y);
            arc = true;
        }
    }
    if (fabs(angle) > 0 && fabs(k) > POLY_K_TH && arc) L = angle / fabs(k);  // update_length
    if (arc && fabs(k) < POLY_K_TH && f < a.nfrags - 1) {  // the refit of a later fragment
        k = 0.0;
        theta = cvl_atan2(P2[1] - ay, P2[0] - ax);
    }
    double *row = info_out + p * 12;
    row[0] = 1.0;   // forward
    row[1] = kmax;  // _ref_pt after compute_best_fit: the best cell's k range
    row[2] = kmin;
    row[3] = T2;    // _ref_theta
    row[4] = ax;    // _pt: the start edge
    row[5] = ay;
    row[6] = theta;
    row[7] = k;
    row[8] = L;
    row[9] = quality;
    row[10] = arc ? cx : 0.0;
    row[11] = arc ? cy : 0.0;
}

}  // namespace cvl
