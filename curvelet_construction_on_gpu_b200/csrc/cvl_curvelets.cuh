// cvl_curvelets.cuh -- sm_100a kernels of the curvelet path for FP64 runs on grids of
// up to 64 cells with 9 offsets: (c) + (d) the pairwise bundles and the chain growth in
// one kernel (k_curvelets, and k_curvelets_exact for the anchors it leaves), and (e) the
// output expansion (k_finalize_exact).
//
// What a run outputs needs few bundle bounds as numbers: a curvelet's k range is one
// cell of its chain's bundles. All other bounds are only compared: whether a pair's
// bundle, or an intersection, has an open cell, and which open cell lies nearest the
// grid's centre. k_curvelets makes those comparisons on single-precision enclosures
// of the bounds, with an error bound proved below; an anchor with a comparison that an
// enclosure leaves undecided goes to k_curvelets_exact, which settles it in FP64 with
// the reference's expressions. k_finalize_exact then evaluates each curvelet's one cell
// in FP64, as the reference computes it. So every decision and every number is the FP64
// path's, bit for bit.
//
// Why: the FP64 transport of every cell of every pair was bound by the FP64 pipe and
// its issue slots (about 170 warp instructions per 32 cells, four IEEE quotients
// among them), and its bundles went through device memory (1 KB per pair).
//
// ---- the enclosures ------------------------------------------------------------
// u = 2^-24 (half an ulp at 1). Inputs are the FP64 values the reference uses, each
// rounded once to single precision (relative error u): X, Y = DX, DY; the trig values
// of T0 -+ dt (c, s) and of T2t_j (cT, sT); the grid offsets d, d^2 and 2d + 2dx. The
// trig values are at most 1; R = hypot(DX, DY) <= Rb = |X| + |Y| up to u; dm = max |d|.
// Every operation below rounds once, fma included.
//   s    = fma(sT, c, cT (-s'))      the sine of T2t - (T0 -+ dt) by the addition
//                                    theorem: |err| <= 2u|sT c| + 3u|cT s'| + u|s| <= 4u
//   t2   = fma(sT, -2X, cT 2Y)       -2 tt: |err| <= 8uR
//   cn   = fma(c, X, s Y)            |err| <= 4uR
//   D    = fma(-s, d, cn)            |err| <= 5uR + 6u dm                     =: dD
//   A    = X^2 + Y^2 - dx^2          |err| <= 5uR^2 + 4u dx^2
//   e1   = fma(d, t2, A + d^2)       |err| <= u (7R^2 + 12 dm R + 3dm^2 + 6dx^2) =: dE
//   N    = t2 + (2d + 2dx)           -2 (tt - d - dx): |err| <= 10uR + 4u (dm + dx)
//   lower k_dx = N (-1 / e1), upper k_dx = fma(-4dx, -1 / e1, lower), k_dt = s / D; the
//   reciprocals by rcp.approx (2u), in lane_bundle those of the two D from one of their
//   product.
// For a quotient of true value k, |err| <= (dN + |k| dE) / |e1| + 8u|k| with dN = N's
// bound + 12u dx (for the upper one's second term), and (4u + |k| dD) / |D| + 8u|k|. With
// e0 = 2^-14 max_k, a cell is accepted when
//   e1 >= Ethr = (dN + max_k dE) / (e0 - 8u max_k), and for both denominators
//   |D| >= Dthr = (4u + max_k dD) / (e0 - 8u max_k),
// so that each bound is off by at most e0 max(1, |k| / max_k): by e0 where it lies
// within [-max_k, max_k]; a larger one is recognised as larger (2^-14 of its size is
// less than its distance past max_k plus e0), and clamps or closes the cell either way.
// |D| below Dthr is accepted too when |s| >= S1 = 2 max_k Dthr + 8u and |D| >= Dtiny > dD
// at the longest pair's R (pair_radius): then |k| > 1.4 max_k with the sign of its
// quotient certain.
// Where a column fails, it is made once more with e1, the numerators, s and D computed in
// FP64 and rounded once each (fine_column). Its roundings to single precision leave a
// quotient off by 12u |k|. Its FP64 quantities differ from the reference's by their own
// rounding and by that of the reference's angles: half an ulp of T2t, and half one of
// T2t - (T0 -+ dt), so at most 2^-52 (|T2| + |T0| + dt + max |dt_j|). With
// eps = 2^-51 (|T2| + |T0| + dt + max |dt_j| + 4) for both,
//   s: eps    D: eps (R + dm) =: fD    N: eps (3R + dm + dx) =: fN
//   e1: eps (R^2 + 3 dm R + dm^2 + dx^2) =: fE
// at the longest pair's R, and, as above, a cell is accepted when
//   e1 >= (fN + max_k fE) / (e0 - 12u max_k),  |D| >= (eps + max_k fD) / (e0 - 12u max_k).
// (2^-27 and 2^-30 for the default parameters and orientations within a turn.)
// The FP64 path's own rounding (2^-50 of these magnitudes), the addition theorem on
// its rounded angles (|theta| <= FAST_ANGLE = 2^20, checked when binning: 2^-31, against 4u
// = 2^-22 in s and likewise in the others) and higher orders of u are covered by 2% on
// Ethr, Dthr and S1.
// Bounds are kept as (n, M): n the negated lower one, so that an intersection takes the
// smaller of both, and a cell is open when M + n > 0. With h = 2.04 e0,
//   min M + min n >  h       every bound considered, the cell is open;
//   min M + min n <= -h      it is closed;
// and anything between is undecided: a few tests in ten thousand.
#pragma once

#include "cvl_enclosures.h"
#include "cvl_path.cuh"
#include "cvl_search.cuh"

namespace cvl {

constexpr int FAST_CAP = 32;     // pairs of a direction run k_curvelets takes (k_curvelets_exact: FAST_WIDE)
// Bundles of an anchor's seeds kept in shared memory (later seeds' are recomputed), warps per
// block and blocks per SM. The kernel is bound by its issue slots; 5 blocks (96 registers, no
// spills) with 16 slots measured best: 1.42 ms on a 735k-edge map and 14.6 ms on a dense
// 3.65M-edge one, against 1.49 and 15.0 ms with 6 blocks (80 registers) and 12 slots, and 1.55
// and 16.1 ms with 7 and 10.
constexpr int FAST_SLOTS = 16;
constexpr int FAST_WARPS = 4;
constexpr int FAST_BLOCKS = 5;
constexpr int FAST_EXACT_BLOCKS = 3;
// bundle slots of a k_curvelets_exact warp, as many as three blocks of an SM have room for (a
// seed past them has its bundle made again at every visit: with 4 slots a 3.65M-edge run's
// two kernels took 14.64 ms, with these 14.48; 16 or 24 in two blocks: 14.82)
constexpr int FAST_WIDE_SLOTS = 14;
constexpr int FAST_TILE = 4;     // consecutive anchors a queue-pulling warp takes at a time

struct FastBinned {
    FastEdge *e;     // [N], bucket order
    double2 *cs2;    // [N] cos(theta), sin(theta)
    int4 *at;        // [N] pixel cell, input index, map
};

// Records of k_curvelets: ids[slot][gms] internal edge indices, the seed's first (its
// bundle starts the chain's), then the chain's after the anchor; meta = len |
// rank of the best cell << 8 | forward << 24.
struct FastArgs {
    Model md;
    FastModel fm;
    EdgeRecords B;
    FastBinned F;
    int a_begin, a_end;
    const unsigned long long *row;      // [N] the anchors' rows (pack_row)
    const int *csr_ids;
    const unsigned char *pcls;          // run | close << 2 | branch1 << 3
    unsigned *rec_ids, *rec_meta;
    unsigned long long arena_cap;       // below 2^32
    unsigned long long *arena_ctr;
    unsigned *rec_base, *run_cnt, *count;  // by input index, as GrowthArgsT
    MapStats *stats;
    int count_only;
    unsigned *err;
    unsigned arena_chunk;               // records a warp reserves at a time
    int tile;                           // consecutive anchors a warp takes at a time
    const RunDims *dims;                // graph runs: the anchors are [0, dims->N)
    unsigned *queue;                    // QUEUE: tiles taken so far
    unsigned *over_cnt;                 // anchors k_curvelets leaves to k_curvelets_exact
    unsigned *over_queue;               // the next of them (0 at start)
    int *over_list;
    const unsigned *unfit;              // UNFIT_*
};

constexpr unsigned L_KMASK = 0x3ffu, L_NOSEED = 0x2000u, L_CLOSE = 0x4000u, L_BRANCH1 = 0x8000u;
constexpr unsigned S_CLOSE = 0x80u;  // in a seed's byte: a close pair
constexpr float CLOSED = -1e30f;     // a bound past the grid's cells

constexpr int SLOT_PITCH = 68;       // 64 cells, and a bank shift between slots: a round's stores conflict nowhere

// Shared memory of one warp.
template <int CAP, int SLOTS>
struct FastSmem {
    // pair constants: -2X, 2Y, A, Ethr | cos, -sin, cn of the lower k_dt bound, Dthr | of the upper, S1
    float4 geo[CAP + 4][3];          // (a round may read past its last pair)
    float2 slot[SLOTS][SLOT_PITCH];  // bounds (n, M) by cell
    float2 trig[8];                  // sin, cos of T2t_j (9 offsets and 64 cells: Q <= 7)
    int nn[CAP];                     // internal neighbour by list position
    unsigned short list[2 * CAP];    // the first run's pairs, then the second's: k | flags
    unsigned char seed[2][CAP];      // list position of each run's seeds
};
struct FastWideSmem : FastSmem<FAST_WIDE, FAST_WIDE_SLOTS> {
    unsigned cur[FAST_WIDE / 32], skip[FAST_WIDE / 32];
    unsigned mask[FAST_WIDE][FAST_WIDE / 32], meta[FAST_WIDE];  // accepted chains
};
// and of the block: cos/sin of each orientation offset; d, d^2, 2d + 2dx by cell
struct FastBlockSmem {
    double2 cs[8];
    float4 cell[64];  // (w: the cell's orientation sample, an integer)
};
template <class W>
constexpr size_t fast_smem_bytes() {
    return sizeof(FastBlockSmem) + FAST_WARPS * sizeof(W);
}

__device__ __forceinline__ float rcp_approx(float x) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// The reference's bounds of one cell of pair (anchor i, neighbour nn), in FP64.
struct CellAnchor {  // the part of a cell that is the anchor's
    double d, T2t, sT, cT;
};
__device__ __forceinline__ CellAnchor cell_anchor(const Model &md, double T2, int cell) {
    CellAnchor c;
    const int ci = cell / md.Q, j = cell - ci * md.Q;
    c.d = grid_offset(md.sx, ci, md.P);
    c.T2t = T2 + grid_offset(md.st, j, md.Q);  // :698-702
    sincos(c.T2t, &c.sT, &c.cT);
    return c;
}
__device__ __forceinline__ void exact_cell(const Model &md, const EdgeRecords &B, double2 cs2, int i, int nn,
                                           const CellAnchor &c, double &m, double &M) {
    const PairGeom g = pair_geom(md, B.x[i], B.y[i], cs2.x, cs2.y, B.x[nn], B.y[nn], B.sp[nn], B.cp[nn], B.sm[nn],
                                 B.cm[nn]);
    if (g.close) {  // the default bundle (:682-687)
        m = -md.max_k;
        M = md.max_k;
        return;
    }
    const double T0 = B.th[nn];
    const double s_m = sin(c.T2t - (T0 - md.dt)), s_p = sin(c.T2t - (T0 + md.dt));  // :728-729
    const double tt = c.sT * g.DX - c.cT * g.DY;  // :705
    bundle_cell_fp64<QUOT_DIVIDE>(md, c.d, 2.0 * c.d, c.d * c.d, transport_column(md, g, tt, s_m, s_p), m, M);
}
__device__ __forceinline__ void exact_cell(const Model &md, const EdgeRecords &B, double2 cs2, int i, int nn,
                                           int cell, double &m, double &M) {
    exact_cell(md, B, cs2, i, nn, cell_anchor(md, B.th[i], cell), m, M);
}

// Out of line, for undecided cells: whether the cell is open in the intersection of the
// bundles of the pair at list position ps, of the seeds in mask, and of the pair at pr
// (pr >= 0).
__device__ __noinline__ bool exact_open(const FastArgs &a, const FastWideSmem &S, int f, int i, int ps,
                                        const unsigned *mask, int pr, int cell) {
    const double2 cs2 = a.F.cs2[i];
    double m, M;
    exact_cell(a.md, a.B, cs2, i, S.nn[ps], cell, m, M);
    for (int w = 0; w < FAST_WIDE / 32; ++w) {
        unsigned b = mask ? mask[w] : 0u;
        while (b) {
            const int s = 32 * w + __ffs(b) - 1;
            b &= b - 1;
            double m2, M2;
            exact_cell(a.md, a.B, cs2, i, S.nn[S.seed[f][s] & ~S_CLOSE], cell, m2, M2);
            if (m < m2) m = m2;
            if (M > M2) M = M2;
        }
    }
    if (pr >= 0) {
        double m2, M2;
        exact_cell(a.md, a.B, cs2, i, S.nn[pr], cell, m2, M2);
        if (m < m2) m = m2;
        if (M > M2) M = M2;
    }
    return M > m;
}

// Out of line: bounds (n, M) of this lane's two cells of a pair the enclosures do not
// cover, from the FP64 bounds, rounded inwards.
__device__ __noinline__ float4 exact_bundle(const FastArgs &a, int i, int nn, int lane) {
    const double2 cs2 = a.F.cs2[i];
    float4 o = make_float4(CLOSED, CLOSED, CLOSED, CLOSED);
    double m, M;
    if (2 * lane < a.md.cells) {
        exact_cell(a.md, a.B, cs2, i, nn, 2 * lane, m, M);
        o.x = __double2float_rd(-m);
        o.y = __double2float_rd(M);
    }
    if (2 * lane + 1 < a.md.cells) {
        exact_cell(a.md, a.B, cs2, i, nn, 2 * lane + 1, m, M);
        o.z = __double2float_rd(-m);
        o.w = __double2float_rd(M);
    }
    return o;
}

// Two single-precision values operated on together (f32x2 instructions: one issue slot for
// two cells), kept as the 64-bit register pair the instructions take.
using f32x2 = unsigned long long;
__device__ __forceinline__ f32x2 pack2(float x, float y) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
    return r;
}
__device__ __forceinline__ f32x2 pack2(float2 v) { return pack2(v.x, v.y); }
__device__ __forceinline__ f32x2 dup2(float x) { return pack2(x, x); }
__device__ __forceinline__ float2 unpack2(f32x2 v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
    f32x2 d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
    f32x2 d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ float min3(float a, float b, float c) {
    float d;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}
__device__ __forceinline__ float max3(float a, float b, float c) {
    float d;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}

// Bounds of two cells of one pair, with the denominators for the acceptance test. nslo,
// nshi: the negated sines of the k_dt bounds.
struct TwoCells {
    float2 e1, dlo, dhi;
    float n0, M0, n1, M1;
};
__device__ __forceinline__ TwoCells two_cells(const FastModel &fm, f32x2 d, f32x2 d2, f32x2 c2, f32x2 t2, f32x2 A,
                                              f32x2 nslo, f32x2 nshi, f32x2 cnlo, f32x2 cnhi) {
    TwoCells o;
    const f32x2 e1 = fma2(d, t2, add2(A, d2)), dlo = fma2(nslo, d, cnlo), dhi = fma2(nshi, d, cnhi);
    o.e1 = unpack2(e1);
    o.dlo = unpack2(dlo);
    o.dhi = unpack2(dhi);
    const f32x2 nre = pack2(rcp_approx(-o.e1.x), rcp_approx(-o.e1.y));
    const f32x2 klo = mul2(add2(t2, c2), nre), khi = fma2(nre, dup2(fm.ndx_4), klo);
    const float2 dd = unpack2(mul2(dlo, dhi));
    const f32x2 nrd = pack2(rcp_approx(-dd.x), rcp_approx(-dd.y));
    const f32x2 tlo = mul2(nslo, mul2(nrd, dhi)), thi = mul2(nshi, mul2(nrd, dlo));  // (-s) (-1 / D)
    const float2 kl = unpack2(klo), kh = unpack2(khi), tl = unpack2(tlo), th = unpack2(thi);
    o.n0 = min3(-kl.x, -tl.x, fm.mk);
    o.n1 = min3(-kl.y, -tl.y, fm.mk);
    o.M0 = min3(kh.x, th.x, fm.mk);
    o.M1 = min3(kh.y, th.y, fm.mk);
    return o;
}

// Bounds (n0, M0, n1, M1) of this lane's two cells (2 lane, 2 lane + 1) of the pair at list
// position p; every lane of the warp calls. covered: the enclosures hold (warp-uniform).
__device__ __forceinline__ float4 lane_bundle(const FastArgs &a, const float4 *geo, const float2 *trig,
                                              const FastBlockSmem &T, int lane, bool &covered) {
    const FastModel &fm = a.fm;
    const float4 g0 = geo[0], g1 = geo[1], g2 = geo[2];
    const int c0 = 2 * lane < a.md.cells ? 2 * lane : 0, c1 = 2 * lane + 1 < a.md.cells ? 2 * lane + 1 : c0;
    const float4 q0 = T.cell[c0], q1 = T.cell[c1];
    const float2 s0 = trig[__float_as_int(q0.w)], s1 = trig[__float_as_int(q1.w)];
    const f32x2 sT = pack2(s0.x, s1.x), cT = pack2(s0.y, s1.y);
    const f32x2 t2 = fma2(sT, dup2(g0.x), mul2(cT, dup2(g0.y)));
    const float2 slo = unpack2(fma2(sT, dup2(g1.x), mul2(cT, dup2(g1.y))));
    const float2 shi = unpack2(fma2(sT, dup2(g2.x), mul2(cT, dup2(g2.y))));
    const TwoCells o = two_cells(fm, pack2(q0.x, q1.x), pack2(q0.y, q1.y), pack2(q0.z, q1.z), t2, dup2(g0.z),
                                 pack2(-slo.x, -slo.y), pack2(-shi.x, -shi.y), dup2(g1.z), dup2(g2.z));
    const float dthr = g1.w, S1 = g2.w;
    const bool ok = fminf(o.e1.x, o.e1.y) >= g0.w && fabsf(o.dlo.x) >= (fabsf(slo.x) >= S1 ? fm.dtiny : dthr) &&
                    fabsf(o.dlo.y) >= (fabsf(slo.y) >= S1 ? fm.dtiny : dthr) &&
                    fabsf(o.dhi.x) >= (fabsf(shi.x) >= S1 ? fm.dtiny : dthr) &&
                    fabsf(o.dhi.y) >= (fabsf(shi.y) >= S1 ? fm.dtiny : dthr);
    covered = __all_sync(FULL, ok);
    return make_float4(2 * lane < a.md.cells ? o.n0 : CLOSED, o.M0, 2 * lane + 1 < a.md.cells ? o.n1 : CLOSED, o.M1);
}

// A column's cells from quantities computed in FP64 and rounded once. Returns whether the
// enclosures hold.
__device__ __forceinline__ bool fine_column(const FastArgs &a, double2 cs, int i, int nn, bool branch1, float2 *b,
                                            float &wmax) {
    const double2 c2 = a.F.cs2[i];
    const FastEdge ae = a.F.e[i];
    const float ang = fabsf((float)a.B.th[i]) + fabsf((float)a.B.th[nn]) + a.fm.fa;
    const float ethr = a.fm.fe * ang, dthr = a.fm.fd * ang;
    const double sT = fma(c2.y, cs.x, c2.x * cs.y), cT = fma(c2.x, cs.x, -(c2.y * cs.y));
    const double X = ae.x - a.F.e[nn].x, Y = ae.y - a.F.e[nn].y;
    const double cm = a.B.cm[nn], sm = a.B.sm[nn], cp = a.B.cp[nn], sp = a.B.sp[nn];
    const double cl = branch1 ? cm : cp, sl = branch1 ? sm : sp, ch = branch1 ? cp : cm, sh = branch1 ? sp : sm;
    const double t2 = -2.0 * fma(sT, X, -(cT * Y));
    const double slo = fma(sT, cl, -(cT * sl)), shi = fma(sT, ch, -(cT * sh));
    const double A = fma(X, X, fma(Y, Y, -a.md.dx2)), cnlo = fma(cl, X, sl * Y), cnhi = fma(ch, X, sh * Y);
    const float slof = (float)slo, shif = (float)shi;
    bool ok = true;
    wmax = CLOSED;
#pragma unroll
    for (int k = 0; k < FAST_P; ++k) {
        const double d = grid_offset(a.md.sx, k, FAST_P);
        const float e1 = (float)fma(d, t2 + d, A);
        const float dlo = (float)fma(-slo, d, cnlo), dhi = (float)fma(-shi, d, cnhi);
        const double N = t2 + 2.0 * d;  // -2 (tt - d)
        const float re = rcp_approx(e1);
        const float n = min3((float)(N + 2.0 * a.md.dx) * re, -(slof * rcp_approx(dlo)), a.fm.mk);
        const float M = min3((float)(2.0 * a.md.dx - N) * re, shif * rcp_approx(dhi), a.fm.mk);
        ok = ok && e1 >= ethr && fabsf(dlo) >= dthr && fabsf(dhi) >= dthr;
        wmax = fmaxf(wmax, n + M);
        b[k] = make_float2(n, M);
    }
    return ok;
}

// The block's tables, filled by all its threads (ends with a barrier).
__device__ __forceinline__ void fast_tables(const Model &md, FastBlockSmem &T) {
    for (int t = threadIdx.x; t < 64; t += blockDim.x) {
        const int c = t < md.cells ? t : 0;
        const double d = grid_offset(md.sx, c / md.Q, md.P);
        T.cell[t] = make_float4((float)d, (float)(d * d), (float)(2.0 * d + 2.0 * md.dx), __int_as_float(c % md.Q));
        if (t < 8) {
            double s, co;
            sincos(grid_offset(md.st, t < md.Q ? t : 0, md.Q), &s, &co);
            T.cs[t] = make_double2(co, s);
        }
    }
    __syncthreads();
}

// sin/cos(T2t_j) of the anchor for the samples j < Q, by the addition theorem in FP64
// (off by 2^-41 at most), a lane each.
__device__ __forceinline__ void fast_trig(const FastBlockSmem &T, double2 t2, int Q, int lane, float2 *trig) {
    if (lane < Q) {
        const double2 o = T.cs[lane];
        trig[lane] = make_float2((float)fma(t2.y, o.x, t2.x * o.y), (float)fma(t2.x, o.x, -(t2.y * o.y)));
    }
}

// The pairs of the anchor's direction runs, in neighbour order, to list: the first run's
// (a perpendicular pair is no seed; it goes with them for its validity), then the second's,
// at cnt0 when all fit in cap places, else at cap.
__device__ __forceinline__ void fast_lists(const unsigned char *pcls, int deg, int cap, int lane, unsigned short *list,
                                           int &cnt0, int &cnt1, unsigned &close_cnt) {
    const unsigned lt_mask = (1u << lane) - 1u;
    auto entry = [](int k, unsigned cl) {
        return (unsigned short)((unsigned)k | ((cl & 4u) ? L_CLOSE : 0u) | ((cl & 8u) ? L_BRANCH1 : 0u) |
                                ((cl & 3u) == 2u ? L_NOSEED : 0u));
    };
    cnt0 = cnt1 = 0;
    close_cnt = 0;
    for (int pass = 0; pass < 2; ++pass) {
        const int base = pass == 0 ? 0 : (deg <= cap ? cnt0 : cap);
        int n = 0;
        for (int k0 = 0; k0 < deg; k0 += 32) {
            const int k = k0 + lane;
            const unsigned cl = k < deg ? pcls[k] : 0u;
            const bool t = k < deg && ((cl & 3u) == 1u) == (pass == 1);
            const unsigned b = __ballot_sync(FULL, t);
            const int at = n + __popc(b & lt_mask);
            if (t && at < cap) list[base + at] = entry(k, cl);
            n += __popc(b);
            close_cnt += __popc(__ballot_sync(FULL, t && (cl & 4u)));
        }
        if (pass == 0) cnt0 = n; else cnt1 = n;
    }
}

// The constants of one pair, to geo. A close pair needs none: its thresholds are always met.
__device__ __forceinline__ void fast_constants(const FastModel &fm, double ax, double ay, const FastEdge &ne, bool close,
                                               bool b1, float4 *geo) {
    const float X = (float)(ax - ne.x), Y = (float)(ay - ne.y);
    const float Rb = fabsf(X) + fabsf(Y);
    // the lower k_dt bound is from T0 - dt in branch 1, else from T0 + dt
    const float cl = b1 ? ne.cm : ne.cp, sl = b1 ? ne.sm : ne.sp;
    const float ch = b1 ? ne.cp : ne.cm, sh = b1 ? ne.sp : ne.sm;
    const float ethr = fmaf(Rb, fmaf(Rb, fm.eRR, fm.eR), fm.e0), dthr = fmaf(Rb, fm.dR, fm.d0);
    const float S1 = fmaf(Rb, fm.sR, fm.s0);
    geo[0] = make_float4(-2.0f * X, 2.0f * Y, fmaf(X, X, fmaf(Y, Y, -fm.dx2)), close ? CLOSED : ethr);
    geo[1] = make_float4(cl, -sl, fmaf(cl, X, sl * Y), close ? -1.0f : dthr);
    geo[2] = make_float4(ch, -sh, fmaf(ch, X, sh * Y), close ? 1e30f : S1);
}

// The same for cnt pairs of a list, a lane each.
__device__ __forceinline__ void fast_list_constants(const FastArgs &a, unsigned long long off, double ax, double ay,
                                                    const unsigned short *list, int cnt, int lane, float4 (*geo)[3],
                                                    int *nns) {
    for (int p = lane; p < cnt; p += 32) {
        const unsigned e = list[p];
        const int nn = a.csr_ids[off + (e & L_KMASK)];
        nns[p] = nn;
        fast_constants(a.fm, ax, ay, a.F.e[nn], e & L_CLOSE, e & L_BRANCH1, geo[p]);
    }
}

// A warp's map counts, flushed when the map changes.
struct FastCounts {
    int map = -1;
    unsigned valid = 0u, close = 0u;
    __device__ __forceinline__ void flush(MapStats *stats, int lane) {
        if (lane == 0 && map >= 0 && (valid | close)) {
            atomicAdd(&stats[map].valid_pairs, valid);
            atomicAdd(&stats[map].close_pairs, close);
        }
    }
    __device__ __forceinline__ void add(MapStats *stats, int lane, int m, unsigned v, unsigned c) {
        if (m != map) {
            flush(stats, lane);
            map = m;
            valid = close = 0u;
        }
        valid += v;
        close += c;
    }
};

// ---------------------------------------------------------------------------
// k_curvelets: a warp per anchor.
//  - Bundles: four pairs at a time, a lane per (pair, orientation sample), which makes
//    the 9 cells of its column in registers, two per f32x2 instruction, with the
//    column's sines and the pair's constants shared by them. The pairs' validity is a
//    ballot; the valid ones' cells go to shared memory, where the growth reads a bundle
//    as two cells per lane.
//  - Growth: seed by seed (:479-545), a vote per intersection (:832-854).
// Both direction runs' bundles are made together when the anchor's pairs fit (32), which
// leaves fewer lanes of the last round idle.
// ---------------------------------------------------------------------------
template <bool QUEUE>
__global__ void __launch_bounds__(FAST_WARPS * 32, FAST_BLOCKS) k_curvelets(const __grid_constant__ FastArgs a) {
    extern __shared__ __align__(16) unsigned char cv_smem[];
    using Smem = FastSmem<FAST_CAP, FAST_SLOTS>;
    const Model &md = a.md;
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    if (*a.unfit) {  // no rows; the host runs the two-kernel path instead, or fails
        if (blockIdx.x == 0 && threadIdx.x == 0) atomicOr(a.err, ERR_ANGLE);
        return;
    }
    FastBlockSmem &T = *(FastBlockSmem *)cv_smem;
    Smem &S = ((Smem *)(cv_smem + sizeof(FastBlockSmem)))[wib];
    fast_tables(md, T);
    for (int k = lane; k < FAST_SLOTS * SLOT_PITCH; k += 32)  // (the cells past the grid stay closed)
        S.slot[0][k] = make_float2(CLOSED, CLOSED);

    constexpr int PPR = 4;                   // pairs per round (9 offsets and 64 cells: Q <= 7 samples)
    const int Q = md.Q, pl = lane & (PPR - 1), jl = lane / PPR;  // the lane's pair and sample
    const unsigned lt_mask = (1u << lane) - 1u;
    const unsigned rank0 = 2 * lane < md.cells ? (unsigned)a.fm.rank[2 * lane] : 0xffffu;
    const unsigned rank1 = 2 * lane + 1 < md.cells ? (unsigned)a.fm.rank[2 * lane + 1] : 0xffffu;
    const float h = a.fm.h;

    FastCounts counts;
    unsigned ch_cur = 0, ch_left = 0;  // the warp's arena chunk: next record, records left

    const int a_end = a.dims ? a.dims->N : a.a_end;
    const int tiles = (a_end - a.a_begin + a.tile - 1) / a.tile;
    auto next_tile = [&](int cur) -> int {
        if constexpr (!QUEUE) return cur + (int)gridDim.x * FAST_WARPS;
        unsigned q = 0;
        if (lane == 0) q = atomicAdd(a.queue, 1u);
        return (int)__shfl_sync(FULL, q, 0);
    };
    for (int t = QUEUE ? next_tile(0) : (int)blockIdx.x * FAST_WARPS + wib; t < tiles; t = next_tile(t))
    for (int i = a.a_begin + t * a.tile, i_end = min(i + a.tile, a_end); i < i_end; ++i) {
        const unsigned long long row = a.row[i];
        if (row == NO_ROW) continue;  // (ERR_CAPACITY is raised: the run is run again)
        const unsigned long long off = row & ((1ull << 48) - 1ull);
        const int deg = (int)(row >> 48);
        const bool joint = deg <= FAST_CAP;  // both runs' pairs in one pass
        __syncwarp();
        fast_trig(T, a.F.cs2[i], Q, lane, S.trig);
        int cnt0 = 0, cnt1 = 0;
        unsigned close_cnt = 0, closes = 0u, noseed = 0u;  // close, perpendicular pairs by list position
        float undecided = CLOSED;  // the largest w of a test that found nothing open, by lane
        if (joint) {
            // a lane per pair: its place in the list (the first run's pairs, perpendicular ones
            // with them, then the second's, each in neighbour order), its constants
            const unsigned cl = lane < deg ? a.pcls[off + lane] : 0u;
            const bool second = (cl & 3u) == 1u;
            const unsigned b1 = __ballot_sync(FULL, second);
            cnt1 = __popc(b1);
            cnt0 = deg - cnt1;
            const int at = second ? cnt0 + __popc(b1 & lt_mask) : __popc(~b1 & lt_mask);
            closes = __reduce_or_sync(FULL, (cl & 4u) ? 1u << at : 0u);
            noseed = __reduce_or_sync(FULL, (cl & 3u) == 2u ? 1u << at : 0u);
            close_cnt = __popc(closes);
            if (lane < deg) {
                const int nn = a.csr_ids[off + lane];
                S.nn[at] = nn;
                S.list[at] = (cl & 8u) ? L_BRANCH1 : 0u;
                fast_constants(a.fm, a.F.e[i].x, a.F.e[i].y, a.F.e[nn], cl & 4u, cl & 8u, S.geo[at]);
            }
        } else {
            fast_lists(a.pcls + off, deg, FAST_CAP, lane, S.list, cnt0, cnt1, close_cnt);
            if (max(cnt0, cnt1) > FAST_CAP) undecided = 1e30f;
        }
        __syncwarp();

        const int orig = a.B.orig[i];
        unsigned valid_cnt = 0;
        const unsigned ch_left0 = ch_left;
        bool new_chunk = false;
        int ns0 = 0, ns1 = 0;  // seeds of each run: seed s of the first is at slot s, of the second at slot ns0 + s
        // Accepted chain z of the anchor (of a run, when not joint) is with lane z. A chain is
        // its set of seeds, a bit mask: the walk takes them in ascending order.
        unsigned my_mask = 0u, my_meta = 0u, n_acc = 0, n_acc0 = 0;
        for (int f = 0; f < 2; ++f) {
            if (__any_sync(FULL, undecided > -h)) break;
            if (f == 0 || !joint) {
                // ---- the bundles of this pass's pairs, round by round
                const int cnt = joint ? deg : (f == 0 ? cnt0 : cnt1);
                const int n_first = joint ? cnt0 : (f == 0 ? cnt : 0);  // the first run's pairs
                const unsigned short *list = S.list + (f == 1 ? FAST_CAP : 0);
                if (!joint) {
                    fast_list_constants(a, off, a.F.e[i].x, a.F.e[i].y, list, cnt, lane, S.geo, S.nn);
                    const unsigned le = lane < cnt ? list[lane] : 0u;
                    closes = __ballot_sync(FULL, le & L_CLOSE);
                    noseed = __ballot_sync(FULL, le & L_NOSEED);
                    __syncwarp();
                }
                const float2 tj = S.trig[jl];
                const int p_end = jl < Q ? cnt : 0;
                unsigned validm = closes, unsurem = 0u;  // by list position; unsurem by lane
                for (int p0 = 0; p0 < cnt; p0 += PPR) {
                    const int p = p0 + pl;
                    const bool on = p < p_end;
                    float2 b[FAST_P];
                    float wmax = CLOSED;
                    const float4 g0 = S.geo[p][0], g1 = S.geo[p][1], g2 = S.geo[p][2];
                    const float t2 = fmaf(tj.x, g0.x, tj.y * g0.y);
                    const float slo = fmaf(tj.x, g1.x, tj.y * g1.y), shi = fmaf(tj.x, g2.x, tj.y * g2.y);
                    {
                        float emin = 1e30f, dlmin = 1e30f, dhmin = 1e30f;
                        float pe = 0.0f, pl_ = 0.0f, ph = 0.0f, pw = 0.0f;  // of the cell before: two cells to a min
#pragma unroll
                        for (int k = 0; k < FAST_P; ++k) {
                            const float e1 = fmaf(a.fm.d[k], t2, g0.z + a.fm.d2[k]);
                            const float dlo = fmaf(-slo, a.fm.d[k], g1.z), dhi = fmaf(-shi, a.fm.d[k], g2.z);
                            const float nre = rcp_approx(-e1);
                            const float klo = (t2 + a.fm.c2[k]) * nre, khi = fmaf(nre, a.fm.ndx_4, klo);
                            const float tlo = slo * rcp_approx(dlo), thi = shi * rcp_approx(dhi);
                            const float n = min3(-klo, -tlo, a.fm.mk), M = min3(khi, thi, a.fm.mk);
                            if (k & 1) {
                                emin = min3(emin, pe, e1);
                                dlmin = min3(dlmin, fabsf(pl_), fabsf(dlo));
                                dhmin = min3(dhmin, fabsf(ph), fabsf(dhi));
                                wmax = max3(wmax, pw, n + M);
                            } else if (k == FAST_P - 1) {
                                emin = fminf(emin, e1);
                                dlmin = fminf(dlmin, fabsf(dlo));
                                dhmin = fminf(dhmin, fabsf(dhi));
                                wmax = fmaxf(wmax, n + M);
                            } else {
                                pe = e1;
                                pl_ = dlo;
                                ph = dhi;
                                pw = n + M;
                            }
                            b[k] = make_float2(n, M);
                        }
                        bool bad = on && !(emin >= g0.w && dlmin >= (fabsf(slo) >= g2.w ? a.fm.dtiny : g1.w) &&
                                           dhmin >= (fabsf(shi) >= g2.w ? a.fm.dtiny : g1.w));
                        if (__any_sync(FULL, bad)) {
                            if (bad && !fine_column(a, T.cs[jl], i, S.nn[p], list[p] & L_BRANCH1, b, wmax))
                                undecided = 1e30f;
                        }
                    }
                    // validity (bundle_valid_check, :821-830): an open cell in any of the pair's
                    // columns, which are every fourth lane's
                    unsigned open = __ballot_sync(FULL, on && wmax > h);
                    open |= open >> 16;
                    open |= open >> 8;
                    open |= open >> 4;
                    validm |= (open & 0xfu) << p0;
                    if (on && wmax > -h) unsurem |= 1u << (p & 31);
                    const unsigned bit = 1u << (p & 31), found = validm & ~noseed;
                    const int s = __popc(found & (bit - 1u));
                    if (on && (found & bit) && s < FAST_SLOTS) {
                        float2 *dst = &S.slot[s][jl];
#pragma unroll
                        for (int k = 0; k < FAST_P; ++k) dst[k * Q] = b[k];
                    }
                }
                if (unsurem & ~validm) undecided = 1e30f;
                valid_cnt += __popc(validm);
                const unsigned seedm = validm & ~noseed;
                const unsigned firsts = n_first >= 32 ? FULL : (1u << n_first) - 1u;
                ns0 = __popc(seedm & firsts);
                ns1 = __popc(seedm & ~firsts);
                __syncwarp();
                if (seedm >> lane & 1u) {
                    const int s = __popc(seedm & lt_mask);
                    const bool close = closes >> lane & 1u;
                    S.seed[lane < n_first ? 0 : 1][lane < n_first ? s : s - ns0] =
                        (unsigned char)((unsigned)lane | (close ? S_CLOSE : 0u));
                }
                for (unsigned m = closes & seedm; m; m &= m - 1) {  // close pairs: the default bundle (:682-687)
                    const int s = __popc(seedm & ((m & -m) - 1u));
                    const float mk = a.fm.mk;
                    if (s < FAST_SLOTS)
                        *(float4 *)&S.slot[s][2 * lane] = make_float4(2 * lane < md.cells ? mk : CLOSED, mk,
                                                                      2 * lane + 1 < md.cells ? mk : CLOSED, mk);
                }
                __syncwarp();
                if (__any_sync(FULL, undecided > -h)) break;
            }

            const int ns = f == 0 ? ns0 : ns1;
            // A curvelet needs the anchor and at least two more edges (:549).
            if (!a.count_only && ns > 1 && md.gms > 2) {
                const unsigned char *seeds = S.seed[f];
                const int slot0 = joint && f ? ns0 : 0;  // (not joint: ns0 is this pass's)
                const int lim = FAST_SLOTS - slot0;      // seeds from here on have no slot
                const float4 *slots = (const float4 *)S.slot[0] + lane + slot0 * (SLOT_PITCH / 2);
                auto load_far = [&](int s) -> float4 {
                    const unsigned p = seeds[s];
                    if (p & S_CLOSE) {
                        const float mk = a.fm.mk;
                        return make_float4(2 * lane < md.cells ? mk : CLOSED, mk, 2 * lane + 1 < md.cells ? mk : CLOSED, mk);
                    }
                    bool covered;
                    const float4 b = lane_bundle(a, S.geo[p], S.trig, T, lane, covered);
                    if (!covered) undecided = 1e30f;
                    return b;
                };
                // The walk of bundle c over seeds [r, r_end): each whose bundle meets c's in an open
                // cell (:832-854) is taken, and c becomes the intersection; at most room.
                auto walk = [&](float4 &c, unsigned &mask, int &room, int r, int r_end) {
                    auto step = [&](float4 b) {
                        b.x = fminf(c.x, b.x);
                        b.y = fminf(c.y, b.y);
                        b.z = fminf(c.z, b.z);
                        b.w = fminf(c.w, b.w);
                        const float w = fmaxf(b.x + b.y, b.z + b.w);
                        if (__any_sync(FULL, w > h)) {
                            c = b;
                            mask |= 1u << r;
                            --room;
                        } else {
                            undecided = fmaxf(undecided, w);
                        }
                    };
                    const float4 *src = slots + r * (SLOT_PITCH / 2);
                    for (const int near = min(r_end, lim); r < near; ++r, src += SLOT_PITCH / 2) {
                        step(*src);
                        if (room == 0) return;
                    }
                    for (; r < r_end && room > 0; ++r) step(load_far(r));
                };
                // a chain of more than two edges that no earlier seed of the run has (first-wins,
                // :876-916): its best cell is the open one of least rank (:202-219)
                auto accept = [&](const float4 &c, unsigned mask, int s) {
                    const float w0 = c.x + c.y, w1 = c.z + c.w;
                    const unsigned own = min(w0 > h ? rank0 : 0xffu, w1 > h ? rank1 : 0xffu);
                    const unsigned best = __reduce_min_sync(FULL, own);
                    if ((rank0 < best && w0 > -h) || (rank1 < best && w1 > -h)) undecided = 1e30f;
                    if (lane == (int)n_acc) {
                        my_mask = mask;
                        my_meta = best | ((unsigned)s << 16) | ((unsigned)f << 24);
                    }
                    ++n_acc;
                };
                const int take = md.gms - 1;  // seeds a chain takes at most (the anchor is its first, :485)
                // Seed 0's chain C. Another seed s of C has the same chain: its walk takes and
                // refuses the same seeds (what it joins is a part of C, whose cells are open
                // together; and for what C's walk refused it holds at least as much). So has a
                // seed after a full C whose bundle meets all of C: its walk fills up with C before
                // it comes to itself. First-wins drops both.
                float4 c0;
                if (lim > 0) c0 = *slots; else c0 = load_far(0);
                unsigned C = 1u;
                int left = take - 1;
                walk(c0, C, left, 1, ns);
                if (take - left >= 2) accept(c0, C, 0);
                const int full_at = left == 0 ? 32 - __clz(C) : ns;  // seeds from here on are after a full C
                for (unsigned rest = ~C & (ns == 32 ? FULL : (1u << ns) - 1u); rest; rest &= rest - 1) {
                    const int s = __ffs(rest) - 1;
                    float4 c;
                    if (s < lim) c = slots[s * (SLOT_PITCH / 2)]; else c = load_far(s);
                    if (s >= full_at) {
                        const float w = fmaxf(fminf(c0.x, c.x) + fminf(c0.y, c.y), fminf(c0.z, c.z) + fminf(c0.w, c.w));
                        if (__any_sync(FULL, w > h)) continue;
                    }
                    unsigned mask = 0u;
                    int room = take;
                    walk(c, mask, room, 0, s);
                    if (room > 0) {  // the seed itself joins without intersection (:496-511)
                        mask |= 1u << s;
                        if (--room > 0) walk(c, mask, room, s + 1, ns);
                    }
                    if (take - room < 2) continue;
                    if (__any_sync(FULL, lane >= (int)n_acc0 && my_mask == mask)) continue;  // equal chains are equal masks
                    accept(c, mask, s);
                }
                if (__any_sync(FULL, undecided > -h)) break;
            }
            // ---- the records, in seed order, to the warp's arena chunk: of both runs together
            // when joint
            if (f == 0 && joint) {
                n_acc0 = n_acc;
                continue;
            }
            unsigned rbase = 0;
            if (n_acc) {
                if (n_acc > ch_left) {
                    const unsigned want = max(n_acc, a.arena_chunk);
                    unsigned long long at = 0;
                    if (lane == 0) at = atomicAdd(a.arena_ctr, (unsigned long long)want);
                    at = __shfl_sync(FULL, at, 0);
                    const bool fits = at + want <= a.arena_cap;
                    if (!fits && lane == 0) atomicOr(a.err, ERR_ARENA);
                    ch_cur = (unsigned)at;
                    ch_left = fits ? want : 0u;
                    new_chunk = true;
                }
                if (n_acc <= ch_left) {
                    rbase = ch_cur;
                    ch_cur += n_acc;
                    ch_left -= n_acc;
                    if (lane < (int)n_acc) {
                        const unsigned char *seeds = S.seed[my_meta >> 24];
                        unsigned *ids = a.rec_ids + (unsigned long long)(rbase + lane) * (unsigned)md.gms;
                        a.rec_meta[rbase + lane] = (unsigned)(1 + __popc(my_mask)) | ((my_meta & 0xffu) << 8) |
                                                   (my_meta >> 24 ? 0u : 1u << 24);
                        *ids++ = (unsigned)S.nn[seeds[my_meta >> 16 & 0xffu] & ~S_CLOSE];
                        for (; my_mask; my_mask &= my_mask - 1)
                            *ids++ = (unsigned)S.nn[seeds[__ffs(my_mask) - 1] & ~S_CLOSE];
                    }
                } else {
                    n_acc = n_acc0 = 0;  // (the arena is full: the run is run again)
                }
            }
            if (!a.count_only && lane == 0) {
                if (joint) {
                    a.rec_base[2 * orig] = rbase;
                    a.run_cnt[2 * orig] = n_acc0;
                    a.rec_base[2 * orig + 1] = rbase + n_acc0;
                    a.run_cnt[2 * orig + 1] = n_acc - n_acc0;
                    a.count[orig] = n_acc;
                } else {
                    a.rec_base[2 * orig + f] = rbase;
                    a.run_cnt[2 * orig + f] = n_acc;
                    if (f == 0) a.count[orig] = n_acc; else a.count[orig] += n_acc;
                }
            }
            if (!joint) {
                n_acc = n_acc0 = 0;
                my_mask = 0u;
            }
            __syncwarp();
        }
        if (__any_sync(FULL, undecided > -h)) {
            // k_curvelets_exact takes the whole anchor; this warp's records of it are dropped
            if (!new_chunk) {
                ch_cur -= ch_left0 - ch_left;
                ch_left = ch_left0;
            }
            if (lane == 0) a.over_list[atomicAdd(a.over_cnt, 1u)] = i;
            continue;
        }
        counts.add(a.stats, lane, a.B.map[i], valid_cnt, close_cnt);
    }
    counts.flush(a.stats, lane);
}

// ---------------------------------------------------------------------------
// k_curvelets_exact: the anchors k_curvelets left (an undecided comparison, a pair whose
// enclosures do not hold, or a run of more than 32 pairs), run by run, a pair's two cells
// per lane. It takes the same comparisons and settles the undecided ones in FP64.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(FAST_WARPS * 32, FAST_EXACT_BLOCKS) k_curvelets_exact(const __grid_constant__ FastArgs a) {
    extern __shared__ __align__(16) unsigned char cv_smem[];
    constexpr int SLOTS = FAST_WIDE_SLOTS;
    const Model &md = a.md;
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    if (*a.unfit) return;
    const int n_over = (int)*a.over_cnt;
    if ((int)blockIdx.x * FAST_WARPS >= n_over) return;
    FastBlockSmem &T = *(FastBlockSmem *)cv_smem;
    FastWideSmem &S = ((FastWideSmem *)(cv_smem + sizeof(FastBlockSmem)))[wib];
    fast_tables(md, T);
    const unsigned rank0 = 2 * lane < md.cells ? (unsigned)a.fm.rank[2 * lane] : 0xffffu;
    const unsigned rank1 = 2 * lane + 1 < md.cells ? (unsigned)a.fm.rank[2 * lane + 1] : 0xffffu;
    const float h = a.fm.h;
    FastCounts counts;
    for (;;) {
        unsigned it = 0;
        if (lane == 0) it = atomicAdd(a.over_queue, 1u);
        it = __shfl_sync(FULL, it, 0);
        if (it >= (unsigned)n_over) break;
        const int i = a.over_list[it];
        const unsigned long long row = a.row[i];
        const unsigned long long off = row & ((1ull << 48) - 1ull);
        const int deg = (int)(row >> 48);
        __syncwarp();
        int cnt0, cnt1;
        unsigned close_cnt;
        fast_lists(a.pcls + off, deg, FAST_WIDE, lane, S.list, cnt0, cnt1, close_cnt);
        fast_trig(T, a.F.cs2[i], md.Q, lane, S.trig);
        __syncwarp();
        const int orig = a.B.orig[i];
        unsigned valid_cnt = 0, n_out = 0;
        for (int f = 0; f < 2; ++f) {
            const int cnt = f == 0 ? cnt0 : cnt1;
            const unsigned short *list = S.list + (f == 1 ? cnt0 : 0);  // (deg <= FAST_WIDE)
            fast_list_constants(a, off, a.F.e[i].x, a.F.e[i].y, list, cnt, lane, S.geo, S.nn);
            __syncwarp();
            auto bundle = [&](int p, bool close) -> float4 {
                if (close) {
                    const float mk = a.fm.mk;
                    return make_float4(2 * lane < md.cells ? mk : CLOSED, mk, 2 * lane + 1 < md.cells ? mk : CLOSED, mk);
                }
                bool covered;
                const float4 b = lane_bundle(a, S.geo[p], S.trig, T, lane, covered);
                return covered ? b : exact_bundle(a, i, S.nn[p], lane);
            };
            unsigned char *seeds = S.seed[f];
            int ns = 0;
            for (int p = 0; p < cnt; ++p) {
                const bool close = list[p] & L_CLOSE;
                const float4 b = bundle(p, close);
                bool valid = true;
                if (!close) {
                    const float w0 = b.x + b.y, w1 = b.z + b.w;
                    valid = __any_sync(FULL, fmaxf(w0, w1) > h);
                    if (!valid && __any_sync(FULL, fmaxf(w0, w1) > -h)) {
                        const bool o = (w0 > -h && exact_open(a, S, f, i, p, nullptr, -1, 2 * lane)) ||
                                       (w1 > -h && exact_open(a, S, f, i, p, nullptr, -1, 2 * lane + 1));
                        valid = __any_sync(FULL, o);
                    }
                }
                if (valid) {
                    ++valid_cnt;
                    if (!(list[p] & L_NOSEED)) {
                        if (ns < SLOTS) *(float4 *)&S.slot[ns][2 * lane] = b;
                        if (lane == 0) seeds[ns] = (unsigned char)(p | (close ? S_CLOSE : 0u));
                        ++ns;
                    }
                }
            }
            __syncwarp();
            unsigned n_acc = 0;
            unsigned long long rbase = 0;
            bool fits = true;
            if (!a.count_only && ns > 1 && md.gms > 2) {
                auto load = [&](int s) -> float4 {
                    if (s < SLOTS) return *(const float4 *)&S.slot[s][2 * lane];
                    return bundle(seeds[s] & ~S_CLOSE, seeds[s] & S_CLOSE);
                };
                for (int s = 0; s < ns; ++s) {
                    if (s > 0 && (S.skip[s >> 5] >> (s & 31) & 1u)) continue;  // (as in k_curvelets)
                    float4 c = load(s);
                    const int ps = seeds[s] & ~S_CLOSE;
                    int left = md.gms - 1;
                    if (lane < FAST_WIDE / 32) S.cur[lane] = 0u;
                    __syncwarp();
                    for (int r = 0; r < ns; ++r) {
                        if (r != s) {
                            const float4 b = load(r);
                            const float4 t = make_float4(fminf(c.x, b.x), fminf(c.y, b.y), fminf(c.z, b.z),
                                                         fminf(c.w, b.w));
                            const float w0 = t.x + t.y, w1 = t.z + t.w;
                            bool take = __any_sync(FULL, fmaxf(w0, w1) > h);
                            if (!take && __any_sync(FULL, fmaxf(w0, w1) > -h)) {
                                const int pr = seeds[r] & ~S_CLOSE;
                                const bool o = (w0 > -h && exact_open(a, S, f, i, ps, S.cur, pr, 2 * lane)) ||
                                               (w1 > -h && exact_open(a, S, f, i, ps, S.cur, pr, 2 * lane + 1));
                                take = __any_sync(FULL, o);
                            }
                            if (!take) continue;
                            c = t;
                        }
                        if (lane == 0) S.cur[r >> 5] |= 1u << (r & 31);
                        __syncwarp();
                        if (--left == 0) break;
                    }
                    if (s == 0) {
                        if (lane < FAST_WIDE / 32) S.skip[lane] = S.cur[lane];
                        __syncwarp();
                    }
                    if (md.gms - 1 - left < 2) continue;
                    bool dup = false;
                    for (unsigned z = lane; z < n_acc; z += 32) {
                        unsigned diff = 0;
                        for (int w = 0; w < FAST_WIDE / 32; ++w) diff |= S.mask[z][w] ^ S.cur[w];
                        dup = dup || diff == 0u;
                    }
                    if (__any_sync(FULL, dup)) continue;
                    const float w0 = c.x + c.y, w1 = c.z + c.w;
                    unsigned best = w0 > h ? rank0 : 0xffu;
                    if (w1 > h && rank1 < best) best = rank1;
                    best = __reduce_min_sync(FULL, best);
                    const bool u0 = rank0 < best && w0 > -h, u1 = rank1 < best && w1 > -h;
                    if (__any_sync(FULL, u0 || u1)) {
                        unsigned bb = best;
                        if (u0 && exact_open(a, S, f, i, ps, S.cur, -1, 2 * lane)) bb = rank0;
                        if (u1 && rank1 < bb && exact_open(a, S, f, i, ps, S.cur, -1, 2 * lane + 1)) bb = rank1;
                        best = __reduce_min_sync(FULL, bb);
                    }
                    if (lane < FAST_WIDE / 32) S.mask[n_acc][lane] = S.cur[lane];
                    if (lane == 0) S.meta[n_acc] = (unsigned)(md.gms - left) | (best << 8) | ((unsigned)s << 16);
                    __syncwarp();
                    ++n_acc;
                }
                if (n_acc) {
                    if (lane == 0) rbase = atomicAdd(a.arena_ctr, (unsigned long long)n_acc);
                    rbase = __shfl_sync(FULL, rbase, 0);
                    fits = rbase + n_acc <= a.arena_cap;
                    if (!fits && lane == 0) atomicOr(a.err, ERR_ARENA);
                    for (unsigned z = lane; fits && z < n_acc; z += 32) {
                        const unsigned meta = S.meta[z];
                        unsigned *ids = a.rec_ids + (rbase + z) * (unsigned long long)md.gms;
                        *ids++ = (unsigned)S.nn[seeds[meta >> 16] & ~S_CLOSE];
                        for (int w = 0; w < FAST_WIDE / 32; ++w)
                            for (unsigned m = S.mask[z][w]; m; m &= m - 1)
                                *ids++ = (unsigned)S.nn[seeds[32 * w + __ffs(m) - 1] & ~S_CLOSE];
                        a.rec_meta[rbase + z] = (meta & 0xffffu) | (f == 0 ? 1u << 24 : 0u);
                    }
                }
            }
            if (!a.count_only && lane == 0) {
                a.rec_base[2 * orig + f] = (unsigned)rbase;
                a.run_cnt[2 * orig + f] = fits ? n_acc : 0u;
            }
            n_out += fits ? n_acc : 0u;
            __syncwarp();
        }
        if (lane == 0 && !a.count_only) a.count[orig] = n_out;
        counts.add(a.stats, lane, a.B.map[i], valid_cnt, close_cnt);
    }
    counts.flush(a.stats, lane);
}

// ---------------------------------------------------------------------------
// (e) finalize of k_curvelets' records: chain rows and info rows at anchor-major
// positions, as k_finalize, with the best cell's k range evaluated here in FP64: the
// seed's bundle, then the chain's in order, each bound selected as :513-527 does.
// k_finalize_exact: a lane per curvelet, a warp per tile of 32 anchors (input order). A round
// of 32 curvelets costs one pair after the other's chain of sines and quotients, which
// enough warps hide on a large run.
// k_finalize_small, for runs of up to 64 Ki edges, where latency is what counts: G lanes
// per curvelet (a power of two, at least group_max_sz), each with one of its pairs, and a
// warp per 8 anchors. The rows of a round's 32 / G curvelets are consecutive, so they are put
// together in shared memory and written as one run. (On a 242k-edge map it takes half as long
// again as k_finalize_exact: what is done once per curvelet leaves most lanes idle.)
// ---------------------------------------------------------------------------
struct FinalArgs {
    Model md;
    EdgeRecords B;
    const double2 *cs2;
    const int *pos_of;  // input index -> internal
    int N, M;
    const int *map_off;
    const unsigned *rec_ids, *rec_meta;
    const unsigned *rec_base, *run_cnt;
    const unsigned long long *out_off;
    unsigned long long out_cap;
    unsigned char cell_of[64];
    const unsigned *err;  // a run with an error is to be run again, or fails: nothing is written
    unsigned *chains;
    double *info;
    const RunDims *dims;
};

// (4 blocks of 256 per SM, 64 registers and some spills: it waits for its gathers. 1.77 ms on a
// dense 3.65M-edge map against 1.85 with 3 blocks and 2.15 with 2.)
__global__ void __launch_bounds__(256, 4) k_finalize_exact(const __grid_constant__ FinalArgs f) {
    const Model &md = f.md;
    if (*f.err) return;
    const int N = f.dims ? f.dims->N : f.N;
    const int W = md.gms + 1;
    const int lane = threadIdx.x & 31;
    const int warp = (int)((blockIdx.x * (unsigned)blockDim.x + threadIdx.x) >> 5);
    const int warps = (int)((gridDim.x * (unsigned)blockDim.x) >> 5);
    for (long long a0 = (long long)warp * 32; a0 < N; a0 += (long long)warps * 32) {
        const int a = (int)a0 + lane;
        unsigned c0 = 0, cnt = 0, rb0 = 0, rb1 = 0;
        unsigned long long dst = 0;
        int moff = 0, pos = 0;
        if (a < N) {
            c0 = f.run_cnt[2 * a];
            const unsigned c1 = f.run_cnt[2 * a + 1];
            dst = f.out_off[a];
            if (c0 + c1 > 0 && dst + c0 + c1 <= f.out_cap) {
                cnt = c0 + c1;
                rb0 = f.rec_base[2 * a];
                rb1 = f.rec_base[2 * a + 1];
                pos = f.pos_of[a];
                moff = f.map_off[f.B.map[pos]];
            }
        }
        unsigned incl = cnt;  // inclusive prefix of the tile's counts
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const unsigned o = __shfl_up_sync(FULL, incl, d);
            if (lane >= d) incl += o;
        }
        const unsigned total = __shfl_sync(FULL, incl, 31);
        for (unsigned e0 = 0; e0 < total; e0 += 32) {
            const unsigned e = e0 + lane;
            int T = 0;  // the anchor of curvelet e: the first lane whose inclusive prefix exceeds e
#pragma unroll
            for (int step = 16; step >= 1; step >>= 1) {
                const unsigned v = __shfl_sync(FULL, incl, T + step - 1);
                if (v <= e) T += step;
            }
            const unsigned r = e - (__shfl_sync(FULL, incl, T) - __shfl_sync(FULL, cnt, T));
            const unsigned lc0 = __shfl_sync(FULL, c0, T);
            const unsigned lrb0 = __shfl_sync(FULL, rb0, T), lrb1 = __shfl_sync(FULL, rb1, T);
            const unsigned long long ldst = __shfl_sync(FULL, dst, T);
            const int lmoff = __shfl_sync(FULL, moff, T);
            const int i = __shfl_sync(FULL, pos, T);
            if (e >= total) continue;
            const int la = (int)a0 + T;
            const unsigned long long s =
                (r < lc0) ? (unsigned long long)lrb0 + r : (unsigned long long)lrb1 + (r - lc0);
            const unsigned long long d = ldst + r;
            const unsigned meta = f.rec_meta[s];
            const int len = (int)(meta & 0xffu);
            const int cell = (int)f.cell_of[(meta >> 8) & 0x3fu];
            const unsigned *ids = f.rec_ids + s * (unsigned long long)md.gms;
            unsigned *row = f.chains + d * (unsigned long long)W;
            // the chain row (record_curvelet_chain, :269-276), the best cell's bounds and the length
            row[0] = (unsigned)(la - lmoff) + 1u;
            row[1] = (unsigned)(la - lmoff) + 1u;
            const double2 cs2 = f.cs2[i];
            const int seed = (int)ids[0];
            const CellAnchor ca = cell_anchor(md, f.B.th[i], cell);
            double k_min, k_max;
            exact_cell(md, f.B, cs2, i, seed, ca, k_min, k_max);
            double length = 0.0, px = f.B.x[i], py = f.B.y[i];
            for (int z = 1; z < len; ++z) {
                const int nn = (int)ids[z];
                row[z + 1] = (unsigned)(f.B.orig[nn] - lmoff) + 1u;
                const double qx = f.B.x[nn], qy = f.B.y[nn];
                length += sqrt(sq_dist(px, py, qx, qy));
                px = qx;
                py = qy;
                if (nn != seed) {
                    double m, Mx;
                    exact_cell(md, f.B, cs2, i, nn, ca, m, Mx);
                    k_min = (k_min < m) ? m : k_min;
                    k_max = (k_max > Mx) ? Mx : k_max;
                }
            }
            for (int z = len + 1; z < W; ++z) row[z] = 0u;
            // fill_curvelet_info (:221-255)
            const double ltheta = f.B.th[i];
            const int mini = cell / md.Q, minj = cell % md.Q;
            const double k = (k_max + k_min) / 2.0;
            const double dx = info_offset(md.sx, mini, md.P);
            const double dt = info_offset(md.st, minj, md.Q);
            const double theta = to_2pi(ltheta + dt);
            const double pt_x = f.B.x[i] - dx * sin(theta);
            const double pt_y = f.B.y[i] + dx * cos(theta);
            const double quality =
                (length > 0.0 && len > 0) ? 2.0 / (1.0 * md.nrad / length + 1.0 * length / (double)len) : 0.0;
            double *inf = f.info + d * 10ull;
            inf[0] = (meta >> 24) & 1u ? 1.0 : 0.0;
            inf[1] = k_max;
            inf[2] = k_min;
            inf[3] = ltheta;
            inf[4] = pt_x;
            inf[5] = pt_y;
            inf[6] = theta;
            inf[7] = k;
            inf[8] = length;
            inf[9] = quality;
        }
    }
}

constexpr int FINAL_WARPS = 8;
constexpr int FINAL_ANCHORS = 8;  // of a warp
template <int G>
__global__ void __launch_bounds__(FINAL_WARPS * 32, 3) k_finalize_small(const __grid_constant__ FinalArgs f) {
    constexpr int PER = 32 / G;  // curvelets per round
    __shared__ double s_info[FINAL_WARPS][PER * 10];
    __shared__ unsigned s_row[FINAL_WARPS][PER * (G + 1)];
    const Model &md = f.md;
    if (*f.err) return;
    const int N = f.dims ? f.dims->N : f.N;
    const int W = md.gms + 1;  // <= G + 1
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const int q = lane & (G - 1), own = lane / G;
    const int warp = (int)((blockIdx.x * (unsigned)blockDim.x + threadIdx.x) >> 5);
    const int warps = (int)((gridDim.x * (unsigned)blockDim.x) >> 5);
    for (long long a0 = (long long)warp * FINAL_ANCHORS; a0 < N; a0 += (long long)warps * FINAL_ANCHORS) {
        const int a = (int)a0 + lane;
        unsigned c0 = 0, cnt = 0, rb0 = 0, rb1 = 0;
        unsigned long long dst = 0;
        int moff = 0, pos = 0;
        if (lane < FINAL_ANCHORS && a < N) {
            c0 = f.run_cnt[2 * a];
            const unsigned c1 = f.run_cnt[2 * a + 1];
            dst = f.out_off[a];
            if (c0 + c1 > 0 && dst + c0 + c1 <= f.out_cap) {
                cnt = c0 + c1;
                rb0 = f.rec_base[2 * a];
                rb1 = f.rec_base[2 * a + 1];
                pos = f.pos_of[a];
                moff = f.map_off[f.B.map[pos]];
            }
        }
        unsigned incl = cnt;  // inclusive prefix of the tile's counts
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const unsigned o = __shfl_up_sync(FULL, incl, d);
            if (lane >= d) incl += o;
        }
        const unsigned total = __shfl_sync(FULL, incl, 31);
        // the tile's first row (of its first anchor with curvelets)
        const unsigned some = __ballot_sync(FULL, cnt > 0);
        const unsigned long long row0 = __shfl_sync(FULL, dst, some ? __ffs(some) - 1 : 0);
        for (unsigned e0 = 0; e0 < total; e0 += PER) {
            const unsigned e = min(e0 + (unsigned)own, total - 1u);
            int T = 0;  // the anchor of curvelet e: the first lane whose inclusive prefix exceeds e
#pragma unroll
            for (int step = 16; step >= 1; step >>= 1) {
                const unsigned v = __shfl_sync(FULL, incl, T + step - 1);
                if (v <= e) T += step;
            }
            const unsigned r = e - (__shfl_sync(FULL, incl, T) - __shfl_sync(FULL, cnt, T));
            const unsigned lc0 = __shfl_sync(FULL, c0, T);
            const unsigned lrb0 = __shfl_sync(FULL, rb0, T), lrb1 = __shfl_sync(FULL, rb1, T);
            const int lmoff = __shfl_sync(FULL, moff, T);
            const int i = __shfl_sync(FULL, pos, T);
            const int la = (int)a0 + T;
            const unsigned long long s =
                (r < lc0) ? (unsigned long long)lrb0 + r : (unsigned long long)lrb1 + (r - lc0);
            const unsigned meta = f.rec_meta[s];
            const int len = (int)(meta & 0xffu);
            const int cell = (int)f.cell_of[(meta >> 8) & 0x3fu];
            const unsigned *ids = f.rec_ids + s * (unsigned long long)md.gms;
            const int seed = (int)ids[0];
            // lane 0: the seed's bounds; lane z: the chain's z-th edge, its step's length and
            // (unless it is the seed) its bounds
            const int nn = q < len ? (int)ids[q] : seed;
            const double ax = f.B.x[i], ay = f.B.y[i];
            double m = 0.0, Mx = 0.0;
            const bool pair = q == 0 || (q < len && nn != seed);
            if (pair) exact_cell(md, f.B, f.cs2[i], i, nn, cell, m, Mx);
            const double qx = f.B.x[nn], qy = f.B.y[nn];
            double px = __shfl_up_sync(FULL, qx, 1, G), py = __shfl_up_sync(FULL, qy, 1, G);
            if (q == 1) {  // the first step is from the anchor
                px = ax;
                py = ay;
            }
            const double step_len = sqrt(sq_dist(px, py, qx, qy));
            // in the chain's order: the bounds, and the length
            double k_min = m, k_max = Mx, length = 0.0;
            const unsigned pairs = __ballot_sync(FULL, pair);
#pragma unroll
            for (int z = 1; z < G; ++z) {
                const double zm = __shfl_sync(FULL, m, z, G), zM = __shfl_sync(FULL, Mx, z, G);
                const double zl = __shfl_sync(FULL, step_len, z, G);
                if (pairs >> (own * G + z) & 1u) {
                    k_min = (k_min < zm) ? zm : k_min;
                    k_max = (k_max > zM) ? zM : k_max;
                }
                if (z < len) length += zl;
            }
            // the chain row (record_curvelet_chain, :269-276)
            unsigned *row = s_row[wib] + own * W;
            if (q == 0) row[0] = (unsigned)(la - lmoff) + 1u;
            if (q + 1 < W) row[q + 1] = q == 0 ? (unsigned)(la - lmoff) + 1u : q < len ? (unsigned)(f.B.orig[nn] - lmoff) + 1u : 0u;
            if (q == 0) {
                // fill_curvelet_info (:221-255)
                const double ltheta = f.B.th[i];
                const int mini = cell / md.Q, minj = cell % md.Q;
                const double k = (k_max + k_min) / 2.0;
                const double dx = info_offset(md.sx, mini, md.P);
                const double dt = info_offset(md.st, minj, md.Q);
                const double theta = to_2pi(ltheta + dt);
                double *inf = s_info[wib] + own * 10;
                inf[0] = (meta >> 24) & 1u ? 1.0 : 0.0;
                inf[1] = k_max;
                inf[2] = k_min;
                inf[3] = ltheta;
                inf[4] = ax - dx * sin(theta);
                inf[5] = ay + dx * cos(theta);
                inf[6] = theta;
                inf[7] = k;
                inf[8] = length;
                inf[9] = (length > 0.0 && len > 0) ? 2.0 / (1.0 * md.nrad / length + 1.0 * length / (double)len) : 0.0;
            }
            __syncwarp();
            const int now = (int)min((unsigned)PER, total - e0);
            for (int k = lane; k < now * 10; k += 32) f.info[(row0 + e0) * 10ull + k] = s_info[wib][k];
            for (int k = lane; k < now * W; k += 32) f.chains[(row0 + e0) * (unsigned long long)W + k] = s_row[wib][k];
            __syncwarp();
        }
    }
}

}  // namespace cvl
