// cvl_enclosures.h -- host side of the single-precision enclosures: the model that
// k_curvelets decides with, its thresholds made from a run's parameters (the error bounds
// are derived in cvl_curvelets.cuh), or ok = 0 where they do not cover them.
#pragma once

#include <algorithm>
#include <cmath>

namespace cvl {

constexpr int FAST_P = 9;        // grid offsets of the column code (the default grid)
constexpr int FAST_WIDE = 128;   // pairs of an anchor (max_candidates <= 128)
// Orientations the enclosures hold for (rad): the reference's rounding of its angles is 2^-31
// there, 0.2% and less of what single precision leaves of the quantities they enter.
constexpr double FAST_ANGLE = 0x1p20;
// e0 / max_k: larger leaves more comparisons undecided, smaller more columns to be made anew
// (2^-13 to 2^-15 measured alike)
constexpr double FAST_E0 = 0x1p-14;

struct FastModel {
    float d[FAST_P], d2[FAST_P], c2[FAST_P];  // each offset's d, d^2, 2d + 2dx
    float mk, h;               // max_k, 2.04 e0
    float dx2, dx_2, ndx_4;    // dx^2, 2 dx, -4 dx
    float e0, eR, eRR;         // Ethr = e0 + eR Rb + eRR Rb^2
    float d0, dR;              // Dthr = d0 + dR Rb
    float s0, sR;              // S1 = s0 + sR Rb
    float dtiny;
    float fe, fd, fa;          // fine_column's thresholds of e1 and D: fe, fd times |T2| + |T0| + fa
    int ok;                    // the model is within the enclosures' range
    unsigned char rank[64];    // best-cell rank of each cell (fill_curvelet_info, :202-219)
    unsigned char cell_of[64]; // and the cell of each rank
};

// The longest distance of a pair: the search's radius, or the corner of its pixel window (two
// positions whose rounded ones differ by w are less than w + 1 apart). It is not nrad: a staged
// call's neighbour lists have a radius and a window of their own.
template <class M>
double pair_radius(const M &md) {
    return std::min(std::sqrt((double)md.rad_sqr), std::sqrt(2.0) * (md.w + 1.0));
}

// The enclosures' constants, or ok = 0: outside them the two-kernel path runs (other
// grids, cells no curvelet may take, extreme parameters).
template <class M>
FastModel make_fast(const M &md) {
    FastModel f{};
    const double u = 0x1p-24, mk = md.max_k, dx = md.dx, up = 1.02;
    const double dm = md.sx * ((double)md.P - 1.0) / 2.0, R = pair_radius(md);
    bool ok = md.P == FAST_P && md.Q >= 3 && md.cells <= 64 && md.max_cand <= FAST_WIDE && mk >= 0x1p-10 &&
              mk <= 0x1p10 && R >= 0x1p-10 && R <= 128.0 && dx >= 0x1p-20 && dx <= 64.0 && dm <= 64.0 &&
              md.dt >= -64.0 && md.dt <= 64.0 && md.st * md.Q <= 128.0;
    for (int c = 0; c < md.cells && ok; ++c) {  // every cell may be the best one (:207-219)
        const double ddx = md.sx * ((double)(c / md.Q) - ((double)md.P - 1.0) / 2.0);
        const double ddt = md.st * ((double)(c % md.Q) - ((double)md.Q - 1.0) / 2.0);
        ok = ddx * ddx + ddt * ddt < 100.0;
    }
    if (!ok) return f;
    for (int i = 0; i < FAST_P; ++i) {
        const double d = md.sx * ((double)i - ((double)md.P - 1.0) / 2.0);
        f.d[i] = (float)d;
        f.d2[i] = (float)(d * d);
        f.c2[i] = (float)(2.0 * d + 2.0 * dx);
    }
    const double e0 = FAST_E0 * mk, den = e0 - 8.0 * u * mk;
    f.mk = (float)mk;
    f.h = (float)(2.04 * e0);
    f.dx2 = (float)md.dx2;
    f.dx_2 = (float)(2.0 * dx);
    f.ndx_4 = (float)(-4.0 * dx);
    f.e0 = (float)(up * u * (4.0 * dm + 16.0 * dx + mk * (3.0 * dm * dm + 6.0 * dx * dx)) / den);
    f.eR = (float)(up * u * (10.0 + mk * 12.0 * dm) / den);
    f.eRR = (float)(up * u * mk * 7.0 / den);
    f.d0 = (float)(up * u * (4.0 + mk * 6.0 * dm) / den);
    f.dR = (float)(up * u * mk * 5.0 / den);
    f.s0 = (float)(up * (2.0 * mk * f.d0 + 8.0 * u));
    f.sR = (float)(up * 2.0 * mk * f.dR);
    f.dtiny = (float)(2.0 * u * (5.0 * R + 6.0 * dm));
    // fine_column: eps = 2^-51 (|T2| + |T0| + fa), the FP64 quantities' errors in its terms
    const double fine = up * 0x1p-51 / (e0 - 12.0 * u * mk);
    f.fe = (float)(fine * (3.0 * R + dm + dx + mk * (R * R + 3.0 * dm * R + dm * dm + dx * dx)));
    f.fd = (float)(fine * (1.0 + mk * (R + dm)));
    f.fa = (float)(up * (4.0 + std::fabs((double)md.dt) + md.st * ((double)md.Q - 1.0) / 2.0));
    // the cells ordered by (d, row-major index), with the reference's arithmetic
    double dist[64];
    for (int c = 0; c < md.cells; ++c) {
        const double ddx = md.sx * ((double)(c / md.Q) - ((double)md.P - 1.0) / 2.0);
        const double ddt = md.st * ((double)(c % md.Q) - ((double)md.Q - 1.0) / 2.0);
        const double a = ddx * ddx, b = ddt * ddt;
        dist[c] = a + b;
    }
    for (int c = 0; c < md.cells; ++c) {
        int r = 0;
        for (int o = 0; o < md.cells; ++o) r += dist[o] < dist[c] || (dist[o] == dist[c] && o < c);
        f.rank[c] = (unsigned char)r;
        f.cell_of[r] = (unsigned char)c;
    }
    f.ok = 1;
    return f;
}

}  // namespace cvl
