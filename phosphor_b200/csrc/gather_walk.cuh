// gather_walk.cuh — a pixel's walk over the photons inside its radius, for the gather and its adjoint.
#pragma once

#include "kernels.hpp"

namespace phx {

// x / y from r = 1 / y, for the many x of one y.  Markstein's theorem ("Computation of elementary functions on
// the IBM RISC System/6000 processor", IBM J. Res. Dev. 34, 1990): if r is 1/y rounded to nearest and q
// within one ulp of x/y, then q + (x - q y) r, each step one fused multiply-add, is x/y rounded to
// nearest.  x r alone is within 1.5 ulp, so a first step brings it within one and the second is exact.
// Needs x/y, x and x 2^-24 in the normal range.
PHX_DI float div_known(float x, float y, float r) {
    float q = x * r;
    q = __fmaf_rn(__fmaf_rn(-q, y, x), r, q);
    return __fmaf_rn(__fmaf_rn(-q, y, x), r, q);
}
// x / GAUSS_DENOM for x = 0 or in [2^-30, 1.5]: one step is enough (tests/test_short_forms.py
// tries every such x).
PHX_DI float div_gauss(float x) {
    constexpr float r = 1.0f / GAUSS_DENOM;
    const float q = x * r;
    return __fmaf_rn(__fmaf_rn(-q, GAUSS_DENOM, x), r, q);
}

// pm_expf for t in [-1, 0]: its operations without its range checks.
PHX_DI float exp_unit(float t) {
    float kf; // 0 or -1
    const float p = pm_exp_frac(t, &kf);
    return kf < 0.0f ? p * 0.5f : p;
}

// The Gaussian weight of a photon at squared distance dsq < r_sq (photon_hash.h:88-95): the reference's
// expression, its quotients formed from reciprocals prepared once a pixel.
struct KernelWeight {
    float denom, rdenom, dsq_min;
    PHX_DI explicit KernelWeight(float r_sq) {
        denom = 2.0f * r_sq;
        rdenom = 1.0f / denom;
        dsq_min = denom > 1e-18f && denom < 1e18f ? 1e-30f : __int_as_float(0x7f800000);
    }
    PHX_DI float operator()(float dsq) const {
        const float x = (-GAUSS_BETA) * dsq;
        const float t = dsq >= dsq_min ? div_known(x, denom, rdenom) : x / denom;
        return GAUSS_ALPHA * (1.0f - div_gauss(1.0f - exp_unit(t)));
    }
};

// The 27 cells around a hit point: an axis's three cell coordinates, a byte each, and the cells within the
// radius (none for a pixel that gathers nothing).
struct NearCells {
    u32 wx = 0, wy = 0, wz = 0, near = 0;
};

PHX_DI NearCells near_cells(const float4 pos, float r_sq, const GridDev &grid) {
    NearCells n;
    float d2[3][3];
    // The 27 cells in the reference's order (photon_hash.h:65-82), each in sorted (canonical)
    // photon order.  A cell whose box lies farther than the search radius from the hit point holds
    // no photon with dsq < r_sq, so it adds nothing and is skipped; the box is widened by 1/1024
    // of a cell on every side so that rounding in get_hash (which decides a photon's cell) and in
    // this test can never skip a photon that would count.
    // get_hash of a neighbour position works axis by axis, and an axis's coordinate only takes the
    // three values pos + {-1, 0, 1} * cell: each axis's three cell coordinates are computed once,
    // with the same operations get_hash applies, and packed one byte per offset; an axis's three
    // squared distances decide the cells together (infinite outside the grid, which has at most 255
    // cells per axis).
    constexpr float M = 1.0f / 1024.0f;
    const float gf = (float)grid.g;
    auto axis_cells = [&](float p, float o, float c, float (&d)[3]) -> u32 {
        const float q0 = (p - o) / c; // the hit point in cell units
        u32 w = 0;
#pragma unroll
        for (int k = 0; k < 3; k++) {
            float q = p;
            q += (float)(k - 1) * c;
            const float f = (q - o) / c;
            const bool in = !(f < 0.0f || f >= gf);
            const u32 ci = in ? (u32)f : 0u;
            const float gap = fmaxf(fmaxf(((float)ci - M) - q0, q0 - ((float)ci + (1.0f + M))), 0.0f) * c;
            d[k] = in ? gap * gap : __int_as_float(0x7f800000);
            w |= ci << (8 * k);
        }
        return w;
    };
    n.wx = axis_cells(pos.x, grid.ox, grid.cx, d2[0]);
    n.wy = axis_cells(pos.y, grid.oy, grid.cy, d2[1]);
    n.wz = axis_cells(pos.z, grid.oz, grid.cz, d2[2]);
#pragma unroll
    for (u32 c = 0; c < 27; c++) {
        const float dx = d2[0][c % 3], dy = d2[1][(c / 3) % 3], dz = d2[2][c / 9];
        if (!((dx + dy) + dz > r_sq) && dx + dy + dz < __int_as_float(0x7f800000))
            n.near |= 1u << c;
    }
    return n;
}

constexpr u32 GQ_CAP = 16, GQ_AHEAD = 4;

// Every lane of the warp walks its cells' photons, GQ_AHEAD at a time, and queues those inside its radius
// ({index, squared distance} in its column of q_k, q_d); flush(n) works the lanes' n queued photons off, all
// lanes together, whenever some lane could not take GQ_AHEAD more and at the end.  All 32 lanes take part.
template <class F>
PHX_DI void walk_photons(const GatherBufs &g, const u32 *cs, u32 G, NearCells nc, const float4 pos, float r_sq,
                         u32 (*q_k)[128], float (*q_d)[128], u32 tid, F &&flush) {
    constexpr u32 FULL = 0xffffffffu;
    const float dw = pos.w - 0.0f;
    // the photon range of the next cell of `near`
    auto next_cell = [&](u32 *lo, u32 *hi) {
        const u32 c = (u32)__ffs(nc.near) - 1u, c3 = c / 3u;
        nc.near &= nc.near - 1u;
        const u32 hx = (nc.wx >> (8u * (c - 3u * c3))) & 0xffu, hy = (nc.wy >> (8u * (c3 % 3u))) & 0xffu,
                  hz = (nc.wz >> (8u * (c / 9u))) & 0xffu;
        const u32 h = G * G * hx + G * hy + hz + 1; // get_hash's cell index
        *lo = min(__ldg(&cs[h]), g.n_cap);
        *hi = min(__ldg(&cs[h + 1]), g.n_cap);
    };
    u32 cnt = 0;
    u32 k = 0, end = 0, n0 = 0, n1 = 0;
    bool ahead = nc.near != 0; // n0, n1: the range of the cell after the current one, loaded ahead
    if (ahead)
        next_cell(&n0, &n1);
    for (;;) {
        while (k >= end && ahead) { // the next cell with photons
            k = n0;
            end = n1;
            ahead = nc.near != 0;
            if (ahead)
                next_cell(&n0, &n1);
        }
        __syncwarp();
        if (!__any_sync(FULL, k < end))
            break;
        if (k < end) {
            float4 p[GQ_AHEAD];
#pragma unroll
            for (u32 u = 0; u < GQ_AHEAD; u++)
                p[u] = __ldg(&g.s_posdir[min(k + u, end - 1u)]);
#pragma unroll
            for (u32 u = 0; u < GQ_AHEAD; u++) {
                const float dx = pos.x - p[u].x, dy = pos.y - p[u].y, dz = pos.z - p[u].z;
                const float dsq = ((dx * dx + dy * dy) + dz * dz) + dw * dw;
                if (dsq < r_sq && k + u < end) {
                    q_k[cnt][tid] = k + u;
                    q_d[cnt][tid] = dsq;
                    cnt++;
                }
            }
            k += GQ_AHEAD;
        }
        if (__any_sync(FULL, cnt > GQ_CAP - GQ_AHEAD)) {
            flush(cnt);
            cnt = 0;
        }
    }
    flush(cnt);
}

} // namespace phx
