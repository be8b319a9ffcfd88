// The energy terms past contact, volume and surface, shared by the tiled
// sweep (sweep.cu) and the direct sweep (direct.cu): length and nematic
// alignment from the exact moment sums, chemotaxis, motility, drift, the
// connectivity veto, and the moment sums' own commits.
#pragma once

#include <cstdint>

#include "device.cuh"
#include "engine.h"
#include "neighbours.cuh"

namespace glz {

// A pass's view of the moment sums: its snapshot (base + prev) and where its
// changes go, and which buffer holds each species' field.
struct TermView {
    const long long *base, *prev;
    unsigned long long *cur;
    unsigned field_cur;
    const float *logs;  // 0, then motility_log of 1 .. kLogs - 1, in shared memory; or null
};

__device__ __forceinline__ const float *field_of(const SweepLaunch &a, unsigned field_cur, int s) {
    return a.field_buf + ((size_t)2 * s + ((field_cur >> s) & 1u)) * (size_t)a.g.sites;
}

// The wrapped coordinates one step either side of a site.
struct Around {
    int xm, xp, ym, yp, zm, zp;
};

template <int DIM>
__device__ __forceinline__ Around around(const Geometry &g, int x, int y, int z) {
    Around r;
    r.xm = x == 0 ? g.w - 1 : x - 1;
    r.xp = x == g.w - 1 ? 0 : x + 1;
    r.ym = y == 0 ? g.h - 1 : y - 1;
    r.yp = y == g.h - 1 ? 0 : y + 1;
    r.zm = DIM == 3 ? (z == 0 ? g.d - 1 : z - 1) : 0;
    r.zp = DIM == 3 ? (z == g.d - 1 ? 0 : z + 1) : 0;
    return r;
}

// The site index of neighbour k of a neighbourhood fixed at compile time.
template <int DIM, int NOFF>
__device__ __forceinline__ uint32_t neighbour_site(const Geometry &g, const Around &r, int x, int y, int z, int k) {
    const int dx = neighbour_offset<DIM, NOFF>(k, 0), dy = neighbour_offset<DIM, NOFF>(k, 1),
              dz = neighbour_offset<DIM, NOFF>(k, 2);
    const int nx = dx < 0 ? r.xm : (dx > 0 ? r.xp : x), ny = dy < 0 ? r.ym : (dy > 0 ? r.yp : y),
              nz = dz < 0 ? r.zm : (dz > 0 ? r.zp : z);
    return (uint32_t)((nz * g.h + ny) * g.w + nx);
}

// The dominant eigenvalue of a symmetric 3x3 by twenty rounds of power
// iteration and a Rayleigh quotient, as the serial engine takes it
// (moments.rs:165-186).
__device__ __noinline__ inline double power_lambda(const double c[3][3]) {
    double v0 = 1.0, v1 = 0.7, v2 = 0.3;
    for (int round = 0; round < 20; ++round) {
        double w0 = c[0][0] * v0 + c[0][1] * v1 + c[0][2] * v2;
        double w1 = c[1][0] * v0 + c[1][1] * v1 + c[1][2] * v2;
        double w2 = c[2][0] * v0 + c[2][1] * v1 + c[2][2] * v2;
        double norm = sqrt(w0 * w0 + w1 * w1 + w2 * w2);
        if (norm < 1e-15) return 0.0;
        v0 = w0 / norm;
        v1 = w1 / norm;
        v2 = w2 / norm;
    }
    double w0 = c[0][0] * v0 + c[0][1] * v1 + c[0][2] * v2;
    double w1 = c[1][0] * v0 + c[1][1] * v1 + c[1][2] * v2;
    double w2 = c[2][0] * v0 + c[2][1] * v1 + c[2][2] * v2;
    double lambda = v0 * w0 + v1 * w1 + v2 * w2;
    return lambda > 0.0 ? lambda : 0.0;
}

// a / n correctly rounded for an integer-valued a below 2^53 and a count n
// with y = 1 / n correctly rounded: q = a y is within two units of the last
// place, one residual step makes it faithful, and the next returns the
// correctly rounded quotient (P. Markstein, "Computation of elementary
// functions on the IBM RISC System/6000 processor", IBM J. Res. Dev. 34(1),
// 1990: with y the rounded reciprocal and q faithful, fma(fma(-n, q, a), y,
// q) rounds as a / n does). The bits are those of a division, so the host
// replay may divide; a cell's five or nine means share one reciprocal and
// carry no branch, so they overlap.
__host__ __device__ __forceinline__ double mean_of(double a, double n, double y) {
    double q = a * y;
    q = fma(fma(-n, q, a), y, q);
    return fma(fma(-n, q, a), y, q);
}

// 4 sqrt(lambda_max) of a cell's covariance from its n sites and exact sums
// (moments.rs:150-155); a plane takes the 2x2 closed form.
template <int DIM>
__device__ __forceinline__ double axis_length(long long n, const long long *m) {
    const double dn = (double)n, y = __drcp_rn(dn);
    double lambda;
    if (DIM == 2) {
        const double mx = mean_of((double)m[0], dn, y), my = mean_of((double)m[1], dn, y);
        const double cxx = mean_of((double)m[2], dn, y) - mx * mx;
        const double cyy = mean_of((double)m[3], dn, y) - my * my;
        const double cxy = mean_of((double)m[4], dn, y) - mx * my;
        const double half = 0.5 * (cxx + cyy), diff = 0.5 * (cxx - cyy);
        lambda = half + sqrt(diff * diff + cxy * cxy);
        lambda = lambda > 0.0 ? lambda : 0.0;
    } else {
        const double mx = mean_of((double)m[0], dn, y), my = mean_of((double)m[1], dn, y),
                     mz = mean_of((double)m[2], dn, y);
        double c[3][3];
        c[0][0] = mean_of((double)m[3], dn, y) - mx * mx;
        c[1][1] = mean_of((double)m[4], dn, y) - my * my;
        c[2][2] = mean_of((double)m[5], dn, y) - mz * mz;
        c[0][1] = c[1][0] = mean_of((double)m[6], dn, y) - mx * my;
        c[0][2] = c[2][0] = mean_of((double)m[7], dn, y) - mx * mz;
        c[1][2] = c[2][1] = mean_of((double)m[8], dn, y) - my * mz;
        lambda = power_lambda(c);
    }
    const double length = 4.0 * sqrt(lambda);
    return n < 2 ? 0.0 : length;
}

template <int DIM>
__device__ __forceinline__ void site_terms(int ux, int uy, int uz, long long *t) {
    if (DIM == 2) {
        t[0] = ux; t[1] = uy; t[2] = (long long)ux * ux; t[3] = (long long)uy * uy; t[4] = (long long)ux * uy;
    } else {
        t[0] = ux; t[1] = uy; t[2] = uz;
        t[3] = (long long)ux * ux; t[4] = (long long)uy * uy; t[5] = (long long)uz * uz;
        t[6] = (long long)ux * uy; t[7] = (long long)ux * uz; t[8] = (long long)uy * uz;
    }
}

// The connectivity veto's full Moore ring (connectivity.rs:23-29).
template <int DIM>
constexpr int kRing = DIM == 2 ? 8 : 26;

// Where neighbour k sits in a 3 x 3 (x 3) cube of bits about the target.
template <int DIM, int NOFF>
__host__ __device__ constexpr int cube_bit(int k) {
    return (neighbour_offset<DIM, NOFF>(k, 0) + 1) + 3 * (neighbour_offset<DIM, NOFF>(k, 1) + 1) +
           (DIM == 3 ? 9 * (neighbour_offset<DIM, NOFF>(k, 2) + 1) : 0);
}

// lib.rs:371-389: whether the ring positions in `present` (bits of the cube)
// are one piece, two positions joined when no coordinate differs by more than
// one. Such steps are a box dilation of the cube's bits, one axis at a time,
// so a round of the flood fill is a dozen bit operations whatever the number
// of positions reached.
template <int DIM>
__host__ __device__ __forceinline__ bool one_piece(uint32_t present) {
    constexpr uint32_t col0 = DIM == 3 ? 0x1249249u : 0x49u;  // bits with dx = -1
    constexpr uint32_t col2 = col0 << 2;
    constexpr uint32_t row0 = DIM == 3 ? 0x1c0e07u : 0x7u;  // bits with dy = -1
    constexpr uint32_t row2 = row0 << 6;
    if ((present & (present - 1u)) == 0u) return true;
    uint32_t reached = present & (~present + 1u);
    for (int round = 0; round < 26; ++round) {
        uint32_t grown = reached | ((reached & ~col2) << 1) | ((reached & ~col0) >> 1);
        grown |= ((grown & ~row2) << 3) | ((grown & ~row0) >> 3);
        if (DIM == 3) grown |= (grown << 9) | (grown >> 9);
        grown &= present;
        if (grown == reached) break;
        reached = grown;
    }
    return reached == present;
}

// The moment-sum terms of the target site in a cell's own frame.
__device__ __forceinline__ int4 anchor_of(const SweepLaunch &a, uint32_t label) {
    return *reinterpret_cast<const int4 *>(&a.anchor[(size_t)label * 4]);
}

template <int DIM>
__device__ __forceinline__ void terms_of(const SweepLaunch &a, const int4 &an, int x, int y, int z, long long *t) {
    site_terms<DIM>(fold_int(x - an.x, a.g.w), fold_int(y - an.y, a.g.h), fold_int(z - an.z, a.g.d), t);
}

// A cell's moment words (and its nematic sums) in the pass snapshot.
template <int DIM>
__device__ __forceinline__ void moments_of(const SweepLaunch &a, const TermView &v, uint32_t label, bool nematic,
                                           long long *m) {
    constexpr int NM = DIM == 2 ? 5 : 9;
    const size_t at = (size_t)label * a.g.nm;
#pragma unroll
    for (int k = 0; k < NM; ++k) m[k] = v.base[at + k] + v.prev[at + k];
    m[NM] = m[NM + 1] = 0;
    if (nematic) {
        m[NM] = v.base[at + NM] + v.prev[at + NM];
        m[NM + 1] = v.base[at + NM + 1] + v.prev[at + NM + 1];
    }
}

// Change in a cell's length energy (cpu.rs:291-305) when the site with sum
// terms `terms` leaves (sign -1) or joins (+1) it, from its moment words m.
template <int DIM>
__device__ __forceinline__ double length_delta(const TypeTables &T, int type, long long n, const long long *m,
                                               const long long *terms, int sign) {
    constexpr int NM = DIM == 2 ? 5 : 9;
    long long after[NM];
#pragma unroll
    for (int k = 0; k < NM; ++k) after[k] = m[k] + sign * terms[k];
    const double tl = T.target_length[type];
    const double before = axis_length<DIM>(n, m) - tl;
    const double now = axis_length<DIM>(n + sign, after) - tl;
    return T.lambda_length[type] * (now * now - before * before);
}

// Change in a cell's nematic energy (cpu.rs:315-332, lib.rs:603-637) when the
// site with sum terms `terms` (its moment terms, then its field components in
// fixed point) leaves (sign -1) or joins (+1) it: -lambda (f' . a' - f . a),
// f the cell's field sum and a its anisotropy, from its moment words m.
template <int DIM>
__device__ __forceinline__ double nematic_delta(const TypeTables &T, int type, long long n, const long long *m,
                                                const long long *terms, int sign) {
    constexpr int NM = DIM == 2 ? 5 : 9;
    long long after[NM + 2];
#pragma unroll
    for (int k = 0; k < NM + 2; ++k) after[k] = m[k] + sign * terms[k];
    double a0, a1, b0, b1;
    anisotropy<DIM>(n, m, a0, a1);
    anisotropy<DIM>(n + sign, after, b0, b1);
    const double scale = 1.0 / 4294967296.0;
    const double before = (double)m[NM] * scale * a0 + (double)m[NM + 1] * scale * a1;
    const double now = (double)after[NM] * scale * b0 + (double)after[NM + 1] * scale * b1;
    return -T.lambda_nematic[type] * (now - before);
}

// The offsets of a neighbourhood along an axis, one more than each in two
// bits, neighbour k's at bit 2 k.
template <int DIM, int NOFF>
__host__ __device__ constexpr uint64_t packed_offsets(int axis) {
    uint64_t bits = 0;
    for (int k = 0; k < NOFF; ++k) bits |= (uint64_t)(neighbour_offset<DIM, NOFF>(k, axis) + 1) << (2 * k);
    return bits;
}

// The offset of neighbour `pick`: a shift of a constant an axis (the
// 26-neighbourhood has a closed form), not a chain of selects or a table.
template <int DIM, int NOFF>
__device__ __forceinline__ void pick_offset(int pick, int &dx, int &dy, int &dz) {
    if constexpr (DIM == 3 && NOFF == 26) {
        dx = neighbour_offset<3, 26>(pick, 0);
        dy = neighbour_offset<3, 26>(pick, 1);
        dz = neighbour_offset<3, 26>(pick, 2);
    } else {
        constexpr uint64_t X = packed_offsets<DIM, NOFF>(0), Y = packed_offsets<DIM, NOFF>(1),
                           Z = packed_offsets<DIM, NOFF>(2);
        if constexpr (2 * NOFF <= 32) {
            dx = (int)((uint32_t)X >> (2 * pick) & 3u) - 1;
            dy = (int)((uint32_t)Y >> (2 * pick) & 3u) - 1;
            dz = DIM == 3 ? (int)((uint32_t)Z >> (2 * pick) & 3u) - 1 : 0;
        } else {
            dx = (int)(X >> (2 * pick) & 3u) - 1;
            dy = (int)(Y >> (2 * pick) & 3u) - 1;
            dz = (int)(Z >> (2 * pick) & 3u) - 1;
        }
    }
}

// Logs of the whole activities an Act memory runs through (it starts at its
// maximum and runs down by one a step): motility_log's own values, taken once
// a block, so a neighbour's log is a table read; the entry of 0 is zero, what
// a neighbour that does not count adds.
constexpr int kLogs = 256;

__device__ __forceinline__ int whole_activity(float v) {
    const int k = (int)v;
    return k < kLogs && (float)k == v ? k : -1;
}

// The geometric mean of the activity over the sites of `label` around `site`
// (x, y, z), the site itself included; zero as soon as one of them has none
// left (lib.rs:391-424, motility.rs:58-79). Labels and activity are the
// pass's starting values: a pass with motility defers its writes.
template <int DIM, int NOFF>
__device__ __noinline__ float activity_mean(const SweepLaunch &a, uint32_t site, int x, int y, int z, uint32_t label) {
    const float here = a.activity[site];
    if (!(here > 0.0f)) return 0.0f;
    const Around r = around<DIM>(a.g, x, y, z);
    float log_sum = motility_log(here), count = 1.0f;
    for (int k = 0; k < NOFF; ++k) {
        const uint32_t n = neighbour_site<DIM, NOFF>(a.g, r, x, y, z, k);
        if (n == site || a.labels[n] != label) continue;
        const float v = a.activity[n];
        if (!(v > 0.0f)) return 0.0f;
        log_sum = __fadd_rn(log_sum, motility_log(v));
        count = __fadd_rn(count, 1.0f);
    }
    return metropolis_exp(__fdiv_rn(log_sum, count));
}

// The same mean from values already read: `here` the site's activity, v its
// neighbours', bit k of `like` whether neighbour k carries the label. `known`
// is false when an activity that counts is not whole (the mean is then not
// taken here).
template <int NOFF>
__device__ __forceinline__ float table_mean(const float *logs, float here, const float *v, uint32_t like, bool &known) {
    known = true;
    if (!(here > 0.0f)) return 0.0f;
    int at[NOFF], least = whole_activity(here);
    bool spent = false;
    const int own = least;
#pragma unroll
    for (int k = 0; k < NOFF; ++k) {
        const bool counts = like >> k & 1u;
        at[k] = counts ? whole_activity(v[k]) : 0;
        least = min(least, at[k]);
        spent |= counts && !(v[k] > 0.0f);
    }
    if (spent) return 0.0f;
    known = least >= 0;
    if (!known) return 0.0f;
    float log_sum = logs[own];
#pragma unroll
    for (int k = 0; k < NOFF; ++k) log_sum = __fadd_rn(log_sum, logs[at[k]]);
    return metropolis_exp(__fdiv_rn(log_sum, (float)(1 + __popc(like))));
}

// The length, nematic, chemotaxis, motility and drift terms of a copy
// (cpu.rs:291-332, 341-395); the motility term with MOTILE.
template <int DIM, int NOFF, bool MOTILE>
__device__ __forceinline__ float extra_terms(const SweepLaunch &a, const TypeTables &T, const TermView &v, uint32_t old, uint32_t nw,
                                             int t_old, int t_new, int vol_old, int vol_new, int x, int y, int z,
                                             int pick, uint32_t target, float delta) {
    constexpr int NM = DIM == 2 ? 5 : 9;
    const int W = a.g.w, H = a.g.h, D = a.g.d;
    // The length and nematic terms, leaving cell first (lib.rs:578-639). A
    // lane takes the side of the copy that states a term, and a second turn
    // only when both do, so a warp whose lanes differ in the side runs the
    // f64 chain once, not once a side.
    if (a.has_length || a.has_nematic) {
        const auto states = [&](uint32_t l, int type) {
            return l != 0 && ((a.has_length && T.lambda_length[type] != 0.0) ||
                              (a.has_nematic && T.lambda_nematic[type] != 0.0));
        };
        int turns = (states(old, t_old) ? 1 : 0) | (states(nw, t_new) ? 2 : 0);
        long long q[2] = {0, 0};
        if (turns && a.has_nematic) {
            q[0] = nematic_fixed(a.nematic[2 * (size_t)target]);
            q[1] = nematic_fixed(a.nematic[2 * (size_t)target + 1]);
        }
        while (turns) {
            const bool leaving = turns & 1;
            turns = leaving ? turns & 2 : 0;
            const uint32_t l = leaving ? old : nw;
            const int type = leaving ? t_old : t_new, n = leaving ? vol_old : vol_new, sign = leaving ? -1 : 1;
            const bool len = a.has_length && T.lambda_length[type] != 0.0;
            const bool nem = a.has_nematic && T.lambda_nematic[type] != 0.0;
            long long m[NM + 2], t[NM + 2];
            moments_of<DIM>(a, v, l, nem, m);
            terms_of<DIM>(a, anchor_of(a, l), x, y, z, t);
            t[NM] = q[0];
            t[NM + 1] = q[1];
            if (len) delta = __fadd_rn(delta, (float)length_delta<DIM>(T, type, n, m, t, sign));
            if (nem) delta = __fadd_rn(delta, (float)nematic_delta<DIM>(T, type, n, m, t, sign));
        }
    }
    int ox, oy, oz;
    pick_offset<DIM, NOFF>(pick, ox, oy, oz);
    const Around r = around<DIM>(a.g, x, y, z);
    const int sx = ox < 0 ? r.xm : (ox > 0 ? r.xp : x), sy = oy < 0 ? r.ym : (oy > 0 ? r.yp : y),
              sz = oz < 0 ? r.zm : (oz > 0 ? r.zp : z);
    const uint32_t source = (uint32_t)((sz * H + sy) * W + sx);
    if (a.has_chemotaxis && nw != 0) {
        for (int s = 0; s < a.n_species; ++s) {
            const float lam = T.chemotaxis[t_new * a.n_species + s];
            if (lam == 0.0f) continue;
            const float *f = field_of(a, v.field_cur, s);
            delta = __fsub_rn(delta, __fmul_rn(lam, __fsub_rn(f[target], f[source])));
        }
    }
    // Motility (cpu.rs:346-352, lib.rs:656-663): the cell's memory pulls it
    // where it has been.
    if (MOTILE && nw != 0) {
        const float lam = T.lambda_activity[t_new], top = T.max_activity[t_new];
        if (lam != 0.0f && top > 0.0f) {
            float into = 0.0f, out_of = 0.0f;
            bool known_into = false, known_out = false;
            if (v.logs) {
                // every value of both means is requested before any is used,
                // a label on the site itself included (a test that reads it
                // only past the site's own holds up the rest: 5.88 and 5.73 ms
                // for 60 MCS of the 64 x 64 x 32 slab)
                const Around rs = around<DIM>(a.g, sx, sy, sz);
                float at_source[NOFF], at_target[NOFF];
                uint32_t like_new = 0, like_old = 0;
#pragma unroll
                for (int k = 0; k < NOFF; ++k) {
                    const uint32_t n = neighbour_site<DIM, NOFF>(a.g, rs, sx, sy, sz, k);
                    const uint32_t m = neighbour_site<DIM, NOFF>(a.g, r, x, y, z, k);
                    at_source[k] = a.activity[n];
                    at_target[k] = a.activity[m];
                    const uint32_t ln = a.labels[n], lm = a.labels[m];
                    like_new |= (uint32_t)((n != source) & (ln == nw)) << k;
                    like_old |= (uint32_t)((m != target) & (lm == old)) << k;
                }
                into = table_mean<NOFF>(v.logs, a.activity[source], at_source, like_new, known_into);
                out_of = table_mean<NOFF>(v.logs, a.activity[target], at_target, like_old, known_out);
            }
            if (!known_into) into = activity_mean<DIM, NOFF>(a, source, sx, sy, sz, nw);
            if (!known_out) out_of = activity_mean<DIM, NOFF>(a, target, x, y, z, old);
            delta = __fsub_rn(delta, __fmul_rn(__fdiv_rn(lam, top), __fsub_rn(into, out_of)));
        }
    }
    // The drift (cpu.rs:360-369, lib.rs:664-673): work e . (target - source),
    // the step folded onto the lattice.
    if (a.has_external && nw != 0) {
        const float ex = T.external[3 * t_new], ey = T.external[3 * t_new + 1], ez = T.external[3 * t_new + 2];
        if (ex != 0.0f || ey != 0.0f || ez != 0.0f) {
            const float fx = (float)fold_int(x - sx, W), fy = (float)fold_int(y - sy, H), fz = (float)fold_int(z - sz, D);
            delta = __fsub_rn(delta, __fadd_rn(__fadd_rn(__fmul_rn(ex, fx), __fmul_rn(ey, fy)), __fmul_rn(ez, fz)));
        }
    }
    return delta;
}

// The moment sums follow an accepted copy: the site leaves `old` and joins
// `nw`, whose anchors the caller has read.
template <int DIM>
__device__ __forceinline__ void commit_moments(const SweepLaunch &a, unsigned long long *cur, uint32_t old,
                                               uint32_t nw, const int4 &an_old, const int4 &an_new, int x, int y,
                                               int z) {
    constexpr int NM = DIM == 2 ? 5 : 9;
    const int nm = a.g.nm;
    long long terms[NM], q[2] = {0, 0};
    if (a.has_nematic) {
        const size_t site = ((size_t)z * a.g.h + y) * a.g.w + x;
        q[0] = nematic_fixed(a.nematic[2 * site]);
        q[1] = nematic_fixed(a.nematic[2 * site + 1]);
    }
    if (old != 0) {
        terms_of<DIM>(a, an_old, x, y, z, terms);
#pragma unroll
        for (int k = 0; k < NM; ++k) atomicAdd(&cur[(size_t)old * nm + k], (unsigned long long)(-terms[k]));
        if (a.has_nematic)
            for (int k = 0; k < 2; ++k) atomicAdd(&cur[(size_t)old * nm + NM + k], (unsigned long long)(-q[k]));
    }
    if (nw != 0) {
        terms_of<DIM>(a, an_new, x, y, z, terms);
#pragma unroll
        for (int k = 0; k < NM; ++k) atomicAdd(&cur[(size_t)nw * nm + k], (unsigned long long)terms[k]);
        if (a.has_nematic)
            for (int k = 0; k < 2; ++k) atomicAdd(&cur[(size_t)nw * nm + NM + k], (unsigned long long)q[k]);
    }
}

}  // namespace glz
