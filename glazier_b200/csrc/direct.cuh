// One copy attempt priced where it lies, shared by the kernels that read the
// lattice in place: the direct sweep (direct.cu), and the cluster and
// direct ensemble sweeps (sweep.cu). A target's neighbours are other
// colours, which no copy in the pass changes, so the labels it reads are the
// pass's.
#pragma once

#include <cstdint>

#include "device.cuh"
#include "engine.h"
#include "neighbours.cuh"
#include "pdl.cuh"
#include "pricing.cuh"
#include "terms.cuh"

namespace glz {

// The per-pass view of the tallies and draws a direct pass reads.
struct PassView {
    int colour;
    uint64_t key_pick, key_accept;
    const int2 *vs_base;
    const long long *vs_prev;
    unsigned long long *vs_cur;
};

// The per-colour guard: whether cell `old` keeps a site of a colour other
// than the pass's own, which no copy in this pass can take.
__device__ __noinline__ inline bool direct_keeps_other_colour(const SweepLaunch &a, int colour, uint32_t old) {
    int other = 0;
    for (int c = 0; c < a.g.ncol; ++c)
        if (c != colour) other += a.vol_by_colour[(size_t)old * a.g.ncol + c];
    return other != 0;
}

// Where a direct pass finds and puts labels and tallies: global memory.
struct GlobalPass {
    const SweepLaunch &a;
    const PassView &v;
    __device__ __forceinline__ uint32_t label(int x, int y, int z) const {
        return a.labels[(z * a.g.h + y) * a.g.w + x];
    }
    __device__ __forceinline__ int type(uint32_t l) const { return a.cell_type[l]; }
    __device__ __forceinline__ int2 base(uint32_t l) const { return v.vs_base[l]; }
    __device__ __forceinline__ long long prev(uint32_t l) const { return v.vs_prev[l]; }
    __device__ __forceinline__ bool keeps_other_colour(uint32_t old) const {
        return direct_keeps_other_colour(a, v.colour, old);
    }
    __device__ __forceinline__ void put(uint32_t target, int, int, int, uint32_t nw) const { a.labels[target] = nw; }
    __device__ __forceinline__ void tally(uint32_t l, int dv, int ds) const {
        atomicAdd(&v.vs_cur[l], pack_delta(dv, ds));
        atomicAdd(&a.vol_by_colour[(size_t)l * a.g.ncol + v.colour], dv);
    }
};

// Site (x, y, z) of target j of colour `colour` in a direct pass.
template <int DIM>
__device__ __forceinline__ void direct_site(const SweepLaunch &a, int colour, int j, int &x, int &y, int &z) {
    const uint32_t row = udiv(a.g.div_hw, (uint32_t)j);
    x = 2 * (int)((uint32_t)j - row * (uint32_t)(a.g.w / 2)) + (colour & 1);
    if constexpr (DIM == 2) {
        y = 2 * (int)row + ((colour >> 1) & 1);
        z = 0;
    } else {
        const uint32_t plane = udiv(a.g.div_hh, row);
        y = 2 * (int)(row - plane * (uint32_t)(a.g.h / 2)) + ((colour >> 1) & 1);
        z = 2 * (int)plane + ((colour >> 2) & 1);
    }
}

// The label of the picked neighbour of (x, y, z).
template <int DIM, int NOFF, class Access>
__device__ __forceinline__ uint32_t picked_label(const SweepLaunch &a, const Access &acc, int x, int y, int z, int pick) {
    int dx, dy, dz;
    pick_offset<DIM, NOFF>(pick, dx, dy, dz);
    const int nx = x + dx < 0 ? a.g.w - 1 : (x + dx >= a.g.w ? 0 : x + dx);
    const int ny = y + dy < 0 ? a.g.h - 1 : (y + dy >= a.g.h ? 0 : y + dy);
    const int nz = DIM == 2 ? 0 : (z + dz < 0 ? a.g.d - 1 : (z + dz >= a.g.d ? 0 : z + dz));
    return acc.label(nx, ny, nz);
}

// The labels of a target's energy neighbours, read as they are asked for.
template <int DIM, int NOFF, class Access>
struct NeighbourReads {
    const Access &acc;
    int x, y, z;
    Around r;
    __device__ __forceinline__ NeighbourReads(const SweepLaunch &a, const Access &access, int px, int py, int pz)
        : acc(access), x(px), y(py), z(pz), r(around<DIM>(a.g, px, py, pz)) {}
    __device__ __forceinline__ uint32_t at(int dx, int dy, int dz) const {
        return acc.label(dx < 0 ? r.xm : (dx > 0 ? r.xp : x), dy < 0 ? r.ym : (dy > 0 ? r.yp : y),
                         dz < 0 ? r.zm : (dz > 0 ? r.zp : z));
    }
    __device__ __forceinline__ uint32_t operator()(int k) const {
        return at(neighbour_offset<DIM, NOFF>(k, 0), neighbour_offset<DIM, NOFF>(k, 1), neighbour_offset<DIM, NOFF>(k, 2));
    }
    // neighbour k of the connectivity veto's ring
    __device__ __forceinline__ uint32_t ring(int k) const {
        constexpr int N = kRing<DIM>;
        return at(neighbour_offset<DIM, N>(k, 0), neighbour_offset<DIM, N>(k, 1), neighbour_offset<DIM, N>(k, 2));
    }
};

// The same labels already in registers.
template <int DIM, int NOFF, class Access>
struct NeighbourLabels : NeighbourReads<DIM, NOFF, Access> {
    uint32_t label[NOFF];
    __device__ __forceinline__ NeighbourLabels(const SweepLaunch &a, const Access &access, int px, int py, int pz)
        : NeighbourReads<DIM, NOFF, Access>(a, access, px, py, pz) {}
    __device__ __forceinline__ void load() {
#pragma unroll
        for (int k = 0; k < NOFF; ++k) label[k] = NeighbourReads<DIM, NOFF, Access>::operator()(k);
    }
    __device__ __forceinline__ uint32_t operator()(int k) const { return label[k]; }
    __device__ __forceinline__ uint32_t picked(int pick) const {
        uint32_t l = label[0];
#pragma unroll
        for (int k = 1; k < NOFF; ++k) l = k == pick ? label[k] : l;
        return l;
    }
};

// The copy attempt at target (x, y, z) whose pick and two labels the caller
// has read earlier in the pass (the target's label changes only by its own
// commit and the neighbour is another colour, so they are still the pass's):
// priced with price_and_commit's arithmetic operation for operation. `terms`
// is used with TERMS only: 0 none past contact, volume and surface, 1 all but
// motility, 2 all.
template <int DIM, int NOFF, bool UNIFORM, class Access, class Labels, int TERMS = 0>
__device__ __forceinline__ void direct_copy(const SweepLaunch &a, const TypeTables &T, const Access &acc,
                                            const Labels &neighbour, uint64_t key_accept, int x, int y, int z, int pick,
                                            uint32_t old, uint32_t nw, const TermView *terms = nullptr) {
    const int W = a.g.w, H = a.g.h;
    const uint32_t target = (uint32_t)((z * H + y) * W + x);
    const int2 base_old = acc.base(old), base_new = acc.base(nw);
    const long long prev_old = acc.prev(old), prev_new = acc.prev(nw);
    const int t_old = UNIFORM ? a.uniform_type : acc.type(old);
    const int t_new = UNIFORM ? a.uniform_type : acc.type(nw);
    // the moment commit's anchors, read here so the commit does not wait
    int4 an_old = make_int4(0, 0, 0, 0), an_new = an_old;
    if (TERMS && a.tracks) {
        an_old = anchor_of(a, old);
        an_new = anchor_of(a, nw);
    }
    float delta = 0.0f;
    int like_old = 0, like_new = 0;
    uint32_t present = 0;  // TERMS: ring positions of `old` among the energy neighbours, as bits of the veto's cube
    if (UNIFORM) {
#pragma unroll
        for (int k = 0; k < NOFF; ++k) {
            const uint32_t ln = neighbour(k);
            like_old += ln == old;
            like_new += ln == nw;
            if (TERMS && ln == old) present |= 1u << cube_bit<DIM, NOFF>(k);
        }
        delta = __fmul_rn(a.uniform_contact, (float)(like_old - like_new));
    } else {
#pragma unroll
        for (int k = 0; k < NOFF; ++k) {
            // no branch: a bond that does not count adds a zero, which leaves
            // the sum's bits alone, and every neighbour's type is read, so
            // that the type and table reads overlap (per MCS, types read only
            // of labels that are neither cell's, and of all: two types 14.4
            // and 13.9 us at 512^2, 21.2 and 19.2 at 1024^2, 146.7 and 136.4
            // at 4096^2; 26 neighbours 47.0 and 35.1 at 64^3, 74.1 and 57.8
            // at 128^3)
            const uint32_t ln = neighbour(k);
            const bool is_old = ln == old, is_new = ln == nw;
            const int tn = acc.type(ln);
            const float j_old = T.contact[t_old * a.n_types + tn], j_new = T.contact[t_new * a.n_types + tn];
            delta = __fsub_rn(delta, is_old ? 0.0f : j_old);
            delta = __fadd_rn(delta, is_new ? 0.0f : j_new);
            like_old += is_old;
            like_new += is_new;
            if (TERMS && is_old) present |= 1u << cube_bit<DIM, NOFF>(k);
        }
    }
    if (old != 0 && like_old == 0 && !acc.keeps_other_colour(old)) return;
    if (TERMS && old != 0 && a.g.ring_n > 0 && T.connected[t_old]) {
        // the connectivity veto (lib.rs:511-521); the ring positions the
        // energy neighbourhood leaves out are read here
#pragma unroll
        for (int k = 0; k < kRing<DIM>; ++k) {
            const int dx = neighbour_offset<DIM, kRing<DIM>>(k, 0), dy = neighbour_offset<DIM, kRing<DIM>>(k, 1),
                      dz = neighbour_offset<DIM, kRing<DIM>>(k, 2);
            const int steps = (dx != 0) + (dy != 0) + (dz != 0);  // axes it differs on: 1 a face, 2 an edge, 3 a corner
            const bool seen = steps <= (NOFF == 4 || NOFF == 6 ? 1 : (NOFF == 8 || NOFF == 18 ? 2 : 3));
            if (!seen && neighbour.ring(k) == old) present |= 1u << cube_bit<DIM, kRing<DIM>>(k);
        }
        if (!one_piece<DIM>(present)) return;
    }
    const int ds_old = 2 * like_old - NOFF;
    const int ds_new = NOFF - 2 * like_new;
    int dv, ds;
    unpack_delta(prev_old, dv, ds);
    const int vol_old = base_old.x + dv, surf_old = base_old.y + ds;
    unpack_delta(prev_new, dv, ds);
    const int vol_new = base_new.x + dv, surf_new = base_new.y + ds;
    delta = size_terms<UNIFORM>(a, T, old, nw, t_old, t_new, vol_old, vol_new, surf_old, surf_new, ds_old, ds_new, delta);
    if (TERMS && (a.has_length || a.has_chemotaxis || a.has_external || TERMS == 2 || a.has_nematic))
        delta = extra_terms<DIM, NOFF, TERMS == 2>(a, T, *terms, old, nw, t_old, t_new, vol_old, vol_new, x, y, z, pick, target, delta);
    const float u = to_f32(draw(key_accept, target));
    if (!(delta <= 0.0f || u < metropolis_exp(__fmul_rn(-delta, a.beta)))) return;
    if (TERMS == 2) {
        const int k = atomicAdd(a.pending_count, 1);
        a.pending[k] = make_uint4(target, nw, __float_as_uint(nw != 0 ? T.max_activity[t_new] : 0.0f), 0u);
    } else {
        acc.put(target, x, y, z, nw);
    }
    if (old != 0) acc.tally(old, -1, ds_old);
    if (nw != 0) acc.tally(nw, 1, ds_new);
    if (TERMS && a.tracks) commit_moments<DIM>(a, terms->cur, old, nw, an_old, an_new, x, y, z);
}

// The whole attempt at target (x, y, z): its pick, its two labels, and the
// copy when they differ.
template <int DIM, int NOFF, bool UNIFORM, class Access, int TERMS = 0>
__device__ __forceinline__ void direct_target(const SweepLaunch &a, const TypeTables &T, const Access &acc, uint64_t key_pick,
                                              uint64_t key_accept, int x, int y, int z,
                                              const TermView *terms = nullptr) {
    const int pick = pick_of<NOFF>(draw(key_pick, (uint32_t)((z * a.g.h + y) * a.g.w + x)));
    const uint32_t old = acc.label(x, y, z), nw = picked_label<DIM, NOFF>(a, acc, x, y, z, pick);
    const NeighbourReads<DIM, NOFF, Access> ln(a, acc, x, y, z);
    if (old != nw)
        direct_copy<DIM, NOFF, UNIFORM, Access, NeighbourReads<DIM, NOFF, Access>, TERMS>(a, T, acc, ln, key_accept, x, y,
                                                                                           z, pick, old, nw, terms);
}

// A direct pass (direct.cu) of the launch's neighbourhood and pricing form.
template <int DIM, int NOFF, bool UNIFORM>
cudaError_t launch_direct(const SweepLaunch &a, cudaStream_t stream);

}  // namespace glz
