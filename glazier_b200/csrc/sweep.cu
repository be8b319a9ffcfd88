// The checkerboard Metropolis copy sweep: the tiled kernel, the cluster sweep of
// small planes, the ensemble's kernels, and the launches that choose between
// these and the direct sweep (direct.cu).
//
// Replaces `cpm_sweep` of the reference device engine (glazier-cuda/src/
// lib.rs:436-716). Same-colour targets are two apart on every axis, outside
// any neighbourhood, so a pass's copies are independent and the labels a
// target reads do not change during the pass.
//
// Layout of the work in the tiled kernel, which one lattice takes on request
// only and whose pieces the ensemble's windowed kernels share:
//   - Persistent CTAs walk the lattice tile by tile. A tile and its one-site
//     halo are staged in shared memory; tiles clear of the periodic edge
//     arrive by a TMA tensor copy issued one tile ahead into the other of two
//     buffers, so the copy of tile i+1 overlaps the work on tile i. Edge
//     tiles, and lattices whose rows are not whole 16-byte units, take
//     wrapped plain loads.
//   - The CTA first draws every target's neighbour pick (one counter-hash
//     draw per target) and keeps only the targets whose neighbour carries
//     another label, about a fifth of them in a tissue, in a shared queue;
//     warps then take the queue 32 copies at a time and price them densely.
//     The expensive path never runs with idle lanes that a light target left
//     behind, and no warp waits on another's share.
//
// Per-cell tallies (volume, surface, exact moment sums) are read from the
// snapshot the rotation in engine.h gives each pass and changed by integer
// atomics whose order does not matter; a pass is therefore deterministic and
// a host replay of the same schedule reproduces it bit for bit.

#include <atomic>
#include <cuda.h>

#include <cstdlib>

#include "device.cuh"
#include "direct.cuh"
#include "engine.h"
#include "neighbours.cuh"
#include "pdl.cuh"
#include "pricing.cuh"
#include "terms.cuh"

namespace glz {

template <int DIM>
struct Tile;

// A plane's tile height (rows of targets and their window), a build-time knob.
#ifndef GLZ_TILE2_TY
#define GLZ_TILE2_TY 32
#endif

template <>
struct Tile<2> {
    static constexpr int TX = 128, TY = GLZ_TILE2_TY, TZ = 1;
    static constexpr int HX = 4;  // x halo rounded up to 16 bytes for the tensor copy
    static constexpr int PX = TX + 2 * HX, PY = TY + 2, PZ = 1;
    static constexpr int HZ = 0;
    static constexpr int NT = (TX / 2) * (TY / 2);
};

template <>
struct Tile<3> {
    static constexpr int TX = 64, TY = 8, TZ = 8;
    static constexpr int HX = 4;
    static constexpr int PX = TX + 2 * HX, PY = TY + 2, PZ = TZ + 2;
    static constexpr int HZ = 1;
    static constexpr int NT = (TX / 2) * (TY / 2) * (TZ / 2);
};

template <int DIM, int NOFF>
__host__ __device__ constexpr int window_offset(int k) {
    return (neighbour_offset<DIM, NOFF>(k, 2) * Tile<DIM>::PY + neighbour_offset<DIM, NOFF>(k, 1)) * Tile<DIM>::PX +
           neighbour_offset<DIM, NOFF>(k, 0);
}

#ifndef GLZ_SWEEP_MIN_BLOCKS
#define GLZ_SWEEP_MIN_BLOCKS 3
#endif

constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;
constexpr long long kWaitLimit = 1LL << 24;

template <int DIM>
struct SweepSmem {
    static constexpr int WIN = Tile<DIM>::PX * Tile<DIM>::PY * Tile<DIM>::PZ;
    // A tensor copy's shared-memory destination must sit on a 128-byte
    // boundary, so each window buffer is padded to a multiple of 32 labels.
    static constexpr int WIN_STRIDE = (WIN + 31) / 32 * 32;
    static constexpr int TPW = Tile<DIM>::NT / kWarps;  // targets per warp per tile
    alignas(128) uint32_t win[2][WIN_STRIDE];
    uint32_t queue[Tile<DIM>::NT];  // the tile's targets whose neighbour carries another label
    int queued, taken;
    float contact[kSmemTypes * kSmemTypes];
    int woff[26];
    int wring[26];
    alignas(8) unsigned long long mbar[2];
};

// Position of target j of a tile: local coordinates in the tile.
template <int DIM>
__device__ __forceinline__ void target_of(int j, int colour, int &lx, int &ly, int &lz) {
    using T = Tile<DIM>;
    const int jx = j % (T::TX / 2);
    const int jy = (j / (T::TX / 2)) % (T::TY / 2);
    const int jz = DIM == 3 ? j / ((T::TX / 2) * (T::TY / 2)) : 0;
    lx = 2 * jx + (colour & 1);
    ly = 2 * jy + ((colour >> 1) & 1);
    lz = DIM == 3 ? 2 * jz + ((colour >> 2) & 1) : 0;
}

// The rare parts of pricing live out of line, so the registers they need do
// not weigh on the common path.

// The per-colour guard: whether cell `old` keeps a site of a colour other than
// the pass's own, which no copy in this pass can take.
__device__ __noinline__ bool keeps_other_colour(const SweepLaunch &a, uint32_t old) {
    int other = 0;
    for (int c = 0; c < a.g.ncol; ++c)
        if (c != a.colour) other += a.vol_by_colour[(size_t)old * a.g.ncol + c];
    return other != 0;
}

// The connectivity veto (lib.rs:511-521): the ring positions of `old` around
// the target must be one piece. `wring` holds the ring's window offsets.
template <int DIM>
__device__ __noinline__ bool ring_one_piece(const int *wring, const uint32_t *win, int wc, uint32_t old) {
    uint32_t present = 0;
#pragma unroll
    for (int k = 0; k < kRing<DIM>; ++k)
        if (win[wc + wring[k]] == old) present |= 1u << cube_bit<DIM, kRing<DIM>>(k);
    return one_piece<DIM>(present);
}

template <int DIM, int NOFF>
__device__ __noinline__ float tile_extra_terms(const SweepLaunch &a, uint32_t old, uint32_t nw, int t_old, int t_new,
                                               int vol_old, int vol_new, int x, int y, int z, int pick,
                                               uint32_t target, float delta) {
    const TermView v{a.mom_base, a.mom_prev, a.mom_cur, a.field_cur, nullptr};
    if (!a.has_motility)
        return extra_terms<DIM, NOFF, false>(a, a.t, v, old, nw, t_old, t_new, vol_old, vol_new, x, y, z, pick, target,
                                             delta);
    return extra_terms<DIM, NOFF, true>(a, a.t, v, old, nw, t_old, t_new, vol_old, vol_new, x, y, z, pick, target, delta);
}

template <int DIM>
__device__ __noinline__ void tile_commit_moments(const SweepLaunch &a, uint32_t old, uint32_t nw, int x, int y, int z) {
    commit_moments<DIM>(a, a.mom_cur, old, nw, anchor_of(a, old), anchor_of(a, nw), x, y, z);
}

// Price one copy attempt whose neighbour pick is known to carry another label
// and commit it if the Metropolis test takes it. UNIFORM: every label carries
// one type, so the contact sum is J times a difference of like-neighbour
// counts (the host has checked that J m is exact in f32 for every count m,
// which makes it the same number the neighbour-by-neighbour sum rounds to)
// and the per-type constants come from the launch parameters.
//
// EXTRAS false compiles out the length, chemotaxis, connectivity and moment
// parts, for launches whose model has none of them. `woff`, `contact` and
// `wring` are the shared-memory tables: window offset of each pick, the
// contact matrix when `small_types`, the connectivity ring.
template <int DIM, int NOFF, bool UNIFORM, bool EXTRAS>
__device__ __forceinline__ void price_and_commit(const SweepLaunch &a, const int *woff, const float *contact,
                                                 const int *wring, const uint32_t *win, uint32_t entry, int x0,
                                                 int y0, int z0, bool small_types) {
    using T = Tile<DIM>;
    const int W = a.g.w, H = a.g.h;
    const int j = (int)(entry & 0xffffu);
    const int pick = (int)(entry >> 16);
    int lx, ly, lz;
    target_of<DIM>(j, a.colour, lx, ly, lz);
    const int x = x0 + lx, y = y0 + ly, z = z0 + lz;
    const uint32_t target = (uint32_t)((z * H + y) * W + x);
    const int wc = ((lz + T::HZ) * T::PY + (ly + 1)) * T::PX + (lx + T::HX);
    const uint32_t old = win[wc];
    const uint32_t nw = win[wc + woff[pick]];

    // The snapshot tallies of both cells, requested before the neighbour loop
    // so their latency hides behind it.
    long long prev_old = 0, prev_new = 0;
    int2 base_old = make_int2(0, 0), base_new = make_int2(0, 0);
    if (old != 0) {
        base_old = a.vs_base[old];
        prev_old = a.vs_prev[old];
    }
    if (nw != 0) {
        base_new = a.vs_base[nw];
        prev_new = a.vs_prev[nw];
    }
    const int t_old = UNIFORM ? a.uniform_type : a.cell_type[old];
    const int t_new = UNIFORM ? a.uniform_type : a.cell_type[nw];

    float delta = 0.0f;
    int like_old = 0, like_new = 0;
    if (UNIFORM) {
#pragma unroll
        for (int k = 0; k < NOFF; ++k) {
            const uint32_t ln = win[wc + window_offset<DIM, NOFF>(k)];
            like_old += ln == old;
            like_new += ln == nw;
        }
        delta = __fmul_rn(a.uniform_contact, (float)(like_old - like_new));
    } else {
#pragma unroll
        for (int k = 0; k < NOFF; ++k) {
            const uint32_t ln = win[wc + window_offset<DIM, NOFF>(k)];
            const int tn = ln == old ? t_old : (ln == nw ? t_new : (int)a.cell_type[ln]);
            if (ln != old) {
                const float j_old =
                    small_types ? contact[t_old * a.n_types + tn] : a.t.contact[t_old * a.n_types + tn];
                delta = __fsub_rn(delta, j_old);
            } else {
                ++like_old;
            }
            if (ln != nw) {
                const float j_new =
                    small_types ? contact[t_new * a.n_types + tn] : a.t.contact[t_new * a.n_types + tn];
                delta = __fadd_rn(delta, j_new);
            } else {
                ++like_new;
            }
        }
    }

    if (old != 0) {
        // A like neighbour is a site of another colour, since every neighbour
        // of a target is; only a target with none needs the per-colour count.
        if (like_old == 0 && !keeps_other_colour(a, old)) return;
        if (EXTRAS && a.g.ring_n > 0 && a.t.connected[t_old] && !ring_one_piece<DIM>(wring, win, wc, old)) return;
    }
    const int ds_old = 2 * like_old - NOFF;
    const int ds_new = NOFF - 2 * like_new;

    int vol_old, surf_old, vol_new, surf_new;
    {
        int dv, ds;
        unpack_delta(prev_old, dv, ds);
        vol_old = base_old.x + dv;
        surf_old = base_old.y + ds;
        unpack_delta(prev_new, dv, ds);
        vol_new = base_new.x + dv;
        surf_new = base_new.y + ds;
    }
    delta = size_terms<UNIFORM>(a, a.t, old, nw, t_old, t_new, vol_old, vol_new, surf_old, surf_new, ds_old, ds_new, delta);
    if (EXTRAS && (a.has_length || a.has_chemotaxis || a.has_external || a.has_motility || a.has_nematic))
        delta = tile_extra_terms<DIM, NOFF>(a, old, nw, t_old, t_new, vol_old, vol_new, x, y, z, pick, target, delta);

    // Metropolis: a copy that lowers the energy (or keeps it) is taken, else
    // with probability exp(-delta / T). The draw and the exponential are
    // computed on every lane, so the test needs no branch; a lane whose delta
    // is not positive takes the copy whatever they say.
    {
        const float u = to_f32(draw(a.key_accept, target));
        if (!(delta <= 0.0f || u < metropolis_exp(__fmul_rn(-delta, a.beta)))) return;
    }

    if (EXTRAS && a.has_motility) {
        const int k = atomicAdd(a.pending_count, 1);
        a.pending[k] = make_uint4(target, nw, __float_as_uint(nw != 0 ? a.t.max_activity[t_new] : 0.0f), 0u);
    } else {
        a.labels[target] = nw;
    }
    if (old != 0) {
        atomicAdd(&a.vs_cur[old], pack_delta(-1, ds_old));
        atomicSub(&a.vol_by_colour[(size_t)old * a.g.ncol + a.colour], 1);
    }
    if (nw != 0) {
        atomicAdd(&a.vs_cur[nw], pack_delta(1, ds_new));
        atomicAdd(&a.vol_by_colour[(size_t)nw * a.g.ncol + a.colour], 1);
    }
    if (EXTRAS && a.tracks) tile_commit_moments<DIM>(a, old, nw, x, y, z);
}

template <int DIM>
__device__ __forceinline__ void tile_origin(int t, int W, int H, int &x0, int &y0, int &z0) {
    using T = Tile<DIM>;
    const int tiles_x = (W + T::TX - 1) / T::TX;
    const int tiles_y = (H + T::TY - 1) / T::TY;
    x0 = (t % tiles_x) * T::TX;
    y0 = ((t / tiles_x) % tiles_y) * T::TY;
    z0 = DIM == 3 ? (t / (tiles_x * tiles_y)) * T::TZ : 0;
}

template <int DIM>
__device__ __forceinline__ bool tile_interior(const SweepLaunch &a, int x0, int y0, int z0) {
    using T = Tile<DIM>;
    return a.use_tma && x0 >= T::HX && x0 + T::TX + T::HX <= a.g.w && y0 >= 1 && y0 + T::TY + 1 <= a.g.h &&
           (DIM == 2 || (z0 >= 1 && z0 + T::TZ + 1 <= a.g.d));
}

// One thread issues the tensor copy of a tile's window into `dst`, arriving
// on `bar` with the byte count the copy will deliver.
template <int DIM>
__device__ __forceinline__ void issue_window(const CUtensorMap &tmap, uint32_t *dst, unsigned long long *bar, int x0,
                                             int y0, int z0) {
    using T = Tile<DIM>;
    const uint32_t b = smem_addr(bar);
    const uint32_t bytes = SweepSmem<DIM>::WIN * sizeof(uint32_t);
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(b), "r"(bytes) : "memory");
    const uint64_t map = reinterpret_cast<uint64_t>(&tmap);
    // x0 - HX is a multiple of 4 labels, i.e. of 16 bytes, as a tensor copy's
    // inner coordinate must be.
    if (DIM == 2) {
        asm volatile(
            "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::
                "r"(smem_addr(dst)),
            "l"(map), "r"(x0 - T::HX), "r"(y0 - 1), "r"(b)
            : "memory");
    } else {
        asm volatile(
            "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], "
            "[%5];" ::"r"(smem_addr(dst)),
            "l"(map), "r"(x0 - T::HX), "r"(y0 - 1), "r"(z0 - 1), "r"(b)
            : "memory");
    }
}

// Wrapped plain loads of a tile's window, for tiles on the periodic edge and
// lattices whose rows are not whole 16-byte units.
template <int DIM>
__device__ __forceinline__ void load_window_plain(const SweepLaunch &a, uint32_t *win, int x0, int y0, int z0) {
    using T = Tile<DIM>;
    using Smem = SweepSmem<DIM>;
    const int tid = threadIdx.x;
    const int W = a.g.w, H = a.g.h, D = a.g.d;
    // Where every window coordinate lies within one lattice span of it (the
    // halo reaches back no further than a span, the last tile's window no
    // further than one span past the end) a compare wraps it; otherwise the
    // remainder does.
    const auto reach = [](int n, int t, int h) { return h <= n && ((n - 1) / t) * t + t + h <= 2 * n; };
    const bool once = reach(W, T::TX, T::HX) && reach(H, T::TY, 1) && (DIM == 2 || reach(D, T::TZ, T::HZ));
    for (int i = tid; i < Smem::WIN; i += blockDim.x) {
        const int px = i % T::PX;
        const int py = (i / T::PX) % T::PY;
        const int pz = i / (T::PX * T::PY);
        int gx = x0 - T::HX + px, gy = y0 - 1 + py, gz = DIM == 3 ? z0 - 1 + pz : 0;
        if (once) {
            gx += gx < 0 ? W : (gx >= W ? -W : 0);
            gy += gy < 0 ? H : (gy >= H ? -H : 0);
            if (DIM == 3) gz += gz < 0 ? D : (gz >= D ? -D : 0);
        } else {
            gx = wrap(gx, W);
            gy = wrap(gy, H);
            gz = DIM == 3 ? wrap(gz, D) : 0;
        }
        win[i] = a.labels[((size_t)gz * H + gy) * W + gx];
    }
    // generic writes to a buffer a later tensor copy will overwrite
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncthreads();
}

// Price every target of the pass's colour in one tile whose window is in
// shared memory: the light pass queues the targets whose neighbour pick
// carries another label, the heavy pass prices and commits the queue.
template <int DIM, int NOFF, bool UNIFORM>
__device__ __forceinline__ void price_tile(const SweepLaunch &a, SweepSmem<DIM> &S, const uint32_t *win, int x0,
                                           int y0, int z0, bool small_types) {
    using T = Tile<DIM>;
    using Smem = SweepSmem<DIM>;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int W = a.g.w, H = a.g.h, D = a.g.d;
    // Light pass: every target's pick; only targets whose neighbour
    // carries another label go into the tile's queue. A warp keeps its
    // entries in registers and reserves queue room once per tile.
    constexpr int PER_LANE = Smem::TPW / 32;
    const bool full = x0 + T::TX <= W && y0 + T::TY <= H && (DIM == 2 || z0 + T::TZ <= D);
    const int tile_base = (z0 * H + y0) * W + x0;
    uint32_t entries[PER_LANE];
    unsigned masks[PER_LANE];
    int total = 0;
#pragma unroll
    for (int k = 0; k < PER_LANE; ++k) {
        const int j = warp * Smem::TPW + k * 32 + lane;
        int lx, ly, lz;
        target_of<DIM>(j, a.colour, lx, ly, lz);
        bool active = false;
        if (full || (x0 + lx < W && y0 + ly < H && (DIM == 2 || z0 + lz < D))) {
            const uint32_t target = (uint32_t)(tile_base + (lz * H + ly) * W + lx);
            const int wc = ((lz + T::HZ) * T::PY + (ly + 1)) * T::PX + (lx + T::HX);
            const int pick = pick_of<NOFF>(draw(a.key_pick, target));
            active = win[wc] != win[wc + S.woff[pick]];
            entries[k] = (uint32_t)j | ((uint32_t)pick << 16);
        }
        masks[k] = __ballot_sync(0xffffffffu, active);
        total += __popc(masks[k]);
    }
    int base = 0;
    if (lane == 0 && total) base = atomicAdd(&S.queued, total);
    base = __shfl_sync(0xffffffffu, base, 0);
    const unsigned below = (1u << lane) - 1u;
#pragma unroll
    for (int k = 0; k < PER_LANE; ++k) {
        if (masks[k] & (1u << lane)) S.queue[base + __popc(masks[k] & below)] = entries[k];
        base += __popc(masks[k]);
    }
    __syncthreads();
    // Heavy pass: warps take the queue 32 copies at a time.
    const int queued = S.queued;
    for (;;) {
        int first = 0;
        if (lane == 0) first = atomicAdd(&S.taken, 32);
        first = __shfl_sync(0xffffffffu, first, 0);
        if (first >= queued) break;
        if (first + lane < queued)
            price_and_commit<DIM, NOFF, UNIFORM, true>(a, S.woff, S.contact, S.wring, win, S.queue[first + lane], x0,
                                                       y0, z0, small_types);
    }
    __syncthreads();
    if (tid == 0) {
        S.queued = 0;
        S.taken = 0;
    }
}

// Wait for phase `parity` of an mbarrier, giving up after kWaitLimit polls.
__device__ __forceinline__ uint32_t wait_parity(unsigned long long *bar, uint32_t parity) {
    const uint32_t b = smem_addr(bar);
    uint32_t done = 0;
    for (long long spin = 0; spin < kWaitLimit && !done; ++spin) {
        asm volatile(
            "{ .reg .pred p; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }"
            : "=r"(done)
            : "r"(b), "r"(parity)
            : "memory");
    }
    return done;
}

// Tally rotation for the next pass, spread over the whole grid: no thread of
// this pass reads what is written here (engine.h).
template <int DIM>
__device__ __forceinline__ void rotate_tallies(const SweepLaunch &a) {
    const int NM = a.g.nm;
    const size_t stride = (size_t)gridDim.x * blockDim.x;
    const size_t n = a.n_live ? (size_t)*a.n_live : (size_t)a.n_labels;
    for (size_t l = (size_t)blockIdx.x * blockDim.x + threadIdx.x; l < n; l += stride) {
        int dv, ds;
        unpack_delta(a.vs_prev[l], dv, ds);
        const int2 b = a.vs_base[l];
        a.vs_next_base[l] = make_int2(b.x + dv, b.y + ds);
        a.vs_clear[l] = 0;
        if (a.tracks) {
#pragma unroll
            for (int k = 0; k < NM; ++k) {
                a.mom_next_base[l * NM + k] = a.mom_base[l * NM + k] + a.mom_prev[l * NM + k];
                a.mom_clear[l * NM + k] = 0;
            }
        }
    }
}

template <int DIM, int NOFF, bool UNIFORM>
__global__ void __launch_bounds__(kThreads, GLZ_SWEEP_MIN_BLOCKS) sweep_kernel(const __grid_constant__ SweepLaunch a,
                                                         const __grid_constant__ CUtensorMap tmap) {
    using T = Tile<DIM>;
    using Smem = SweepSmem<DIM>;
    static_assert(Smem::WIN_STRIDE * sizeof(uint32_t) % 128 == 0, "window buffers must stay 128-byte aligned");
    extern __shared__ __align__(128) unsigned char smem_raw[];
    // The launch asks for 128 spare bytes so the layout can start on a
    // 128-byte boundary whatever the dynamic region's own alignment.
    const uint32_t raw = smem_addr(smem_raw);
    Smem &S = *reinterpret_cast<Smem *>(smem_raw + ((128u - (raw & 127u)) & 127u));

    const int tid = threadIdx.x;
    if (smem_addr(S.win[0]) & 127u) {  // never true by construction; refuse rather than copy misaligned
        if (tid == 0) atomicExch(a.error_flag, 3);
        return;
    }
    const int W = a.g.w, H = a.g.h, D = a.g.d;

    const bool small_types = a.n_types <= kSmemTypes;
    if (small_types)
        for (int i = tid; i < a.n_types * a.n_types; i += blockDim.x) S.contact[i] = a.t.contact[i];
    if (tid < NOFF) S.woff[tid] = (a.g.off[tid][2] * T::PY + a.g.off[tid][1]) * T::PX + a.g.off[tid][0];
    if (tid < kRing<DIM>) S.wring[tid] = window_offset<DIM, kRing<DIM>>(tid);
    if (tid == 0) {
        S.queued = 0;
        S.taken = 0;
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(&S.mbar[0])));
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(&S.mbar[1])));
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    // Nothing above reads what the previous pass writes; a programmatic launch
    // may have started this grid before it ended (see launch).
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    rotate_tallies<DIM>(a);
    __syncthreads();

    const int tiles = ((W + T::TX - 1) / T::TX) * ((H + T::TY - 1) / T::TY) * (DIM == 3 ? (D + T::TZ - 1) / T::TZ : 1);
    int waited[2] = {0, 0};
    bool pending[2] = {false, false};  // a copy issued into the buffer and not yet waited for
    int t = blockIdx.x;
    if (t < tiles) {
        int x0, y0, z0;
        tile_origin<DIM>(t, W, H, x0, y0, z0);
        if (tile_interior<DIM>(a, x0, y0, z0)) {
            if (tid == 0) issue_window<DIM>(tmap, S.win[0], &S.mbar[0], x0, y0, z0);
            pending[0] = true;
        }
    }
    for (int it = 0; t < tiles; t += gridDim.x, ++it) {
        const int buf = it & 1;
        int x0, y0, z0;
        tile_origin<DIM>(t, W, H, x0, y0, z0);
        const int next = t + gridDim.x;
        if (next < tiles) {
            int nx0, ny0, nz0;
            tile_origin<DIM>(next, W, H, nx0, ny0, nz0);
            if (tile_interior<DIM>(a, nx0, ny0, nz0)) {
                if (tid == 0) issue_window<DIM>(tmap, S.win[buf ^ 1], &S.mbar[buf ^ 1], nx0, ny0, nz0);
                pending[buf ^ 1] = true;
            }
        }
        uint32_t *win = S.win[buf];
        if (tile_interior<DIM>(a, x0, y0, z0)) {
            // Bounded wait: a copy that never lands sets the error flag and the
            // CTA stops rather than spinning for ever.
            const uint32_t done = wait_parity(&S.mbar[buf], waited[buf] & 1);
            waited[buf] += 1;
            pending[buf] = false;
            if (!__syncthreads_and(done)) {
                // Before leaving, give a copy still in flight into the other
                // buffer its own bounded wait, so no copy lands after exit.
                if (pending[buf ^ 1]) wait_parity(&S.mbar[buf ^ 1], waited[buf ^ 1] & 1);
                if (tid == 0) atomicExch(a.error_flag, 1);
                return;
            }
        } else {
            load_window_plain<DIM>(a, win, x0, y0, z0);
        }
        price_tile<DIM, NOFF, UNIFORM>(a, S, win, x0, y0, z0, small_types);
    }
}

// ---------------------------------------------------------------- the lean windows
//
// Replicas whose copies price only contact, volume and surface terms can be
// swept by the lean ensemble kernel (below): the draws, copies and commits of
// sweep_kernel, with the work laid out so that no CTA-wide barrier stands
// between tiles.
//   - Each warp owns a fixed share of every tile's targets (two rows of them
//     in a plane) and prices it alone: light pass, its own queue, heavy pass.
//     Warps drift apart by up to the depth of the window ring.
//   - Windows arrive through a ring of kLeanStages buffers, by tensor copies
//     issued up to kLeanStages tiles ahead; the last warp to finish with a
//     buffer issues the next copy into it.
//   - A tile on the periodic edge takes the copy with its out-of-lattice
//     cells filled, then the warps overwrite those cells with the wrapped
//     labels, each a disjoint share of window rows, and meet on an mbarrier
//     (a bounded wait) before pricing. Without tensor copies (rows that are
//     not whole 16-byte units, or a lattice smaller than a window) every cell
//     of every window is loaded that way.
// One lattice's lean passes take the streaming form of direct.cu instead,
// which measured faster at every size.
#ifndef GLZ_LEAN_STAGES
#define GLZ_LEAN_STAGES 3
#endif
constexpr int kLeanStages = GLZ_LEAN_STAGES;
#ifndef GLZ_LEAN_WARPS
#define GLZ_LEAN_WARPS 8
#endif
#ifndef GLZ_LEAN_MIN_BLOCKS
#define GLZ_LEAN_MIN_BLOCKS 3
#endif
constexpr int kLeanWarps = GLZ_LEAN_WARPS;
constexpr int kLeanThreads = 32 * kLeanWarps;
constexpr int kRotate = 2;  // labels per thread whose rotation reads are copied in ahead

template <int DIM>
struct LeanSmem {
    static constexpr int WIN = SweepSmem<DIM>::WIN;
    static constexpr int WIN_STRIDE = SweepSmem<DIM>::WIN_STRIDE;
    static constexpr int TPW = Tile<DIM>::NT / kLeanWarps;  // targets per warp per tile
    alignas(128) uint32_t win[kLeanStages][WIN_STRIDE];
    uint32_t queue[kLeanWarps][TPW + 32];  // a tile's entries after fewer than 32 held from the tile before
    int woff[26];
    int done[kLeanStages];    // warps finished with the buffer's current tile
    int issued[kLeanStages];  // copies issued into the buffer
    alignas(8) unsigned long long full[kLeanStages];     // the buffer's copy has landed
    alignas(8) unsigned long long patched[kLeanStages];  // every warp has patched its rows
    // the tally rotation's first kRotate labels per thread, copied in while the tiles run
    alignas(16) int2 rot_base[2 * kLeanThreads];
    alignas(16) long long rot_prev[2 * kLeanThreads];
};

// Tensor copies for every tile, edge tiles included: the lattice's rows are
// whole 16-byte units and the lattice is at least a window on every axis, so
// an edge window wraps at most once per axis.
template <int DIM>
__device__ __forceinline__ bool lean_copies(const SweepLaunch &a) {
    using T = Tile<DIM>;
    return a.use_tma && a.g.w >= T::PX && a.g.h >= T::PY && (DIM == 2 || a.g.d >= T::PZ);
}

// The warp's rows of an edge tile's window (rows warp, warp + kLeanWarps, ...):
// in a row whose y (and z) lie in the lattice only the cells the copy left
// filled, else every cell, from the wrapped labels.
template <int DIM>
__device__ __forceinline__ void lean_patch(const SweepLaunch &a, uint32_t *win, int x0, int y0, int z0, bool copies) {
    using T = Tile<DIM>;
    const int W = a.g.w, H = a.g.h, D = a.g.d;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    // Whether every window coordinate is at most one lattice span outside it
    // (the halo reaches back no further than a span, the last tile's window
    // no further than one span past the end), so one step wraps it.
    const auto reach = [](int n, int t, int h) { return h <= n && ((n - 1) / t) * t + t + h <= 2 * n; };
    const bool once = reach(W, T::TX, T::HX) && reach(H, T::TY, 1) && (DIM == 2 || reach(D, T::TZ, T::HZ));
    int lo = 0, hi = 0;  // window columns [lo, hi) lie inside the lattice
    if (copies) {
        lo = T::HX - x0 > 0 ? T::HX - x0 : 0;
        hi = W - x0 + T::HX < T::PX ? W - x0 + T::HX : T::PX;
    }
    for (int r = warp; r < T::PY * T::PZ; r += kLeanWarps) {
        const int py = r % T::PY, pz = r / T::PY;
        const int gy = y0 - 1 + py, gz = DIM == 3 ? z0 - T::HZ + pz : 0;
        const bool inside = copies && gy >= 0 && gy < H && gz >= 0 && gz < D;
        const auto wr = [once](int v, int n) { return once ? (v < 0 ? v + n : (v >= n ? v - n : v)) : wrap(v, n); };
        const uint32_t *row = a.labels + ((size_t)(DIM == 3 ? wr(gz, D) : 0) * H + wr(gy, H)) * W;
        uint32_t *dst = win + r * T::PX;
        const int n = inside ? lo + (T::PX - hi) : T::PX;
        for (int c = lane; c < n; c += 32) {
            const int px = inside && c >= lo ? hi + (c - lo) : c;
            dst[px] = row[wr(x0 - T::HX + px, W)];
        }
    }
}

// A grid barrier for the ensemble's cooperative launches.
// polls of the barrier word (each an L2 round trip, so the limit is seconds)
constexpr long long kBarrierLimit = 1LL << 22;

// Barrier number k of the launch (k = 0, 1, ...): false if it timed out.
__device__ __forceinline__ bool grid_barrier(unsigned *bar, unsigned k) {
    __shared__ int ok;
    __syncthreads();
    if (threadIdx.x == 0) {
        ok = 1;
        __threadfence();
        if (atomicAdd(&bar[0], 1u) + 1u == gridDim.x * (k + 1u)) {
            __threadfence();
            atomicExch(&bar[1], k + 1u);
        } else {
            long long spin = 0;
            for (;;) {
                unsigned g;
                asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(g) : "l"(&bar[1]) : "memory");
                if (g >= k + 1u || ++spin > kBarrierLimit) {
                    ok = g >= k + 1u;
                    break;
                }
            }
        }
        __threadfence();
    }
    __syncthreads();
    return ok != 0;
}

// ---------------------------------------------------------------- the cluster sweep
//
// A small plane of a lean model with nothing between its colour passes (no
// fields, division, death or infection) runs every MCS of a call in ONE
// thread-block cluster, its lattice and tallies in the CTAs' shared memory:
//   - The lattice is split by rows over the CTAs, an even number of rows
//     each, with a copy of the row either side. A copy committed to a CTA's
//     first or last row is also written to the neighbour's copy of it, so
//     every label a pass reads is in the CTA's own shared memory.
//   - The tallies are dealt by label (label l in CTA l mod C), read and
//     changed through distributed shared memory. Cell types are held whole by
//     every CTA.
//   - Each thread's targets are the same sites of every pass but for the
//     colour's offset, and the next pass's picks are drawn between the
//     cluster barrier's arrive and its wait, so a pass starts at its label
//     reads. The unlike targets go into the CTA's queue with their labels,
//     and whole warps price it.
// The copies, draws and tally rotation are the direct sweep's; the lattice
// and tallies go back to global memory at the end. What bounds a pass is its
// chain: labels, queue, the two cells' tallies across the cluster, pricing,
// the commits' atomics, the barrier (1.5 us a pass at 128^2; 2.4 when every
// label was read through a table of row pointers into the CTAs, the picks
// were drawn at the pass's start and a target's coordinates divided out).

constexpr int kClusterThreads = 1024;  // a CTA's threads at most
constexpr int kClusterMost = 16;       // CTAs of a cluster at most (16 is the non-portable limit)
constexpr int kClusterSmem = 200 * 1024;
constexpr int kClusterPerThread = 4;  // a thread's targets a pass at most

// Shared-memory layout of one CTA of a C-CTA cluster sweep (bytes from the
// start): delta[3][Lc] (i64), base[2][Lc] (int2), the queue (uint4 each),
// slab[R + 2][W] (u32), volc[Lc][4] (i32), the types, the queue's two fill
// counters.
struct ClusterLayout {
    int C, R, Lc, qcap;
    size_t delta, base, queue, slab, volc, types, qn, bytes;
    __host__ __device__ ClusterLayout(int w, int h, int n_labels, int c) : C(c) {
        R = 2 * ((h / 2 + c - 1) / c);
        Lc = (n_labels + c - 1) / c;
        qcap = R / 2 * (w / 2);
        delta = 0;
        base = delta + 3 * (size_t)Lc * 8;
        queue = (base + 2 * (size_t)Lc * 8 + 15) / 16 * 16;
        slab = queue + (size_t)qcap * 16;
        volc = slab + ((size_t)(R + 2) * w * 4 + 15) / 16 * 16;
        types = volc + (size_t)Lc * 16;
        qn = types + ((size_t)n_labels + 15) / 16 * 16;
        bytes = qn + 16;
    }
};

// The address of a CTA's own shared memory as it appears in CTA `rank` of the
// cluster, and the reads and changes that take such an address.
__device__ __forceinline__ uint32_t cluster_addr(uint32_t own, int rank) {
    uint32_t a;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(own), "r"(rank));
    return a;
}

__device__ __forceinline__ int2 cluster_ld_int2(uint32_t a) {
    int2 v;
    asm volatile("ld.shared::cluster.v2.s32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(a));
    return v;
}

__device__ __forceinline__ long long cluster_ld_i64(uint32_t a) {
    long long v;
    asm volatile("ld.shared::cluster.s64 %0, [%1];" : "=l"(v) : "r"(a));
    return v;
}

__device__ __forceinline__ int cluster_ld_int(uint32_t a) {
    int v;
    asm volatile("ld.shared::cluster.s32 %0, [%1];" : "=r"(v) : "r"(a));
    return v;
}

__device__ __forceinline__ void cluster_st(uint32_t a, uint32_t v) {
    asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(a), "r"(v) : "memory");
}

__device__ __forceinline__ void cluster_add(uint32_t a, unsigned long long v) {
    asm volatile("red.relaxed.cluster.shared::cluster.add.u64 [%0], %1;" ::"r"(a), "l"(v) : "memory");
}

__device__ __forceinline__ void cluster_add(uint32_t a, int v) {
    asm volatile("red.relaxed.cluster.shared::cluster.add.s32 [%0], %1;" ::"r"(a), "r"(v) : "memory");
}

__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire;" ::: "memory"); }

// Labels and tallies of a cluster pass. `row` is the target's row of the
// slab, set per copy.
struct ClusterPass {
    uint32_t base_at, prev_at, cur_at, volc_at;  // this pass's slots in the CTA's own shared memory
    const uint8_t *types;
    int shift, mask, colour;
    uint32_t *slab_row;         // the target's row in the slab
    uint32_t halo_up, halo_dn;  // the neighbours' copies of the CTA's first and last row
    bool first, last;           // the target's row is the CTA's first, last
    __device__ __forceinline__ int type(uint32_t l) const { return types[l]; }
    __device__ __forceinline__ int2 base(uint32_t l) const {
        return cluster_ld_int2(cluster_addr(base_at + (l >> shift) * 8, (int)(l & mask)));
    }
    __device__ __forceinline__ long long prev(uint32_t l) const {
        return cluster_ld_i64(cluster_addr(prev_at + (l >> shift) * 8, (int)(l & mask)));
    }
    __device__ __forceinline__ bool keeps_other_colour(uint32_t old) const {
        const uint32_t v = cluster_addr(volc_at + (old >> shift) * 16, (int)(old & mask));
        int other = 0;
        for (int c = 0; c < 4; ++c)
            if (c != colour) other += cluster_ld_int(v + 4 * c);
        return other != 0;
    }
    __device__ __forceinline__ void put(uint32_t, int x, int, int, uint32_t nw) const {
        slab_row[x] = nw;
        if (first) cluster_st(halo_up + 4 * x, nw);
        if (last) cluster_st(halo_dn + 4 * x, nw);
    }
    __device__ __forceinline__ void tally(uint32_t l, int dv, int ds) const {
        cluster_add(cluster_addr(cur_at + (l >> shift) * 8, (int)(l & mask)), pack_delta(dv, ds));
        cluster_add(cluster_addr(volc_at + (l >> shift) * 16 + 4 * colour, (int)(l & mask)), dv);
    }
};

// A target's energy neighbours in the slab: its row and the rows either side.
template <int NOFF>
struct SlabLabels {
    const uint32_t *row;
    int W, x, xm, xp;
    __device__ __forceinline__ uint32_t operator()(int k) const {
        const int dx = neighbour_offset<2, NOFF>(k, 0), dy = neighbour_offset<2, NOFF>(k, 1);
        return row[dy * W + (dx < 0 ? xm : (dx > 0 ? xp : x))];
    }
    __device__ __forceinline__ uint32_t ring(int) const { return 0; }
};

template <int NOFF, bool UNIFORM, int TPT>
__global__ void __launch_bounds__(kClusterThreads, 1) cluster_sweep_kernel(const __grid_constant__ ResidentLaunch r) {
    const SweepLaunch &a = r.a;
    int C, rank;
    asm("mov.u32 %0, %%cluster_nctaid.x;" : "=r"(C));
    asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
    const int W = a.g.w, H = a.g.h, n_labels = a.n_labels, hw = W / 2;
    const ClusterLayout L(W, H, n_labels, C);
    const int tid = threadIdx.x, nth = blockDim.x, lane = tid & 31;
    __shared__ TypeSmem<false> tables;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    long long *delta = reinterpret_cast<long long *>(smem_raw + L.delta);
    int2 *base = reinterpret_cast<int2 *>(smem_raw + L.base);
    uint4 *queue = reinterpret_cast<uint4 *>(smem_raw + L.queue);
    uint32_t *slab = reinterpret_cast<uint32_t *>(smem_raw + L.slab);  // row y0 - 1 first
    int *volc = reinterpret_cast<int *>(smem_raw + L.volc);
    uint8_t *types = smem_raw + L.types;
    int *qn = reinterpret_cast<int *>(smem_raw + L.qn);
    const TypeTables T = UNIFORM ? a.t : load_types<false>(a, tables);
    const int y0 = min(H, rank * L.R), y1 = min(H, y0 + L.R), rows = y1 - y0;
    if (tid < 2) qn[tid] = 0;

    // this CTA's rows and the two about them, its labels' tallies, the types
    if (rows > 0)
        for (int i = tid; i < (rows + 2) * W; i += nth) {
            const int k = i / W, y = y0 - 1 + k;
            slab[i] = a.labels[(size_t)(y < 0 ? H - 1 : (y >= H ? y - H : y)) * W + (i - k * W)];
        }
    for (int i = tid; i < L.Lc; i += nth) {
        const int l = i * C + rank;
        const bool in = l < n_labels;
        for (int k = 0; k < 2; ++k) base[k * L.Lc + i] = in ? r.vs_base[k][l] : make_int2(0, 0);
        for (int k = 0; k < 3; ++k) delta[k * L.Lc + i] = in ? r.vs_delta[k][l] : 0;
        for (int c = 0; c < 4; ++c) volc[i * 4 + c] = in ? a.vol_by_colour[(size_t)l * 4 + c] : 0;
    }
    if (!UNIFORM)
        for (int i = tid; i < n_labels; i += nth) types[i] = a.cell_type[i];
    // The CTA's first row is the row after the CTA before's last, its last
    // row the one before the next's first.
    const int filled = (H - 1) / L.R;  // the last CTA with rows
    const int up = rank == 0 ? filled : rank - 1, dn = rank >= filled ? 0 : rank + 1;
    const int up_rows = min(H, (up + 1) * L.R) - up * L.R;
    ClusterPass acc;
    acc.types = types;
    acc.shift = __ffs(C) - 1;
    acc.mask = C - 1;
    acc.volc_at = smem_addr(volc);
    acc.halo_up = cluster_addr(smem_addr(slab) + (uint32_t)((up_rows + 1) * W) * 4u, up);
    acc.halo_dn = cluster_addr(smem_addr(slab), dn);
    const uint32_t base_at = smem_addr(base), delta_at = smem_addr(delta);

    // this thread's targets, the same in every pass but for the colour's offset
    const int count = rows / 2 * hw;
    int tx[TPT], ty[TPT], pick[TPT];
#pragma unroll
    for (int k = 0; k < TPT; ++k) {
        const int t = k * nth + tid, j = t / hw;
        tx[k] = t < count ? 2 * (t - j * hw) : -1;
        ty[k] = 2 * j;
    }
    const auto draw_picks = [&](uint64_t key, int c) {
#pragma unroll
        for (int k = 0; k < TPT; ++k)
            if (tx[k] >= 0)
                pick[k] = pick_of<NOFF>(
                    draw(key, (uint32_t)((y0 + ty[k] + ((c >> 1) & 1)) * W + tx[k] + (c & 1))));
    };
    uint32_t step = (uint32_t)r.step0;
    draw_picks(stream_key(r.seed, (int32_t)step, 0, 0), 0);
    cluster_arrive();  // every CTA's part in place before any is read
    cluster_wait();

    int b = (int)(r.pass0 % 2), cur = (int)(r.pass0 % 3), parity = 0;
    for (int m = 0; m < r.mcs; ++m) {
        for (int c = 0; c < 4; ++c) {
            const int next = cur == 2 ? 0 : cur + 1, prev = cur == 0 ? 2 : cur - 1;
            const int cx = c & 1, cy = (c >> 1) & 1;
            acc.colour = c;
            acc.base_at = base_at + (uint32_t)(b * L.Lc) * 8u;
            acc.prev_at = delta_at + (uint32_t)(prev * L.Lc) * 8u;
            acc.cur_at = delta_at + (uint32_t)(cur * L.Lc) * 8u;
            const uint64_t key_accept = stream_key(r.seed, (int32_t)step, c, 1);
            // Light step: the two labels of every target; the unlike go into
            // the queue (a warp's slots reserved at once). A pass's copies
            // read only its snapshot and other colours' labels and commit by
            // atomics, so the queue's order changes nothing.
            int *fill = qn + parity;
            uint2 ln[TPT];
            unsigned masks[TPT];
            int mine = 0;
#pragma unroll
            for (int k = 0; k < TPT; ++k) {
                ln[k] = make_uint2(0u, 0u);
                if (tx[k] >= 0) {
                    int dx, dy, dz;
                    pick_offset<2, NOFF>(pick[k], dx, dy, dz);
                    const int x = tx[k] + cx, sx = x + dx;
                    const uint32_t *row = slab + (ty[k] + cy + 1) * W;
                    ln[k] = make_uint2(row[x], row[dy * W + (sx < 0 ? W - 1 : (sx >= W ? 0 : sx))]);
                }
            }
#pragma unroll
            for (int k = 0; k < TPT; ++k) {
                masks[k] = __ballot_sync(0xffffffffu, ln[k].x != ln[k].y);
                mine += __popc(masks[k]);
            }
            int slot = 0;
            if (lane == 0 && mine) slot = atomicAdd(fill, mine);
            slot = __shfl_sync(0xffffffffu, slot, 0);
#pragma unroll
            for (int k = 0; k < TPT; ++k) {
                if (masks[k] & (1u << lane))
                    queue[slot + __popc(masks[k] & ((1u << lane) - 1u))] =
                        make_uint4((uint32_t)(tx[k] + cx), (uint32_t)(ty[k] + cy) | ((uint32_t)pick[k] << 28), ln[k].x,
                                   ln[k].y);
                slot += __popc(masks[k]);
            }
            __syncthreads();
            const int total = *fill;
            if (tid == 0) qn[parity ^ 1] = 0;  // the next pass's counter; no thread reads it before the cluster barrier
            // this CTA's labels' rotation for the next pass, which no thread
            // of this one reads, from the last thread back
            for (int i = nth - 1 - tid; i < L.Lc; i += nth) {
                int dv, ds;
                unpack_delta(delta[prev * L.Lc + i], dv, ds);
                const int2 v = base[b * L.Lc + i];
                base[(b ^ 1) * L.Lc + i] = make_int2(v.x + dv, v.y + ds);
                delta[next * L.Lc + i] = 0;
            }
            for (int e = tid; e < total; e += nth) {
                const uint4 q = queue[e];
                const int x = (int)q.x, row = (int)(q.y & 0xfffffffu);
                acc.slab_row = slab + (row + 1) * W;
                acc.first = row == 0;
                acc.last = row == rows - 1;
                const SlabLabels<NOFF> labels{acc.slab_row, W, x, x == 0 ? W - 1 : x - 1, x == W - 1 ? 0 : x + 1};
                direct_copy<2, NOFF, UNIFORM>(a, T, acc, labels, key_accept, x, y0 + row, 0, (int)(q.y >> 28), q.z, q.w);
            }
            cluster_arrive();
            // the next pass's picks while the others arrive
            if (c == 3) ++step;
            const int nc = (c + 1) & 3;
            draw_picks(stream_key(r.seed, (int32_t)step, nc, 0), nc);
            cluster_wait();
            b ^= 1;
            cur = next;
            parity ^= 1;
        }
    }

    // back to global memory: this CTA's rows and labels
    for (int i = tid; i < rows * W; i += nth) a.labels[(size_t)y0 * W + i] = slab[W + i];
    for (int i = tid; i < L.Lc; i += nth) {
        const int l = i * C + rank;
        if (l >= n_labels) continue;
        for (int k = 0; k < 2; ++k) r.vs_base[k][l] = base[k * L.Lc + i];
        for (int k = 0; k < 3; ++k) r.vs_delta[k][l] = delta[k * L.Lc + i];
        for (int c = 0; c < 4; ++c) a.vol_by_colour[(size_t)l * 4 + c] = volc[i * 4 + c];
    }
}

// The widest cluster of `kernel` the device schedules with the most shared
// memory and threads, or 0.
template <class Kernel>
static int widest_cluster(Kernel kernel) {
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kClusterSmem) ||
        cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1)) {
        cudaGetLastError();
        return 0;
    }
    for (int c = kClusterMost; c >= 1; c /= 2) {
        cudaLaunchConfig_t cfg{};
        cfg.gridDim = dim3(c);
        cfg.blockDim = dim3(kClusterThreads);
        cfg.dynamicSmemBytes = kClusterSmem;
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = c;
        at[0].val.clusterDim.y = 1;
        at[0].val.clusterDim.z = 1;
        cfg.attrs = at;
        cfg.numAttrs = 1;
        int clusters = 0;
        if (cudaOccupancyMaxActiveClusters(&clusters, kernel, &cfg) == cudaSuccess && clusters >= 1) return c;
        cudaGetLastError();
    }
    return 0;
}

// Run `mcs` MCS of a small 2D lean model in one cluster; cudaErrorNotSupported
// (nothing launched) when the plane or its labels do not fit one. A plane
// takes the widest cluster (100 MCS at 128^2: 0.60 ms on 16 CTAs, 0.63 on 8,
// 0.82 on 4), a thread one target while a CTA's targets are no more than its
// threads can be.
template <int NOFF, bool UNIFORM, int TPT>
static cudaError_t launch_cluster(const ResidentLaunch &r, cudaStream_t stream) {
    const SweepLaunch &a = r.a;
    auto kernel = cluster_sweep_kernel<NOFF, UNIFORM, TPT>;
    static std::atomic<int> widest{-1};  // handles on other host threads may launch too
    int C = widest.load(std::memory_order_acquire);
    if (C < 0) {
        C = widest_cluster(kernel);
        widest.store(C, std::memory_order_release);
    }
    while (C > 1 && C > a.g.h / 2) C /= 2;  // a CTA holds two rows at least
    if (C < 1) return cudaErrorNotSupported;
    const ClusterLayout L(a.g.w, a.g.h, a.n_labels, C);
    if (L.bytes > (size_t)kClusterSmem) return cudaErrorNotSupported;
    if (L.qcap > TPT * kClusterThreads)
        return TPT < kClusterPerThread ? launch_cluster<NOFF, UNIFORM, kClusterPerThread>(r, stream)
                                       : cudaErrorNotSupported;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(C);
    cfg.blockDim = dim3(((L.qcap + TPT - 1) / TPT + 31) / 32 * 32);
    cfg.dynamicSmemBytes = L.bytes;
    cfg.stream = stream;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = C;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, r);
}

cudaError_t launch_cluster_sweep(const ResidentLaunch &r, cudaStream_t stream) {
    const SweepLaunch &a = r.a;
    if (a.g.dim != 2 || a.g.ncol != 4) return cudaErrorNotSupported;
    for (int k = 0; k < a.g.n_off; ++k)
        for (int axis = 0; axis < 3; ++axis) {
            const int want = a.g.n_off == 4 ? neighbour_offset<2, 4>(k, axis) : neighbour_offset<2, 8>(k, axis);
            if (a.g.off[k][axis] != want) return cudaErrorInvalidValue;
        }
    const bool uniform = a.uniform_type >= 0 && a.uniform_contact_exact;
    if (a.g.n_off == 4) return uniform ? launch_cluster<4, true, 1>(r, stream) : launch_cluster<4, false, 1>(r, stream);
    if (a.g.n_off == 8) return uniform ? launch_cluster<8, true, 1>(r, stream) : launch_cluster<8, false, 1>(r, stream);
    return cudaErrorNotSupported;
}

template <int DIM, int NOFF, bool UNIFORM>
static cudaError_t launch(const SweepLaunch &a, cudaStream_t stream) {
    // the compile-time neighbourhood must be the one the host built
    for (int k = 0; k < NOFF; ++k)
        for (int axis = 0; axis < 3; ++axis)
            if (a.g.off[k][axis] != neighbour_offset<DIM, NOFF>(k, axis)) return cudaErrorInvalidValue;
    CUtensorMap tmap;
    if (a.use_tma && a.tensor_map)
        tmap = *static_cast<const CUtensorMap *>(a.tensor_map);
    else
        memset(&tmap, 0, sizeof tmap);
    if (a.direct) return launch_direct<DIM, NOFF, UNIFORM>(a, stream);
    using T = Tile<DIM>;
    static std::atomic<int> grid_cap_once{0};  // handles on other host threads may launch too
    const size_t smem = sizeof(SweepSmem<DIM>) + 128;
    if (!grid_cap_once.load(std::memory_order_acquire)) {
        cudaError_t e = cudaFuncSetAttribute(sweep_kernel<DIM, NOFF, UNIFORM>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)smem);
        if (e) return e;
        int dev = 0, sms = 0, per_sm = 0;
        if ((e = cudaGetDevice(&dev))) return e;
        if ((e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev))) return e;
        if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, sweep_kernel<DIM, NOFF, UNIFORM>, kThreads, smem)))
            return e;
        grid_cap_once.store(sms * (per_sm > 0 ? per_sm : 1), std::memory_order_release);
    }
    const int tiles = ((a.g.w + T::TX - 1) / T::TX) * ((a.g.h + T::TY - 1) / T::TY) *
                      (DIM == 3 ? (a.g.d + T::TZ - 1) / T::TZ : 1);
    const int grid_cap = grid_cap_once.load(std::memory_order_acquire);
    int grid = tiles < grid_cap ? tiles : grid_cap;
    if (a.max_ctas > 0 && grid > a.max_ctas) grid = a.max_ctas;
    // Programmatic launch: the grid may start its prologue while the previous
    // kernel on the stream ends (the kernel waits before it reads pass data).
    // GLAZIER_SWEEP_PDL=0 launches it plainly.
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = programmatic_launch();
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, sweep_kernel<DIM, NOFF, UNIFORM>, a, tmap);
}

template <bool UNIFORM>
static cudaError_t launch_any(const SweepLaunch &a, cudaStream_t stream) {
    if (a.g.dim == 2) {
        if (a.g.n_off == 4) return launch<2, 4, UNIFORM>(a, stream);
        if (a.g.n_off == 8) return launch<2, 8, UNIFORM>(a, stream);
    } else {
        if (a.g.n_off == 6) return launch<3, 6, UNIFORM>(a, stream);
        if (a.g.n_off == 18) return launch<3, 18, UNIFORM>(a, stream);
        if (a.g.n_off == 26) return launch<3, 26, UNIFORM>(a, stream);
    }
    return cudaErrorInvalidValue;
}

// The pass's listed copies (target, new label, its type's maximum); the other
// pass parity's count, which the copies before these emptied, is set to zero
// for the next pass. An entry is requested beside the count, so a copy is one
// round trip and its writes.
__global__ void __launch_bounds__(256) apply_copies_kernel(const __grid_constant__ SweepLaunch a, float *activity, int most) {
    grid_wait();
    int k = blockIdx.x * blockDim.x + threadIdx.x;
    uint4 p = k < most ? a.pending[k] : make_uint4(0u, 0u, 0u, 0u);
    const int count = *a.pending_count;
    if (k == 0) *a.pending_clear = 0;
    while (k < count) {
        a.labels[p.x] = p.y;
        const float top = __uint_as_float(p.z);
        if (top > 0.0f) activity[p.x] = top;
        k += gridDim.x * blockDim.x;
        if (k < count) p = a.pending[k];
    }
}

cudaError_t launch_apply_copies(const SweepLaunch &a, float *activity, cudaStream_t stream) {
    // at most one copy per target, and a pass has sites / colours targets; an
    // accepted one is rare enough that a fraction of that grid covers them
    const int most = a.g.sites / a.g.ncol + 1;
    return launch_after(apply_copies_kernel, dim3((unsigned)((most + 2047) / 2048)), 256, stream, a, activity, most);
}

__global__ void activity_decay_kernel(float *activity, int sites) {
    grid_wait();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= sites) return;
    const float v = activity[i];
    activity[i] = v > 0.0f ? __fsub_rn(v, 1.0f) : 0.0f;
}

cudaError_t launch_activity_decay(float *activity, int sites, cudaStream_t stream) {
    return launch_after(activity_decay_kernel, dim3((unsigned)((sites + 255) / 256)), 256, stream, activity, sites);
}

cudaError_t launch_sweep(const SweepLaunch &a, cudaStream_t stream) {
    return a.uniform_type >= 0 && a.uniform_contact_exact ? launch_any<true>(a, stream) : launch_any<false>(a, stream);
}


// ---------------------------------------------------------------- the ensemble

template <int DIM>
struct EnsembleSmem {
    SweepSmem<DIM> s;
    SweepLaunch desc;  // the current replica's launch, per-pass fields patched
    int replica;       // the replica `desc` holds, -1 before the first tile
    int next_replica;
};

// The schedule position of tile t: the last prefix entry at or below it.
__device__ __forceinline__ int replica_of_tile(const int *prefix, int n, int t) {
    int lo = 0, hi = n - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (prefix[mid] <= t)
            lo = mid;
        else
            hi = mid - 1;
    }
    return lo;
}

template <int DIM, int NOFF, bool UNIFORM>
__global__ void __launch_bounds__(kThreads, GLZ_SWEEP_MIN_BLOCKS)
    ensemble_sweep_kernel(const __grid_constant__ EnsembleLaunch e) {
    using T = Tile<DIM>;
    using Smem = SweepSmem<DIM>;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    const uint32_t raw = smem_addr(smem_raw);
    EnsembleSmem<DIM> &E = *reinterpret_cast<EnsembleSmem<DIM> *>(smem_raw + ((128u - (raw & 127u)) & 127u));
    Smem &S = E.s;
    const int tid = threadIdx.x;
    if (smem_addr(S.win[0]) & 127u) {
        if (tid == 0) atomicExch(e.error_flag, 3);
        return;
    }
    const long long step = e.clock->step;
    const long long pass = e.clock->pass + e.colour;

    // Tally rotation for the next pass over every replica's cells at once.
    {
        const size_t stride = (size_t)gridDim.x * blockDim.x;
        int2 *const base = e.vs_base[pass % 2];
        const long long *const prev = e.vs_delta[(pass + 2) % 3];
        int2 *const next_base = e.vs_base[(pass + 1) % 2];
        long long *const clear = e.vs_delta[(pass + 1) % 3];
        for (size_t l = (size_t)blockIdx.x * blockDim.x + tid; l < (size_t)e.total_cells; l += stride) {
            int dv, ds;
            unpack_delta(prev[l], dv, ds);
            const int2 b = base[l];
            next_base[l] = make_int2(b.x + dv, b.y + ds);
            clear[l] = 0;
        }
    }
    if (tid < NOFF) S.woff[tid] = window_offset<DIM, NOFF>(tid);
    if (tid == 0) {
        S.queued = 0;
        S.taken = 0;
        E.replica = -1;
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(&S.mbar[0])));
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(&S.mbar[1])));
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();

    const CUtensorMap *maps = static_cast<const CUtensorMap *>(e.maps);
    int waited[2] = {0, 0};
    bool pending[2] = {false, false};
    // The position, origin and tensor-copy eligibility of global tile t.
    auto locate = [&](int t, int &pos, int &x0, int &y0, int &z0) -> bool {
        pos = replica_of_tile(e.tile_prefix, e.n, t);
        const SweepLaunch &ra = e.replicas[e.order[pos]].a;
        tile_origin<DIM>(t - e.tile_prefix[pos], ra.g.w, ra.g.h, x0, y0, z0);
        return maps != nullptr && tile_interior<DIM>(ra, x0, y0, z0);
    };
    // Each CTA takes a contiguous run of the schedule's tiles (runs differ by
    // at most one tile), so consecutive tiles mostly share a replica and its
    // launch stays in shared memory.
    const int per = e.total_tiles / (int)gridDim.x, extra = e.total_tiles % (int)gridDim.x;
    const int first = (int)blockIdx.x * per + ((int)blockIdx.x < extra ? (int)blockIdx.x : extra);
    const int last = first + per + ((int)blockIdx.x < extra ? 1 : 0);
    int t = first;
    if (t < last) {
        int pos, x0, y0, z0;
        if (locate(t, pos, x0, y0, z0)) {
            if (tid == 0) issue_window<DIM>(maps[e.order[pos]], S.win[0], &S.mbar[0], x0, y0, z0);
            pending[0] = true;
        }
    }
    for (int it = 0; t < last; ++t, ++it) {
        const int buf = it & 1;
        int pos, x0, y0, z0;
        const bool interior = locate(t, pos, x0, y0, z0);
        const int r = e.order[pos];
        const int next = t + 1;
        if (next < last) {
            int npos, nx0, ny0, nz0;
            if (locate(next, npos, nx0, ny0, nz0)) {
                if (tid == 0) issue_window<DIM>(maps[e.order[npos]], S.win[buf ^ 1], &S.mbar[buf ^ 1], nx0, ny0, nz0);
                pending[buf ^ 1] = true;
            }
        }
        if (r != E.replica) {
            // Bring this replica's launch into shared memory and patch the
            // per-pass fields: keys, tally rotation, colour, step.
            __syncthreads();
            const EnsembleReplica &rep = e.replicas[r];
            const int *src = reinterpret_cast<const int *>(&rep.a);
            int *dst = reinterpret_cast<int *>(&E.desc);
            for (int i = tid; i < (int)(sizeof(SweepLaunch) / sizeof(int)); i += blockDim.x) dst[i] = src[i];
            __syncthreads();
            if (tid == 0) {
                SweepLaunch &d = E.desc;
                d.colour = e.colour;
                d.step = (int32_t)step;
                d.key_pick = stream_key(rep.seed, d.step, e.colour, 0);
                d.key_accept = stream_key(rep.seed, d.step, e.colour, 1);
                d.vs_base = e.vs_base[pass % 2] + rep.cell_off;
                d.vs_prev = e.vs_delta[(pass + 2) % 3] + rep.cell_off;
                d.vs_cur = reinterpret_cast<unsigned long long *>(e.vs_delta[pass % 3] + rep.cell_off);
                E.replica = r;
            }
            const bool small = rep.a.n_types <= kSmemTypes;
            if (small)
                for (int i = tid; i < rep.a.n_types * rep.a.n_types; i += blockDim.x) S.contact[i] = rep.a.t.contact[i];
            __syncthreads();
        }
        const SweepLaunch &a = E.desc;
        uint32_t *win = S.win[buf];
        if (interior) {
            const uint32_t done = wait_parity(&S.mbar[buf], waited[buf] & 1);
            waited[buf] += 1;
            pending[buf] = false;
            if (!__syncthreads_and(done)) {
                if (pending[buf ^ 1]) wait_parity(&S.mbar[buf ^ 1], waited[buf ^ 1] & 1);
                if (tid == 0) atomicExch(e.error_flag, 1);
                return;
            }
        } else {
            load_window_plain<DIM>(a, win, x0, y0, z0);
        }
        price_tile<DIM, NOFF, UNIFORM>(a, S, win, x0, y0, z0, a.n_types <= kSmemTypes);
    }
}

// ---------------------------------------------------------------- the lean ensemble
//
// The layout above over an ensemble: warp-owned target shares, the
// window ring refilled by the last warp out, queue entries carried into the
// warp's next tile. Warps may be on different tiles, so each ring slot holds
// its own copy of the tile's replica launch, with the pass's fields patched
// in; the warp that refills a slot copies the next tile's launch in first.
// Each CTA takes a contiguous run of the schedule's tiles.
template <int DIM>
struct LeanEnsembleSmem {
    LeanSmem<DIM> s;
    SweepLaunch desc[kLeanStages];  // the slot's tile's replica launch
    int org[kLeanStages][4];        // the slot's tile: origin x, y, z, replica
};

// The schedule's tile t: its replica's launch (pass fields patched) and
// origin into slot `slot`, by the whole warp; lane 0 then starts its window
// (a tensor copy, or a bare arrival when the replica's window takes plain
// loads).
template <int DIM>
__device__ __forceinline__ void lean_ens_fill(const EnsembleLaunch &e, LeanEnsembleSmem<DIM> &E, int t, int slot,
                                              long long step, long long pass) {
    using T = Tile<DIM>;
    const int lane = threadIdx.x & 31;
    const int pos = replica_of_tile(e.tile_prefix, e.n, t);
    const int r = e.order[pos];
    const EnsembleReplica &rep = e.replicas[r];
    const int *src = reinterpret_cast<const int *>(&rep.a);
    int *dst = reinterpret_cast<int *>(&E.desc[slot]);
    for (int i = lane; i < (int)(sizeof(SweepLaunch) / sizeof(int)); i += 32) dst[i] = src[i];
    __syncwarp();
    if (lane == 0) {
        SweepLaunch &d = E.desc[slot];
        d.colour = e.colour;
        d.step = (int32_t)step;
        d.key_pick = stream_key(rep.seed, d.step, e.colour, 0);
        d.key_accept = stream_key(rep.seed, d.step, e.colour, 1);
        d.vs_base = e.vs_base[pass % 2] + rep.cell_off;
        d.vs_prev = e.vs_delta[(pass + 2) % 3] + rep.cell_off;
        d.vs_cur = reinterpret_cast<unsigned long long *>(e.vs_delta[pass % 3] + rep.cell_off);
        int x0, y0, z0;
        tile_origin<DIM>(t - e.tile_prefix[pos], d.g.w, d.g.h, x0, y0, z0);
        E.org[slot][0] = x0;
        E.org[slot][1] = y0;
        E.org[slot][2] = z0;
        E.org[slot][3] = r;
        E.s.issued[slot] += 1;
        const CUtensorMap *maps = static_cast<const CUtensorMap *>(e.maps);
        if (maps && lean_copies<DIM>(d))
            issue_window<DIM>(maps[r], E.s.win[slot], &E.s.full[slot], x0, y0, z0);
        else
            asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_addr(&E.s.full[slot])) : "memory");
    }
}

template <int DIM, int NOFF, bool UNIFORM>
__global__ void __launch_bounds__(kLeanThreads, GLZ_LEAN_MIN_BLOCKS)
    lean_ensemble_kernel(const __grid_constant__ EnsembleLaunch e) {
    using T = Tile<DIM>;
    using Smem = LeanSmem<DIM>;
    constexpr int PER_LANE = Smem::TPW / 32;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    const uint32_t raw = smem_addr(smem_raw);
    LeanEnsembleSmem<DIM> &E = *reinterpret_cast<LeanEnsembleSmem<DIM> *>(smem_raw + ((128u - (raw & 127u)) & 127u));
    Smem &S = E.s;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (smem_addr(S.win[0]) & 127u) {
        if (tid == 0) atomicExch(e.error_flag, 3);
        return;
    }
    const long long step = e.clock->step;
    const long long pass = e.clock->pass + e.colour;
    const int per = e.total_tiles / (int)gridDim.x, extra = e.total_tiles % (int)gridDim.x;
    const int first = (int)blockIdx.x * per + ((int)blockIdx.x < extra ? (int)blockIdx.x : extra);
    const int mine = per + ((int)blockIdx.x < extra ? 1 : 0);

    if (tid == 0) {
        for (int k = 0; k < kLeanStages; ++k) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(&S.full[k])));
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(&S.patched[k])), "r"(kLeanWarps));
            S.done[k] = 0;
            S.issued[k] = 0;
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
#pragma unroll
    for (int k = 0; k < NOFF; ++k)
        if (tid == k) S.woff[k] = window_offset<DIM, NOFF>(k);
    __syncthreads();
    if (warp == 0)
        for (int i = 0; i < kLeanStages && i < mine; ++i) lean_ens_fill<DIM>(e, E, first + i, i, step, pass);
    // the tally rotation over every replica's cells, its reads copied in ahead
    const size_t rot_stride = (size_t)gridDim.x * blockDim.x;
    const size_t rot_first = (size_t)blockIdx.x * blockDim.x + tid;
    const int2 *rot_base = e.vs_base[pass % 2];
    const long long *rot_prev = e.vs_delta[(pass + 2) % 3];
#pragma unroll
    for (int k = 0; k < kRotate; ++k) {
        const size_t l = rot_first + k * rot_stride;
        if (l < (size_t)e.total_cells) {
            asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(smem_addr(&S.rot_base[k * kLeanThreads + tid])),
                         "l"(rot_base + l)
                         : "memory");
            asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(smem_addr(&S.rot_prev[k * kLeanThreads + tid])),
                         "l"(rot_prev + l)
                         : "memory");
        }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");

    uint32_t *queue = S.queue[warp];
    const unsigned below = (1u << lane) - 1u;
    uint32_t patch_parity = 0;
    int held = 0, held_slot = -1;

    for (int i = 0; i < mine; ++i) {
        const int slot = i % kLeanStages;
        uint32_t *win = S.win[slot];
        bool ok = wait_parity(&S.full[slot], (uint32_t)(i / kLeanStages) & 1u) != 0;
        const SweepLaunch &a = E.desc[slot];
        const int x0 = E.org[slot][0], y0 = E.org[slot][1], z0 = E.org[slot][2];
        const int W = a.g.w, H = a.g.h, D = a.g.d;
        const bool copies = e.maps != nullptr && lean_copies<DIM>(a);
        const bool edge = !copies || !(x0 >= T::HX && x0 + T::TX + T::HX <= W && y0 >= 1 && y0 + T::TY + 1 <= H &&
                                       (DIM == 2 || (z0 >= 1 && z0 + T::TZ + 1 <= D)));
        if (edge && __all_sync(0xffffffffu, ok)) {
            lean_patch<DIM>(a, win, x0, y0, z0, copies);
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0)
                asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_addr(&S.patched[slot])) : "memory");
            ok = wait_parity(&S.patched[slot], (patch_parity >> slot) & 1u) != 0;
            patch_parity ^= 1u << slot;
        }
        if (!__all_sync(0xffffffffu, ok)) {
            if (lane == 0) {
                atomicExch(e.error_flag, 1);
                for (int k = 0; k < kLeanStages; ++k)
                    if (S.issued[k] > 0) wait_parity(&S.full[k], (uint32_t)(S.issued[k] - 1) & 1u);
            }
            asm volatile("cp.async.wait_all;" ::: "memory");
            return;
        }

        // light pass over this warp's share, behind the entries held over
        const bool full = x0 + T::TX <= W && y0 + T::TY <= H && (DIM == 2 || z0 + T::TZ <= D);
        const uint32_t tile_base = (uint32_t)((z0 * H + y0) * W + x0);
        uint32_t entries[PER_LANE];
        unsigned masks[PER_LANE];
#pragma unroll
        for (int k = 0; k < PER_LANE; ++k) {
            const int j = warp * Smem::TPW + k * 32 + lane;
            int lx, ly, lz;
            target_of<DIM>(j, e.colour, lx, ly, lz);
            const bool in = full || (x0 + lx < W && y0 + ly < H && (DIM == 2 || z0 + lz < D));
            bool active = false;
            int pick = 0;
            if (in) {
                const int wc = ((lz + T::HZ) * T::PY + (ly + 1)) * T::PX + (lx + T::HX);
                pick = pick_of<NOFF>(draw(a.key_pick, tile_base + (uint32_t)((lz * H + ly) * W + lx)));
                active = win[wc] != win[wc + S.woff[pick]];
            }
            entries[k] = (uint32_t)j | ((uint32_t)pick << 16);
            masks[k] = __ballot_sync(0xffffffffu, active);
        }
        int total = held;
#pragma unroll
        for (int k = 0; k < PER_LANE; ++k) {
            if (masks[k] & (1u << lane)) queue[total + __popc(masks[k] & below)] = entries[k];
            total += __popc(masks[k]);
        }
        __syncwarp();
        int taken = 0;
        for (;;) {
            const int n = total - taken;
            if (n < 32 && taken >= held) break;
            const int q = taken + lane;
            if (q < total) {
                const int s_ = q < held ? held_slot : slot;
                price_and_commit<DIM, NOFF, UNIFORM, false>(E.desc[s_], S.woff, nullptr, nullptr, S.win[s_], queue[q],
                                                            E.org[s_][0], E.org[s_][1], E.org[s_][2], false);
            }
            taken += n < 32 ? n : 32;
        }
        __syncwarp();
        if (held_slot >= 0) {
            // release the previous tile's slot; the last warp out refills it
            int last_out = 0;
            if (lane == 0) {
                __threadfence_block();
                last_out = atomicAdd(&S.done[held_slot], 1) == kLeanWarps - 1;
                if (last_out) S.done[held_slot] = 0;
            }
            last_out = __shfl_sync(0xffffffffu, last_out, 0);
            if (last_out && i - 1 + kLeanStages < mine) {
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                lean_ens_fill<DIM>(e, E, first + i - 1 + kLeanStages, held_slot, step, pass);
            }
        }
        const int keep = total - taken;
        if (taken > 0 && keep > 0) {
            const uint32_t v = lane < keep ? queue[taken + lane] : 0u;
            __syncwarp();
            if (lane < keep) queue[lane] = v;
            __syncwarp();
        }
        held = keep;
        held_slot = slot;
    }
    if (mine > 0) {
        if (lane < held)
            price_and_commit<DIM, NOFF, UNIFORM, false>(E.desc[held_slot], S.woff, nullptr, nullptr, S.win[held_slot],
                                                        queue[lane], E.org[held_slot][0], E.org[held_slot][1],
                                                        E.org[held_slot][2], false);
        __syncwarp();
        if (lane == 0) {
            __threadfence_block();
            atomicAdd(&S.done[held_slot], 1);
        }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    int2 *next_base = e.vs_base[(pass + 1) % 2];
    long long *clear = e.vs_delta[(pass + 1) % 3];
#pragma unroll
    for (int k = 0; k < kRotate; ++k) {
        const size_t l = rot_first + k * rot_stride;
        if (l < (size_t)e.total_cells) {
            int dv, ds;
            unpack_delta(S.rot_prev[k * kLeanThreads + tid], dv, ds);
            const int2 b = S.rot_base[k * kLeanThreads + tid];
            next_base[l] = make_int2(b.x + dv, b.y + ds);
            clear[l] = 0;
        }
    }
    for (size_t l = rot_first + kRotate * rot_stride; l < (size_t)e.total_cells; l += rot_stride) {
        int dv, ds;
        unpack_delta(rot_prev[l], dv, ds);
        const int2 b = rot_base[l];
        next_base[l] = make_int2(b.x + dv, b.y + ds);
        clear[l] = 0;
    }
}

// ---------------------------------------------------------------- the direct ensemble
//
// Tile t of colour pass `colour` (pass number `pass`, step `step`): the
// block finds the tile's replica, patches the replica's launch into `d` and
// prices the tile's targets.
template <int NOFF, bool UNIFORM, int BX, int BY>
__device__ __forceinline__ void direct_ensemble_tile(const EnsembleLaunch &e, SweepLaunch &d, int *where, int t,
                                                     int colour, long long step, long long pass) {
    if (threadIdx.x == 0) {
        const int pos = replica_of_tile(e.tile_prefix, e.n, t);
        where[0] = pos;
        where[1] = e.order[pos];
    }
    __syncthreads();
    const int pos = where[0];
    const EnsembleReplica &rep = e.replicas[where[1]];
    {
        const int *src = reinterpret_cast<const int *>(&rep.a);
        int *dst = reinterpret_cast<int *>(&d);
        for (int i = threadIdx.x; i < (int)(sizeof(SweepLaunch) / sizeof(int)); i += blockDim.x) dst[i] = src[i];
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        d.colour = colour;
        d.step = (int32_t)step;
        d.key_pick = stream_key(rep.seed, d.step, colour, 0);
        d.key_accept = stream_key(rep.seed, d.step, colour, 1);
        d.vs_base = e.vs_base[pass % 2] + rep.cell_off;
        d.vs_prev = e.vs_delta[(pass + 2) % 3] + rep.cell_off;
        d.vs_cur = reinterpret_cast<unsigned long long *>(e.vs_delta[pass % 3] + rep.cell_off);
    }
    __syncthreads();
    const int lt = t - e.tile_prefix[pos];
    const int hw = d.g.w / 2, hh = d.g.h / 2;
    const int tiles_x = (hw + BX - 1) / BX;
    const int jx = (lt % tiles_x) * BX + (int)threadIdx.x % BX;
    const int jy = (lt / tiles_x) * BY + (int)threadIdx.x / BX;
    if (jx < hw && jy < hh) {
        const PassView v{colour, d.key_pick, d.key_accept, d.vs_base, d.vs_prev, d.vs_cur};
        direct_target<2, NOFF, UNIFORM, GlobalPass, false>(d, d.t, GlobalPass{d, v}, v.key_pick, v.key_accept,
                                                           2 * jx + (colour & 1), 2 * jy + ((colour >> 1) & 1), 0);
    }
    __syncthreads();  // `d` and `where` serve the block's next tile
}

// The tally rotation over every replica's cells for the pass numbered `pass`,
// which no thread of that pass reads, spread over the grid.
__device__ __forceinline__ void ensemble_rotate(const EnsembleLaunch &e, long long pass) {
    int2 *next_base = e.vs_base[(pass + 1) % 2];
    long long *clear = e.vs_delta[(pass + 1) % 3];
    const int2 *base = e.vs_base[pass % 2];
    const long long *prev = e.vs_delta[(pass + 2) % 3];
    const size_t stride = (size_t)gridDim.x * blockDim.x;
    for (size_t l = (size_t)blockIdx.x * blockDim.x + threadIdx.x; l < (size_t)e.total_cells; l += stride) {
        int dv, ds;
        unpack_delta(prev[l], dv, ds);
        const int2 b = base[l];
        next_base[l] = make_int2(b.x + dv, b.y + ds);
        clear[l] = 0;
    }
}

// A plane ensemble's pass with one block per tile of BX x BY targets of one
// replica, priced where they lie (direct_target, as the direct kernel does).
// The tile shape sets which sites a block's loads share; the autotuner picks
// it by time, since the results do not depend on it.
template <int NOFF, bool UNIFORM, int BX, int BY>
__global__ void __launch_bounds__(BX *BY) direct_ensemble_kernel(const __grid_constant__ EnsembleLaunch e) {
    __shared__ SweepLaunch d;
    __shared__ int where[2];  // the tile's place in the schedule, its replica
    const long long step = e.clock->step;
    const long long pass = e.clock->pass + e.colour;
    direct_ensemble_tile<NOFF, UNIFORM, BX, BY>(e, d, where, (int)blockIdx.x, e.colour, step, pass);
    ensemble_rotate(e, pass);
}

// Every colour pass of a step in one cooperative launch: blocks stride over
// the tiles, a grid barrier between passes (the tallies a pass reads are its
// snapshot, complete once every block has finished the pass before).
template <int NOFF, bool UNIFORM, int BX, int BY>
__global__ void __launch_bounds__(BX *BY) direct_ensemble_step_kernel(const __grid_constant__ EnsembleLaunch e) {
    __shared__ SweepLaunch d;
    __shared__ int where[2];
    const long long step = e.clock->step;
    for (int c = 0; c < e.ncol; ++c) {
        const long long pass = e.clock->pass + c;
        for (int t = (int)blockIdx.x; t < e.total_tiles; t += (int)gridDim.x)
            direct_ensemble_tile<NOFF, UNIFORM, BX, BY>(e, d, where, t, c, step, pass);
        ensemble_rotate(e, pass);
        if (c + 1 < e.ncol && !grid_barrier(e.barrier, (unsigned)c)) {
            if (threadIdx.x == 0) atomicExch(e.error_flag, 4);
            return;
        }
    }
}

template <int NOFF, bool UNIFORM, int BX, int BY>
static cudaError_t direct_ensemble_shape(const EnsembleLaunch &e, cudaStream_t stream) {
    if (!e.one_launch) {
        direct_ensemble_kernel<NOFF, UNIFORM, BX, BY><<<e.total_tiles, BX * BY, 0, stream>>>(e);
        return cudaGetLastError();
    }
    static std::atomic<int> most_once{0};  // blocks that can all be resident at once
    if (!most_once.load(std::memory_order_acquire)) {
        int dev = 0, sms = 0, per_sm = 0;
        if (cudaError_t x = cudaGetDevice(&dev)) return x;
        if (cudaError_t x = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) return x;
        if (cudaError_t x = cudaOccupancyMaxActiveBlocksPerMultiprocessor(
                &per_sm, direct_ensemble_step_kernel<NOFF, UNIFORM, BX, BY>, BX * BY, 0))
            return x;
        most_once.store(sms * per_sm, std::memory_order_release);
    }
    const int most = most_once.load(std::memory_order_acquire);
    if (most < 1) return cudaErrorCooperativeLaunchTooLarge;
    const int grid = e.total_tiles < most ? e.total_tiles : most;
    if (cudaError_t x = cudaMemsetAsync(e.barrier, 0, 2 * sizeof(unsigned), stream)) return x;
    void *args[] = {const_cast<EnsembleLaunch *>(&e)};
    return cudaLaunchCooperativeKernel((const void *)direct_ensemble_step_kernel<NOFF, UNIFORM, BX, BY>, dim3(grid),
                                       dim3(BX * BY), args, 0, stream);
}

// ---------------------------------------------------------------- runs of the ensemble
//
// One block per run of kEnsembleRun consecutive targets of a replica: the
// direct sweep's warp-queued pass over every replica's runs at once. The
// block copies its replica's launch into shared memory and draws its picks
// before the programmatic wait (nothing of the step writes a launch or the
// clock); every warp draws and compares its 128 targets, queues the unlike
// ones with their labels and prices the queue. A replica's last run is all it
// can waste, where the windowed kernel's tiles lose a quarter of their sites
// on replicas of uneven sides, and each of its tiles waits for its launch to
// be found and copied (64 monolayers of 128 to 1024 a side, 12.7 M sites: 254
// us per MCS windowed, 278 in blocks of 32 x 8 targets priced where they lie).
constexpr int kRunEach = kEnsembleRun / 256;  // targets a lane

template <int DIM, int NOFF, bool UNIFORM>
__global__ void __launch_bounds__(256, 4) run_ensemble_kernel(const __grid_constant__ EnsembleLaunch e) {
    __shared__ SweepLaunch d;
    __shared__ TypeSmem<false> types;
    __shared__ uint2 pair[8][32 * kRunEach];  // (old, new) labels of each queued copy
    __shared__ int queue[8][32 * kRunEach];
    __shared__ uint8_t picks[8][32 * kRunEach];
    const int tid = (int)threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const unsigned below = (1u << lane) - 1u;
    const int2 run = e.runs[blockIdx.x];
    const EnsembleReplica &rep = e.replicas[run.x];
    const EnsembleClock clock = *e.clock;
    {
        const int *src = reinterpret_cast<const int *>(&rep.a);
        int *dst = reinterpret_cast<int *>(&d);
        for (int i = tid; i < (int)(sizeof(SweepLaunch) / sizeof(int)); i += 256) dst[i] = src[i];
    }
    const unsigned long long pass = (unsigned long long)(clock.pass + e.colour);
    const int32_t step = (int32_t)clock.step;
    const int b = (int)(pass % 2), cur = (int)(pass % 3), next = cur == 2 ? 0 : cur + 1, prev = cur == 0 ? 2 : cur - 1;
    const PassView v{e.colour,
                     stream_key(rep.seed, step, e.colour, 0),
                     stream_key(rep.seed, step, e.colour, 1),
                     e.vs_base[b] + rep.cell_off,
                     e.vs_delta[prev] + rep.cell_off,
                     reinterpret_cast<unsigned long long *>(e.vs_delta[cur] + rep.cell_off)};
    __syncthreads();
    const TypeTables T = UNIFORM ? d.t : load_types<false>(d, types);
    const GlobalPass acc{d, v};
    const int targets = (d.g.w / 2) * (d.g.h / 2) * (DIM == 3 ? d.g.d / 2 : 1);
    const int first = run.y + warp * 32 * kRunEach;
    int pick[kRunEach];
#pragma unroll
    for (int k = 0; k < kRunEach; ++k) {
        const int j = first + k * 32 + lane;
        pick[k] = 0;
        if (j < targets) {
            int x, y, z;
            direct_site<DIM>(d, e.colour, j, x, y, z);
            pick[k] = pick_of<NOFF>(draw(v.key_pick, (uint32_t)((z * d.g.h + y) * d.g.w + x)));
        }
    }
    grid_wait();
    if (!UNIFORM) __syncthreads();  // the tables are in place
    uint2 labels[kRunEach];
#pragma unroll
    for (int k = 0; k < kRunEach; ++k) {
        const int j = first + k * 32 + lane;
        labels[k] = make_uint2(0u, 0u);
        if (j < targets) {
            int x, y, z;
            direct_site<DIM>(d, e.colour, j, x, y, z);
            labels[k] = make_uint2(acc.label(x, y, z), picked_label<DIM, NOFF>(d, acc, x, y, z, pick[k]));
        }
    }
    int total = 0;
#pragma unroll
    for (int k = 0; k < kRunEach; ++k) {
        const bool unlike = labels[k].x != labels[k].y;
        const unsigned m = __ballot_sync(0xffffffffu, unlike);
        if (unlike) {
            const int at = total + __popc(m & below);
            queue[warp][at] = first + k * 32 + lane;
            picks[warp][at] = (uint8_t)pick[k];
            pair[warp][at] = labels[k];
        }
        total += __popc(m);
    }
    __syncwarp();
    for (int q = lane; q < total; q += 32) {
        int x, y, z;
        direct_site<DIM>(d, e.colour, queue[warp][q], x, y, z);
        const NeighbourReads<DIM, NOFF, GlobalPass> ln(d, acc, x, y, z);
        direct_copy<DIM, NOFF, UNIFORM>(d, T, acc, ln, v.key_accept, x, y, z, picks[warp][q], pair[warp][q].x,
                                        pair[warp][q].y);
    }
    // this block's share of the tally rotation over every replica's cells,
    // which no thread of this pass reads
    const int2 *base = e.vs_base[b];
    int2 *next_base = e.vs_base[b ^ 1];
    const long long *last_delta = e.vs_delta[prev];
    long long *clear = e.vs_delta[next];
    const long long share = (e.total_cells + gridDim.x - 1) / gridDim.x;
    const long long from = share * blockIdx.x, to = from + share < e.total_cells ? from + share : e.total_cells;
    for (long long l = from + tid; l < to; l += 256) {
        int dv, ds;
        unpack_delta(last_delta[l], dv, ds);
        const int2 t = base[l];
        next_base[l] = make_int2(t.x + dv, t.y + ds);
        clear[l] = 0;
    }
}

template <int NOFF, bool UNIFORM>
static cudaError_t direct_ensemble_launch(const EnsembleLaunch &e, cudaStream_t stream) {
    if (e.total_tiles <= 0) return cudaSuccess;
    if (e.tile_shape == 1) return direct_ensemble_shape<NOFF, UNIFORM, 32, 8>(e, stream);
    if (e.tile_shape == 2) return direct_ensemble_shape<NOFF, UNIFORM, 16, 16>(e, stream);
    return direct_ensemble_shape<NOFF, UNIFORM, 64, 4>(e, stream);
}

__global__ void clock_advance_kernel(EnsembleClock *clock, int ncol) {
    clock->step += 1;
    clock->pass += ncol;
}

template <int DIM, int NOFF, bool UNIFORM>
static int ensemble_cap() {
    static std::atomic<int> cap{0};  // handles on other host threads may launch too
    if (!cap.load(std::memory_order_acquire)) {
        const size_t smem = sizeof(EnsembleSmem<DIM>) + 128;
        if (cudaFuncSetAttribute(ensemble_sweep_kernel<DIM, NOFF, UNIFORM>,
                                 cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem))
            return 0;
        int dev = 0, sms = 0, per_sm = 0;
        if (cudaGetDevice(&dev) || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) return 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, ensemble_sweep_kernel<DIM, NOFF, UNIFORM>, kThreads,
                                                          smem))
            return 0;
        cap.store(sms * (per_sm > 0 ? per_sm : 1), std::memory_order_release);
    }
    return cap.load(std::memory_order_acquire);
}

// Whether ensembles take the lean kernel (GLAZIER_ENSEMBLE_LEAN=0: the
// barrier-per-tile one).
static bool lean_ensemble() {
    static const bool on = [] {
        const char *env = std::getenv("GLAZIER_ENSEMBLE_LEAN");
        return !(env && env[0] == '0');
    }();
    return on;
}

template <int DIM, int NOFF, bool UNIFORM>
static int lean_ensemble_cap() {
    static std::atomic<int> cap{0};  // handles on other host threads may launch too
    if (!cap.load(std::memory_order_acquire)) {
        const size_t smem = sizeof(LeanEnsembleSmem<DIM>) + 128;
        if (cudaFuncSetAttribute(lean_ensemble_kernel<DIM, NOFF, UNIFORM>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)smem))
            return 0;
        int dev = 0, sms = 0, per_sm = 0;
        if (cudaGetDevice(&dev) || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) return 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, lean_ensemble_kernel<DIM, NOFF, UNIFORM>,
                                                          kLeanThreads, smem))
            return 0;
        cap.store(sms * (per_sm > 0 ? per_sm : 1), std::memory_order_release);
    }
    return cap.load(std::memory_order_acquire);
}

template <int DIM, int NOFF, bool UNIFORM>
static cudaError_t ensemble_launch(const EnsembleLaunch &e, cudaStream_t stream) {
    if (e.tile_shape == kEnsembleRuns)
        return launch_after(run_ensemble_kernel<DIM, NOFF, UNIFORM>, dim3((unsigned)e.total_tiles), 256, stream, e);
    if (lean_ensemble()) {
        const int cap = lean_ensemble_cap<DIM, NOFF, UNIFORM>();
        if (!cap) return cudaErrorInvalidConfiguration;
        int grid = e.total_tiles < cap ? e.total_tiles : cap;
        if (e.max_ctas > 0 && grid > e.max_ctas) grid = e.max_ctas;
        const size_t smem = sizeof(LeanEnsembleSmem<DIM>) + 128;
        lean_ensemble_kernel<DIM, NOFF, UNIFORM><<<grid, kLeanThreads, smem, stream>>>(e);
        return cudaGetLastError();
    }
    const int cap = ensemble_cap<DIM, NOFF, UNIFORM>();
    if (!cap) return cudaErrorInvalidConfiguration;
    int grid = e.total_tiles < cap ? e.total_tiles : cap;
    if (e.max_ctas > 0 && grid > e.max_ctas) grid = e.max_ctas;
    const size_t smem = sizeof(EnsembleSmem<DIM>) + 128;
    ensemble_sweep_kernel<DIM, NOFF, UNIFORM><<<grid, kThreads, smem, stream>>>(e);
    return cudaGetLastError();
}

template <bool UNIFORM>
static cudaError_t ensemble_any(const EnsembleLaunch &e, int dim, int n_off, cudaStream_t stream) {
    if (e.tile_shape > 0 && e.tile_shape != kEnsembleRuns) {
        if (dim != 2 || e.tile_shape > 3) return cudaErrorInvalidValue;
        return n_off == 4 ? direct_ensemble_launch<4, UNIFORM>(e, stream) : direct_ensemble_launch<8, UNIFORM>(e, stream);
    }
    if (dim == 2) {
        if (n_off == 4) return ensemble_launch<2, 4, UNIFORM>(e, stream);
        if (n_off == 8) return ensemble_launch<2, 8, UNIFORM>(e, stream);
    } else {
        if (n_off == 6) return ensemble_launch<3, 6, UNIFORM>(e, stream);
        if (n_off == 18) return ensemble_launch<3, 18, UNIFORM>(e, stream);
        if (n_off == 26) return ensemble_launch<3, 26, UNIFORM>(e, stream);
    }
    return cudaErrorInvalidValue;
}

cudaError_t launch_ensemble_sweep(const EnsembleLaunch &e, int dim, int n_off, bool uniform, cudaStream_t stream) {
    return uniform ? ensemble_any<true>(e, dim, n_off, stream) : ensemble_any<false>(e, dim, n_off, stream);
}

cudaError_t launch_clock_advance(EnsembleClock *clock, int ncol, cudaStream_t stream) {
    clock_advance_kernel<<<1, 1, 0, stream>>>(clock, ncol);
    return cudaGetLastError();
}

template <int DIM, int NOFF, bool UNIFORM>
static int grid_cap_of() {
    return lean_ensemble() ? lean_ensemble_cap<DIM, NOFF, UNIFORM>() : ensemble_cap<DIM, NOFF, UNIFORM>();
}

template <bool UNIFORM>
static int cap_any(int dim, int n_off) {
    if (dim == 2) return n_off == 4 ? grid_cap_of<2, 4, UNIFORM>() : grid_cap_of<2, 8, UNIFORM>();
    if (n_off == 6) return grid_cap_of<3, 6, UNIFORM>();
    if (n_off == 18) return grid_cap_of<3, 18, UNIFORM>();
    return grid_cap_of<3, 26, UNIFORM>();
}

int ensemble_grid_cap(int dim, int n_off, bool uniform) { return uniform ? cap_any<true>(dim, n_off) : cap_any<false>(dim, n_off); }

// The box a sweep tile's tensor copy moves: the tile plus its halo.
int sweep_box(int dim, uint32_t box[3]) {
    if (dim == 2) {
        box[0] = Tile<2>::PX;
        box[1] = Tile<2>::PY;
        box[2] = 1;
    } else {
        box[0] = Tile<3>::PX;
        box[1] = Tile<3>::PY;
        box[2] = Tile<3>::PZ;
    }
    return 0;
}

}  // namespace glz
