// Per-cell tallies from the lattice: the recount, the settle that folds the
// pending deltas into the base, and the medium's own counts.
//
// The recount replaces `recount` (glazier-cuda/src/lib.rs:144-172) and the
// host-side `assemble` (glazier-core/src/cpu.rs:178-217) that seeds every
// counter before a run. Besides volume and surface it counts each cell's
// sites per checkerboard colour (the sweep's guard reads these), fixes each
// cell's anchor at its first site in scan order (the frame moments.rs
// unwraps a cell in), and accumulates the exact int64 moment sums about it.

#include <climits>

#include "device.cuh"
#include "engine.h"
#include "neighbours.cuh"
#include "pdl.cuh"
#include "tally.cuh"

namespace glz {

// A lattice holds fewer than 2^31 sites, so 32-bit division suffices.
__device__ __forceinline__ void coords_of(const Geometry &g, size_t i, int &x, int &y, int &z) {
    const uint32_t s = (uint32_t)i;
    const uint32_t row = udiv(g.div_w, s);
    const uint32_t plane = udiv(g.div_h, row);
    x = (int)(s - row * (uint32_t)g.w);
    y = (int)(row - plane * (uint32_t)g.h);
    z = (int)plane;
}

// The label count a recount covers: the live count in device memory for a
// population model, else the launch's.
__device__ __forceinline__ int recount_labels(const RecountLaunch &a) { return a.n_live ? *a.n_live : a.n_labels; }

__global__ void __launch_bounds__(256) clear_tallies_kernel(const __grid_constant__ RecountLaunch a) {
    const int l = blockIdx.x * blockDim.x + threadIdx.x;
    if (l >= recount_labels(a)) return;
    clear_tallies(a, l);
    a.first[l] = INT_MAX;
}

__global__ void __launch_bounds__(256) first_sites_kernel(const __grid_constant__ RecountLaunch a) {
    grid_wait();
    const uint32_t n_labels = (uint32_t)recount_labels(a);
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    uint32_t l = i < (size_t)a.g.sites ? a.labels[i] : 0u;
    if (l >= n_labels) {
        a.labels[i] = l = 0u;
        atomicExch(a.error_flag, 2);
    }
    first_site(a.first, l, (int)i);
}

// Sum of (u0 + k)^2 for k = 0 .. n - 1.
__device__ __forceinline__ long long squares_from(long long u0, long long n) {
    return n * u0 * u0 + u0 * n * (n - 1) + (n - 1) * n * (2 * n - 1) / 6;
}

// A run of `len` sites of label l along x from (x, y, z), into its moment
// words about its first site: the offsets along a run are consecutive unless
// the run crosses the fold half a span away, so its sums are closed forms
// and the run is one atomic a word, not one a site.
template <int DIM>
__device__ __forceinline__ void run_moments(const RecountLaunch &a, uint32_t l, int x, int y, int z, int len) {
    const uint32_t f = (uint32_t)a.first[l];
    const uint32_t row = udiv(a.g.div_w, f), pl = udiv(a.g.div_h, row);
    const int ax = (int)(f - row * (uint32_t)a.g.w), ay = (int)(row - pl * (uint32_t)a.g.h), az = (int)pl;
    const long long u0 = fold_int(x - ax, a.g.w), u1 = fold_int(x + len - 1 - ax, a.g.w);
    const long long uy = fold_int(y - ay, a.g.h), uz = fold_int(z - az, a.g.d);
    long long s1 = 0, s2 = 0;
    if (u1 - u0 == len - 1) {
        s1 = len * (u0 + u1) / 2;
        s2 = squares_from(u0, len);
    } else {
        for (int k = 0; k < len; ++k) {
            const long long u = fold_int(x + k - ax, a.g.w);
            s1 += u;
            s2 += u * u;
        }
    }
    const long long words[9] = {s1,      len * uy, DIM == 2 ? s2 : len * uz, DIM == 2 ? len * uy * uy : s2,
                                DIM == 2 ? s1 * uy : len * uy * uy, len * uz * uz, s1 * uy, s1 * uz, len * uy * uz};
    unsigned long long *m = reinterpret_cast<unsigned long long *>(&a.mom_base[(size_t)l * a.g.nm]);
#pragma unroll
    for (int k = 0; k < (DIM == 2 ? 5 : 9); ++k) atomicAdd(&m[k], (unsigned long long)words[k]);
}

// Unlike-label neighbours of site i (label l) at (x, y, z), in 32-bit index
// arithmetic: the wrapped coordinates one step either side are formed once
// and each offset picks among them. A neighbour that wraps onto the site
// itself is not a bond.
__device__ __forceinline__ int unlike_neighbours(const Geometry &g, const uint32_t *labels, uint32_t i, uint32_t l,
                                                 int x, int y, int z) {
    const int W = g.w, H = g.h, D = g.d;
    const int xm = x == 0 ? W - 1 : x - 1, xp = x == W - 1 ? 0 : x + 1;
    const int ym = y == 0 ? H - 1 : y - 1, yp = y == H - 1 ? 0 : y + 1;
    const int zm = z == 0 ? D - 1 : z - 1, zp = z == D - 1 ? 0 : z + 1;
    int bonds = 0;
    for (int k = 0; k < g.n_off; ++k) {
        const int dx = g.off[k][0], dy = g.off[k][1], dz = g.off[k][2];
        const uint32_t nx = (uint32_t)(dx < 0 ? xm : (dx > 0 ? xp : x));
        const uint32_t ny = (uint32_t)(dy < 0 ? ym : (dy > 0 ? yp : y));
        const uint32_t nz = (uint32_t)(dz < 0 ? zm : (dz > 0 ? zp : z));
        const uint32_t n = (nz * (uint32_t)H + ny) * (uint32_t)W + nx;
        bonds += n != i && labels[n] != l;
    }
    return bonds;
}

// Volume, unlike-bond surface, per-colour volume and moment sums of every
// label, and its anchor (its first site). The medium has no tally (its counts
// are medium_count_kernel's). Blocks run along lattice rows (x across threads, one row per block
// row), so a warp holds 32 consecutive sites of one row and a cell usually
// covers a run of lanes: each run adds its counts through its first lane,
// one atomic per run, not per site.
// Along a row only x changes, so a run's sites alternate between two
// colours, starting with its first lane's. A label that comes back later in
// the warp starts another run. Neighbour addresses are the compile-time
// neighbourhood's offsets over the wrapped rows and columns either side.
template <int DIM, int NOFF>
__global__ void recount_counts_kernel(const __grid_constant__ RecountLaunch a) {
    constexpr uint32_t kNone = 0xffffffffu;
    grid_wait();
    if (a.flags && !a.flags[(a.clock ? a.clock->step : a.step) & 1]) return;
    const uint32_t n_labels = (uint32_t)recount_labels(a);
    const int W = a.g.w, H = a.g.h, D = a.g.d;
    const int lane = threadIdx.x & 31;
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    const int xm = x == 0 ? W - 1 : x - 1, xp = x == W - 1 ? 0 : x + 1;
    for (int row = blockIdx.y; row < H * D; row += gridDim.y) {
        const int y = row % H, z = row / H;
        const uint32_t i = (uint32_t)row * (uint32_t)W + (uint32_t)x;
        uint32_t l = x < W ? a.labels[i] : kNone;
        if (l != kNone && l >= n_labels) {
            atomicExch(a.error_flag, 2);
            l = kNone;
        }
        int bonds = 0;
        if (l == 0) l = kNone;
        if (l != kNone) {
            const int ym = y == 0 ? H - 1 : y - 1, yp = y == H - 1 ? 0 : y + 1;
            const int zm = z == 0 ? D - 1 : z - 1, zp = z == D - 1 ? 0 : z + 1;
#pragma unroll
            for (int k = 0; k < NOFF; ++k) {
                const int dx = neighbour_offset<DIM, NOFF>(k, 0), dy = neighbour_offset<DIM, NOFF>(k, 1),
                          dz = neighbour_offset<DIM, NOFF>(k, 2);
                const uint32_t nx = (uint32_t)(dx < 0 ? xm : (dx > 0 ? xp : x));
                const uint32_t ny = (uint32_t)(dy < 0 ? ym : (dy > 0 ? yp : y));
                const uint32_t nz = (uint32_t)(dz < 0 ? zm : (dz > 0 ? zp : z));
                const uint32_t n = (nz * (uint32_t)H + ny) * (uint32_t)W + nx;
                // a neighbour that wraps onto the site itself is not a bond
                bonds += n != i && a.labels[n] != l;
            }
        }
        const int colour = (x & 1) | ((y & 1) << 1) | (DIM == 3 ? ((z & 1) << 2) : 0);
        const unsigned full = 0xffffffffu;
        const uint32_t before = __shfl_up_sync(full, l, 1);
        const bool head = lane == 0 || l != before;
        const unsigned heads = __ballot_sync(full, head);
        // inclusive prefix sum of the bond counts over the warp
        int scan = bonds;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(full, scan, o);
            if (lane >= o) scan += v;
        }
        const unsigned later = heads & ~(full >> (31 - lane));  // heads after this lane
        const int last = later ? __ffs(later) - 2 : 31;          // this lane's run ends here
        const int scan_last = __shfl_sync(full, scan, last);
        if (head && l != kNone) {
            const int len = last - lane + 1;
            const int run_bonds = scan_last - scan + bonds;
            atomicAdd(&a.vs_base[l].x, len);
            if (run_bonds) atomicAdd(&a.vs_base[l].y, run_bonds);
            if (a.first[l] == (int)i)
                *reinterpret_cast<int4 *>(&a.anchor[4 * (size_t)l]) = make_int4(x, y, z, (int)i);
            if (a.tracks) run_moments<DIM>(a, l, x, y, z, len);
            int *by_colour = &a.vol_by_colour[(size_t)l * a.g.ncol];
            atomicAdd(&by_colour[colour], (len + 1) / 2);
            if (len > 1) atomicAdd(&by_colour[colour ^ 1], len / 2);
        }
        if (a.nematic && l != kNone) {
            constexpr int NM = DIM == 2 ? 5 : 9;
            unsigned long long *m = reinterpret_cast<unsigned long long *>(&a.mom_base[(size_t)l * a.g.nm]);
            atomicAdd(&m[NM], (unsigned long long)nematic_fixed(a.nematic[2 * (size_t)i]));
            atomicAdd(&m[NM + 1], (unsigned long long)nematic_fixed(a.nematic[2 * (size_t)i + 1]));
        }
    }
}

template <int DIM, int NOFF>
static cudaError_t launch_counts(const RecountLaunch &a, cudaStream_t stream) {
    for (int k = 0; k < NOFF; ++k)
        for (int axis = 0; axis < 3; ++axis)
            if (a.g.off[k][axis] != neighbour_offset<DIM, NOFF>(k, axis)) return cudaErrorInvalidValue;
    const int bx = a.g.w >= 256 ? 256 : (a.g.w + 31) / 32 * 32;
    // at a step's end few blocks, which mostly find no event
    const int rows = a.g.h * a.g.d, across = (a.g.w + bx - 1) / bx;
    const int most = a.flags && a.g.sites <= (1 << 20) ? (296 * (256 / bx) + across - 1) / across : 65535;
    const dim3 grid((unsigned)across, (unsigned)(rows < most ? rows : most));
    return launch_after(recount_counts_kernel<DIM, NOFF>, grid, bx, stream, a);
}

static cudaError_t launch_counts_any(const RecountLaunch &a, cudaStream_t stream) {
    if (a.g.dim == 2) {
        if (a.g.n_off == 4) return launch_counts<2, 4>(a, stream);
        if (a.g.n_off == 8) return launch_counts<2, 8>(a, stream);
    } else {
        if (a.g.n_off == 6) return launch_counts<3, 6>(a, stream);
        if (a.g.n_off == 18) return launch_counts<3, 18>(a, stream);
        if (a.g.n_off == 26) return launch_counts<3, 26>(a, stream);
    }
    return cudaErrorInvalidValue;
}

cudaError_t launch_recount(const RecountLaunch &a, cudaStream_t stream) {
    if (!a.first || !a.anchor) return cudaErrorInvalidValue;
    if (!a.flags) {
        const size_t n = (size_t)a.n_labels;  // the count, or the capacity with n_live
        clear_tallies_kernel<<<(int)((n + 255) / 256), 256, 0, stream>>>(a);
        if (cudaError_t e = cudaGetLastError()) return e;
        if (cudaError_t e =
                launch_after(first_sites_kernel, dim3((unsigned)((a.g.sites + 255) / 256)), 256, stream, a))
            return e;
    }
    return launch_counts_any(a, stream);
}

__device__ __forceinline__ void settle_one(int l, int2 *vs_base, long long *vs_delta, long long *mom_base,
                                           long long *mom_delta, int nm, int tracks);

__global__ void settle_kernel(int2 *vs_base, long long *vs_delta, long long *mom_base, long long *mom_delta, int nm,
                              int n, int tracks, const int *n_live) {
    const int l = blockIdx.x * blockDim.x + threadIdx.x;
    if (l >= (n_live ? *n_live : n)) return;
    settle_one(l, vs_base, vs_delta, mom_base, mom_delta, nm, tracks);
}

__global__ void engine_clock_kernel(EngineClock *clock, int ncol) {
    grid_wait();
    clock->step += 1;
    clock->pass += ncol;
    clock->field_cur ^= clock->field_flip;
}

cudaError_t launch_engine_clock_advance(EngineClock *clock, int ncol, cudaStream_t stream) {
    return launch_after(engine_clock_kernel, dim3(1), 1, stream, clock, ncol);
}

__device__ __forceinline__ void settle_one(int l, int2 *vs_base, long long *vs_delta, long long *mom_base,
                                           long long *mom_delta, int nm, int tracks) {
    int dv, ds;
    unpack_delta(vs_delta[l], dv, ds);
    int2 b = vs_base[l];
    vs_base[l] = make_int2(b.x + dv, b.y + ds);
    vs_delta[l] = 0;
    if (tracks)
        for (int k = 0; k < nm; ++k) {
            mom_base[(size_t)l * nm + k] += mom_delta[(size_t)l * nm + k];
            mom_delta[(size_t)l * nm + k] = 0;
        }
}

cudaError_t launch_settle(int2 *vs_base, long long *vs_delta, long long *mom_base, long long *mom_delta, int nm,
                          int n_labels, int tracks, const int *n_live, cudaStream_t stream) {
    if (n_labels <= 0) return cudaSuccess;
    settle_kernel<<<(n_labels + 255) / 256, 256, 0, stream>>>(vs_base, vs_delta, mom_base, mom_delta, nm, n_labels,
                                                              tracks, n_live);
    return cudaGetLastError();
}

__global__ void medium_count_kernel(const __grid_constant__ Geometry g, const uint32_t *labels,
                                    unsigned long long *out) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    unsigned long long sites = 0, bonds = 0;
    if (i < (size_t)g.sites && labels[i] == 0) {
        int x, y, z;
        coords_of(g, i, x, y, z);
        sites = 1;
        bonds = (unsigned long long)unlike_neighbours(g, labels, (uint32_t)i, 0u, x, y, z);
    }
    for (int o = 16; o > 0; o >>= 1) {
        sites += __shfl_down_sync(0xffffffffu, sites, o);
        bonds += __shfl_down_sync(0xffffffffu, bonds, o);
    }
    if ((threadIdx.x & 31) == 0 && (sites || bonds)) {
        atomicAdd(&out[0], sites);
        atomicAdd(&out[1], bonds);
    }
}

cudaError_t launch_medium_count(const Geometry &g, const uint32_t *labels, unsigned long long *out,
                                cudaStream_t stream) {
    cudaError_t e = cudaMemsetAsync(out, 0, 2 * sizeof(unsigned long long), stream);
    if (e) return e;
    medium_count_kernel<<<(g.sites + 255) / 256, 256, 0, stream>>>(g, labels, out);
    return cudaGetLastError();
}

}  // namespace glz
