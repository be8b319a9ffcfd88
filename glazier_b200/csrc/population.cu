// The per-label end of a Monte Carlo step: the infection rule's switches, and
// division and death, planned per cell on the device.
//
// Replaces `run_population` (glazier-cuda/src/lib.rs:1362-1461) and its
// kernels `cell_circular_sums`, `cell_moments` and `apply_population`
// (lib.rs:66-142), which took five host round trips every Monte Carlo step.
// Here every decision is made on the device from the exact moment sums, in
// four kernels, the last three of which return at once in a step that plans
// no event:
//   labels  per cell: the infection rule; the step's pending deltas folded
//           into the tallies; then a live cell at or past its division volume
//           (and of at least four sites, cpu.rs:681) plans a cut through its
//           centroid perpendicular to its major axis (power iteration on the
//           covariance, moments.rs:165-186), and any other live cell of a
//           type with a death rate dies when its counter-hash draw falls
//           under the rate (the reference's `else if`, lib.rs:1406-1423).
//   count   per site: how many sites each planned cut would move. The last
//           block to finish decides, in label order: a cut that moves nothing
//           or everything is no division (cpu.rs:697-703); the rest take
//           daughter labels n, n + 1, ... in their mothers' order. The live
//           label count stays in device memory, so no host read stands
//           between steps.
//   apply   per site: death to medium, the far side of a cut to the daughter;
//           every tally zeroed and each label's first site found.
//   recount (tally.cu) the tallies from the lattice (cpu.rs:649-653).
// On a small lattice these are chains of a few reads each, so their number is
// what they cost: a whole run of the 256^2 infection model (200 MCS) takes
// 11.3 ms with these and the four-site field kernel, 15 with eleven kernels.

#include "device.cuh"
#include "engine.h"
#include "pdl.cuh"
#include "tally.cuh"
#include "terms.cuh"

namespace glz {

constexpr int kDeath = 1, kDivision = 2;  // a step's event flags

__device__ __forceinline__ double along_cut(const Geometry &g, const int *anchor, const double *plan, uint32_t l,
                                            uint32_t i) {
    const uint32_t row = udiv(g.div_w, i), z = udiv(g.div_h, row), x = i - row * (uint32_t)g.w,
                   y = row - z * (uint32_t)g.h;
    const int4 an = *reinterpret_cast<const int4 *>(&anchor[4 * (size_t)l]);
    const double ux = (double)fold_int((int)x - an.x, g.w);
    const double uy = (double)fold_int((int)y - an.y, g.h);
    const double uz = (double)fold_int((int)z - an.z, g.d);
    const double *p = &plan[6 * (size_t)l];
    return (ux - p[0]) * p[3] + (uy - p[1]) * p[4] + (uz - p[2]) * p[5];
}

// What cell l (of a population model) plans: 0 nothing, kDivision (its cut
// into the plan table) or kDeath.
__device__ __forceinline__ int plan_of(const PopulationLaunch &a, int l, double div_vol, double death_rate, int v,
                                       const long long *m) {
    if (v <= 0) return 0;
    if (div_vol > 0.0 && (double)v >= div_vol && v >= 4) {
        const double dn = (double)v;
        double c[3][3], mean[3];
        if (a.g.dim == 2) {
            mean[0] = (double)m[0] / dn;
            mean[1] = (double)m[1] / dn;
            mean[2] = 0.0;
            c[0][0] = (double)m[2] / dn - mean[0] * mean[0];
            c[1][1] = (double)m[3] / dn - mean[1] * mean[1];
            c[0][1] = c[1][0] = (double)m[4] / dn - mean[0] * mean[1];
            c[2][2] = c[0][2] = c[2][0] = c[1][2] = c[2][1] = 0.0;
        } else {
            mean[0] = (double)m[0] / dn;
            mean[1] = (double)m[1] / dn;
            mean[2] = (double)m[2] / dn;
            c[0][0] = (double)m[3] / dn - mean[0] * mean[0];
            c[1][1] = (double)m[4] / dn - mean[1] * mean[1];
            c[2][2] = (double)m[5] / dn - mean[2] * mean[2];
            c[0][1] = c[1][0] = (double)m[6] / dn - mean[0] * mean[1];
            c[0][2] = c[2][0] = (double)m[7] / dn - mean[0] * mean[2];
            c[1][2] = c[2][1] = (double)m[8] / dn - mean[1] * mean[2];
        }
        double v0 = 1.0, v1 = 0.7, v2 = 0.3;
        bool degenerate = false;
        for (int round = 0; round < 20; ++round) {
            const double w0 = c[0][0] * v0 + c[0][1] * v1 + c[0][2] * v2;
            const double w1 = c[1][0] * v0 + c[1][1] * v1 + c[1][2] * v2;
            const double w2 = c[2][0] * v0 + c[2][1] * v1 + c[2][2] * v2;
            const double norm = sqrt(w0 * w0 + w1 * w1 + w2 * w2);
            if (norm < 1e-15) {
                degenerate = true;
                break;
            }
            v0 = w0 / norm;
            v1 = w1 / norm;
            v2 = w2 / norm;
        }
        if (degenerate) {
            v0 = 1.0;
            v1 = 0.0;
            v2 = 0.0;
        }
        double *p = &a.plan[6 * (size_t)l];
        p[0] = mean[0];
        p[1] = mean[1];
        p[2] = mean[2];
        p[3] = v0;
        p[4] = v1;
        p[5] = v2;
        return kDivision;
    }
    if (death_rate > 0.0) {
        const uint64_t key =
            a.clock ? stream_key(a.seed, (int32_t)a.clock->step, kPopulationStream, 0) : a.key_death;
        if (to_f64(draw(key, (uint32_t)l)) < death_rate) return kDeath;
    }
    return 0;
}

// Every read of a label is requested at once, the label live or not (the
// arrays hold the capacity), and the types' rates come from shared memory:
// the count, then the tallies, types, dose and rates each behind the one
// before were six round trips.
__global__ void __launch_bounds__(128) labels_kernel(const __grid_constant__ PopulationLaunch a) {
    __shared__ double rates[2][kSmemTypes];  // division volume, death rate
    const bool held = a.has_pop && a.n_types <= kSmemTypes;
    if (held && (int)threadIdx.x < a.n_types) {
        rates[0][threadIdx.x] = a.t.division_volume[threadIdx.x];
        rates[1][threadIdx.x] = a.t.death_rate[threadIdx.x];
    }
    const double *const division = held ? rates[0] : a.t.division_volume;
    const double *const death = held ? rates[1] : a.t.death_rate;
    // the slots at the end of the step's passes (the clock advances after it)
    const long long p = a.clock ? a.clock->pass + a.g.ncol : a.pass;
    int2 *const base = a.tal.vs_base[p % 2];
    long long *const delta = a.tal.vs_delta[(p + 2) % 3];
    const int l = blockIdx.x * blockDim.x + threadIdx.x;
    const bool room = l < (a.n_live ? a.cap : a.n_labels);
    __syncthreads();
    grid_wait();
    int t = room ? a.cell_type[l] : 0;
    const long long dose = room && a.infect_from >= 0 ? (long long)a.dose[l] : 0;
    const long long change = room && a.has_pop ? delta[l] : 0;
    int2 b = room && a.has_pop ? base[l] : make_int2(0, 0);
    const int n = a.n_live ? *a.n_live : a.n_labels;
    if (a.has_pop && l == 0 && a.seen_step >= 0) *a.seen = ((unsigned long long)a.seen_step << 32) | (unsigned)n;
    int event = 0;
    if (l < n) {
        if (a.infect_from >= 0 && l > 0 && t == a.infect_from && dose >= a.infect_threshold) {
            t = a.infect_to;
            a.cell_type[l] = (uint8_t)t;
        }
        if (a.has_pop) {
            int dv, ds;
            unpack_delta(change, dv, ds);
            b = make_int2(b.x + dv, b.y + ds);
            base[l] = b;
            delta[l] = 0;
            long long m[11];
            if (a.tracks) {
                long long *const mom = a.tal.mom_base[p % 2] + (size_t)l * a.g.nm;
                long long *const mom_delta = a.tal.mom_delta[(p + 2) % 3] + (size_t)l * a.g.nm;
#pragma unroll
                for (int k = 0; k < 11; ++k)
                    if (k < a.g.nm) m[k] = mom[k] + mom_delta[k];
#pragma unroll
                for (int k = 0; k < 11; ++k)
                    if (k < a.g.nm) {
                        mom[k] = m[k];
                        mom_delta[k] = 0;
                    }
            }
            if (l > 0) event = plan_of(a, l, division[t], death[t], b.x, m);
            a.mode[l] = (unsigned char)event;
            a.moved[l] = 0;
        }
    }
    if (a.has_pop) {
        const int any = __reduce_or_sync(0xffffffffu, (unsigned)event);
        if (any && (threadIdx.x & 31) == 0) atomicOr(&a.flags[population_parity(a)], any);
    }
}

// Give each kept division the next daughter label, in label order, and add
// the daughters to the live count; one block.
__device__ void decide(const PopulationLaunch &a, int *flag) {
    constexpr int kEach = 8;  // consecutive labels a thread takes
    __shared__ int warp_total[32];
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, warps = blockDim.x >> 5;
    const int n = *a.n_live;
    int running = 0, events = 0;
    for (int base = 0; base < n; base += (int)blockDim.x * kEach) {
        int keep = 0, mine = 0;
#pragma unroll
        for (int k = 0; k < kEach; ++k) {
            const int l = base + tid * kEach + k;
            const int m = l < n ? __ldcg(&a.mode[l]) : 0;
            if (m == kDeath) events |= kDeath;
            if (m == kDivision) {
                const int moved = __ldcg(&a.moved[l]);
                const int volume = a.tal.vs_base[a.base_slot][l].x;
                if (moved > 0 && moved < volume) {
                    keep |= 1 << k;
                    ++mine;
                } else {
                    a.mode[l] = 0;
                }
            }
        }
        int scan = mine;
        for (int o = 1; o < 32; o <<= 1) {
            const int up = __shfl_up_sync(0xffffffffu, scan, o);
            if (lane >= o) scan += up;
        }
        __syncthreads();  // the totals of the chunk before have been read
        if (lane == 31) warp_total[wid] = scan;
        __syncthreads();
        int before = running + scan - mine;
        for (int w = 0; w < warps; ++w) {
            before += w < wid ? warp_total[w] : 0;
            running += warp_total[w];
        }
#pragma unroll
        for (int k = 0; k < kEach; ++k)
            if (keep >> k & 1) {
                const int l = base + tid * kEach + k;
                const uint32_t d = (uint32_t)(n + before++);
                a.daughter[l] = d;
                a.cell_type[d] = a.cell_type[l];
            }
    }
    const int death = __syncthreads_or(events);
    if (tid == 0) {
        *flag = (death ? kDeath : 0) | (running ? kDivision : 0);
        *a.n_live = n + running;
    }
}

__global__ void __launch_bounds__(256) count_kernel(const __grid_constant__ PopulationLaunch a) {
    __shared__ bool last;
    grid_wait();
    const int par = population_parity(a);
    int *const flag = &a.flags[par];
    if (blockIdx.x == 0 && threadIdx.x == 0) a.flags[par ^ 1] = 0;  // the next step's, read by no kernel of this one
    const int events = *flag;
    if (!events) return;
    const size_t stride = (size_t)gridDim.x * blockDim.x, first = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    // each label's first site starts past them all (apply finds it)
    for (size_t l = first; l < (size_t)a.cap; l += stride) a.first[l] = INT_MAX;
    if (!(events & kDivision)) return;
    for (size_t i = first; i < (size_t)a.g.sites; i += stride) {
        const uint32_t l = a.labels[i];
        if (l != 0 && a.mode[l] == kDivision && along_cut(a.g, a.anchor, a.plan, l, (uint32_t)i) > 0.0)
            atomicAdd(&a.moved[l], 1);
    }
    // the last block to arrive sees every other block's counts
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) last = atomicAdd(a.ticket, 1) == (int)gridDim.x - 1;
    __syncthreads();
    if (!last) return;
    __threadfence();
    decide(a, flag);
    if (threadIdx.x == 0) *a.ticket = 0;
}

__global__ void __launch_bounds__(256) apply_kernel(const __grid_constant__ PopulationLaunch a) {
    grid_wait();
    if (!a.flags[population_parity(a)]) return;
    const size_t stride = (size_t)gridDim.x * blockDim.x, begin = (size_t)blockIdx.x * blockDim.x;
    for (size_t base = begin; base < (size_t)a.g.sites; base += stride) {
        const size_t i = base + threadIdx.x;
        uint32_t l = i < (size_t)a.g.sites ? a.labels[i] : 0u;
        if (l != 0) {
            const unsigned char m = a.mode[l];
            if (m == kDeath) {
                a.labels[i] = l = 0;
            } else if (m == kDivision && along_cut(a.g, a.anchor, a.plan, l, (uint32_t)i) > 0.0) {
                a.labels[i] = l = a.daughter[l];
            }
        }
        first_site(a.first, l, (int)i);
    }
    RecountLaunch r{};
    r.g = a.g;
    r.vs_base = a.tal.vs_base[a.base_slot];
    r.mom_base = a.tal.mom_base[a.base_slot];
    for (int k = 0; k < 3; ++k) {
        r.vs_delta[k] = a.tal.vs_delta[k];
        r.mom_delta[k] = a.tal.mom_delta[k];
    }
    r.vol_by_colour = a.vol_by_colour;
    r.tracks = a.tracks;
    for (size_t l = begin + threadIdx.x; l < (size_t)*a.n_live; l += stride) clear_tallies(r, (int)l);
}

cudaError_t launch_step_labels(const PopulationLaunch &a, cudaStream_t stream) {
    const int n = a.n_live ? a.cap : a.n_labels;
    if (cudaError_t e = launch_after(labels_kernel, dim3((unsigned)((n + 127) / 128)), 128, stream, a)) return e;
    if (!a.has_pop) return cudaSuccess;
    // at most two blocks an SM up to 2^20 sites, so a step without an event
    // starts few, and eight past it
    const long long sites = ((long long)a.g.sites + 255) / 256, most = a.g.sites <= (1 << 20) ? 296 : 1184;
    const dim3 grid((unsigned)(sites < most ? sites : most));
    if (cudaError_t e = launch_after(count_kernel, grid, 256, stream, a)) return e;
    return launch_after(apply_kernel, grid, 256, stream, a);
}

}  // namespace glz
