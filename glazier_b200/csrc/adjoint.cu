// The adjoint of the chemical-field step, conditioned on a recorded lattice
// trajectory, behind glz_adj_* in include/glazier_gpu.h.
//
// Forward, one Monte Carlo step per species s (the engine's field step,
// field.rs:99-149, in its f32 operation order):
//   k_s sub-steps   u' = u + d (sum of faces - faces u) - e u,  d = D/k, e = decay/k
//   exchange        v1 = u + sec[t];  v2 = v1 - upt[t] v1;  v = max(v2, 0)
// on sites owned by a cell of type t (owner 255 is the medium: no exchange).
// The discrete Metropolis sweep itself is never differentiated: the owners of
// every step come from a trajectory the caller recorded.
//
// Backward, per step in reverse, per species:
//   exchange        lambda_v1 = lambda_v [v2 >= 0] (1 - upt);  d/dsec += lambda_v1;
//                   d/dupt += -lambda_v [v2 >= 0] v1
//   sub-step        lambda_u = lambda' + d (sum of faces of lambda' - faces lambda') - e lambda'
//                   (the periodic Laplacian is its own transpose);
//                   d/dd += lambda' (sum of faces of u - faces u);  d/de += -lambda' u
// and dD = dd / k, d(decay) = de / k. The forward state is kept at every
// `checkpoint_every`-th step; the backward recomputes each segment's sub-step
// inputs from its checkpoint, but for the last segment, whose sub-step states
// the forward keeps as it goes. Adjoint fields are f32; parameter gradients are
// summed in f64 in an order fixed by the lattice alone.
//
// One launch runs one sub-step round of every species that has a sub-step
// left (the engine's round structure), so with one sub-step per species a
// step is one launch forward and one backward. The backward of a species'
// last round applies the exchange adjoint on the fly at the site and its
// faces (it is pointwise), so it needs no launch of its own.
//
// No reference counterpart: glazier has no differentiable field step.

#include <cuda_runtime.h>

#include <cmath>
#include <cstdio>
#include <string>
#include <vector>

#include "../../include/glazier_gpu.h"
#include "device.cuh"
#include "engine.h"

namespace {

int fail(int code, const std::string &msg) {
    glz::set_last_error(msg);
    return code;
}

#define CU(call)                                                                                          \
    do {                                                                                                  \
        cudaError_t e_ = (call);                                                                          \
        if (e_ != cudaSuccess) return fail(GLZ_DRIVER, std::string(#call) + ": " + cudaGetErrorString(e_)); \
    } while (0)

constexpr int kThreads = 256;
constexpr uint8_t kMedium = 255;

struct Grid {
    int w, h, d, dim, sites;
    glz::Divider div_w, div_h;  // w and h as multiply-shift dividers
};

__device__ __forceinline__ void faces_of(const Grid &g, size_t i, size_t nb[6]) {
    const int W = g.w, H = g.h, D = g.d;
    // fewer than 2^31 sites: 32-bit quotients
    const uint32_t r = glz::udiv(g.div_w, (uint32_t)i), pl = glz::udiv(g.div_h, r);
    const int x = (int)((uint32_t)i - r * (uint32_t)W), y = (int)(r - pl * (uint32_t)H), z = (int)pl;
    const size_t row = ((size_t)z * H + y) * W;
    nb[0] = row + (x == 0 ? W - 1 : x - 1);
    nb[1] = row + (x == W - 1 ? 0 : x + 1);
    nb[2] = ((size_t)z * H + (y == 0 ? H - 1 : y - 1)) * W + x;
    nb[3] = ((size_t)z * H + (y == H - 1 ? 0 : y + 1)) * W + x;
    if (g.dim == 3) {
        nb[4] = ((size_t)(z == 0 ? D - 1 : z - 1) * H + y) * W + x;
        nb[5] = ((size_t)(z == D - 1 ? 0 : z + 1) * H + y) * W + x;
    }
}

__device__ __forceinline__ float face_sum(const Grid &g, const float *u, const size_t nb[6]) {
    float sum = u[nb[0]];
    sum = __fadd_rn(sum, u[nb[1]]);
    sum = __fadd_rn(sum, u[nb[2]]);
    sum = __fadd_rn(sum, u[nb[3]]);
    if (g.dim == 3) {
        sum = __fadd_rn(sum, u[nb[4]]);
        sum = __fadd_rn(sum, u[nb[5]]);
    }
    return sum;
}

// Every kernel here may be launched before the one ahead of it on the stream
// has finished (programmatic dependent launch, `launch_after`): it waits for
// that grid and its memory first, then lets the next launch start.
__device__ __forceinline__ void grid_wait() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

template <class Kernel, class... Args>
cudaError_t launch_blocks(Kernel kernel, dim3 grid, int threads, size_t smem, cudaStream_t stream, Args... args) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = dim3((unsigned)threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, args...);
}

template <class Kernel, class... Args>
cudaError_t launch_after(Kernel kernel, int grid, size_t smem, cudaStream_t stream, Args... args) {
    return launch_blocks(kernel, dim3((unsigned)grid), kThreads, smem, stream, args...);
}

struct Species {
    const float *in;    // the sub-step's input
    float *out;         // its output (after the exchange in the last round); may be null
    float *keep;        // last round: where to keep the exchange input; may be null
    int active, last;
};

// The per-sub-step diffusion and decay of each species live in device
// memory (`de`: d for every species, then e), like the rate tables, so a
// captured sequence of rounds serves any parameters with the same sub-step
// counts.
struct ForwardRound {
    Grid g;
    int n_species;
    const uint8_t *owner;  // this step's owner types
    const float *sec, *upt, *de;
    Species sp[glz::kMaxSpecies];
};

// One sub-step round of the field step; the exchange on a species' last round.
__global__ void __launch_bounds__(kThreads) forward_round(const __grid_constant__ ForwardRound a) {
    grid_wait();
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (size_t)a.g.sites) return;
    size_t nb[6];
    faces_of(a.g, i, nb);
    const float faces = a.g.dim == 3 ? 6.0f : 4.0f;
    int t = -1;
    for (int s = 0; s < a.n_species; ++s) {
        const Species &p = a.sp[s];
        if (!p.active) continue;
        const float here = p.in[i];
        const float sum = face_sum(a.g, p.in, nb);
        const float d = a.de[s], e = a.de[a.n_species + s];
        float v = __fsub_rn(__fadd_rn(here, __fmul_rn(d, __fsub_rn(sum, __fmul_rn(faces, here)))), __fmul_rn(e, here));
        if (p.last) {
            if (p.keep) p.keep[i] = v;
            if (t < 0) t = a.owner[i];
            if (t != kMedium) {
                v = __fadd_rn(v, a.sec[t * a.n_species + s]);
                v = __fsub_rn(v, __fmul_rn(a.upt[t * a.n_species + s], v));
                v = v < 0.0f ? 0.0f : v;
            }
        }
        if (p.out) p.out[i] = v;
    }
}

// Lattices whose rows are whole multiples of four sites take the round
// kernels in four-site form: a thread takes sites x0 .. x0 + 3 of a row (x0
// a multiple of 4), reads the row and the rows across its y (and z) faces as
// float4 and the two x neighbours past its ends as scalars, so neighbouring
// sites share their loads. Each site's arithmetic is the one-site kernel's,
// operation for operation, so both forms give the same field bits.
struct Quad {
    size_t c;     // the first of the four sites
    size_t l, r;  // the x neighbour before the first and after the last
    size_t f[4];  // the same four x in the rows across the y-1, y+1, z-1 and z+1 faces
};

__device__ __forceinline__ Quad quad_of(const Grid &g, size_t q) {
    const int W = g.w, H = g.h, D = g.d;
    const uint32_t i = (uint32_t)(4 * q);  // fewer than 2^31 sites
    const uint32_t rw = glz::udiv(g.div_w, i), pl = glz::udiv(g.div_h, rw);
    const int x0 = (int)(i - rw * (uint32_t)W), y = (int)(rw - pl * (uint32_t)H), z = (int)pl;
    const size_t row = ((size_t)z * H + y) * W;
    Quad o;
    o.c = row + x0;
    o.l = row + (x0 == 0 ? W - 1 : x0 - 1);
    o.r = row + (x0 + 4 == W ? 0 : x0 + 4);
    o.f[0] = ((size_t)z * H + (y == 0 ? H - 1 : y - 1)) * W + x0;
    o.f[1] = ((size_t)z * H + (y == H - 1 ? 0 : y + 1)) * W + x0;
    o.f[2] = g.dim == 3 ? ((size_t)(z == 0 ? D - 1 : z - 1) * H + y) * W + x0 : 0;
    o.f[3] = g.dim == 3 ? ((size_t)(z == D - 1 ? 0 : z + 1) * H + y) * W + x0 : 0;
    return o;
}

__device__ __forceinline__ void ld4(const float *p, float v[4]) {
    const float4 t = *reinterpret_cast<const float4 *>(p);
    v[0] = t.x;
    v[1] = t.y;
    v[2] = t.z;
    v[3] = t.w;
}

__device__ __forceinline__ void st4(float *p, const float v[4]) {
    *reinterpret_cast<float4 *>(p) = make_float4(v[0], v[1], v[2], v[3]);
}

__device__ __forceinline__ void ld4(const uint8_t *p, int v[4]) {
    const uchar4 t = *reinterpret_cast<const uchar4 *>(p);
    v[0] = t.x;
    v[1] = t.y;
    v[2] = t.z;
    v[3] = t.w;
}

// The four sites' face sums, in face_sum's order, from their own values h,
// the x neighbours past the ends xl and xr, and the rows across the faces.
__device__ __forceinline__ void quad_sums(bool volume, const float h[4], float xl, float xr, const float fy0[4],
                                          const float fy1[4], const float fz0[4], const float fz1[4], float sum[4]) {
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        float v = __fadd_rn(k == 0 ? xl : h[k - 1], k == 3 ? xr : h[k + 1]);
        v = __fadd_rn(v, fy0[k]);
        v = __fadd_rn(v, fy1[k]);
        if (volume) {
            v = __fadd_rn(v, fz0[k]);
            v = __fadd_rn(v, fz1[k]);
        }
        sum[k] = v;
    }
}

__global__ void __launch_bounds__(kThreads) forward_quads(const __grid_constant__ ForwardRound a) {
    grid_wait();
    const size_t q = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= (size_t)a.g.sites / 4) return;
    const Quad o = quad_of(a.g, q);
    const bool volume = a.g.dim == 3;
    const float faces = volume ? 6.0f : 4.0f;
    int own[4];
    bool have_own = false;
    for (int s = 0; s < a.n_species; ++s) {
        const Species &p = a.sp[s];
        if (!p.active) continue;
        float h[4], fy0[4], fy1[4], fz0[4] = {}, fz1[4] = {}, sum[4], v[4];
        ld4(p.in + o.c, h);
        ld4(p.in + o.f[0], fy0);
        ld4(p.in + o.f[1], fy1);
        if (volume) {
            ld4(p.in + o.f[2], fz0);
            ld4(p.in + o.f[3], fz1);
        }
        quad_sums(volume, h, p.in[o.l], p.in[o.r], fy0, fy1, fz0, fz1, sum);
        const float d = a.de[s], e = a.de[a.n_species + s];
#pragma unroll
        for (int k = 0; k < 4; ++k)
            v[k] = __fsub_rn(__fadd_rn(h[k], __fmul_rn(d, __fsub_rn(sum[k], __fmul_rn(faces, h[k])))), __fmul_rn(e, h[k]));
        if (p.last) {
            if (p.keep) st4(p.keep + o.c, v);
            if (!have_own) {
                ld4(a.owner + o.c, own);
                have_own = true;
            }
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const int t = own[k];
                if (t != kMedium) {
                    v[k] = __fadd_rn(v[k], a.sec[t * a.n_species + s]);
                    v[k] = __fsub_rn(v[k], __fmul_rn(a.upt[t * a.n_species + s], v[k]));
                    v[k] = v[k] < 0.0f ? 0.0f : v[k];
                }
            }
        }
        if (p.out) st4(p.out + o.c, v);
    }
}

// Parameter gradients are summed without atomics, in an order fixed by the
// lattice alone, so a backward is bit-reproducible and independent of the
// checkpoint interval: the backward kernel runs on a fixed grid of at most
// `kBlocks` blocks striding over the sites, each block adds its own totals
// into its own row of `partial` (blocks x n_grads f64; a row is touched by
// one block only and launches are ordered on one stream), and
// `reduce_partials` sums the rows in block order at the end.
constexpr int kBlocks = 148 * 8;
constexpr int kWarps = kThreads / 32;
constexpr int kMostTypes = 254;  // of a handle: an owner is a byte, and 255 the medium

__device__ __forceinline__ double warp_sum(double v) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    return v;
}

// The block's sum of one f64 per thread, in a fixed order, on thread 0.
__device__ __forceinline__ double block_sum(double v, double *scratch) {
    v = warp_sum(v);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (lane == 0) scratch[warp] = v;
    __syncthreads();
    double total = 0.0;
    if (threadIdx.x == 0)
        for (int w = 0; w < kWarps; ++w) total += scratch[w];
    __syncthreads();
    return total;
}

struct Adjoint {
    const float *u;     // the sub-step's input
    const float *exch;  // last round: the exchange input
    const float *lam;   // the adjoint of the round's output (of the step's output in the last round)
    float *lam_in;      // the adjoint of the sub-step's input
    int active, last;
};

struct BackwardRound {
    Grid g;
    int n_species, n_types, n_grads;
    const uint8_t *owner;
    const float *sec, *upt, *de;
    double *partial;
    Adjoint sp[glz::kMaxSpecies];
};

// The exchange adjoint at site j: the adjoint of the exchange input from the
// adjoint `l` of its output, with v1 and the clamp gate for the gradients.
__device__ __forceinline__ float exchange_adjoint(const BackwardRound &a, const Adjoint &p, int s, size_t j, float l,
                                                  float *v1_out, float *lv_out) {
    const uint8_t t = a.owner[j];
    if (t == kMedium) return l;
    const float q = a.upt[t * a.n_species + s];
    const float v1 = __fadd_rn(p.exch[j], a.sec[t * a.n_species + s]);
    const float v2 = __fsub_rn(v1, __fmul_rn(q, v1));
    const float lv = v2 < 0.0f ? 0.0f : l;
    if (v1_out) {
        *v1_out = v1;
        *lv_out = lv;
    }
    return __fmul_rn(lv, __fsub_rn(1.0f, q));
}

// One sub-step round backward, last rounds first: lambda of every active
// species through its exchange (last round) and sub-step, and the gradients.
// Each warp reduces the exchange gradients of one owner type at a time (the
// types present in its 32 sites, in lane order of first appearance); lane 0
// adds them to the warp's own shared row. The block's row of `partial` is
// copied into shared memory as the launch starts, summed into there, and
// written back at the end, so no read of it waits at the tail.
__global__ void __launch_bounds__(kThreads) backward_round(const __grid_constant__ BackwardRound a) {
    grid_wait();
    extern __shared__ double acc[];  // kWarps rows of 2 * n_types (sec then upt), then the block's n_grads row
    __shared__ double scratch[kWarps];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int T = a.n_types, S = a.n_species;
    const float faces = a.g.dim == 3 ? 6.0f : 4.0f;
    const size_t stride = (size_t)gridDim.x * blockDim.x;
    double *global_row = a.partial + (size_t)blockIdx.x * a.n_grads;
    double *row = acc + (size_t)kWarps * 2 * T;
    for (int k = threadIdx.x; k < a.n_grads; k += blockDim.x)
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((uint32_t)__cvta_generic_to_shared(row + k)), "l"(global_row + k)
                     : "memory");
    asm volatile("cp.async.commit_group;" ::: "memory");
    double *mine = acc + (size_t)warp * 2 * T;
    for (int s = 0; s < S; ++s) {
        const Adjoint &p = a.sp[s];
        if (!p.active) continue;
        if (p.last) {
            for (int k = threadIdx.x; k < kWarps * 2 * T; k += blockDim.x) acc[k] = 0.0;
            __syncthreads();
        }
        double gd = 0.0, ge = 0.0;
        // every lane of a warp takes the same number of trips
        for (size_t base = (size_t)blockIdx.x * blockDim.x; base < (size_t)a.g.sites; base += stride) {
            const size_t i = base + threadIdx.x;
            const bool in = i < (size_t)a.g.sites;
            float l1 = 0.0f, dupt = 0.0f;
            int t = kMedium;
            if (in) {
                size_t nb[6];
                faces_of(a.g, i, nb);
                float l = p.lam[i];
                float ls;
                if (p.last) {
                    float v1 = 0.0f, lv = 0.0f;
                    t = a.owner[i];
                    l = exchange_adjoint(a, p, s, i, l, &v1, &lv);
                    if (t != kMedium) {
                        l1 = l;
                        dupt = -__fmul_rn(lv, v1);
                    }
                    ls = exchange_adjoint(a, p, s, nb[0], p.lam[nb[0]], nullptr, nullptr);
                    const int nf = a.g.dim == 3 ? 6 : 4;
                    for (int f = 1; f < nf; ++f)
                        ls = __fadd_rn(ls, exchange_adjoint(a, p, s, nb[f], p.lam[nb[f]], nullptr, nullptr));
                } else {
                    ls = face_sum(a.g, p.lam, nb);
                }
                const float d = a.de[s], e = a.de[S + s];
                p.lam_in[i] = __fsub_rn(__fadd_rn(l, __fmul_rn(d, __fsub_rn(ls, __fmul_rn(faces, l)))), __fmul_rn(e, l));
                const float here = p.u[i];
                const float us = face_sum(a.g, p.u, nb);
                gd += (double)__fmul_rn(l, __fsub_rn(us, __fmul_rn(faces, here)));
                ge -= (double)__fmul_rn(l, here);
            }
            if (p.last) {
                unsigned todo = __ballot_sync(0xffffffffu, t != kMedium);
                while (todo) {
                    const int leader = __ffs(todo) - 1;
                    const int tt = __shfl_sync(0xffffffffu, t, leader);
                    const bool same = t == tt;
                    const double x = warp_sum(same ? (double)l1 : 0.0);
                    const double y = warp_sum(same ? (double)dupt : 0.0);
                    if (lane == 0) {
                        mine[tt] += x;
                        mine[T + tt] += y;
                    }
                    todo &= ~__ballot_sync(0xffffffffu, same);
                }
            }
        }
        // gradient layout: d, e per species, then sec, upt per (type, species);
        // the row's copy has landed once every thread has waited for its own
        // part and block_sum's barrier has passed
        asm volatile("cp.async.wait_all;" ::: "memory");
        const double td = block_sum(gd, scratch);
        const double te = block_sum(ge, scratch);
        if (threadIdx.x == 0) {
            row[s] += td;
            row[S + s] += te;
        }
        if (p.last) {
            __syncthreads();
            for (int k = threadIdx.x; k < 2 * T; k += blockDim.x) {
                double v = 0.0;
                for (int w = 0; w < kWarps; ++w) v += acc[(size_t)w * 2 * T + k];
                const int tt = k % T;
                row[(k < T ? 2 * S : 2 * S + T * S) + tt * S + s] += v;
            }
            __syncthreads();
        }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    for (int k = threadIdx.x; k < a.n_grads; k += blockDim.x) global_row[k] = row[k];
}

// A species' rates for owner type t: from registers holding the first TMAX
// types (TMAX > 0, every type below TMAX), else from the tables.
template <int TMAX>
struct Rates {
    float sec[TMAX > 0 ? TMAX : 1], upt[TMAX > 0 ? TMAX : 1];
    const float *gsec, *gupt;  // the tables at the species, stride n_species
    int stride;
    __device__ __forceinline__ void load(const float *sec_table, const float *upt_table, int s, int n_species,
                                         int n_types) {
        gsec = sec_table + s;
        gupt = upt_table + s;
        stride = n_species;
#pragma unroll
        for (int tt = 0; tt < (TMAX > 0 ? TMAX : 1); ++tt) {
            sec[tt] = TMAX > 0 && tt < n_types ? gsec[tt * stride] : 0.0f;
            upt[tt] = TMAX > 0 && tt < n_types ? gupt[tt * stride] : 0.0f;
        }
    }
    __device__ __forceinline__ void of(int t, float &s_out, float &u_out) const {
        if (TMAX > 0) {
            s_out = sec[0];
            u_out = upt[0];
#pragma unroll
            for (int tt = 1; tt < (TMAX > 0 ? TMAX : 1); ++tt)
                if (t == tt) {
                    s_out = sec[tt];
                    u_out = upt[tt];
                }
        } else {
            s_out = gsec[t * stride];
            u_out = gupt[t * stride];
        }
    }
};

// The exchange adjoint of one site of type t (kMedium: none) whose exchange
// input was x: exchange_adjoint with the owner, the input and the rates
// already read.
template <int TMAX>
__device__ __forceinline__ float exchange_adjoint_at(const Rates<TMAX> &r, int t, float x, float l, float *v1_out,
                                                     float *lv_out) {
    if (t == kMedium) return l;
    float sec, q;
    r.of(t, sec, q);
    const float v1 = __fadd_rn(x, sec);
    const float v2 = __fsub_rn(v1, __fmul_rn(q, v1));
    const float lv = v2 < 0.0f ? 0.0f : l;
    *v1_out = v1;
    *lv_out = lv;
    return __fmul_rn(lv, __fsub_rn(1.0f, q));
}

// backward_round in four-site form. Each thread adds its four sites'
// gradient terms in x order. With TMAX > 0 (every owner type below TMAX)
// each thread also keeps its exchange gradients per owner type in registers
// across its trips, and each warp sums them once at the end of a species;
// with TMAX 0 the warps reduce them type by type on every trip, as
// backward_round does. Either way the order is fixed by the lattice.
template <int TMAX>
__global__ void __launch_bounds__(kThreads) backward_quads(const __grid_constant__ BackwardRound a) {
    grid_wait();
    extern __shared__ double acc[];  // kWarps rows of 2 * n_types (sec then upt), then the block's n_grads row
    __shared__ double scratch[kWarps];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int T = a.n_types, S = a.n_species;
    const bool volume = a.g.dim == 3;
    const float faces = volume ? 6.0f : 4.0f;
    const size_t quads = (size_t)a.g.sites / 4, stride = (size_t)gridDim.x * blockDim.x;
    double *global_row = a.partial + (size_t)blockIdx.x * a.n_grads;
    double *row = acc + (size_t)kWarps * 2 * T;
    for (int k = threadIdx.x; k < a.n_grads; k += blockDim.x)
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((uint32_t)__cvta_generic_to_shared(row + k)),
                     "l"(global_row + k)
                     : "memory");
    asm volatile("cp.async.commit_group;" ::: "memory");
    double *mine = acc + (size_t)warp * 2 * T;
    for (int s = 0; s < S; ++s) {
        const Adjoint &p = a.sp[s];
        if (!p.active) continue;
        if (p.last) {
            for (int k = threadIdx.x; k < kWarps * 2 * T; k += blockDim.x) acc[k] = 0.0;
            __syncthreads();
        }
        double gd = 0.0, ge = 0.0;
        double tsec[TMAX > 0 ? TMAX : 1] = {}, tupt[TMAX > 0 ? TMAX : 1] = {};  // per owner type, TMAX > 0
        const float d = a.de[s], e = a.de[S + s];
        Rates<TMAX> rates;
        rates.load(a.sec, a.upt, s, S, T);
        // every lane of a warp takes the same number of trips
        for (size_t base = (size_t)blockIdx.x * blockDim.x; base < quads; base += stride) {
            const size_t q = base + threadIdx.x;
            const bool in = q < quads;
            float l1[4] = {}, dupt[4] = {};
            int t[4] = {kMedium, kMedium, kMedium, kMedium};
            if (in) {
                const Quad o = quad_of(a.g, q);
                float l[4], fy0[4], fy1[4], fz0[4] = {}, fz1[4] = {}, ls[4];
                ld4(p.lam + o.c, l);
                ld4(p.lam + o.f[0], fy0);
                ld4(p.lam + o.f[1], fy1);
                if (volume) {
                    ld4(p.lam + o.f[2], fz0);
                    ld4(p.lam + o.f[3], fz1);
                }
                float xl = p.lam[o.l], xr = p.lam[o.r];
                // the sub-step input, read before anything is written
                float u[4], uy0[4], uy1[4], uz0[4] = {}, uz1[4] = {}, us[4];
                ld4(p.u + o.c, u);
                ld4(p.u + o.f[0], uy0);
                ld4(p.u + o.f[1], uy1);
                if (volume) {
                    ld4(p.u + o.f[2], uz0);
                    ld4(p.u + o.f[3], uz1);
                }
                const float ul = p.u[o.l], ur = p.u[o.r];
                if (p.last) {
                    float x[4], v1, lv;
                    ld4(a.owner + o.c, t);
                    ld4(p.exch + o.c, x);
                    int ty0[4], ty1[4], tz0[4] = {}, tz1[4] = {};
                    float xy0[4], xy1[4], xz0[4] = {}, xz1[4] = {};
                    ld4(a.owner + o.f[0], ty0);
                    ld4(p.exch + o.f[0], xy0);
                    ld4(a.owner + o.f[1], ty1);
                    ld4(p.exch + o.f[1], xy1);
                    if (volume) {
                        ld4(a.owner + o.f[2], tz0);
                        ld4(p.exch + o.f[2], xz0);
                        ld4(a.owner + o.f[3], tz1);
                        ld4(p.exch + o.f[3], xz1);
                    }
                    const int tl = a.owner[o.l], tr = a.owner[o.r];
                    const float xxl = p.exch[o.l], xxr = p.exch[o.r];
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        l[k] = exchange_adjoint_at(rates, t[k], x[k], l[k], &v1, &lv);
                        if (t[k] != kMedium) {
                            l1[k] = l[k];
                            dupt[k] = -__fmul_rn(lv, v1);
                        }
                        fy0[k] = exchange_adjoint_at(rates, ty0[k], xy0[k], fy0[k], &v1, &lv);
                        fy1[k] = exchange_adjoint_at(rates, ty1[k], xy1[k], fy1[k], &v1, &lv);
                        if (volume) {
                            fz0[k] = exchange_adjoint_at(rates, tz0[k], xz0[k], fz0[k], &v1, &lv);
                            fz1[k] = exchange_adjoint_at(rates, tz1[k], xz1[k], fz1[k], &v1, &lv);
                        }
                    }
                    xl = exchange_adjoint_at(rates, tl, xxl, xl, &v1, &lv);
                    xr = exchange_adjoint_at(rates, tr, xxr, xr, &v1, &lv);
                }
                quad_sums(volume, l, xl, xr, fy0, fy1, fz0, fz1, ls);
                float li[4];
#pragma unroll
                for (int k = 0; k < 4; ++k)
                    li[k] = __fsub_rn(__fadd_rn(l[k], __fmul_rn(d, __fsub_rn(ls[k], __fmul_rn(faces, l[k])))),
                                      __fmul_rn(e, l[k]));
                st4(p.lam_in + o.c, li);
                quad_sums(volume, u, ul, ur, uy0, uy1, uz0, uz1, us);
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    gd += (double)__fmul_rn(l[k], __fsub_rn(us[k], __fmul_rn(faces, u[k])));
                    ge -= (double)__fmul_rn(l[k], u[k]);
                }
            }
            if (TMAX > 0 && p.last) {
#pragma unroll
                for (int k = 0; k < 4; ++k)
#pragma unroll
                    for (int tt = 0; tt < (TMAX > 0 ? TMAX : 1); ++tt) {
                        tsec[tt] += t[k] == tt ? (double)l1[k] : 0.0;
                        tupt[tt] += t[k] == tt ? (double)dupt[k] : 0.0;
                    }
            } else if (p.last) {
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    unsigned todo = __ballot_sync(0xffffffffu, t[k] != kMedium);
                    while (todo) {
                        const int leader = __ffs(todo) - 1;
                        const int tt = __shfl_sync(0xffffffffu, t[k], leader);
                        const bool same = t[k] == tt;
                        const double x = warp_sum(same ? (double)l1[k] : 0.0);
                        const double y = warp_sum(same ? (double)dupt[k] : 0.0);
                        if (lane == 0) {
                            mine[tt] += x;
                            mine[T + tt] += y;
                        }
                        todo &= ~__ballot_sync(0xffffffffu, same);
                    }
                }
            }
        }
        if (TMAX > 0 && p.last) {
#pragma unroll
            for (int tt = 0; tt < (TMAX > 0 ? TMAX : 1); ++tt) {
                const double x = warp_sum(tsec[tt]), y = warp_sum(tupt[tt]);
                if (lane == 0 && tt < T) {
                    mine[tt] = x;
                    mine[T + tt] = y;
                }
            }
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
        const double td = block_sum(gd, scratch);
        const double te = block_sum(ge, scratch);
        if (threadIdx.x == 0) {
            row[s] += td;
            row[S + s] += te;
        }
        if (p.last) {
            __syncthreads();
            for (int k = threadIdx.x; k < 2 * T; k += blockDim.x) {
                double v = 0.0;
                for (int w = 0; w < kWarps; ++w) v += acc[(size_t)w * 2 * T + k];
                const int tt = k % T;
                row[(k < T ? 2 * S : 2 * S + T * S) + tt * S + s] += v;
            }
            __syncthreads();
        }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    for (int k = threadIdx.x; k < a.n_grads; k += blockDim.x) global_row[k] = row[k];
}

// Planes take several rounds a launch (tile_plane says which): a block holds a
// tile of kTileX by kTileY sites of one species with kHalo sites about it in shared memory and runs up to kHalo rounds there,
// each valid one site less far out than the round before, so a round costs a
// block barrier and not a launch, and neighbouring tiles repeat the rounds of
// their common margin (1.4 times the sites at 64 x 32 with a halo of 4).
// Species do not meet in a field step, so each has blocks of its own. A round
// of a 512^2 field was a launch of a few dependent reads on L2-resident data:
// 3.8 us forward and 9.4 backward, whatever the arithmetic. At 512^2 with two
// species, 50 steps and a checkpoint every 10 (host clock of the calls) the
// forward takes 135 us (189 one round a launch) and the backward 415 (686); at
// 1024^2, 286 (377) and 1410 (2025). Issue slots and shared-memory latency
// bound a round now. Tiles of 16, 24 or 40 rows, blocks of 256, 320 or 512
// threads, and two quads a thread one under the other were all slower at
// 512^2, and so was copying each round's inputs in a round ahead.
// Each site's arithmetic is the one-round kernels', operation for operation.
constexpr int kHalo = 4;  // rounds a launch at most; a whole quad, so tiles stay aligned
constexpr int kTileX = 64, kTileY = 32;
constexpr int kRegionX = kTileX + 2 * kHalo, kRegionY = kTileY + 2 * kHalo;
constexpr int kRegionQuads = kRegionX / 4;
constexpr int kTileThreads = 384;
constexpr int kQuadsEach = (kRegionY * kRegionQuads + kTileThreads - 1) / kTileThreads;
constexpr int kTileTypes = 16;  // owner types whose rates and sums a tile kernel holds at most

struct TileForward {
    Grid g;
    int n_species, n_types, steps;
    const uint8_t *owner;  // the first step's owner types
    const float *sec, *upt, *de;
    int k[glz::kMaxSpecies];             // sub-steps a step
    const float *in[glz::kMaxSpecies];   // the first step's input
    float *keep[glz::kMaxSpecies][kHalo];  // by round: where to keep the exchange input (null: nowhere)
    float *post[glz::kMaxSpecies][kHalo];  // by round: where to store its output (null: nowhere)
};

struct TileBackward {
    Grid g;
    int n_species, n_types, steps;
    const uint8_t *owner;  // the first step's owner types (the last the launch takes back)
    const float *sec, *upt, *de;
    int k[glz::kMaxSpecies];
    const float *lam[glz::kMaxSpecies];
    float *lam_in[glz::kMaxSpecies];
    const float *u[glz::kMaxSpecies][kHalo];     // by round, last first: its sub-step's input
    const float *exch[glz::kMaxSpecies][kHalo];  // by round, a step's last: the exchange input
    double *sums;  // each thread's running gradient sums: [block][value][thread]
    int fresh;     // the sums start at zero
};

// A thread's quads of a tile's region: region row and first column, the
// lattice site they wrap to, and whether they are the tile's own. On rows of
// whole quads (WHOLE) a quad is four sites in a line, read and written at
// once; on others it may run past its row's end, from cell bend on at the
// row's start, and the tile's own cells of the last are the first `count`.
template <bool WHOLE>
struct TileQuads {
    int w;
    int bend[kQuadsEach], count[kQuadsEach];
    int cell[kQuadsEach];  // offset in the region, -1 past its end
    int row[kQuadsEach], col[kQuadsEach];
    uint32_t site[kQuadsEach];
    bool mine[kQuadsEach];
    __device__ __forceinline__ TileQuads(const Grid &g, int x0, int y0) : w(g.w) {
#pragma unroll
        for (int n = 0; n < kQuadsEach; ++n) {
            const int q = (int)threadIdx.x + n * kTileThreads;
            row[n] = q / kRegionQuads;
            col[n] = q - row[n] * kRegionQuads;
            cell[n] = row[n] < kRegionY ? 4 * q : -1;
            const int y = y0 - kHalo + row[n], x = x0 - kHalo + 4 * col[n];
            site[n] = (uint32_t)glz::wrap(y, g.h) * (uint32_t)g.w + (uint32_t)glz::wrap(x, g.w);
            mine[n] = row[n] >= kHalo && row[n] < kHalo + kTileY && col[n] >= 1 && col[n] < kRegionQuads - 1 &&
                      y < g.h && x < g.w;
            bend[n] = g.w - glz::wrap(x, g.w);
            count[n] = mine[n] ? g.w - x : 0;
        }
    }
    // cell c of quad n is the tile's own
    __device__ __forceinline__ bool own(int n, int c) const { return WHOLE ? mine[n] : c < count[n]; }
    // quad n's cells of a lattice array, its first cell at site `at` of it
    template <class T, class V>
    __device__ __forceinline__ void load(const T *p, uint32_t at, int n, V v[4]) const {
        if constexpr (WHOLE) {
            ld4(p + at, v);
        } else {
#pragma unroll
            for (int c = 0; c < 4; ++c) v[c] = p[at + c - (c >= bend[n] ? (uint32_t)w : 0u)];
        }
    }
    template <class T, class V>
    __device__ __forceinline__ void load(const T *p, int n, V v[4]) const {
        load(p, site[n], n, v);
    }
    // the tile's own cells of quad n to a lattice array
    __device__ __forceinline__ void store(float *p, int n, const float v[4]) const {
        if constexpr (WHOLE) {
            if (mine[n]) st4(p + site[n], v);
        } else {
#pragma unroll
            for (int c = 0; c < 4; ++c)
                if (c < count[n]) p[site[n] + c] = v[c];
        }
    }
    // whether quad n has a site within `margin` of the tile
    __device__ __forceinline__ bool within(int n, int margin) const {
        return cell[n] >= 0 && row[n] >= kHalo - margin && row[n] < kHalo + kTileY + margin &&
               (margin > 0 || (col[n] >= 1 && col[n] < kRegionQuads - 1));
    }
};

// The diffusion and decay of a quad of region cells, from `b`.
__device__ __forceinline__ void quad_step(const float *b, int cell, float d, float e, float h[4], float v[4]) {
    float up[4], dn[4], none[4] = {}, sum[4];
    ld4(b + cell, h);
    ld4(b + cell - kRegionX, up);
    ld4(b + cell + kRegionX, dn);
    quad_sums(false, h, b[cell - 1], b[cell + 4], up, dn, none, none, sum);
#pragma unroll
    for (int c = 0; c < 4; ++c)
        v[c] = __fsub_rn(__fadd_rn(h[c], __fmul_rn(d, __fsub_rn(sum[c], __fmul_rn(4.0f, h[c])))), __fmul_rn(e, h[c]));
}

// The species' rates by owner type, (sec, upt), in shared memory, and the slot
// of owner `o`: the medium's has none of either.
__device__ __forceinline__ void tile_rates(const float *sec, const float *upt, int s, int n_species, int n_types,
                                           float2 *rates) {
    const int t = (int)threadIdx.x;
    if (t <= n_types)
        rates[t] = t < n_types ? make_float2(sec[t * n_species + s], upt[t * n_species + s]) : make_float2(0.0f, 0.0f);
}

template <bool WHOLE>
__global__ void __launch_bounds__(kTileThreads) tile_forward(const __grid_constant__ TileForward a) {
    __shared__ alignas(16) float region[2][kRegionX * kRegionY];
    __shared__ float2 rates[kTileTypes + 1];
    const int s = (int)blockIdx.z, k = a.k[s], rounds = a.steps * k;
    const TileQuads<WHOLE> Q(a.g, (int)blockIdx.x * kTileX, (int)blockIdx.y * kTileY);
    grid_wait();
    tile_rates(a.sec, a.upt, s, a.n_species, a.n_types, rates);
    const float d = a.de[s], e = a.de[a.n_species + s];
#pragma unroll
    for (int n = 0; n < kQuadsEach; ++n)
        if (Q.cell[n] >= 0) {
            float v[4];
            Q.load(a.in[s], n, v);
            st4(region[0] + Q.cell[n], v);
        }
    int at = 0;
    for (int t = 0, r = 0; t < a.steps; ++t) {
        int own[kQuadsEach][4];
#pragma unroll
        for (int n = 0; n < kQuadsEach; ++n)
            if (Q.cell[n] >= 0) Q.load(a.owner + (size_t)t * a.g.sites, n, own[n]);
        for (int j = 0; j < k; ++j, ++r) {
            __syncthreads();  // the round before is in place (and the rates)
            const float *b = region[at];
            float *next = region[at ^ 1];
            float *const keep = a.keep[s][r], *const post = a.post[s][r];
            const bool last = j == k - 1;
#pragma unroll
            for (int n = 0; n < kQuadsEach; ++n) {
                if (!Q.within(n, rounds - 1 - r)) continue;
                float h[4], v[4];
                quad_step(b, Q.cell[n], d, e, h, v);
                if (last) {
                    if (keep) Q.store(keep, n, v);
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        const bool cell = own[n][c] != kMedium;
                        const float2 rate = rates[cell ? own[n][c] : a.n_types];
                        float w = __fadd_rn(v[c], rate.x);
                        w = __fsub_rn(w, __fmul_rn(rate.y, w));
                        w = w < 0.0f ? 0.0f : w;
                        v[c] = cell ? w : v[c];
                    }
                }
                st4(next + Q.cell[n], v);
                if (post) Q.store(post, n, v);
            }
            at ^= 1;
        }
    }
}

// The rounds of `steps` steps backward. Each thread adds its quads' gradient
// terms, round by round and in x order, to running sums that it takes up from
// the launch before and leaves for the next: whatever the checkpoint interval
// cuts launches into, a thread adds the same terms in the same order. The
// sums by owner type sit in shared memory, a column a thread (a select among
// registers cost more than the rest of the exchange).
__host__ __device__ constexpr size_t tile_backward_smem(int n_types) {
    return sizeof(double) * 2 * kTileThreads * (n_types + 1) + sizeof(float) * 2 * kRegionX * kRegionY;
}

template <bool WHOLE>
__global__ void __launch_bounds__(kTileThreads, 2) tile_backward(const __grid_constant__ TileBackward a) {
    extern __shared__ __align__(16) unsigned char dynamic[];
    __shared__ float2 rates[kTileTypes + 1];
    const int T = a.n_types, tid = (int)threadIdx.x;
    float *const region = reinterpret_cast<float *>(dynamic);  // two of kRegionX * kRegionY
    // [type][sec, upt][thread], the medium's slot last (its sums go nowhere)
    double *const by_type = reinterpret_cast<double *>(region + 2 * kRegionX * kRegionY) + tid;
    const int s = (int)blockIdx.z, k = a.k[s], rounds = a.steps * k;
    const int block = ((int)blockIdx.z * (int)gridDim.y + (int)blockIdx.y) * (int)gridDim.x + (int)blockIdx.x;
    const TileQuads<WHOLE> Q(a.g, (int)blockIdx.x * kTileX, (int)blockIdx.y * kTileY);
    grid_wait();
    tile_rates(a.sec, a.upt, s, a.n_species, T, rates);
    const float d = a.de[s], e = a.de[a.n_species + s];
    double *const sums = a.sums + (size_t)block * (2 + 2 * T) * kTileThreads + tid;
    double gd = 0.0, ge = 0.0;
    if (!a.fresh) {
        gd = sums[0];
        ge = sums[kTileThreads];
    }
    for (int v = 0; v < 2 * T; ++v) by_type[v * kTileThreads] = a.fresh ? 0.0 : sums[(2 + v) * kTileThreads];
    by_type[2 * T * kTileThreads] = by_type[(2 * T + 1) * kTileThreads] = 0.0;
#pragma unroll
    for (int n = 0; n < kQuadsEach; ++n)
        if (Q.cell[n] >= 0) {
            float v[4];
            Q.load(a.lam[s], n, v);
            st4(region + Q.cell[n], v);
        }
    __syncthreads();
    int at = 0;
    for (int t = a.steps - 1, r = 0; t >= 0; --t) {
        for (int j = k - 1; j >= 0; --j, ++r) {
            const int margin = rounds - 1 - r;
            float *const b = region + at * kRegionX * kRegionY, *const next = region + (at ^ 1) * kRegionX * kRegionY;
            const float *const u = a.u[s][r];
            if (j == k - 1) {
                // through the exchange, at the site
                const float *const exch = a.exch[s][r];
                float x[kQuadsEach][4];
                int own[kQuadsEach][4];
#pragma unroll
                for (int n = 0; n < kQuadsEach; ++n)
                    if (Q.within(n, margin + 1)) {
                        Q.load(exch, n, x[n]);
                        Q.load(a.owner + (size_t)t * a.g.sites, n, own[n]);
                    }
#pragma unroll
                for (int n = 0; n < kQuadsEach; ++n) {
                    if (!Q.within(n, margin + 1)) continue;
                    float l[4];
                    ld4(b + Q.cell[n], l);
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        const bool cell = own[n][c] != kMedium;
                        const int o = cell ? own[n][c] : T;
                        const float2 rate = rates[o];
                        const float v1 = __fadd_rn(x[n][c], rate.x);
                        const float v2 = __fsub_rn(v1, __fmul_rn(rate.y, v1));
                        const float lv = v2 < 0.0f ? 0.0f : l[c];
                        const float l1 = __fmul_rn(lv, __fsub_rn(1.0f, rate.y));
                        l[c] = cell ? l1 : l[c];
                        if (Q.own(n, c)) {
                            double *const sum = by_type + 2 * o * kTileThreads;
                            sum[0] += (double)l1;
                            sum[kTileThreads] -= (double)__fmul_rn(lv, v1);
                        }
                    }
                    st4(b + Q.cell[n], l);
                }
                __syncthreads();
            }
#pragma unroll
            for (int n = 0; n < kQuadsEach; ++n) {
                if (!Q.within(n, margin)) continue;
                float l[4], li[4];
                quad_step(b, Q.cell[n], d, e, l, li);
                st4(next + Q.cell[n], li);
                if (Q.mine[n]) {
                    const uint32_t W = (uint32_t)a.g.w, all = (uint32_t)a.g.sites, site = Q.site[n];
                    const uint32_t x = site - glz::udiv(a.g.div_w, site) * W;
                    float h[4], hu[4], hd[4], none[4] = {}, us[4];
                    Q.load(u, site, n, h);
                    Q.load(u, site < W ? site + all - W : site - W, n, hu);
                    Q.load(u, site + W >= all ? site + W - all : site + W, n, hd);
                    quad_sums(false, h, u[x == 0 ? site + W - 1 : site - 1], u[x + 4 >= W ? site + 4 - W : site + 4], hu,
                              hd, none, none, us);
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        if (!Q.own(n, c)) continue;
                        gd += (double)__fmul_rn(l[c], __fsub_rn(us[c], __fmul_rn(4.0f, h[c])));
                        ge -= (double)__fmul_rn(l[c], h[c]);
                    }
                }
            }
            __syncthreads();
            at ^= 1;
        }
    }
#pragma unroll
    for (int n = 0; n < kQuadsEach; ++n)
        if (Q.mine[n]) {
            float v[4];
            ld4(region + at * kRegionX * kRegionY + Q.cell[n], v);
            Q.store(a.lam_in[s], n, v);
        }
    sums[0] = gd;
    sums[kTileThreads] = ge;
    for (int v = 0; v < 2 * T; ++v) sums[(2 + v) * kTileThreads] = by_type[v * kTileThreads];
}

// Gradient blockIdx.x from every thread's sums: thread i adds thread i's (and
// i + kThreads's) of each of its species' tiles in order, then the block's
// threads are summed.
__global__ void __launch_bounds__(kThreads) tile_gradients(const double *__restrict__ sums, int tiles, int n_species,
                                                           int n_types, double *__restrict__ grads) {
    __shared__ double scratch[kWarps];
    grid_wait();
    // gradient layout: d, e per species, then sec, upt per (type, species);
    // a species' values: d, e, then (sec, upt) by type
    const int S = n_species, g = (int)blockIdx.x, values = 2 + 2 * n_types;
    int s = g % S, v = g / S;
    if (g >= 2 * S) {
        const int i = g - 2 * S, table = i / (n_types * S), t = (i - table * n_types * S) / S;
        v = 2 + 2 * t + table;
    }
    const double *p = sums + ((size_t)s * tiles * values + v) * kTileThreads;
    const size_t stride = (size_t)values * kTileThreads;
    double total = 0.0;
    for (int i = (int)threadIdx.x; i < kTileThreads; i += kThreads) {
#pragma unroll 8
        for (int b = 0; b < tiles; ++b) total += p[(size_t)b * stride + i];
    }
    total = block_sum(total, scratch);
    if (threadIdx.x == 0) grads[g] = total;
}

// grads[k] = the sum over blocks of partial[b][k], one warp per k: lane l
// adds rows l, l + 32, ... in order, then the warp's lanes are summed by the
// fixed shuffle tree, so the order depends on the block count alone.
__global__ void __launch_bounds__(kThreads) reduce_partials(const double *__restrict__ partial, int blocks, int n_grads,
                                                            double *__restrict__ grads) {
    grid_wait();
    const int k = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
    if (k >= n_grads) return;  // whole warps leave together
    double v = 0.0;
#pragma unroll 8
    for (int b = lane; b < blocks; b += 32) v += partial[(size_t)b * n_grads + k];
    v = warp_sum(v);
    if (lane == 0) grads[k] = v;
}

// field.rs:155-160
int substeps(double diffusion, int dimensions) {
    if (diffusion <= 0.0) return 1;
    double k = std::ceil(diffusion / (1.0 / (2.0 * (double)dimensions)));
    return k < 1.0 ? 1 : (int)k;
}

}  // namespace

struct glz_adj {
    Grid g{};
    int n_species = 0, n_types = 0, steps = 0, every = 1;
    cudaStream_t stream = nullptr;
    uint8_t *owner = nullptr;  // steps * sites
    bool have_trajectory = false;
    float *ckpt = nullptr;     // ceil(steps / every) checkpoints of n_species * sites
    float *seg = nullptr;      // a segment's sub-step states: every * (kmax + 1) * n_species * sites
    float *tmp[2] = {};        // n_species * sites each: sub-step outputs inside a step
    float *work[2] = {};       // step outputs between checkpoints
    float *lam[2] = {};        // the adjoint fields
    float *d_sec = nullptr, *d_upt = nullptr;  // d_sec starts the one allocation of the rate tables
    float *staging = nullptr;                  // pinned: the rate tables on their way in
    float *d_de = nullptr;      // per-sub-step d then e per species
    float *final_out = nullptr; // n_species * sites: the forward's last step, copied to the caller
    double *partial = nullptr;  // kBlocks rows of n_grads, or the tile kernels' running sums
    double *d_grads = nullptr;  // n_grads: d, e per species, then sec, upt per (type, species)
    std::vector<double> params;
    std::vector<int> k;
    int kmax = 0;
    int seg_kmax = -1;          // the kmax `seg` was sized for
    bool forward_done = false;
    // The forward and backward sequences as CUDA graphs, captured for the
    // sub-step counts in `graph_k` and replayed for any parameters with them.
    cudaGraphExec_t fwd_exec = nullptr, bwd_exec = nullptr;
    std::vector<int> graph_k;
    int bwd_cur[glz::kMaxSpecies] = {};  // after a backward: which lam buffer holds each species
};

namespace {

size_t field_floats(const glz_adj *h) { return (size_t)h->n_species * h->g.sites; }
int n_grads(const glz_adj *h) { return 2 * h->n_species + 2 * h->n_types * h->n_species; }
// Rows of whole multiples of four sites take the four-site kernels.
bool quads(const glz_adj *h) { return h->g.w % 4 == 0; }
int blocks_for(const glz_adj *h) {
    const long long items = quads(h) ? h->g.sites / 4 : h->g.sites;
    return (int)((items + kThreads - 1) / kThreads);
}

// Planes that take the tile kernels, which pay up to about 1400^2 sites: past
// it the running sums that every launch reads and writes (15 bytes a site of a
// species at four types) no longer stay in L2 beside the fields. Forward and backward, a round a launch and
// in tiles, us, 20 steps of two species: of four types 83 + 220 and 65 + 123
// at 8 x 512, 88 + 224 and 66 + 127 at 16 x 512, 98 + 283 and 77 + 189 at
// 512^2, 178 + 805 and 149 + 607 at 1024^2, 192 + 883 and 181 + 776 at 1100^2,
// 275 + 1198 and 247 + 1169 at 1400^2, 506 + 2143 and 438 + 2303 at 2048^2
// (one species 336 + 1143 and 252 + 1399); of 16 types 98 + 775 and 77 + 283
// at 512^2, 178 + 2623 and 152 + 1059 at 1024^2, 503 + 8395 and 442 + 3990 at
// 2048^2. The line is a size at which both few and many types gain.
// Rows that are not whole quads take them with more than one species or from
// 2^16 sites (510 x 512 of two species, 50 steps, 274 + 1117 and 176 + 514;
// 98 x 96 of two, 30 steps, 115 + 319 and 90 + 243; of one species 101 + 228
// and 89 + 225 at 258 x 256, but 98 + 224 and 89 + 249 at 194 x 200).
bool tile_plane(const glz_adj *h) {
    const bool rows = quads(h) || (h->g.w >= 8 && (h->n_species > 1 || h->g.sites >= (1 << 16)));
    return h->g.dim == 2 && rows && h->n_types <= kTileTypes && h->g.sites <= (1 << 20);
}
// ... when every species' sub-steps fit a launch's rounds.
bool tiled(const glz_adj *h) { return tile_plane(h) && h->kmax <= kHalo; }
int steps_each(const glz_adj *h) { return kHalo / h->kmax; }
dim3 tile_grid(const glz_adj *h) {
    return dim3((unsigned)((h->g.w + kTileX - 1) / kTileX), (unsigned)((h->g.h + kTileY - 1) / kTileY),
                (unsigned)h->n_species);
}
size_t partial_doubles(const glz_adj *h) {
    const size_t rows = (size_t)kBlocks * n_grads(h);
    if (!tile_plane(h)) return rows;
    const dim3 grid = tile_grid(h);
    const size_t sums = (size_t)grid.x * grid.y * grid.z * (2 + 2 * h->n_types) * kTileThreads;
    return sums > rows ? sums : rows;
}

int launch_forward(glz_adj *h, const ForwardRound &a) {
    CU(quads(h) ? launch_after(forward_quads, blocks_for(h), 0, h->stream, a)
                : launch_after(forward_round, blocks_for(h), 0, h->stream, a));
    return GLZ_OK;
}
// the rate tables in one run: sec and upt per (type, species), d and e per species
size_t table_floats(const glz_adj *h) { return (size_t)2 * h->n_types * h->n_species + 2 * h->n_species; }

// The sub-step state j of species s at step `local` of the segment starting
// at checkpoint `sg`: j < k[s] the input of sub-step j, j = k[s] the exchange
// input. State 0 of the segment's first step is the checkpoint itself.
float *seg_state(glz_adj *h, int sg, int local, int j, int s) {
    if (local == 0 && j == 0) return h->ckpt + ((size_t)sg * h->n_species + s) * (size_t)h->g.sites;
    return h->seg + (((size_t)local * (h->kmax + 1) + j) * h->n_species + s) * (size_t)h->g.sites;
}

void drop_graphs(glz_adj *h) {
    if (h->fwd_exec) cudaGraphExecDestroy(h->fwd_exec);
    if (h->bwd_exec) cudaGraphExecDestroy(h->bwd_exec);
    h->fwd_exec = h->bwd_exec = nullptr;
    h->graph_k.clear();
}

int set_params(glz_adj *h, const double *params) {
    const int S = h->n_species, T = h->n_types;
    for (int s = 0; s < S; ++s)
        if (!(params[s] >= 0.0) || !(params[S + s] >= 0.0) || !std::isfinite(params[s]) ||
            !std::isfinite(params[S + s]))
            return fail(GLZ_INVALID, "diffusion and decay must be finite and >= 0");
    h->params.assign(params, params + n_grads(h));
    h->k.resize(S);
    h->kmax = 0;
    for (int s = 0; s < S; ++s) {
        h->k[s] = substeps(params[s], h->g.dim);
        h->kmax = h->k[s] > h->kmax ? h->k[s] : h->kmax;
    }
    // sec, upt, then d and e per species, staged in pinned memory: every
    // forward ends in a stream synchronize, so the previous copy out of the
    // staging has landed before it is written again
    float *sec = h->staging, *upt = sec + T * S, *de = upt + T * S;
    for (int i = 0; i < T * S; ++i) {
        sec[i] = (float)params[2 * S + i];
        upt[i] = (float)params[2 * S + T * S + i];
    }
    for (int sp = 0; sp < S; ++sp) {
        de[sp] = (float)(params[sp] / (double)h->k[sp]);
        de[S + sp] = (float)(params[S + sp] / (double)h->k[sp]);
    }
    CU(cudaMemcpyAsync(h->d_sec, h->staging, table_floats(h) * 4, cudaMemcpyHostToDevice, h->stream));
    if (h->seg_kmax != h->kmax) {
        drop_graphs(h);  // they name the buffer freed here, and outlive it if the new one is refused
        cudaFree(h->seg);
        h->seg = nullptr;
        h->seg_kmax = -1;
        CU(cudaMalloc(&h->seg, (size_t)h->every * (h->kmax + 1) * field_floats(h) * sizeof(float)));
        h->seg_kmax = h->kmax;
    }
    return GLZ_OK;
}

// One step forward of every species, owners of step t, from `in` to `out`
// (n_species * sites each, distinct buffers).
int step_forward(glz_adj *h, int t, const float *in, float *out) {
    const size_t n = h->g.sites;
    ForwardRound a{};
    a.g = h->g;
    a.n_species = h->n_species;
    a.owner = h->owner + (size_t)t * n;
    a.sec = h->d_sec;
    a.upt = h->d_upt;
    a.de = h->d_de;
    const float *cur[glz::kMaxSpecies];
    for (int s = 0; s < h->n_species; ++s) cur[s] = in + (size_t)s * n;
    for (int r = 0; r < h->kmax; ++r) {
        for (int s = 0; s < h->n_species; ++s) {
            Species &p = a.sp[s];
            p.active = r < h->k[s];
            p.last = r == h->k[s] - 1;
            p.in = cur[s];
            p.keep = nullptr;
            p.out = p.last ? out + (size_t)s * n : h->tmp[r & 1] + (size_t)s * n;
            if (p.active) cur[s] = p.out;
        }
        if (int rc = launch_forward(h, a)) return rc;
    }
    return GLZ_OK;
}

// Step `local` of segment `sg` forward, keeping every sub-step state in the
// segment buffers; the output of the segment's last step goes to `last_out`
// (not kept: null).
int keep_step(glz_adj *h, int sg, int local, int len, float *last_out) {
    ForwardRound a{};
    a.g = h->g;
    a.n_species = h->n_species;
    a.sec = h->d_sec;
    a.upt = h->d_upt;
    a.de = h->d_de;
    a.owner = h->owner + (size_t)(sg * h->every + local) * h->g.sites;
    for (int r = 0; r < h->kmax; ++r) {
        for (int s = 0; s < h->n_species; ++s) {
            Species &p = a.sp[s];
            p.active = r < h->k[s];
            p.last = r == h->k[s] - 1;
            if (!p.active) continue;
            p.in = seg_state(h, sg, local, r, s);
            if (p.last) {
                p.keep = seg_state(h, sg, local, h->k[s], s);
                p.out = local + 1 < len ? seg_state(h, sg, local + 1, 0, s)
                                        : (last_out ? last_out + (size_t)s * h->g.sites : nullptr);
            } else {
                p.keep = nullptr;
                p.out = seg_state(h, sg, local, r + 1, s);
            }
        }
        if (int rc = launch_forward(h, a)) return rc;
    }
    return GLZ_OK;
}

// Steps `local` .. `local + n - 1` of segment `sg` in one tile launch, keeping
// every sub-step state as keep_step does; `out` may name where a step's output
// goes besides (the last of the segment, or none).
int tile_keep(glz_adj *h, int sg, int local, int n, int len, float *last_out) {
    TileForward a{};
    a.g = h->g;
    a.n_species = h->n_species;
    a.n_types = h->n_types;
    a.steps = n;
    a.owner = h->owner + (size_t)(sg * h->every + local) * h->g.sites;
    a.sec = h->d_sec;
    a.upt = h->d_upt;
    a.de = h->d_de;
    for (int s = 0; s < h->n_species; ++s) {
        a.k[s] = h->k[s];
        a.in[s] = seg_state(h, sg, local, 0, s);
        for (int i = 0, r = 0; i < n; ++i)
            for (int j = 0; j < h->k[s]; ++j, ++r) {
                const int step = local + i;
                if (j < h->k[s] - 1) {
                    a.post[s][r] = seg_state(h, sg, step, j + 1, s);
                    continue;
                }
                a.keep[s][r] = seg_state(h, sg, step, h->k[s], s);
                a.post[s][r] = step + 1 < len ? seg_state(h, sg, step + 1, 0, s)
                                              : (last_out ? last_out + (size_t)s * h->g.sites : nullptr);
            }
    }
    CU(launch_blocks(quads(h) ? tile_forward<true> : tile_forward<false>, tile_grid(h), kTileThreads, 0, h->stream, a));
    return GLZ_OK;
}

// keep_step for a whole segment.
int keep_segment(glz_adj *h, int sg, int len, float *last_out) {
    if (tiled(h)) {
        for (int local = 0; local < len; local += steps_each(h)) {
            const int n = len - local < steps_each(h) ? len - local : steps_each(h);
            if (int rc = tile_keep(h, sg, local, n, len, last_out)) return rc;
        }
        return GLZ_OK;
    }
    for (int local = 0; local < len; ++local)
        if (int rc = keep_step(h, sg, local, len, last_out)) return rc;
    return GLZ_OK;
}

// Every step forward up to the last segment's first, tile launches of several
// steps each: the checkpoints on the way, and each launch's last output to a
// work buffer when it is no checkpoint.
int tile_forward_to(glz_adj *h, int t_last) {
    const size_t n_all = field_floats(h), sites = h->g.sites;
    const float *cur = h->ckpt;
    for (int t = 0; t < t_last; t += steps_each(h)) {
        const int n = t_last - t < steps_each(h) ? t_last - t : steps_each(h);
        TileForward a{};
        a.g = h->g;
        a.n_species = h->n_species;
        a.n_types = h->n_types;
        a.steps = n;
        a.owner = h->owner + (size_t)t * sites;
        a.sec = h->d_sec;
        a.upt = h->d_upt;
        a.de = h->d_de;
        float *dst = nullptr;
        for (int i = 1; i <= n; ++i) {
            float *to = (t + i) % h->every == 0 ? h->ckpt + (size_t)((t + i) / h->every) * n_all : nullptr;
            if (i == n) {
                if (!to) to = cur == h->work[0] ? h->work[1] : h->work[0];
                dst = to;
            }
            for (int s = 0; to && s < h->n_species; ++s) a.post[s][i * h->k[s] - 1] = to + (size_t)s * sites;
        }
        for (int s = 0; s < h->n_species; ++s) {
            a.k[s] = h->k[s];
            a.in[s] = cur + (size_t)s * sites;
        }
        CU(launch_blocks(quads(h) ? tile_forward<true> : tile_forward<false>, tile_grid(h), kTileThreads, 0, h->stream, a));
        cur = dst;
    }
    return GLZ_OK;
}

// Record what `body` queues on the handle's stream as a graph, instantiated
// into *exec; the capture ends whatever the body returns.
int capture(glz_adj *h, cudaGraphExec_t *exec, int (*body)(glz_adj *)) {
    CU(cudaStreamBeginCapture(h->stream, cudaStreamCaptureModeThreadLocal));
    const int rc = body(h);
    cudaGraph_t graph = nullptr;
    const cudaError_t e = cudaStreamEndCapture(h->stream, &graph);
    if (rc) {
        if (graph) cudaGraphDestroy(graph);
        return rc;
    }
    if (e != cudaSuccess) return fail(GLZ_DRIVER, std::string("adjoint capture: ") + cudaGetErrorString(e));
    const cudaError_t ei = cudaGraphInstantiate(exec, graph, 0);
    cudaGraphDestroy(graph);
    if (ei != cudaSuccess) return fail(GLZ_DRIVER, std::string("adjoint graph: ") + cudaGetErrorString(ei));
    return GLZ_OK;
}

// Every step forward from checkpoint 0: a step's output goes to the next
// checkpoint, to the work buffer the step did not read, or (the last) to
// final_out. The last segment's steps keep their sub-step states as a
// recompute would, so the backward starts without recomputing it.
int forward_sequence(glz_adj *h) {
    const size_t n = field_floats(h);
    const int last = (h->steps - 1) / h->every, t_last = last * h->every;
    const float *cur = h->ckpt;
    if (tiled(h))
        if (int rc = tile_forward_to(h, t_last)) return rc;
    for (int t = tiled(h) ? t_last : 0; t < t_last; ++t) {
        float *dst;
        if ((t + 1) % h->every == 0)
            dst = h->ckpt + (size_t)((t + 1) / h->every) * n;
        else
            dst = cur == h->work[0] ? h->work[1] : h->work[0];
        if (int rc = step_forward(h, t, cur, dst)) return rc;
        cur = dst;
    }
    return keep_segment(h, last, h->steps - t_last, h->final_out);
}

// Let `kernel` take up to `most` bytes of dynamic shared memory, the most any
// handle asks of it: the setting is the kernel's, so a handle that set its own
// need could leave it too low for one launching on another thread.
template <class Kernel>
int allow_smem(Kernel kernel, size_t most) {
    CU(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most));
    return GLZ_OK;
}

// The backward rounds' dynamic shared memory: each warp's (sec, upt) sums by
// type, then the block's gradients.
constexpr size_t round_backward_smem(int n_types, int n_species) {
    return ((size_t)kWarps * 2 * n_types + 2 * n_species + (size_t)2 * n_types * n_species) * sizeof(double);
}

// backward_sequence by tile launches of several steps each.
int tile_backward_sequence(glz_adj *h) {
    const int S = h->n_species;
    int cur = 0;
    TileBackward a{};
    a.g = h->g;
    a.n_species = S;
    a.n_types = h->n_types;
    a.sec = h->d_sec;
    a.upt = h->d_upt;
    a.de = h->d_de;
    a.sums = h->partial;
    a.fresh = 1;
    const dim3 grid = tile_grid(h);
    const size_t smem = tile_backward_smem(h->n_types);
    const auto backward = quads(h) ? tile_backward<true> : tile_backward<false>;
    if (int rc = allow_smem(backward, tile_backward_smem(kTileTypes))) return rc;
    const int nseg = (h->steps + h->every - 1) / h->every;
    for (int sg = nseg - 1; sg >= 0; --sg) {
        const int t0 = sg * h->every, len = (t0 + h->every < h->steps ? t0 + h->every : h->steps) - t0;
        // the forward left the last segment's states in place
        if (sg < nseg - 1)
            if (int rc = keep_segment(h, sg, len, nullptr)) return rc;
        for (int end = len; end > 0; end -= steps_each(h)) {
            const int n = end < steps_each(h) ? end : steps_each(h), local = end - n;
            a.steps = n;
            a.owner = h->owner + (size_t)(t0 + local) * h->g.sites;
            for (int s = 0; s < S; ++s) {
                a.k[s] = h->k[s];
                a.lam[s] = h->lam[cur] + (size_t)s * h->g.sites;
                a.lam_in[s] = h->lam[1 - cur] + (size_t)s * h->g.sites;
                for (int step = end - 1, r = 0; step >= local; --step)
                    for (int j = h->k[s] - 1; j >= 0; --j, ++r) {
                        a.u[s][r] = seg_state(h, sg, step, j, s);
                        a.exch[s][r] = seg_state(h, sg, step, h->k[s], s);
                    }
            }
            CU(launch_blocks(backward, grid, kTileThreads, smem, h->stream, a));
            a.fresh = 0;
            cur = 1 - cur;
        }
    }
    CU(launch_after(tile_gradients, n_grads(h), 0, h->stream, (const double *)h->partial, (int)(grid.x * grid.y), S,
                    h->n_types, h->d_grads));
    for (int s = 0; s < S; ++s) h->bwd_cur[s] = cur;
    return GLZ_OK;
}

// The backward from lam[0] (the loss gradient at the final fields), segment
// by segment from the last: recompute the segment's sub-step states, then
// its rounds backward; the per-block gradient rows summed at the end.
int backward_sequence(glz_adj *h) {
    if (tiled(h)) return tile_backward_sequence(h);
    const int S = h->n_species, T = h->n_types, G = n_grads(h);
    const size_t sites = h->g.sites;
    const int grid = blocks_for(h) < kBlocks ? blocks_for(h) : kBlocks;
    CU(cudaMemsetAsync(h->partial, 0, (size_t)grid * G * 8, h->stream));
    int cur[glz::kMaxSpecies] = {};  // which lam buffer holds each species' adjoint
    BackwardRound a{};
    a.g = h->g;
    a.n_species = S;
    a.n_types = T;
    a.n_grads = G;
    a.sec = h->d_sec;
    a.upt = h->d_upt;
    a.de = h->d_de;
    a.partial = h->partial;
    const size_t smem = round_backward_smem(T, S);
    // owner types held in registers up to 4 or 8 types, else reduced per trip
    auto *backward = !quads(h) ? backward_round
                     : T <= 4  ? backward_quads<4>
                     : T <= 8  ? backward_quads<8>
                               : backward_quads<0>;
    if (int rc = allow_smem(backward, round_backward_smem(kMostTypes, glz::kMaxSpecies))) return rc;
    const int nseg = (h->steps + h->every - 1) / h->every;
    for (int sg = nseg - 1; sg >= 0; --sg) {
        const int t0 = sg * h->every, len = (t0 + h->every < h->steps ? t0 + h->every : h->steps) - t0;
        // the forward left the last segment's states in place
        if (sg < nseg - 1)
            if (int rc = keep_segment(h, sg, len, nullptr)) return rc;
        for (int local = len - 1; local >= 0; --local) {
            a.owner = h->owner + (size_t)(t0 + local) * sites;
            for (int r = h->kmax - 1; r >= 0; --r) {
                for (int s = 0; s < S; ++s) {
                    Adjoint &p = a.sp[s];
                    p.active = r < h->k[s];
                    p.last = r == h->k[s] - 1;
                    if (!p.active) continue;
                    p.u = seg_state(h, sg, local, r, s);
                    p.exch = seg_state(h, sg, local, h->k[s], s);
                    p.lam = h->lam[cur[s]] + (size_t)s * sites;
                    p.lam_in = h->lam[1 - cur[s]] + (size_t)s * sites;
                    cur[s] = 1 - cur[s];
                }
                CU(launch_after(backward, grid, smem, h->stream, a));
            }
        }
        CU(cudaGetLastError());
    }
    CU(launch_after(reduce_partials, (G + kWarps - 1) / kWarps, 0, h->stream, (const double *)h->partial, grid, G,
                     h->d_grads));
    for (int s = 0; s < S; ++s) h->bwd_cur[s] = cur[s];
    return GLZ_OK;
}

}  // namespace

extern "C" {

int glz_adj_create(int width, int height, int depth, int n_species, int n_types, int steps, int checkpoint_every,
                   glz_adj **out) {
    if (!out) return fail(GLZ_INVALID, "null output handle");
    *out = nullptr;
    if (width <= 0 || height <= 0 || depth <= 0) return fail(GLZ_INVALID, "the lattice has a zero dimension");
    if (n_species < 1 || n_species > glz::kMaxSpecies || n_types < 1 || n_types > kMostTypes || steps < 1 ||
        checkpoint_every < 1)
        return fail(GLZ_INVALID, "species 1..8, types 1..254, steps and checkpoint interval >= 1");
    const long long sites = (long long)width * height * depth;
    if (sites >= (1LL << 31)) return fail(GLZ_INVALID, "the lattice has 2^31 sites or more");
    glz_adj *h = new glz_adj();
    h->g = Grid{width, height, depth, depth > 1 ? 3 : 2, (int)sites, glz::make_divider((uint32_t)width),
                glz::make_divider((uint32_t)height)};
    h->n_species = n_species;
    h->n_types = n_types;
    h->steps = steps;
    h->every = checkpoint_every < steps ? checkpoint_every : steps;
    const size_t n = field_floats(h);
    const int nckpt = (steps + h->every - 1) / h->every;
    auto bail = [&](int rc) {
        glz_adj_destroy(h);
        return rc;
    };
    if (cudaStreamCreateWithFlags(&h->stream, cudaStreamNonBlocking) != cudaSuccess ||
        cudaMalloc(&h->owner, (size_t)steps * sites) != cudaSuccess ||
        cudaMalloc(&h->ckpt, (size_t)nckpt * n * sizeof(float)) != cudaSuccess ||
        cudaMalloc(&h->tmp[0], n * sizeof(float)) != cudaSuccess ||
        cudaMalloc(&h->tmp[1], n * sizeof(float)) != cudaSuccess ||
        cudaMalloc(&h->work[0], n * sizeof(float)) != cudaSuccess ||
        cudaMalloc(&h->work[1], n * sizeof(float)) != cudaSuccess ||
        cudaMalloc(&h->lam[0], n * sizeof(float)) != cudaSuccess ||
        cudaMalloc(&h->lam[1], n * sizeof(float)) != cudaSuccess ||
        cudaMalloc(&h->d_sec, table_floats(h) * 4) != cudaSuccess ||
        cudaMallocHost(&h->staging, table_floats(h) * 4) != cudaSuccess ||
        cudaMalloc(&h->final_out, n * sizeof(float)) != cudaSuccess ||
        cudaMalloc(&h->partial, partial_doubles(h) * 8) != cudaSuccess ||
        cudaMalloc(&h->d_grads, (size_t)n_grads(h) * 8) != cudaSuccess)
        return bail(fail(GLZ_DRIVER, "adjoint allocation failed"));
    h->d_upt = h->d_sec + (size_t)n_types * n_species;
    h->d_de = h->d_upt + (size_t)n_types * n_species;
    *out = h;
    return GLZ_OK;
}

int glz_adj_set_trajectory(glz_adj *h, const uint8_t *owner_types) {
    if (!h || !owner_types) return fail(GLZ_INVALID, "null handle or trajectory");
    const size_t bytes = (size_t)h->steps * h->g.sites;
    for (size_t i = 0; i < bytes; ++i)
        if (owner_types[i] != kMedium && owner_types[i] >= h->n_types)
            return fail(GLZ_INVALID, "an owner type past the type count (255 is the medium)");
    CU(cudaMemcpyAsync(h->owner, owner_types, bytes, cudaMemcpyHostToDevice, h->stream));
    CU(cudaStreamSynchronize(h->stream));
    h->have_trajectory = true;
    h->forward_done = false;
    return GLZ_OK;
}

int glz_adj_forward(glz_adj *h, const double *params, const float *fields0, float *fields_final) {
    if (!h || !params || !fields0 || !fields_final) return fail(GLZ_INVALID, "null argument");
    if (!h->have_trajectory) return fail(GLZ_INVALID, "no trajectory set");
    if (fields0 == fields_final) return fail(GLZ_INVALID, "the initial and final fields share a buffer");
    h->forward_done = false;
    if (int rc = set_params(h, params)) return rc;
    // the graphs hold the sub-step structure (and the segment buffers sized
    // for it): new sub-step counts take new graphs
    if (h->graph_k != h->k) drop_graphs(h);
    if (!h->fwd_exec) {
        if (int rc = capture(h, &h->fwd_exec, forward_sequence)) return rc;
        h->graph_k = h->k;
    }
    const size_t n = field_floats(h);
    CU(cudaMemcpyAsync(h->ckpt, fields0, n * 4, cudaMemcpyDeviceToDevice, h->stream));  // checkpoint 0
    CU(cudaGraphLaunch(h->fwd_exec, h->stream));
    CU(cudaMemcpyAsync(fields_final, h->final_out, n * 4, cudaMemcpyDeviceToDevice, h->stream));
    CU(cudaStreamSynchronize(h->stream));
    h->forward_done = true;
    return GLZ_OK;
}

int glz_adj_backward(glz_adj *h, const float *grad_final, double *grad_params, float *grad_fields0) {
    if (!h || !grad_final || !grad_params) return fail(GLZ_INVALID, "null argument");
    if (!h->forward_done) return fail(GLZ_INVALID, "backward before forward");
    const int S = h->n_species, G = n_grads(h);
    const size_t n = field_floats(h), sites = h->g.sites;
    if (!h->bwd_exec)
        if (int rc = capture(h, &h->bwd_exec, backward_sequence)) return rc;
    CU(cudaMemcpyAsync(h->lam[0], grad_final, n * 4, cudaMemcpyDeviceToDevice, h->stream));
    CU(cudaGraphLaunch(h->bwd_exec, h->stream));
    if (grad_fields0)
        for (int s = 0; s < S; ++s)
            CU(cudaMemcpyAsync(grad_fields0 + (size_t)s * sites, h->lam[h->bwd_cur[s]] + (size_t)s * sites, sites * 4,
                               cudaMemcpyDeviceToDevice, h->stream));
    std::vector<double> g(G);
    CU(cudaMemcpyAsync(g.data(), h->d_grads, (size_t)G * 8, cudaMemcpyDeviceToHost, h->stream));
    CU(cudaStreamSynchronize(h->stream));
    // d = D / k and e = decay / k, so the D and decay gradients are the
    // per-sub-step ones over k
    for (int s = 0; s < S; ++s) {
        grad_params[s] = g[s] / h->k[s];
        grad_params[S + s] = g[S + s] / h->k[s];
    }
    for (int i = 2 * S; i < G; ++i) grad_params[i] = g[i];
    return GLZ_OK;
}

void *glz_adj_stream(glz_adj *h) { return h ? (void *)h->stream : nullptr; }

void glz_adj_destroy(glz_adj *h) {
    if (!h) return;
    if (h->stream) cudaStreamSynchronize(h->stream);
    drop_graphs(h);
    cudaFree(h->final_out);
    cudaFree(h->owner);
    cudaFree(h->ckpt);
    cudaFree(h->seg);
    cudaFree(h->tmp[0]);
    cudaFree(h->tmp[1]);
    cudaFree(h->work[0]);
    cudaFree(h->work[1]);
    cudaFree(h->lam[0]);
    cudaFree(h->lam[1]);
    cudaFree(h->d_sec);
    cudaFreeHost(h->staging);
    cudaFree(h->partial);
    cudaFree(h->d_grads);
    if (h->stream) cudaStreamDestroy(h->stream);
    delete h;
}

}  // extern "C"
