// The chemical-field step: FTCS diffusion and decay, with secretion and
// uptake by the cell that owns each site folded into each species' last
// sub-step.
//
// Replaces `field_diffuse` and `field_exchange` (glazier-cuda/src/lib.rs
// 314-363) and their driver `run_fields` (lib.rs:1147-1189). One launch runs
// one sub-step round for every species that still has a sub-step left, so a
// model whose species all take one sub-step (the common case) reads its
// labels and every species once per Monte Carlo step:
//   out = u + d (sum of faces - faces u) - decay u          (field.rs:110-130)
//   on owned sites: v = out + sec; v -= upt v; v = max(v, 0) (field.rs:133-149)
// With an infection rule set (glz_gpu_set_infection, an extension), the
// uptake upt v of the rule's species by cells of the rule's type is summed
// per cell in fixed point, and the step's per-label kernel (population.cu)
// switches the cells whose sum has reached the threshold.
// Exchange reads only its own species, so running it right after that
// species' last sub-step is the reference's order.

#include "device.cuh"
#include "engine.h"
#include "pdl.cuh"

namespace glz {

// Add each lane's `amount` into dose[label] through the first lane of each
// run of equal labels in the warp: one atomic per run. Every lane of the warp
// takes part; a lane with nothing to add passes label kNoDose.
constexpr uint32_t kNoDose = 0xffffffffu;

__device__ __forceinline__ void add_dose(unsigned long long *dose, uint32_t label, long long amount) {
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const uint32_t before = __shfl_up_sync(full, label, 1);
    const bool head = lane == 0 || label != before;
    const unsigned heads = __ballot_sync(full, head);
    long long scan = amount;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const long long v = __shfl_up_sync(full, scan, o);
        if (lane >= o) scan += v;
    }
    const unsigned later = heads & ~(full >> (31 - lane));
    const int last = later ? __ffs(later) - 2 : 31;
    const long long scan_last = __shfl_sync(full, scan, last);
    if (head && label != kNoDose) {
        const long long run = scan_last - scan + amount;
        if (run != 0) atomicAdd(&dose[label], (unsigned long long)run);
    }
}

template <int DIM>
__global__ void __launch_bounds__(256) field_round_kernel(const __grid_constant__ FieldLaunch a) {
    grid_wait();
    const int W = a.g.w, H = a.g.h, D = a.g.d;
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    const bool in = i < (size_t)a.g.sites;
    // with an infection rule every lane stays for the warp's dose sums
    if (!in && a.infect_species < 0) return;
    const size_t c = in ? i : 0;
    // fewer than 2^31 sites: 32-bit quotients by the geometry's dividers
    const uint32_t qw = udiv(a.g.div_w, (uint32_t)c), plane = udiv(a.g.div_h, qw);
    const int x = (int)((uint32_t)c - qw * (uint32_t)W);
    const int y = (int)(qw - plane * (uint32_t)H);
    const int z = DIM == 3 ? (int)plane : 0;
    const size_t row = ((size_t)z * H + y) * W;
    const size_t xm = row + (x == 0 ? W - 1 : x - 1);
    const size_t xp = row + (x == W - 1 ? 0 : x + 1);
    const size_t ym = ((size_t)z * H + (y == 0 ? H - 1 : y - 1)) * W + x;
    const size_t yp = ((size_t)z * H + (y == H - 1 ? 0 : y + 1)) * W + x;
    size_t zm = 0, zp = 0;
    if (DIM == 3) {
        zm = ((size_t)(z == 0 ? D - 1 : z - 1) * H + y) * W + x;
        zp = ((size_t)(z == D - 1 ? 0 : z + 1) * H + y) * W + x;
    }
    const float faces = DIM == 3 ? 6.0f : 4.0f;
    int type = -1;
    uint32_t label = 0;
    const unsigned cur = a.clock ? a.clock->field_cur : a.field_cur;
    for (int s = 0; s < a.n_species; ++s) {
        if (!a.active[s]) continue;
        long long taken = 0;  // this site's uptake of the infection species, fixed point
        // a species active in this round has flipped once a round before it
        const unsigned from = ((cur >> s) & 1u) ^ ((unsigned)a.round & 1u);
        float *const out = a.field_buf + ((size_t)2 * s + (from ^ 1u)) * (size_t)a.g.sites;
        if (in) {
            const float *__restrict__ u = a.field_buf + ((size_t)2 * s + from) * (size_t)a.g.sites;
            const float here = u[i];
            float sum = u[xm];
            sum = __fadd_rn(sum, u[xp]);
            sum = __fadd_rn(sum, u[ym]);
            sum = __fadd_rn(sum, u[yp]);
            if (DIM == 3) {
                sum = __fadd_rn(sum, u[zm]);
                sum = __fadd_rn(sum, u[zp]);
            }
            float v = __fsub_rn(__fadd_rn(here, __fmul_rn(a.d[s], __fsub_rn(sum, __fmul_rn(faces, here)))),
                                __fmul_rn(a.decay[s], here));
            if (a.last[s]) {
                if (type < 0) {
                    label = a.labels[i];
                    type = label == 0 ? 0x7fffffff : a.cell_type[label];
                }
                if (type != 0x7fffffff) {
                    v = __fadd_rn(v, a.secretion[type * a.n_species + s]);
                    const float amount = __fmul_rn(a.uptake[type * a.n_species + s], v);
                    if (s == a.infect_species && type == a.infect_from)
                        taken = __float2ll_rn(__fmul_rn(amount, kDoseScale));
                    v = __fsub_rn(v, amount);
                    v = v < 0.0f ? 0.0f : v;
                }
            }
            out[i] = v;
        }
        if (s == a.infect_species && a.last[s])
            add_dose(a.dose, in && type == a.infect_from ? label : kNoDose, taken);
    }
}

// Lattices whose rows are whole multiples of four sites: a thread takes four
// sites of a row, so its row and the rows across its faces are one 16-byte
// read each and two more reads give the sites past its ends; the labels are
// read beside them, and the rates sit in shared memory. Each site's
// arithmetic is the one-site kernel's, operation for operation. Bound by
// memory where the fields do not fit L2 and by its two round trips where they
// do (whole steps of the two-field tissue, the one-site kernel then this: 214 ->
// 171 us at 2048^2, of which the field was 62 and is about 19). The grid's y takes a species each where a lattice
// has too few sites to fill the device with them one after another.
constexpr int kRateTypes = 16;  // rates of up to this many types are held in shared memory

__device__ __forceinline__ void four(const float *p, float v[4]) {
    const float4 t = *reinterpret_cast<const float4 *>(p);
    v[0] = t.x;
    v[1] = t.y;
    v[2] = t.z;
    v[3] = t.w;
}

template <int DIM>
__global__ void __launch_bounds__(128) field_quads_kernel(const __grid_constant__ FieldLaunch a) {
    __shared__ float rates[2][kRateTypes * kMaxSpecies];
    const bool held = a.n_types <= kRateTypes;
    if (held)
        for (int k = threadIdx.x; k < a.n_types * a.n_species; k += blockDim.x) {
            rates[0][k] = a.secretion[k];
            rates[1][k] = a.uptake[k];
        }
    const float *const secretion = held ? rates[0] : a.secretion, *const uptake = held ? rates[1] : a.uptake;
    const uint32_t q = blockIdx.x * blockDim.x + threadIdx.x;
    const bool in = q < (uint32_t)a.g.sites / 4u;
    const uint32_t c = in ? 4u * q : 0u;
    const uint32_t W = (uint32_t)a.g.w, H = (uint32_t)a.g.h, D = (uint32_t)a.g.d;
    const uint32_t r = udiv(a.g.div_w, c), z = DIM == 3 ? udiv(a.g.div_h, r) : 0u, y = r - z * H, x = c - r * W;
    const uint32_t row = c - x, plane = W * H;
    const uint32_t left = row + (x == 0 ? W - 1 : x - 1), right = row + (x + 4 == W ? 0 : x + 4);
    const uint32_t ym = y == 0 ? c + (H - 1) * W : c - W, yp = y == H - 1 ? c - (H - 1) * W : c + W;
    const uint32_t zm = DIM == 3 ? (z == 0 ? c + (D - 1) * plane : c - plane) : 0u;
    const uint32_t zp = DIM == 3 ? (z == D - 1 ? c - (D - 1) * plane : c + plane) : 0u;
    const float faces = DIM == 3 ? 6.0f : 4.0f;
    __syncthreads();
    grid_wait();
    uint32_t label[4] = {0u, 0u, 0u, 0u};
    int type[4];
    bool have = false;
    const unsigned cur = a.clock ? a.clock->field_cur : a.field_cur;
    for (int s = (int)blockIdx.y; s < a.n_species; s += (int)gridDim.y) {
        if (!a.active[s]) continue;
        // a species active in this round has flipped once a round before it
        const unsigned from = ((cur >> s) & 1u) ^ ((unsigned)a.round & 1u);
        const float *__restrict__ u = a.field_buf + ((size_t)2 * s + from) * (size_t)a.g.sites;
        float *const out = a.field_buf + ((size_t)2 * s + (from ^ 1u)) * (size_t)a.g.sites;
        float h[4] = {}, f0[4] = {}, f1[4] = {}, f2[4] = {}, f3[4] = {}, v[4] = {}, ul = 0.0f, ur = 0.0f;
        if (in) {
            four(u + c, h);
            four(u + ym, f0);
            four(u + yp, f1);
            ul = u[left];
            ur = u[right];
            if (DIM == 3) {
                four(u + zm, f2);
                four(u + zp, f3);
            }
        }
        if (a.last[s] && !have) {
            have = true;
            if (in) {
                const uint4 l = *reinterpret_cast<const uint4 *>(a.labels + c);
                label[0] = l.x;
                label[1] = l.y;
                label[2] = l.z;
                label[3] = l.w;
            }
#pragma unroll
            for (int k = 0; k < 4; ++k) type[k] = label[k] != 0 ? (int)a.cell_type[label[k]] : -1;
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            float sum = __fadd_rn(k == 0 ? ul : h[k - 1], k == 3 ? ur : h[k + 1]);
            sum = __fadd_rn(sum, f0[k]);
            sum = __fadd_rn(sum, f1[k]);
            if (DIM == 3) {
                sum = __fadd_rn(sum, f2[k]);
                sum = __fadd_rn(sum, f3[k]);
            }
            v[k] = __fsub_rn(__fadd_rn(h[k], __fmul_rn(a.d[s], __fsub_rn(sum, __fmul_rn(faces, h[k])))),
                             __fmul_rn(a.decay[s], h[k]));
        }
        if (a.last[s]) {
            const bool doses = s == a.infect_species;
            long long taken[4] = {0, 0, 0, 0};
#pragma unroll
            for (int k = 0; k < 4; ++k)
                if (type[k] >= 0) {
                    v[k] = __fadd_rn(v[k], secretion[type[k] * a.n_species + s]);
                    const float amount = __fmul_rn(uptake[type[k] * a.n_species + s], v[k]);
                    if (doses && type[k] == a.infect_from) taken[k] = __float2ll_rn(__fmul_rn(amount, kDoseScale));
                    v[k] = __fsub_rn(v[k], amount);
                    v[k] = v[k] < 0.0f ? 0.0f : v[k];
                }
            if (doses) {
                // the sites that share the fourth's label in one sum, which
                // neighbouring threads join; the others each on their own
                long long joined = 0;
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    if (label[k] == label[3])
                        joined += taken[k];
                    else if (taken[k] != 0)
                        atomicAdd(&a.dose[label[k]], (unsigned long long)taken[k]);
                }
                add_dose(a.dose, in && type[3] >= 0 && type[3] == a.infect_from ? label[3] : kNoDose, joined);
            }
        }
        if (in) *reinterpret_cast<float4 *>(out + c) = make_float4(v[0], v[1], v[2], v[3]);
    }
}

cudaError_t launch_field_round(const FieldLaunch &a, cudaStream_t stream) {
    if (a.g.w % 4 == 0) {
        const int blocks = (a.g.sites / 4 + 127) / 128;
        const dim3 grid((unsigned)blocks, (unsigned)(a.g.sites <= (1 << 20) ? a.n_species : 1));
        return launch_after(a.g.dim == 2 ? field_quads_kernel<2> : field_quads_kernel<3>, grid, 128, stream, a);
    }
    const int blocks = (a.g.sites + 255) / 256;
    return launch_after(a.g.dim == 2 ? field_round_kernel<2> : field_round_kernel<3>, dim3((unsigned)blocks), 256, stream,
                        a);
}

}  // namespace glz
