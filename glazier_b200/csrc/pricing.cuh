// Pricing pieces shared by the sweep kernels (sweep.cu, band.cu): the
// volume and surface energy terms, and the shared-memory address helper.
#pragma once

#include <cstdint>

#include "engine.h"

namespace glz {

// Shared memory for the tables of up to kSmemTypes types. A launch's tables
// are few bytes read by every copy, each behind the one before it (a type's
// weight, then its target): read where they lie they cost a cold kernel a
// chain of up to eight L2 round trips.
template <bool EXTRAS>
struct alignas(8) TypeSmem {
    unsigned char bytes[EXTRAS ? TypeLayout(kSmemTypes, kMaxSpecies).bytes : TypeLayout(kSmemTypes, 0).lean];
};

// Copy the launch's tables in (all of the block's threads; the caller's next
// block barrier publishes them) and give where to read them. Reads nothing a
// pass writes, so it may come before a programmatic wait.
template <bool EXTRAS>
__device__ __forceinline__ TypeTables load_types(const SweepLaunch &a, TypeSmem<EXTRAS> &S) {
    TypeTables t = a.t;
    if (a.n_types > kSmemTypes) return t;
    const TypeLayout L(a.n_types, a.n_species);
    const uint32_t *src = reinterpret_cast<const uint32_t *>(a.t.contact);
    uint32_t *dst = reinterpret_cast<uint32_t *>(S.bytes);
    for (int i = threadIdx.x; i < (EXTRAS ? L.bytes : L.lean) / 4; i += blockDim.x) dst[i] = src[i];
    t.contact = reinterpret_cast<const float *>(S.bytes + L.contact);
    t.target_volume = reinterpret_cast<const float *>(S.bytes + L.target_volume);
    t.lambda_volume = reinterpret_cast<const float *>(S.bytes + L.lambda_volume);
    t.target_surface = reinterpret_cast<const float *>(S.bytes + L.target_surface);
    t.lambda_surface = reinterpret_cast<const float *>(S.bytes + L.lambda_surface);
    if (EXTRAS) {
        t.target_length = reinterpret_cast<const double *>(S.bytes + L.target_length);
        t.lambda_length = reinterpret_cast<const double *>(S.bytes + L.lambda_length);
        t.lambda_nematic = reinterpret_cast<const double *>(S.bytes + L.lambda_nematic);
        t.max_activity = reinterpret_cast<const float *>(S.bytes + L.max_activity);
        t.lambda_activity = reinterpret_cast<const float *>(S.bytes + L.lambda_activity);
        t.external = reinterpret_cast<const float *>(S.bytes + L.external);
        t.chemotaxis = reinterpret_cast<const float *>(S.bytes + L.chemotaxis);
        t.connected = S.bytes + L.connected;
    }
    return t;
}

__device__ __forceinline__ uint32_t smem_addr(const void *p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// The volume and surface parts of a copy's energy change, added to `delta`
// in a fixed order (old cell's volume, new cell's volume, old cell's
// surface, new cell's surface), correctly rounded f32 throughout so a host
// replay gets the same bits; the medium (label 0) has neither term.
//   volume:  lambda ((v -/+ 1 - V_t)^2 - (v - V_t)^2) = lambda (1 -/+ 2 (v - V_t))
//   surface: lambda ((s + ds - S_t)^2 - (s - S_t)^2) = lambda ds (2 (s - S_t) + ds)
template <bool UNIFORM>
__device__ __forceinline__ float size_terms(const SweepLaunch &a, const TypeTables &t, uint32_t old, uint32_t nw, int t_old, int t_new,
                                            int vol_old, int vol_new, int surf_old, int surf_new, int ds_old,
                                            int ds_new, float delta) {
    // Every term is formed, so that their reads and products overlap, and the
    // medium's side is left out at its add. A type whose weight is zero has a
    // zero target in the tables (weighted_target), so its term is a zero,
    // which leaves the sum's bits alone. A weight of zero for the medium, or
    // targets as the model states them, would not do: where a target is not
    // finite, or not in f32, 0 * inf is no zero. (Selecting between the term
    // and a zero instead costs 1112 against 1102 us for 10 MCS at 4096^2.)
    const float lv_old = UNIFORM ? a.u_lambda_volume : t.lambda_volume[t_old];
    const float lv_new = UNIFORM ? a.u_lambda_volume : t.lambda_volume[t_new];
    const float ls_old = UNIFORM ? a.u_lambda_surface : t.lambda_surface[t_old];
    const float ls_new = UNIFORM ? a.u_lambda_surface : t.lambda_surface[t_new];
    const float ev_old = __fsub_rn((float)vol_old, UNIFORM ? a.u_target_volume : t.target_volume[t_old]);
    const float ev_new = __fsub_rn((float)vol_new, UNIFORM ? a.u_target_volume : t.target_volume[t_new]);
    const float es_old = __fsub_rn((float)surf_old, UNIFORM ? a.u_target_surface : t.target_surface[t_old]);
    const float es_new = __fsub_rn((float)surf_new, UNIFORM ? a.u_target_surface : t.target_surface[t_new]);
    const float d_old = (float)ds_old, d_new = (float)ds_new;
    const float v_old = __fmul_rn(lv_old, __fsub_rn(1.0f, __fmul_rn(2.0f, ev_old)));
    const float v_new = __fmul_rn(lv_new, __fadd_rn(__fmul_rn(2.0f, ev_new), 1.0f));
    const float s_old = __fmul_rn(ls_old, __fmul_rn(d_old, __fadd_rn(__fmul_rn(2.0f, es_old), d_old)));
    const float s_new = __fmul_rn(ls_new, __fmul_rn(d_new, __fadd_rn(__fmul_rn(2.0f, es_new), d_new)));
    if (old != 0) delta = __fadd_rn(delta, v_old);
    if (nw != 0) delta = __fadd_rn(delta, v_new);
    if (old != 0) delta = __fadd_rn(delta, s_old);
    if (nw != 0) delta = __fadd_rn(delta, s_new);
    return delta;
}

}  // namespace glz
