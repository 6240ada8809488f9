// gc_pack.cuh — one particle's FP32 sweep record (the layouts of rec_quads and
// pos_quads in gc_force.h), shared by the pack kernel and the fused half step.
#pragma once

#include "gc_force.h"
#include "gc_update.h"

namespace gc {

// One record of ND dimensions in mode MODE (NS stress components for the
// Cauchy functor): with all known at compile time it stays in registers.
template <int ND, int MODE, int NS>
__device__ __forceinline__ void pack_rec(const PackArgs& a, int64_t g, const float* h, const float* l) {
    const int64_t N = a.N;
    constexpr int RQ = rec_quads(ND, MODE);
    const double r = a.rho[g];
    float v[ND];
#pragma unroll
    for (int d = 0; d < ND; ++d) v[d] = (float)a.v[d * N + g];
    float w0, w1, w2 = 0.f;
    if (MODE == AUX_P_OVER_RHO2) {
        w0 = a.p ? (float)(-(a.p[g] / (r * r))) : 0.f;  // boundaries may have no pressure
        w1 = (float)(1.0 / r);
        w2 = (float)r;
    } else if (MODE == AUX_MASS_OVER_RHO) {
        w0 = (float)(a.mass[a.inst_of[g]] / r);
        w1 = 0.f;
    } else {
        w0 = (float)(1.0 / r);
        w1 = (float)r;
    }
    float s[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    if (MODE == AUX_INV_RHO2 && a.stress) {
        const double i2 = 1.0 / (r * r);
#pragma unroll
        for (int q = 0; q < NS; ++q) s[q] = (float)(a.stress[q * N + g] * i2);
    }
    float4* o = a.rec + g * RQ;
    if (ND == 2) {
        o[0] = make_float4(h[0], h[1], l[0], l[1]);
        o[1] = make_float4(v[0], v[1], w0, w1);
        if (MODE == AUX_P_OVER_RHO2) o[2] = make_float4(w2, 0.f, 0.f, 0.f);
        if (MODE == AUX_INV_RHO2) o[2] = make_float4(s[0], s[1], s[NS == 3 ? 2 : 3], 0.f);
    } else {
        o[0] = make_float4(h[0], h[1], h[ND - 1], w0);
        o[1] = make_float4(l[0], l[1], l[ND - 1], w1);
        o[2] = make_float4(v[0], v[1], v[ND - 1], MODE == AUX_INV_RHO2 ? s[0] : w2);
        if (MODE == AUX_INV_RHO2) {
            o[3] = make_float4(s[1], s[2], s[3], s[4]);
            o[4] = make_float4(s[5], 0.f, 0.f, 0.f);
        }
    }
}

__device__ __forceinline__ void pack_one(const PackArgs& a, int64_t g) {
    const int64_t N = a.N;
    float h[MAXD], l[MAXD];
#pragma unroll
    for (int d = 0; d < MAXD; ++d) {
        const double x = d < a.nd ? a.x[d * N + g] : 0.0;
        h[d] = (float)x;
        l[d] = (float)(x - (double)h[d]);
    }
#pragma unroll
    for (int d = 0; d < MAXD; ++d)
        if (d < a.nd) a.hpos[d * N + g] = h[d];
    if (a.pos) {
        float4* o = a.pos + g * pos_quads(a.nd);
        if (a.nd == 2) {
            o[0] = make_float4(h[0], h[1], l[0], l[1]);
        } else {
            o[0] = make_float4(h[0], h[1], h[2], 0.f);
            o[1] = make_float4(l[0], l[1], l[2], 0.f);
        }
    }
    if (!a.rec) return;
    // (other shapes of stress have no sweep: the launch refuses them)
    if (a.nd == 3) {
        if (a.mode == AUX_P_OVER_RHO2) pack_rec<3, AUX_P_OVER_RHO2, 0>(a, g, h, l);
        else if (a.mode == AUX_MASS_OVER_RHO) pack_rec<3, AUX_MASS_OVER_RHO, 0>(a, g, h, l);
        else if (a.ns == 6) pack_rec<3, AUX_INV_RHO2, 6>(a, g, h, l);
    } else {
        if (a.mode == AUX_P_OVER_RHO2) pack_rec<2, AUX_P_OVER_RHO2, 0>(a, g, h, l);
        else if (a.mode == AUX_MASS_OVER_RHO) pack_rec<2, AUX_MASS_OVER_RHO, 0>(a, g, h, l);
        else if (a.ns == 3) pack_rec<2, AUX_INV_RHO2, 3>(a, g, h, l);
        else if (a.ns == 4) pack_rec<2, AUX_INV_RHO2, 4>(a, g, h, l);
    }
}

}  // namespace gc
