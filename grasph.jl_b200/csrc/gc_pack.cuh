// gc_pack.cuh — one particle's sweep record (the layouts of rec_quads and
// pos_quads in gc_force.h), shared by the pack kernel and the fused half step.
#pragma once

#include "gc_force.h"
#include "gc_update.h"

namespace gc {

__device__ __forceinline__ float4 quad_of(double a, double b) {
    return make_float4(__int_as_float(__double2loint(a)), __int_as_float(__double2hiint(a)),
                       __int_as_float(__double2loint(b)), __int_as_float(__double2hiint(b)));
}

// One record of ND dimensions in mode MODE (NS stress components for the
// Cauchy functor): with all known at compile time it stays in registers.
template <int ND, int MODE, int NS>
__device__ __forceinline__ void pack_rec(const PackArgs& a, int64_t g, const double* x, const float* h,
                                         const float* l) {
    const int64_t N = a.N;
    const double r = a.rho[g];
    double v[ND];
#pragma unroll
    for (int d = 0; d < ND; ++d) v[d] = a.v[d * N + g];
    double w0, w1, w2 = 0.0, w3 = 0.0;
    if (MODE == AUX_P_OVER_RHO2) {
        w3 = a.p ? a.p[g] : 0.0;  // boundaries may have no pressure
        w0 = -(w3 / (r * r));
        w1 = 1.0 / r;
        w2 = r;
    } else if (MODE == AUX_MASS_OVER_RHO) {
        w0 = a.mass[a.inst_of[g]] / r;
        w1 = 0.0;
    } else {
        w0 = 1.0 / r;
        w1 = r;
    }
    double s[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
    if (MODE == AUX_INV_RHO2 && a.stress) {
        const double i2 = 1.0 / (r * r);
#pragma unroll
        for (int q = 0; q < NS; ++q) s[q] = a.stress[q * N + g] * i2;
    }
    const double sxy = s[NS == 3 ? 2 : 3];  // 2-D
    if (!a.fp32) {
        float4* o = a.rec + g * rec_quads(ND, MODE, false);
        if (ND == 2) {
            o[0] = quad_of(x[0], x[1]);
            o[1] = quad_of(v[0], v[1]);
        } else {
            o[0] = quad_of(x[0], x[1]);
            o[1] = quad_of(x[ND - 1], v[0]);
            o[2] = quad_of(v[1], v[ND - 1]);
        }
        o[ND] = quad_of(w0, w1);
        if (MODE == AUX_P_OVER_RHO2) o[ND + 1] = quad_of(w2, w3);
        if (MODE == AUX_INV_RHO2) {
            o[ND + 1] = quad_of(s[0], s[1]);
            o[ND + 2] = ND == 2 ? quad_of(sxy, 0.0) : quad_of(s[2], s[3]);
            if (ND == 3) o[ND + 3] = quad_of(s[4], s[5]);
        }
        return;
    }
    float4* o = a.rec + g * rec_quads(ND, MODE, true);
    const float f0 = (float)w0, f1 = (float)w1;
    if (ND == 2) {
        o[0] = make_float4(h[0], h[1], l[0], l[1]);
        o[1] = make_float4((float)v[0], (float)v[1], f0, f1);
        if (MODE == AUX_P_OVER_RHO2) o[2] = make_float4((float)w2, 0.f, 0.f, 0.f);
        if (MODE == AUX_INV_RHO2) o[2] = make_float4((float)s[0], (float)s[1], (float)sxy, 0.f);
    } else {
        o[0] = make_float4(h[0], h[1], h[ND - 1], f0);
        o[1] = make_float4(l[0], l[1], l[ND - 1], f1);
        o[2] = make_float4((float)v[0], (float)v[1], (float)v[ND - 1], (float)(MODE == AUX_INV_RHO2 ? s[0] : w2));
        if (MODE == AUX_INV_RHO2) {
            o[3] = make_float4((float)s[1], (float)s[2], (float)s[3], (float)s[4]);
            o[4] = make_float4((float)s[5], 0.f, 0.f, 0.f);
        }
    }
}

__device__ __forceinline__ void pack_one(const PackArgs& a, int64_t g) {
    const int64_t N = a.N;
    double x[MAXD];
    float h[MAXD], l[MAXD];
#pragma unroll
    for (int d = 0; d < MAXD; ++d) {
        x[d] = d < a.nd ? a.x[d * N + g] : 0.0;
        if (a.fp32) x[d] -= a.origin[a.inst_of[g] * MAXD + d];
        h[d] = (float)x[d];
        l[d] = (float)(x[d] - (double)h[d]);
    }
#pragma unroll
    for (int d = 0; d < MAXD; ++d)
        if (d < a.nd) a.hpos[d * N + g] = h[d];
    if (a.pos) {
        float4* o = a.pos + g * pos_quads(a.nd, a.fp32);
        if (!a.fp32) {
            o[0] = quad_of(x[0], x[1]);
            if (a.nd == 3) o[1] = quad_of(x[2], 0.0);
        } else if (a.nd == 2) {
            o[0] = make_float4(h[0], h[1], l[0], l[1]);
        } else {
            o[0] = make_float4(h[0], h[1], h[2], 0.f);
            o[1] = make_float4(l[0], l[1], l[2], 0.f);
        }
    }
    if (!a.rec) return;
    // (other shapes of stress have no sweep: the launch refuses them)
    if (a.nd == 3) {
        if (a.mode == AUX_P_OVER_RHO2) pack_rec<3, AUX_P_OVER_RHO2, 0>(a, g, x, h, l);
        else if (a.mode == AUX_MASS_OVER_RHO) pack_rec<3, AUX_MASS_OVER_RHO, 0>(a, g, x, h, l);
        else if (a.ns == 6) pack_rec<3, AUX_INV_RHO2, 6>(a, g, x, h, l);
    } else {
        if (a.mode == AUX_P_OVER_RHO2) pack_rec<2, AUX_P_OVER_RHO2, 0>(a, g, x, h, l);
        else if (a.mode == AUX_MASS_OVER_RHO) pack_rec<2, AUX_MASS_OVER_RHO, 0>(a, g, x, h, l);
        else if (a.ns == 3) pack_rec<2, AUX_INV_RHO2, 3>(a, g, x, h, l);
        else if (a.ns == 4) pack_rec<2, AUX_INV_RHO2, 4>(a, g, x, h, l);
    }
}

}  // namespace gc
