// k_sweep_f32.cuh — the FP32-compensated pair sweep.
//
// The walk is k_force_impl.cuh's (one warp per group of up to 32 consecutive
// particles of one grid column, the union of its lanes' candidates), but a
// warp takes the strips of a whole window at once: the three strips of one
// row of the 3-D stencil, or the whole 2-D stencil.  It copies a chunk of the
// window's candidates (FP32 records, gc_force.h) into shared memory, tests
// them against every lane, and then each lane evaluates its accepted
// candidates from the copies.
//
// What bounds it is instruction issue (65% of the slots, the FMA pipe half
// busy, shared memory half busy), so the walk and the pair term are written
// for few instructions and even lanes:
//   * a window of three strips at once: lanes accept different numbers of a
//     single strip's candidates, and a warp's pair loop runs as long as its
//     busiest lane (on a jittered 3-D lattice at h = 1.2 spacings 119 rounds a
//     group strip by strip, 88 by windows, 55 if all lanes were busy);
//   * positions are FP32 pairs whose difference is the FP64 one rounded to
//     FP32 (a few adds per pair instead of eight FP64 operations and four
//     conversions), and a record is two or three 16-byte quads;
//   * dv·∇W is W'·(dv·dx), so ∇W itself is never formed; the kernel's constant
//     factor multiplies the sums, not the terms;
//   * components go through packed FP32x2 arithmetic;
//   * the interactions in reach are found by one lane each.
// Three-dimensional dam break of a million jittered particles: 894 us a launch
// with strips staged one at a time and FP64 differences, 704-716 us with this
// kernel; 64 batched columns (1.07 M particles) 292 to 226 us; a
// Lennard-Jones box of 18 k particles 72 to 46 us.  Sixteen warps per SM (128
// registers, chunks of 192) beat eighteen to twenty-four at 80-96 registers,
// whose spills cost more than the occupancy gives.
//
// The neighbour sets stay exact: a pair whose FP32 r² lies within a small
// band of the cutoff takes the reference's FP64 test on the FP64 positions
// (and the reference's own strip range), outside the band the FP32 r² cannot
// be wrong about it.
#pragma once
#include <cfloat>

#include "k_force_impl.cuh"

namespace gc {

__device__ __forceinline__ float rsqrt_fast(float x) {
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float rcp_fast(float x) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float2 bc2(float x) { return make_float2(x, x); }
// a - b, exactly rounded (b·(−1) is exact)
__device__ __forceinline__ float2 sub2(float2 a, float2 b) { return __ffma2_rn(b, bc2(-1.0f), a); }

template <int ND>
__device__ __forceinline__ double dot_exact(const double* a, const double* b) {
    double s = __dmul_rn(a[0], b[0]);
#pragma unroll
    for (int d = 1; d < ND; ++d) s = __dadd_rn(s, __dmul_rn(a[d], b[d]));
    return s;
}

template <int ND, int NS, int PFN, int KK>
struct PhysF32 {
    static constexpr int MODE = aux_mode(PFN);
    static constexpr int NQ = rec_quads(ND, MODE), NQP = pos_quads(ND);
    static constexpr bool FLUID = fluid_pfn<PFN>(), CAUCHY = PFN == GC_PFN_CAUCHY_FLUID;
    static constexpr bool VORT = PFN == GC_PFN_STRAIN_RATE_VORTICITY;
    // Stress components a Cauchy term uses, as the record orders them
    static constexpr int NSA = CAUCHY ? (ND == 2 ? 3 : 6) : 1;
    // One particle's record, own or neighbour.
    struct Rec {
        float2 h, l, v;   // x and y components
        float hz, lz, vz;
        float aux, irho, rho;  // aux: −p/ρ² (fluid) or m/ρ (strain rate)
        float a[NSA];
    };
    // quad(q): the record's q-th 16-byte quad; has3 = false leaves the 2-D
    // fluid's third quad unread
    template <class Q>
    static __device__ __forceinline__ void rec_read(const Q& quad, bool has3, Rec& w) {
        const float4 q0 = quad(0), q1 = quad(1);
        w.h = make_float2(q0.x, q0.y);
        if (ND == 2) {
            w.l = make_float2(q0.z, q0.w);
            w.v = make_float2(q1.x, q1.y);
            if (FLUID) {
                w.aux = q1.z;
                w.irho = q1.w;
                w.rho = has3 ? quad(2).x : 0.f;
            } else if (CAUCHY) {
                const float4 q2 = quad(2);
                w.irho = q1.z;
                w.rho = q1.w;
                const float t[3] = {q2.x, q2.y, q2.z};
#pragma unroll
                for (int q = 0; q < NSA && q < 3; ++q) w.a[q] = t[q];
            } else {
                w.aux = q1.z;
            }
        } else {
            const float4 q2 = quad(2);
            w.hz = q0.z;
            w.l = make_float2(q1.x, q1.y);
            w.lz = q1.z;
            w.v = make_float2(q2.x, q2.y);
            w.vz = q2.z;
            if (FLUID) {
                w.aux = q0.w;
                w.irho = q1.w;
                w.rho = q2.w;
            } else if (CAUCHY) {
                const float4 q3 = quad(3), q4 = quad(4);
                w.irho = q0.w;
                w.rho = q1.w;
                const float t[6] = {q2.w, q3.x, q3.y, q3.z, q3.w, q4.x};
#pragma unroll
                for (int q = 0; q < NSA; ++q) w.a[q] = t[q];
            } else {
                w.aux = q0.w;
            }
        }
    }
    // the position's quads alone (a dynamic boundary's record)
    template <class Q>
    static __device__ __forceinline__ void pos_read(const Q& quad, Rec& w) {
        const float4 q0 = quad(0);
        w.h = make_float2(q0.x, q0.y);
        if (ND == 2) {
            w.l = make_float2(q0.z, q0.w);
        } else {
            const float4 q1 = quad(1);
            w.hz = q0.z;
            w.l = make_float2(q1.x, q1.y);
            w.lz = q1.z;
        }
    }

    // The constants of one interaction, folded.
    struct Par {
        float cut, band;  // (2h)², and how near to it the FP64 test decides
        float qs;         // kernel argument's factor
        // the gradient's factor (with the term's mass for dv/dt and dρ/dt), by
        // which the sums are multiplied at the end; a Lennard-Jones wall's terms
        // take it one by one (kq, with kf = 1)
        float kq;
        double kf;
        float eps, am, beta;  // 0.01·h², α·c̄·h, β·h² of the artificial viscosity
        float dd;             // 2·δ·c̄·h of the density diffusion (0: none)
        float ljc;            // 0.01·c² of the Lennard-Jones wall
        int bt;
    };
    static __device__ __forceinline__ Par params(const ForceArgs& A, const InterRef& r, const GridInst& G,
                                                 const PfnInst& P, int k, float xmax) {
        Par p;
        p.bt = r.btype;
        p.cut = (float)G.cutoff_sq;
        // FP32 r² is off by less than 1e-6 of the cutoff's, plus what the
        // FP32 pairs lose of coordinates |x| (2^-48·|x| each)
        p.band = p.cut * (2e-6f + 1e-13f * xmax * (float)G.inv_cell);
        p.qs = G.f_qs;
        p.kf = G.kq;
        const float ca = A.a_cf[k];
        p.eps = p.am = p.beta = p.dd = 0.f;
        p.ljc = 0.01f * ca * ca;
        if (FLUID || CAUCHY) {
            const bool two = PFN == PFN_FLUID2 && P.two;
            const float cb = ((CAUCHY && r.btype == BT_GHOST) || two) ? G.f_bc : ca;
            p.kf *= r.btype == BT_SELF || r.btype == BT_DYNAMIC ? A.a_mass[k] : G.bmass;
            p.eps = P.f_h2eps;
            p.am = P.f_alpha * (0.5f * (ca + cb)) * P.f_h;
            p.beta = P.f_beta * P.f_h * P.f_h;
            if (P.has_delta) p.dd = 2.f * P.f_delta * (two ? 0.5f * (ca + cb) : ca) * P.f_h;
        }
        p.kq = (float)p.kf;
        if ((FLUID || CAUCHY) && r.btype == BT_STATIC) p.kf = 1.0;
        return p;
    }
    // ∇W = kq·kgrad·dx for a pair at r² (ri = 1/r)
    static __device__ __forceinline__ float kgrad(const Par& p, float rr, float ri) {
        const float r = rr * ri;
        if (KK == GC_KERNEL_CUBIC_SPLINE) {
            // −3·(¼(2−q)² − (1−q)²): with s = q/2, −3·((1−s)² − (1−2s)²)
            const float a = fmaf(r, -p.qs, 1.f), b = __saturatef(fmaf(r, -2.f * p.qs, 1.f));
            return ri * fmaf(a, a, -(b * b));
        } else {
            const float a = fmaxf(fmaf(r, -p.qs, 2.f), 0.f);
            return a * a * a;
        }
    }
    static __device__ __forceinline__ float dot(float2 a, float az, float2 b, float bz) {
        float s = a.x * b.x;
        s = fmaf(a.y, b.y, s);
        if (ND == 3) s = fmaf(az, bz, s);
        return s;
    }

    // Running compensated sums of one lane, component pairs together: (x, y)
    // and (z, dρ/dt); or (xx, yy), (xy, yx), (zz, xz), (zx, yz), (zy, -).
    static constexpr int NP = FLUID || CAUCHY || ND == 2 ? 2 : 5;
    struct Acc {
        float2 s[NP], c[NP];  // Kahan: the sum, and minus its rounding error
    };
    static __device__ __forceinline__ void zero(Acc& a) {
#pragma unroll
        for (int q = 0; q < NP; ++q) a.s[q] = a.c[q] = make_float2(0.f, 0.f);
    }
    // sum q += y - (its error so far): y already carries a.c[q]
    static __device__ __forceinline__ void put(Acc& a, int q, float2 y) {
        const float2 t = __fadd2_rn(a.s[q], y);
        a.c[q] = sub2(y, sub2(t, a.s[q]));
        a.s[q] = t;
    }
    // sum q += u·v
    static __device__ __forceinline__ void add(Acc& a, int q, float2 u, float2 v) { put(a, q, __ffma2_rn(u, v, a.c[q])); }
    static __device__ __forceinline__ double total(const Acc& a, int j) {
        const float s = j & 1 ? a.s[j >> 1].y : a.s[j >> 1].x, c = j & 1 ? a.c[j >> 1].y : a.c[j >> 1].x;
        return (double)s + (double)c;
    }
    // The sums, times `f` in FP64, onto system_a's rates.
    static __device__ __forceinline__ void store(const ForceArgs& A, int64_t gi, const Acc& acc, double f) {
        const int64_t N = A.aN;
        // one lane alone adds to a word, in order, so fire-and-forget reductions
        // give the bits of a load, an add and a store without waiting for the load
        auto put = [&](double* to, int q, double x) { atomicAdd(to + q * N + gi, x); };
        auto sum = [&](int j) { return f * total(acc, j < 2 * NP ? j : 0); };
        if (FLUID || CAUCHY) {
            put(A.advdt, 0, sum(0));
            put(A.advdt, 1, sum(1));
            if (ND == 3) put(A.advdt, 2, sum(2));
            put(A.adrhodt, 0, sum(3));
        } else {
            put(A.asr, 0, sum(0));
            put(A.asr, 1, sum(1));
            if (ND == 3) put(A.asr, 2, sum(4));
            put(A.asr, ND == 3 ? 3 : NS == 4 ? 3 : 2, 0.5 * (sum(2) + sum(3)));
            if (ND == 3) {
                put(A.asr, 4, 0.5 * (sum(5) + sum(6)));
                put(A.asr, 5, 0.5 * (sum(7) + sum(8)));
            }
            if (VORT) {
                put(A.avort, 0, 0.5 * (sum(2) - sum(3)));
                if (ND == 3) {
                    put(A.avort, 1, 0.5 * (sum(5) - sum(6)));
                    put(A.avort, 2, 0.5 * (sum(7) - sum(8)));
                }
            }
        }
    }

    // A dynamic boundary's particle as seen from o (src/PairwiseFunctors.jl:53,
    // 111,222,334): mirrored velocity, own density and stress.
    static __device__ __forceinline__ void mirror(const GridInst& G, const Rec& o, float da, float2 d, float dz,
                                                  Rec& b) {
        float db = da - d.x * G.f_normal[0] - d.y * G.f_normal[1];
        if (ND == 3) db -= dz * G.f_normal[2];
        const float m = -fminf(G.f_beta, fabsf(__fdividef(db, da)));
        b.v = __fmul2_rn(bc2(m), o.v);
        b.vz = m * o.vz;
        b.aux = o.aux;
        b.irho = o.irho;
        b.rho = o.rho;
#pragma unroll
        for (int q = 0; q < NSA; ++q) b.a[q] = o.a[q];
    }

    // The difference of two FP32-pair positions, and r².
    static __device__ __forceinline__ float delta(const Rec& o, const Rec& b, float2& d, float& dz) {
        const float2 h = sub2(o.h, b.h), l = sub2(o.l, b.l);
        d = __fadd2_rn(h, l);
        const float hz = ND == 3 ? o.hz - b.hz : 0.f, lz = ND == 3 ? o.lz - b.lz : 0.f;
        dz = hz + lz;
        // h² + 2hl, not d²: d's rounding stays out of r²
        float s = dot(h, hz, l, lz);
        s += s;
        s = fmaf(h.x, h.x, s);
        s = fmaf(h.y, h.y, s);
        if (ND == 3) s = fmaf(hz, hz, s);
        return s;
    }
    static __device__ __forceinline__ float delta64(const Rec& o, const Rec& b) {
        const double x = (double)(o.h.x - b.h.x) + (double)(o.l.x - b.l.x);
        const double y = (double)(o.h.y - b.h.y) + (double)(o.l.y - b.l.y);
        const double z = ND == 3 ? (double)(o.hz - b.hz) + (double)(o.lz - b.lz) : 0.0;
        return (float)(x * x + y * y + z * z);
    }

    // r² of a pair exactly as pair() computes it
    template <class Q>
    static __device__ __forceinline__ float dist2(const Rec& o, const Q& quad) {
        Rec b;
        pos_read(quad, b);
        float2 d;
        float dz;
        return delta(o, b, d, dz);
    }

    // One candidate: r² from the FP32 pairs, then the functor's term when it
    // lies below the band around the cutoff (returns 1); `nearest` keeps how
    // near to the cutoff an r² came.  The pairs inside the band are left to
    // the caller to count: the kernel's gradient there is below 1e-11 of its
    // peak, so their terms vanish in FP32.  Only a Lennard-Jones wall, whose
    // force need not, has exact() decide them here.  o: own record; da: own
    // distance to a dynamic boundary's plane.  BTK: the system_b kind when
    // known at compile time (BT_SELF then has no density diffusion).
    template <int BTK, class Q, class Exact>
    static __device__ __forceinline__ int pair(const Par& p, const GridInst& G, const PfnInst& P, const Rec& o,
                                               float da, bool has3, const Q& quad, const Exact& exact, float& nearest,
                                               Acc& acc) {
        const int bt = BTK >= 0 ? BTK : p.bt;
        Rec b;
        if (bt == BT_DYNAMIC) pos_read(quad, b);
        else rec_read(quad, has3, b);
        float2 d;
        float dz;
        float rr = delta(o, b, d, dz);
        // a Lennard-Jones force goes with r^-14: its r² from FP64
        if (bt == BT_STATIC) rr = delta64(o, b);
        const float off = rr - p.cut;
        bool in = off < -p.band;
        if (bt == BT_STATIC) {
            if (fabsf(off) <= p.band) in = exact();
        } else {
            nearest = fminf(nearest, fabsf(off));
        }
        term<BTK>(p, G, P, o, da, b, d, dz, rr, in, acc);
        return in ? 1 : 0;
    }

    // The functor's term of a pair at distance (d, dz), r² = rr, onto the
    // sums; a pair that is not `in` adds exact zeros.  b: system_b's record
    // (a dynamic boundary's is made here).
    template <int BTK>
    static __device__ __forceinline__ void term(const Par& p, const GridInst& G, const PfnInst& P, const Rec& o,
                                                float da, Rec& b, float2 d, float dz, float rr, bool in, Acc& acc) {
        const int bt = BTK >= 0 ? BTK : p.bt;
        if (bt == BT_DYNAMIC) mirror(G, o, da, d, dz, b);
        const float ri = rsqrt_fast(rr);
        const float g = kgrad(p, rr, ri);
        const float2 dv = sub2(o.v, b.v);
        const float dvz = ND == 3 ? o.vz - b.vz : 0.f;
        if constexpr (!FLUID && !CAUCHY) {
            // strain rate and vorticity: f·(v_j − v_i)⊗∇W, f = m_j/ρ_j
            const float f = in ? -g * b.aux : 0.f;
            const float2 u = make_float2(in ? dv.x : 0.f, in ? dv.y : 0.f);
            const float2 w = __fmul2_rn(bc2(f), d);
            add(acc, 0, u, w);
            add(acc, 1, u, make_float2(w.y, w.x));
            if constexpr (ND == 3) {
                const float uz = in ? dvz : 0.f, wz = f * dz;
                add(acc, 2, make_float2(uz, u.x), bc2(wz));
                add(acc, 3, make_float2(uz, u.y), make_float2(w.x, wz));
                add(acc, 4, make_float2(uz, 0.f), make_float2(w.y, 0.f));
            }
        } else {
            // dv·∇W = g·(dv·dx); artificial viscosity src/PairwisePhysics.jl:29-34
            const float vr = dot(d, dz, dv, dvz);
            const float mu = fminf(vr, 0.f) * rcp_fast(rr + p.eps);
            const float pj = fmaf(p.beta, mu, -p.am) * mu * (2.f * o.irho);  // π·ρ_j
            if (bt == BT_STATIC) {
                // Lennard-Jones wall, src/PairwiseFunctors.jl:210-219 (kq with system_b's mass)
                const float x = G.f_ljcut * ri, x2 = x * x, x6 = x2 * x2 * x2;
                const float lj = x > 1.f ? p.ljc * __fdividef(x6 * x6 - x6, rr) : 0.f;
                const float s = in ? lj - p.kq * g * pj * b.irho : 0.f;
                add(acc, 0, bc2(s), d);
                if (ND == 3) add(acc, 1, make_float2(s, 0.f), make_float2(dz, 0.f));
                return;
            }
            float q = vr;
            // density diffusion (the specialised self form is without it)
            if (BTK != BT_SELF && p.dd != 0.f) q = fmaf(p.dd * (o.rho - b.rho), b.irho, q);
            q = in ? q : 0.f;
            const float gs = in ? g : 0.f;
            if constexpr (FLUID) {
                float e;
                if (PFN == PFN_FLUID2 && P.two) {
                    e = o.aux + b.aux;  // −p_i/ρ_i² − p_j/ρ_j²
                    if (P.fs)           // the fluid's pressure p = (p/ρ²)·ρ² on both sides
                        e = G.side_b ? b.aux + (b.aux * b.rho * b.rho) * o.irho * o.irho
                                     : o.aux + (o.aux * o.rho * o.rho) * b.irho * b.irho;
                    // artificial surface tension ε·(−(|p_i| + |p_j|)/(ρ_i ρ_j))
                    if (P.has_eps) e -= P.f_eps * (fabsf(o.aux) * o.rho * b.irho + fabsf(b.aux) * b.rho * o.irho);
                    e -= pj * b.irho;
                } else {
                    e = o.aux + fmaf(-pj, b.irho, b.aux);  // −p_i/ρ_i² − p_j/ρ_j² − π
                }
                const float s = in ? g * e : 0.f;
                add(acc, 0, bc2(s), d);
                add(acc, 1, make_float2(s, gs), make_float2(dz, q));
            } else {
                // (σ'_i + σ'_j − π·I)·∇W
                const float pi = pj * b.irho;
                const float2 w = __fmul2_rn(bc2(gs), d);
                if constexpr (ND == 2) {
                    const float2 n = __fadd2_rn(__fadd2_rn(make_float2(o.a[0], o.a[NSA > 1 ? 1 : 0]),
                                                           make_float2(b.a[0], b.a[NSA > 1 ? 1 : 0])),
                                                bc2(-pi));
                    const float2 t = make_float2(in ? n.x : 0.f, in ? n.y : 0.f);
                    const float xy = in ? o.a[NSA > 2 ? 2 : 0] + b.a[NSA > 2 ? 2 : 0] : 0.f;
                    put(acc, 0, __ffma2_rn(bc2(xy), make_float2(w.y, w.x), __ffma2_rn(t, w, acc.c[0])));
                    add(acc, 1, make_float2(0.f, gs), make_float2(0.f, q));
                } else {
                    const float wz = gs * dz;
                    float a[6];
#pragma unroll
                    for (int c = 0; c < 6; ++c) a[c] = o.a[c < NSA ? c : 0] + b.a[c < NSA ? c : 0];
                    if (in) {
                        const float2 y0 = make_float2(fmaf(a[3], w.y, fmaf(a[4], wz, acc.c[0].x)),
                                                      fmaf(a[3], w.x, fmaf(a[5], wz, acc.c[0].y)));
                        put(acc, 0, __ffma2_rn(make_float2(a[0] - pi, a[1] - pi), w, y0));
                        const float y1 = fmaf(a[4], w.x, fmaf(a[5], w.y, acc.c[1].x));
                        put(acc, 1, __ffma2_rn(make_float2(a[2] - pi, gs), make_float2(wz, q),
                                               make_float2(y1, acc.c[1].y)));
                    }
                }
            }
        }
    }
};

// Conservative prefilter of a batch of mb <= 32 candidates (batch_hits of
// k_force_impl.cuh), bit 31 − t set when candidate t may be within the
// cutoff: the pair loop then takes them in order by counting leading zeros.
template <int ND>
__device__ __forceinline__ unsigned batch_hits_lead(const float* cb, int stride, int mb, const float* xi,
                                                    float cut_f) {
    const float2 neg1 = make_float2(-1.0f, -1.0f);
    const float2 ncut = make_float2(-cut_f, -cut_f);
    unsigned hits = 0;
    int t0 = 0;
#pragma unroll
    for (int g = 0; g < 4; ++g) {
        if (8 * g < mb) {  // warp-uniform
#pragma unroll
            for (int t = 0; t < 8; t += 4) {
                float2 ra = ncut, rb = ncut;  // candidates t, t+1 and t+2, t+3
#pragma unroll
                for (int d = 0; d < ND; ++d) {
                    const float4 q = *reinterpret_cast<const float4*>(cb + d * stride + 8 * g + t);
                    const float2 xo = make_float2(xi[d], xi[d]);
                    const float2 da = __ffma2_rn(make_float2(q.x, q.y), neg1, xo);
                    const float2 db = __ffma2_rn(make_float2(q.z, q.w), neg1, xo);
                    ra = __ffma2_rn(da, da, ra);
                    rb = __ffma2_rn(db, db, rb);
                }
                hits = __funnelshift_l(__float_as_uint(ra.x), hits, 1);
                hits = __funnelshift_l(__float_as_uint(ra.y), hits, 1);
                hits = __funnelshift_l(__float_as_uint(rb.x), hits, 1);
                hits = __funnelshift_l(__float_as_uint(rb.y), hits, 1);
            }
            t0 += 8;
        }
    }
    return t0 == 32 ? hits : hits << (32 - t0);
}

// Min and max over the warp of a finite float.
__device__ __forceinline__ void warp_minmax(float v, float& lo, float& hi) {
    const int b = __float_as_int(v), key = b ^ ((b >> 31) & 0x7fffffff);
    const int kl = __reduce_min_sync(0xffffffffu, key), kh = __reduce_max_sync(0xffffffffu, key);
    lo = __int_as_float(kl ^ ((kl >> 31) & 0x7fffffff));
    hi = __int_as_float(kh ^ ((kh >> 31) & 0x7fffffff));
}

// Shared memory of one warp: the chunk's records ([NQ][CH] quads), the
// candidates' FP32 positions ([ND][CH]) and each lane's non-empty hit masks
// with the empty one that ends them.
template <int ND, int NQ, int CH>
__host__ __device__ constexpr int win_warp_bytes() {
    return NQ * CH * 16 + ND * CH * 4 + (CH / 32 + 1) * 128;
}

template <class Phys, int ND, int PFN, int MINB, int CH>
__global__ void __launch_bounds__(WIN_TPB, MINB) k_sweep_win(ForceArgs A) {
    pdl_enter();
    static_assert(CH % 32 == 0 && CH / 32 <= 8, "a lane's masks are numbered by batch, four bits each in a word");
    constexpr int NQ = Phys::NQ;
    constexpr int NSTR = 3, NWIN = ND == 2 ? 1 : 3;  // strips per window, windows
    constexpr int WB = win_warp_bytes<ND, NQ, CH>();
    constexpr int L = ND - 1;
    extern __shared__ float4 sstg[];
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    char* wbase = reinterpret_cast<char*>(sstg) + (threadIdx.x >> 5) * WB;
    float4* slots = reinterpret_cast<float4*>(wbase);
    float* cand = reinterpret_cast<float*>(wbase + NQ * CH * 16);
    unsigned* masks = reinterpret_cast<unsigned*>(wbase + NQ * CH * 16 + ND * CH * 4) + lane;
    const int64_t ngroups = *A.ngroups;
    const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    int64_t wg = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    int2 next = wg < ngroups ? A.groups[wg] : group_of(0, 0, 0);
    for (; wg < ngroups; wg += nwarps) {
        const int2 grp = next;
        if (wg + nwarps < ngroups) next = A.groups[wg + nwarps];
        const bool active = lane < group_count(grp);
        const int32_t gi = grp.x + (active ? lane : 0);  // packed indices fit int32
        const int k = group_inst(grp);
        typename Phys::Rec o;
        {
            const float4* rec = A.arec + (int64_t)gi * NQ;
            Phys::rec_read([&](int q) { return rec[q]; }, true, o);
        }
        float xi[ND], xmax = 0.f;
        xi[0] = o.h.x;
        xi[1] = o.h.y;
        if (ND == 3) xi[L] = o.hz;
        unsigned visit;
        {
            float glo[ND], ghi[ND];
#pragma unroll
            for (int d = 0; d < ND; ++d) {
                warp_minmax(xi[d], glo[d], ghi[d]);
                xmax = fmaxf(xmax, fmaxf(fabsf(glo[d]), fabsf(ghi[d])));
            }
            // the interactions whose system_b comes within reach of the group,
            // one lane each (a 0.1% margin, so no pair is lost)
            bool reach = lane < A.nref;
            if (reach && A.ref[lane].bbox) {
                const SysInst& B = A.ref[lane].bbox[k];
                const double m = 1.001 * A.ref[lane].gi[k].cell + 2.4e-7 * xmax;
                reach = B.n > 0;
#pragma unroll
                for (int d = 0; d < ND; ++d)
                    reach = reach & ((double)ghi[d] >= B.bbmin[d] - m) & ((double)glo[d] <= B.bbmax[d] + m);
            }
            visit = __ballot_sync(FULL, reach);
        }
        // the next group's state on its way to this SM
        {
            const int64_t gn = next.x + (lane < group_count(next) ? lane : 0);
            asm volatile("prefetch.global.L1 [%0];" ::"l"(A.arec + gn * NQ));
#pragma unroll
            for (int d = 0; d < ND; ++d) asm volatile("prefetch.global.L1 [%0];" ::"l"(A.ax + d * A.aN + gn));
        }

        for (int ri = 0; ri < A.nref; ++ri) {
            const InterRef& r = A.ref[ri];
            const GridInst& G = r.gi[k];
            int32_t accepted = 0;
            if ((visit >> ri & 1u) && G.cellbase + G.ncells > r.cs_cells) {
                if (lane == 0) atomicOr(A.err, ERR_CAPACITY);
            } else if (visit >> ri & 1u) {
                const PfnInst& P = r.pi[k];
                // cell coordinates (a grid has < 2^31 cells, so they fit int32)
                double x[ND];
#pragma unroll
                for (int d = 0; d < ND; ++d) x[d] = A.ax[d * A.aN + gi];
                int32_t c[ND];
                const bool ok = cells_of<ND>(G, x, c);
                float da = 0.f;
                if (r.btype == BT_DYNAMIC) {
                    double t = (x[0] - G.point[0]) * G.normal[0];
#pragma unroll
                    for (int d = 1; d < ND; ++d) t += (x[d] - G.point[d]) * G.normal[d];
                    da = (float)t;
                }
                if (active && !ok) atomicOr(A.err, ERR_CAPACITY);
                const int32_t c0 = __shfl_sync(FULL, c[0], 0), c1 = ND == 3 ? __shfl_sync(FULL, c[1], 0) : 0;
                const bool same = ok && c[0] == c0 && (ND == 2 || c[1] == c1);
                // positions over 2^20 cells from the origin, of which an FP32 pair
                // would lose more than FP32 arithmetic does, take FP64 differences
                const bool far = xmax * (float)G.inv_cell > 1048576.f;
                const bool coop = !far && __all_sync(FULL, !active || same);
                const bool self = r.btype == BT_SELF;
                typename Phys::Acc acc;
                Phys::zero(acc);
                const typename Phys::Par par = Phys::params(A, r, G, P, k, xmax + 2.f * (float)G.cell);
                // the 2-D fluid record's third quad (ρ) only for the forms that read it
                const bool has3 = ND == 3 || !Phys::FLUID || PFN == PFN_FLUID2 || par.dd != 0.f;
                const int32_t cz = c[L];
                const int32_t ngl = (int32_t)G.ng[L], ng1 = ND == 3 ? (int32_t)G.ng[1] : 0;
                const int32_t* cs = r.cs + G.cellbase;
                // the reference's test of candidate j (src/Interaction.jl:546-548)
                auto exact_test = [&](int32_t j, double* y, double& r2) {
#pragma unroll
                    for (int q = 0; q < ND; ++q) y[q] = __dsub_rn(A.ax[q * A.aN + gi], r.bx[q * r.bN + j]);
                    r2 = dot_exact<ND>(y, y);
                    return r2 < G.cutoff_sq;
                };
                if (coop) {
                    const int nq = r.btype == BT_DYNAMIC ? Phys::NQP : (has3 ? NQ : 2);
                    // conservative cutoff of the candidate test: 0.1% plus the coordinates' rounding
                    const float ce = (float)G.cell + 4.8e-7f * (xmax + 2.f * (float)G.cell);
                    const float cut_f = 1.001f * ce * ce;
                    // every strip's warp-wide candidate range, lane s holding strip s's
                    int32_t su0 = 0, sn = 0, zlo, zhi;
                    warp_zrange<ND>(c, active, zlo, zhi);
                    if (lane < NSTR * NWIN) {
                        const int32_t b2 =
                            (ND == 2 ? c0 + lane - 1 : (c0 + lane / 3 - 1) * ng1 + (c1 + lane % 3 - 1)) * ngl;
                        su0 = cs[b2 + zlo - 1];
                        sn = max(cs[b2 + zhi + 2] - su0, 0);
                    }
                    // window wi's slots: strip s holds [e[s], e[s + 1]), its slot t candidate u[s] + t
                    auto window = [&](int wi, int32_t* u, int32_t* e) {
                        e[0] = 0;
#pragma unroll
                        for (int s = 0; s < NSTR; ++s) {
                            e[s + 1] = e[s] + __shfl_sync(FULL, sn, NSTR * wi + s);
                            u[s] = __shfl_sync(FULL, su0, NSTR * wi + s) - e[s];
                        }
                    };
                    // the reference's test of slot t of window wi's chunk at ch, which has
                    // to lie in this lane's own strip [cs[z-1], cs[z+2])
                    auto exact_slot = [&](int wi, int32_t ch, int32_t t) {
                        t += ch;
                        int32_t lo = 0, hi = 0, j = 0, e = 0;
#pragma unroll 1
                        for (int s = NSTR * wi; s < NSTR * (wi + 1); ++s) {
                            const int32_t b2 =
                                (ND == 2 ? c0 + s - 1 : (c0 + s / 3 - 1) * ng1 + (c1 + s % 3 - 1)) * ngl + cz;
                            const int32_t u0 = cs[b2 - cz + zlo - 1], n = max(cs[b2 - cz + zhi + 2] - u0, 0);
                            if (t >= e && t < e + n) {
                                j = u0 + t - e;
                                lo = cs[b2 - 1];
                                hi = cs[b2 + 2];
                            }
                            e += n;
                        }
                        double y[ND], r2;
                        return j >= lo && j < hi && exact_test(j, y, r2);
                    };
                    // f(slot, candidate) for this lane's share of the chunk at ch
                    auto chunk = [&](const int32_t* u, const int32_t* e, int32_t ch, auto f) {
#pragma unroll
                        for (int s = 0; s < NSTR; ++s) {
                            const int32_t t1 = min(e[s + 1], ch + CH);
                            for (int32_t t = max(e[s], ch) + lane; t < t1; t += 32) f(t - ch, u[s] + t);
                        }
                    };
                    auto rows = [&](int t, int32_t j) {
#pragma unroll
                        for (int d = 0; d < ND; ++d)
                            __pipeline_memcpy_async(cand + d * CH + t, r.bh + d * r.bN + j, 4);
                    };
                    auto records = [&](int t, int32_t j) {
                        const float4* src = r.brec + (int64_t)j * r.brq;
#pragma unroll
                        for (int q = 0; q < NQ; ++q)
                            if (q < nq) __pipeline_memcpy_async(slots + q * CH + t, src + q, 16);
                    };
                    // The chunks in turn.  A chunk's records are on their way while its
                    // positions are tested, and the next chunk's positions while its
                    // accepted candidates are evaluated, so neither copy is waited out.
                    int wi = -1;
                    int32_t ch = 0, u[NSTR], e[NSTR + 1];
                    auto advance = [&]() {  // to the next window that holds candidates
                        do {
                            if (++wi == NWIN) return;
                            window(wi, u, e);
                        } while (e[NSTR] == 0);
                    };
                    advance();
                    if (wi < NWIN) chunk(u, e, ch, rows);
                    __pipeline_commit();
                    while (wi < NWIN) {
                        window(wi, u, e);
                        const int m = min(e[NSTR] - ch, CH);
                        // this lane's own slot (self interaction, centre strip)
                        const int32_t own = self && wi == NWIN / 2 ? gi - u[1] - ch : -1;
                        chunk(u, e, ch, records);
                        __pipeline_commit();
                        __pipeline_wait_prior(1);
                        __syncwarp();
                        // this lane's non-empty masks and, four bits each, their batch
                        // numbers; an empty one ends the list
                        int nm = 0;
                        unsigned bn = 0;
                        for (int b = 0; 32 * b < m; ++b) {
                            const int mb = min(m - 32 * b, 32);
                            unsigned hits = batch_hits_lead<ND>(cand + 32 * b, CH, mb, xi, cut_f);
                            hits &= active ? 0xffffffffu << (32 - mb) : 0u;
                            const unsigned ts = (unsigned)(own - 32 * b);
                            if (ts < 32u) hits &= ~(0x80000000u >> ts);
                            if (hits) {
                                masks[nm * 32] = hits;
                                bn |= (unsigned)b << (4 * nm);
                                ++nm;
                            }
                        }
                        masks[nm * 32] = 0u;
                        __syncwarp();  // every lane has tested the chunk
                        const int wc = wi;
                        const int32_t cc = ch;
                        ch += CH;
                        if (ch >= e[NSTR]) {
                            ch = 0;
                            advance();
                        }
                        if (wi < NWIN) chunk(u, e, ch, rows);
                        __pipeline_commit();
                        __pipeline_wait_prior(1);
                        __syncwarp();
                        // the accepted candidates, from the copies, in increasing order; the
                        // next mask is loaded while the current one is worked through
                        float nearest = FLT_MAX;
                        auto pairs = [&](auto btk) {
                            const unsigned* mp = masks;
                            unsigned cur = 0, nxt = *mp, bq = bn;
                            const float4* batch = slots;
                            while (cur | nxt) {
                                if (cur == 0) {
                                    cur = nxt;
                                    batch = slots + (bq & 15u) * 32;
                                    bq >>= 4;
                                    mp += 32;
                                    nxt = *mp;
                                }
                                const int t = __clz(cur);
                                cur ^= 0x80000000u >> t;
                                const float4* slot = batch + t;
                                accepted += Phys::template pair<decltype(btk)::value>(
                                    par, G, P, o, da, has3, [&](int q) { return slot[q * CH]; },
                                    [&]() { return exact_slot(wc, cc, (int)(slot - slots)); }, nearest, acc);
                            }
                        };
                        if (self && par.dd == 0.f) pairs(std::integral_constant<int, BT_SELF>{});
                        else pairs(std::integral_constant<int, -1>{});
                        // rare: candidates so near the cutoff that FP64 decides (counts them)
                        if (nearest <= par.band) {
                            for (int mi = 0; mi < nm; ++mi) {
                                const int b = (bn >> (4 * mi) & 15u) * 32;
                                for (unsigned cur = masks[mi * 32]; cur;) {
                                    const int t = b + __clz(cur);
                                    cur ^= 0x80000000u >> (t - b);
                                    const float rr = Phys::dist2(o, [&](int q) { return slots[q * CH + t]; });
                                    if (fabsf(rr - par.cut) <= par.band && exact_slot(wc, cc, t)) ++accepted;
                                }
                            }
                        }
                        __syncwarp();  // every lane is done with the chunk before the next one lands
                    }
                    __pipeline_wait_prior(0);
                } else if (active && ok) {
                    // rare (far, or lanes that disagree on the column in this grid): each
                    // lane walks its own strips, on FP64 differences
                    for (int s = 0; s < NSTR * NWIN; ++s) {
                        const int32_t base =
                            (ND == 2 ? c[0] + s - 1 : (c[0] + s / 3 - 1) * ng1 + (c[1] + s % 3 - 1)) * ngl;
                        const int32_t hi = cs[base + cz + 2];
                        for (int32_t j = cs[base + cz - 1]; j < hi; ++j) {
                            double y[ND], r2;
                            if ((self && j == gi) || !exact_test(j, y, r2)) continue;
                            const float4* rec = r.brec + (int64_t)j * r.brq;
                            typename Phys::Rec b;
                            if (r.btype != BT_DYNAMIC) Phys::rec_read([&](int q) { return rec[q]; }, has3, b);
                            Phys::template term<-1>(par, G, P, o, da, b, make_float2((float)y[0], (float)y[1]),
                                                    ND == 3 ? (float)y[L] : 0.f, (float)r2, true, acc);
                            ++accepted;
                        }
                    }
                }
                if (active) Phys::store(A, gi, acc, par.kf);
            }
            __syncwarp();
            if (active && r.counts) r.counts[gi] = accepted;
        }
        __syncwarp();
    }
}

template <class Phys, int ND, int PFN, int C>
static void launch_win(const ForceArgs& A, cudaStream_t s) {
    constexpr ForceCfg cf = FORCE_CFGS[C];
    int64_t blocks = (A.aN * 32 + WIN_TPB - 1) / WIN_TPB;
    if (blocks > (int64_t)A.num_sms * cf.wminb * 4) blocks = (int64_t)A.num_sms * cf.wminb * 4;
    if (blocks < 1) blocks = 1;
    constexpr size_t smem = (size_t)(WIN_TPB / 32) * win_warp_bytes<ND, Phys::NQ, cf.wch>();
    auto kern = k_sweep_win<Phys, ND, PFN, cf.wminb, cf.wch>;
    if (smem > 48 * 1024) {
        static bool opted = false;
        if (!opted) {
            cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
            opted = true;
        }
    }
    kern<<<(int)blocks, WIN_TPB, smem, s>>>(A);
    g_launches.fetch_add(1, std::memory_order_relaxed);
}

template <int ND, int NS, int PFN, int KK>
static int launch_win_cfg(const ForceArgs& A, cudaStream_t s) {
    using Phys = PhysF32<ND, NS, PFN, KK>;
    switch (A.cfg) {
        case 1: launch_win<Phys, ND, PFN, 1>(A, s); break;
        case 2: launch_win<Phys, ND, PFN, 2>(A, s); break;
        case 3: launch_win<Phys, ND, PFN, 3>(A, s); break;
        default: launch_win<Phys, ND, PFN, 0>(A, s); break;
    }
    return 0;
}

template <int ND, int KK>
static int launch_win_nd(const ForceArgs& A, cudaStream_t s) {
    if (A.pfn == GC_PFN_FLUID) return launch_win_cfg<ND, 0, GC_PFN_FLUID, KK>(A, s);
    if (A.pfn == PFN_FLUID2) return launch_win_cfg<ND, 0, PFN_FLUID2, KK>(A, s);
    auto stress = [&](auto ns) -> int {
        constexpr int NS = decltype(ns)::value;
        if (A.pfn == GC_PFN_CAUCHY_FLUID) return launch_win_cfg<ND, NS, GC_PFN_CAUCHY_FLUID, KK>(A, s);
        if (A.pfn == GC_PFN_STRAIN_RATE) return launch_win_cfg<ND, NS, GC_PFN_STRAIN_RATE, KK>(A, s);
        if (A.pfn == GC_PFN_STRAIN_RATE_VORTICITY)
            return launch_win_cfg<ND, NS, GC_PFN_STRAIN_RATE_VORTICITY, KK>(A, s);
        return GC_ERR_UNSUPPORTED;
    };
    if constexpr (ND == 2) {
        if (A.ns == 3) return stress(std::integral_constant<int, 3>{});
        if (A.ns == 4) return stress(std::integral_constant<int, 4>{});
    } else {
        if (A.ns == 6) return stress(std::integral_constant<int, 6>{});
    }
    return GC_ERR_UNSUPPORTED;
}

// One translation unit per dimension: defines launch_force_<ND>d_f32.
#define GC_DEFINE_FORCE_F32_TU(NDIM, NAME)                                                          \
    int NAME(const ForceArgs& A, bool, cudaStream_t s) {                                            \
        if (A.kk == GC_KERNEL_CUBIC_SPLINE) return launch_win_nd<NDIM, GC_KERNEL_CUBIC_SPLINE>(A, s); \
        return launch_win_nd<NDIM, GC_KERNEL_WENDLAND_C2>(A, s);                                    \
    }

}  // namespace gc
