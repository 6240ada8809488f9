// k_sweep_f32.cuh — the FP32-compensated arithmetic of the window sweep.
//
// What bounds it is instruction issue (65% of the slots, the FMA pipe half
// busy, shared memory half busy), so the pair term is written for few
// instructions:
//   * positions are FP32 pairs whose difference is the FP64 one to within two
//     roundings to FP32 (one where the pairs' high parts subtract exactly, as
//     they do but next to the origin), by a few adds per pair instead of eight
//     FP64 operations and four conversions; a record is two or three 16-byte
//     quads;
//   * dv·∇W is W'·(dv·dx), so ∇W itself is never formed; the kernel's constant
//     factor multiplies the sums, not the terms;
//   * components go through packed FP32x2 arithmetic.
// Three-dimensional dam break of a million jittered particles: 920 us a launch
// with strips staged one at a time and FP64 differences, 709 us with this
// kernel; 64 batched columns (1.07 M particles) 292 to 230 us; a Lennard-Jones
// box of 30 k particles 82 to 51 us.  Sixteen warps per SM (128
// registers, chunks of 192) beat eighteen to twenty-four at 80-96 registers,
// whose spills cost more than the occupancy gives.
//
// The neighbour sets stay exact: a pair whose FP32 r² lies within a small
// band of the cutoff takes the reference's FP64 test on the FP64 positions
// (and the reference's own strip range), outside the band the FP32 r² cannot
// be wrong about it.
#pragma once
#include "k_sweep_win.cuh"

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
__device__ __forceinline__ float min3(float a, float b, float c) {
    float y;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(y) : "f"(a), "f"(b), "f"(c));
    return y;
}
__device__ __forceinline__ float2 bc2(float x) { return make_float2(x, x); }
// a - b, exactly rounded (b·(−1) is exact)
__device__ __forceinline__ float2 sub2(float2 a, float2 b) { return __ffma2_rn(b, bc2(-1.0f), a); }

template <int ND, int NS, int PFN, int KK>
struct PhysF32 {
    static constexpr int MODE = aux_mode(PFN);
    static constexpr bool EXACT = false;
    using Real = float;
    static constexpr bool FLUID = fluid_pfn<PFN>(), CAUCHY = PFN == GC_PFN_CAUCHY_FLUID;
    // quads of a record, of a dynamic boundary's, and of what the functor reads
    // (the plain fluid in 2-D not the third, ρ)
    static constexpr int RQ = rec_quads(ND, MODE, true), NQP = pos_quads(ND, true);
    static constexpr int NQ = PFN == GC_PFN_FLUID && ND == 2 ? 2 : RQ;
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
    static __device__ __forceinline__ float h(const Rec& w, int d) { return d == 0 ? w.h.x : d == 1 ? w.h.y : w.hz; }
    // quad(q): the record's q-th 16-byte quad
    template <class Q>
    static __device__ __forceinline__ void rec_read(const Q& quad, Rec& w) {
        const float4 q0 = quad(0), q1 = quad(1);
        w.h = make_float2(q0.x, q0.y);
        if (ND == 2) {
            w.l = make_float2(q0.z, q0.w);
            w.v = make_float2(q1.x, q1.y);
            if (FLUID) {
                w.aux = q1.z;
                w.irho = q1.w;
                w.rho = NQ > 2 ? quad(2).x : 0.f;
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
        // FP32 r² is off by less than 1e-6 of the cutoff's (ten roundings of
        // terms below 1.3 of it: 8e-7), plus what the FP32 pairs lose of
        // coordinates |x| (2^-47·|x| each, so less than 3e-14·|x|/2h of r²)
        p.band = p.cut * (2e-6f + (float)strip_doubt<ND>(G) + 1e-13f * xmax * (float)G.inv_cell);
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
            const float a = fmaf(r, -p.qs, 2.f);  // (only pairs with r < 2h are added)
            return a * a * a;
        }
    }
    static __device__ __forceinline__ float dot(float2 a, float az, float2 b, float bz, float s0 = 0.f) {
        float s = fmaf(a.x, b.x, s0);
        s = fmaf(a.y, b.y, s);
        if (ND == 3) s = fmaf(az, bz, s);
        return s;
    }

    // Running compensated sums of one lane, component pairs together: (x, y)
    // and (z, dρ/dt); or (xx, yy), (xy, yx), (zz, xz), (zx, yz), (zy, -).
    static constexpr int NP = FLUID || CAUCHY || ND == 2 ? 2 : 5;
    // Beside a strain rate with a zz component, Σ f·0.
    static constexpr bool ZZ = !FLUID && !CAUCHY && ND == 2 && NS == 4;
    struct Acc {
        float2 s[NP], c[NP];  // Kahan: the sum, and minus its rounding error
        float zz;
    };
    static __device__ __forceinline__ void zero(Acc& a) {
        a.zz = 0.f;
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
    // The sums, times kf in FP64, onto system_a's rates.
    static __device__ __forceinline__ void store(const ForceArgs& A, const InterRef&, const GridInst&, int, const Par& p,
                                                 int64_t gi, const Acc& acc) {
        const int64_t N = A.aN;
        const double f = p.kf;
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
            if (ZZ && acc.zz != 0.f) put(A.asr, 2, (double)acc.zz);
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
        // h² + (2h + l)·l, not d²: d's rounding stays out of r².  l counts in
        // full: it reaches an ulp of the coordinate, 3% of 2h at 2^18 cells from
        // the origin.  (2h + l does not wait for d = h + l: 712 us on the million
        // particles, 729 as d + h, 711 with 2h·l alone.)
        // FLT_MIN keeps r² of particles nearly at one place out of the subnormals
        // (whose 1/r the seed cannot give) and is lost in any other.
        float s = dot(__ffma2_rn(h, bc2(2.f), l), fmaf(2.f, hz, lz), l, lz, FLT_MIN);
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

    static __device__ __forceinline__ bool diffuses(const Par& p) { return p.dd != 0.f; }
    static __device__ __forceinline__ float band(const Par& p) { return p.band; }
    static __device__ __forceinline__ bool lj_wall(int bt) { return (FLUID || CAUCHY) && bt == BT_STATIC; }
    // The sums of a lane with a neighbour at no distance: NaN (a Lennard-Jones
    // wall's terms are so by themselves).
    static __device__ __forceinline__ void spoil(const Par& p, Acc& a) {
        if (lj_wall(p.bt)) return;
#pragma unroll
        for (int q = 0; q < NP; ++q) a.s[q] = bc2(CUDART_NAN_F);
    }
    // whether pair<.., LIST>() did not count this candidate
    template <class Q>
    static __device__ __forceinline__ bool not_counted(const Par& p, const Rec& o, const Q& quad) {
        Rec b;
        float2 d;
        float dz;
        pos_read(quad, b);
        const float rr = delta(o, b, d, dz);
        return !(rr - p.cut < -p.band && rr > FLT_MIN);
    }
    // whether pair() left this candidate to the FP64 test, next to the cutoff or
    // where the FP32 pairs of the two positions are equal
    template <class Q>
    static __device__ __forceinline__ bool left_over(const Par& p, const Rec& o, const Q& quad, Acc&) {
        Rec b;
        float2 d;
        float dz;
        pos_read(quad, b);
        const float rr = delta(o, b, d, dz);
        return fabsf(rr - p.cut) <= p.band || rr <= FLT_MIN;
    }

    // One candidate: r² from the FP32 pairs, then the functor's term when it
    // lies below the band around the cutoff (returns 1); `nearest` keeps how
    // near to the cutoff, or to 0, an r² came (one three-input minimum).  The
    // pairs inside the band are left to the caller to count: the kernel's
    // gradient there is below 1e-11 of its peak, so their terms vanish in FP32.
    // Only a Lennard-Jones wall, whose force need not, has exact() decide them
    // here.  o: own record; da: own distance to a dynamic boundary's plane.  BTK:
    // the system_b kind when known at compile time (BT_SELF then has no density
    // diffusion).
    // LIST: the caller keeps a list of what this does not count, which a pair at
    // no distance is among, and `nearest` is not kept.
    template <int BTK, bool LIST, class Q, class Exact>
    static __device__ __forceinline__ int pair(const Par& p, const GridInst& G, const PfnInst& P, const Rec& o,
                                               float da, const Q& quad, const Exact& exact, float& nearest,
                                               Acc& acc) {
        const int bt = BTK >= 0 ? BTK : p.bt;
        Rec b;
        if (bt == BT_DYNAMIC) pos_read(quad, b);
        else rec_read(quad, b);
        float2 d;
        float dz;
        float rr = delta(o, b, d, dz);
        // a Lennard-Jones force goes with r^-14: its r² from FP64
        if (lj_wall(bt)) rr = delta64(o, b);
        const float off = rr - p.cut;
        bool in = off < -p.band;
        if (lj_wall(bt)) {
            if (fabsf(off) <= p.band) in = exact();
        } else if (!LIST) {
            nearest = min3(nearest, fabsf(off), rr);
        }
        term<BTK>(p, G, P, o, da, b, d, dz, rr, in, acc);
        return LIST && !lj_wall(bt) ? in && rr > FLT_MIN : in;
    }

    // The term of an accepted pair from its FP64 differences.
    static __device__ __forceinline__ void walked(const Par& p, const GridInst& G, const PfnInst& P, const Rec& o,
                                                  float da, Rec& b, const double* y, double r2, Acc& acc) {
        const float rr = lj_wall(p.bt) ? (float)r2 : fmaxf((float)r2, FLT_MIN);
        term<-1>(p, G, P, o, da, b, make_float2((float)y[0], (float)y[1]), ND == 3 ? (float)y[ND - 1] : 0.f, rr, true,
                 acc);
        if ((float)r2 == 0.f) spoil(p, acc);
    }

    // The functor's term of a pair at distance (d, dz), r² = rr, onto the
    // sums; a pair that is not `in` adds exact zeros.  b: system_b's record
    // (a dynamic boundary's is made here).
    template <int BTK>
    static __device__ __forceinline__ void term(const Par& p, const GridInst& G, const PfnInst& P, const Rec& o,
                                                float da, Rec& b, float2 d, float dz, float rr, bool in, Acc& acc) {
        const int bt = BTK >= 0 ? BTK : p.bt;
        if (bt == BT_DYNAMIC) mirror(G, o, da, d, dz, b);
        float ri = rsqrt_fast(rr);
        // One Newton step: the seed's error, the same for every pair at a
        // distance, would be the largest of the term (dρ/dt of a resting 3-D
        // lattice 2.1e-7 of scale, 0.7e-7 with it; 1.6% of the sweep).
        ri = fmaf(0.5f * ri, fmaf(-(rr * ri), ri, 1.f), ri);
        const float g = kgrad(p, rr, ri);
        const float2 dv = sub2(o.v, b.v);
        const float dvz = ND == 3 ? o.vz - b.vz : 0.f;
        if constexpr (!FLUID && !CAUCHY) {
            // strain rate and vorticity: f·(v_j − v_i)⊗∇W, f = m_j/ρ_j
            const float f = in ? -g * b.aux : 0.f;
            if (ZZ) acc.zz = fmaf(f, 0.f, acc.zz);  // NaN beside a neighbour of no finite volume
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
            if (lj_wall(bt)) {
                // Lennard-Jones wall, src/PairwiseFunctors.jl:210-219 (kq with system_b's mass)
                const float x = G.f_ljcut * ri, x2 = x * x, x6 = x2 * x2 * x2;
                const float lj = x > 1.f ? p.ljc * __fdividef(x6 * x6 - x6, rr) : 0.f;
                const float s = in ? lj - p.kq * g * pj * b.irho : 0.f;
                add(acc, 0, bc2(s), d);
                if (ND == 3) add(acc, 1, make_float2(s, 0.f), make_float2(dz, 0.f));
                return;
            }
            float q = vr;
            // density diffusion (the plain fluid and the specialised self form are without it)
            if (PFN != GC_PFN_FLUID && BTK != BT_SELF && p.dd != 0.f) q = fmaf(p.dd * (o.rho - b.rho), b.irho, q);
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

// One translation unit per dimension: defines launch_force_<ND>d_f32.
#define GC_DEFINE_FORCE_F32_TU(NDIM, NAME)                                                                       \
    int NAME(const ForceArgs& A, cudaStream_t s) {                                                         \
        if (A.kk == GC_KERNEL_CUBIC_SPLINE) return launch_win_nd<PhysF32, NDIM, GC_KERNEL_CUBIC_SPLINE>(A, s);   \
        return launch_win_nd<PhysF32, NDIM, GC_KERNEL_WENDLAND_C2>(A, s);                                        \
    }

}  // namespace gc
