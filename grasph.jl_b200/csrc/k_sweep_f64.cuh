// k_sweep_f64.cuh — the plain FP64 arithmetic of the window sweep.
//
// What bounds it is instruction issue and the FP64 chains' latency, and the
// reference's expressions spend most of both on square roots and divisions
// (about 390 instructions a pair).  The same terms are evaluated here with
// one reciprocal square root and one reciprocal a pair, each a hardware seed
// and two Newton-Raphson steps (2^-20 squared twice, so the last rounding is
// what is left), with fused multiply-adds, dv·∇W as W'·(dv·dx), and the
// kernel's constant factor on the sums.  Every quantity stays FP64; a term
// differs from the reference's expression by a few units in the last place.
// Sweep of 224 k particles of 3-D water 885 -> 261 us, of 5,000 in 2-D 63.5 ->
// 24.5 us, of an 80 k column 81 -> 44 us a launch (jittered starts).  The first
// configuration (twelve warps per SM) is mostly the fastest: up to 168
// registers, and only the 3-D Cauchy terms spill (92 bytes; every
// configuration of theirs does).
// The acceptance test keeps the reference's unfused r² < (2h)², so the
// neighbour sets are bit-identical.
#pragma once
#include "k_sweep_win.cuh"

namespace gc {

// 1/x and 1/sqrt(x) of a positive normal x, by Newton-Raphson.  (1/sqrt of a
// smaller x, whose seed is infinite, is some number above 2^511.)
__device__ __forceinline__ double rcp_newton(double x) {
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    y = fma(y, fma(-x, y, 1.0), y);
    return fma(y, fma(-x, y, 1.0), y);
}
__device__ __forceinline__ double rsqrt_newton(double x) {
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    y = __hiloint2double(min(__double2hiint(y), 0x5fe00000), __double2loint(y));
    const double h = -0.5 * x;
    y = fma(y, fma(h * y, y, 0.5), y);
    return fma(y, fma(h * y, y, 0.5), y);
}

template <int ND, int NS, int PFN, int KK>
struct PhysF64 {
    static constexpr int MODE = aux_mode(PFN);
    static constexpr bool EXACT = true;
    using Real = double;
    static constexpr bool FLUID = fluid_pfn<PFN>(), CAUCHY = PFN == GC_PFN_CAUCHY_FLUID;
    static constexpr bool VORT = PFN == GC_PFN_STRAIN_RATE_VORTICITY;
    // quads of a record, of a dynamic boundary's, and of what the functor reads
    // (the plain fluid not the last, ρ and p)
    static constexpr int RQ = rec_quads(ND, MODE, false), NQP = pos_quads(ND, false);
    static constexpr int NQ = PFN == GC_PFN_FLUID ? RQ - 1 : RQ;
    static constexpr int NSA = CAUCHY ? (ND == 2 ? 3 : 6) : 1;
    static constexpr int NV = (2 * ND + 1) / 2;  // quads of x and v

    struct Rec {
        double x[ND], v[ND];
        double aux, irho, rho, p;  // aux: −p/ρ² (fluid) or m/ρ (strain rate)
        double a[NSA];
    };
    static __device__ __forceinline__ float h(const Rec& w, int d) { return (float)w.x[d]; }
    template <class Q>
    static __device__ __forceinline__ double at(const Q& quad, int e) {  // double e of the record
        const float4 q = quad(e >> 1);
        return e & 1 ? __hiloint2double(__float_as_int(q.w), __float_as_int(q.z))
                     : __hiloint2double(__float_as_int(q.y), __float_as_int(q.x));
    }
    template <class Q>
    static __device__ __forceinline__ void rec_read(const Q& quad, Rec& w) {
        constexpr int E = 2 * NV;
#pragma unroll
        for (int d = 0; d < ND; ++d) {
            w.x[d] = at(quad, d);
            w.v[d] = at(quad, ND + d);
        }
        if (FLUID) {
            w.aux = at(quad, E);
            w.irho = at(quad, E + 1);
            if (NQ == RQ) {
                w.rho = at(quad, E + 2);
                w.p = at(quad, E + 3);
            }
        } else if (CAUCHY) {
            w.irho = at(quad, E);
            w.rho = at(quad, E + 1);
#pragma unroll
            for (int q = 0; q < NSA; ++q) w.a[q] = at(quad, E + 2 + q);
        } else {
            w.aux = at(quad, E);
        }
    }
    template <class Q>
    static __device__ __forceinline__ void pos_read(const Q& quad, Rec& w) {
#pragma unroll
        for (int d = 0; d < ND; ++d) w.x[d] = at(quad, d);
    }

    struct Par {
        double cut, sure;    // (2h)²; below `sure` the strip range cannot matter
        double qs, qs_lo;    // kernel argument's factor
        double kq;           // the gradient's factor with system_b's mass (Lennard-Jones wall)
        double eps, am, beta;  // 0.01·h², α·c̄·h, β·h² of the artificial viscosity
        double dd;             // 2·δ·c̄·h of the density diffusion (0: none)
        double c;              // system_a's sound speed
        int bt;
    };
    static __device__ __forceinline__ Par params(const ForceArgs& A, const InterRef& r, const GridInst& G,
                                                 const PfnInst& P, int k, float) {
        Par p;
        p.bt = r.btype;
        p.cut = G.cutoff_sq;
        p.sure = G.cutoff_sq * (1.0 - strip_doubt<ND>(G));
        p.qs = G.qs;
        p.qs_lo = G.qs_lo;
        p.eps = p.am = p.beta = p.dd = 0.0;
        if (FLUID || CAUCHY) {
            const double ca = A.a_c[k];
            p.c = ca;
            const bool two = PFN == PFN_FLUID2 && P.two;
            const double cm = (CAUCHY && r.btype == BT_GHOST) || two ? 0.5 * (ca + G.bc) : ca;
            p.eps = (P.h * P.h) * 0.01;
            p.am = P.alpha * cm * P.h;
            p.beta = P.beta * P.h * P.h;
            if (P.has_delta) p.dd = 2.0 * P.delta * (two ? cm : ca) * P.h;
        }
        p.kq = G.kq * G.bmass;
        return p;
    }
    static __device__ __forceinline__ bool diffuses(const Par& p) { return p.dd != 0.0; }
    // (pair()'s `nearest` is r²'s high word, as a float: subnormal or 0 up to this)
    static __device__ __forceinline__ float band(const Par&) { return __int_as_float(0x000fffff); }

    // ∇W = (the kernel's factor)·kgrad·dx for a pair at r² (ri = 1/r)
    static __device__ __forceinline__ double kgrad(const Par& p, double rr, double ri) {
        const double r = rr * ri;
        if (KK == GC_KERNEL_CUBIC_SPLINE) {
            // −3·(¼(2−q)² − (1−q)²): with s = q/2, −3·((1−s)² − (1−2s)²)
            // (1/2h in two parts: rounded once, it would shift every pair's alike.
            // With the sums' factor in two, FP64 errors of one sweep against long
            // double 5-35% below what they were, and no larger than separately
            // rounded square roots and divisions gave; 1.4% of the sweep.)
            const double a0 = fma(-r, p.qs, 1.0), a = fma(-r, p.qs_lo, a0), b = fma(2.0, a0, -1.0);
            const double bb = b > 0.0 ? b * b : 0.0;
            return ri * fma(a, a, -bb);
        } else {
            const double a = fma(-r, p.qs_lo, fma(-r, p.qs, 2.0));
            return a * a * a;
        }
    }
    static __device__ __forceinline__ double dot(const double* a, const double* b) {
        double s = a[0] * b[0];
#pragma unroll
        for (int d = 1; d < ND; ++d) s = fma(a[d], b[d], s);
        return s;
    }

    // Sums: dv/dt then dρ/dt; or the products f·dv_a·∂W_b (row a, column b)
    static constexpr int NSUM = FLUID || CAUCHY ? ND + 1 : ND * ND;
    // ... and, beside a strain rate with a zz component, Σ f·0
    static constexpr bool ZZ = !FLUID && !CAUCHY && ND == 2 && NS == 4;
    struct Acc {
        double s[NSUM];
        double zz;
    };
    static __device__ __forceinline__ void zero(Acc& a) {
        a.zz = 0.0;
#pragma unroll
        for (int q = 0; q < NSUM; ++q) a.s[q] = 0.0;
    }
    // The sums of a lane with a neighbour at no distance: NaN (a Lennard-Jones
    // wall's terms are so by themselves).
    static __device__ __forceinline__ void spoil(const Par& p, Acc& a) {
        if ((FLUID || CAUCHY) && p.bt == BT_STATIC) return;
#pragma unroll
        for (int q = 0; q < NSUM; ++q) a.s[q] = CUDART_NAN;
    }
    template <class Q>
    static __device__ __forceinline__ bool left_over(const Par& p, const Rec& o, const Q& quad, Acc& a) {
        Rec b;
        pos_read(quad, b);
        double d[ND];
#pragma unroll
        for (int q = 0; q < ND; ++q) d[q] = o.x[q] - b.x[q];
        if (dot_exact<ND>(d, d) == 0.0) spoil(p, a);
        return false;
    }
    // The sums' factor, f + lo: the gradient's, with the terms' mass for dv/dt
    // and dρ/dt.  A Lennard-Jones wall's terms carry it themselves (its mass,
    // which may be 0, is not the force's).  Both halves: rounded once, it would
    // put its error on every sum alike.
    static __device__ __forceinline__ void factor(const ForceArgs& A, const InterRef& r, const GridInst& G, int k,
                                                  double& f, double& lo) {
        f = G.kq;
        lo = G.kq_lo;
        if (!FLUID && !CAUCHY) return;
        const double m = r.btype == BT_SELF || r.btype == BT_DYNAMIC ? A.a_mass[k] : G.bmass, t = f * m;
        lo = fma(f, m, -t) + lo * m;
        f = t;
        if (r.btype == BT_STATIC) {
            f = 1.0;
            lo = 0.0;
        }
    }
    static __device__ __forceinline__ void store(const ForceArgs& A, const InterRef& r, const GridInst& G, int k,
                                                 const Par&, int64_t gi, const Acc& acc) {
        const int64_t N = A.aN;
        double f, lo;
        factor(A, r, G, k, f, lo);
        // (reductions, as in the FP32 policy)
        auto put = [&](double* to, int q, double x) { atomicAdd(to + q * N + gi, fma(f, x, lo * x)); };
        auto m = [&](int a, int b) { return acc.s[(a * ND + b) % NSUM]; };
        if (FLUID || CAUCHY) {
#pragma unroll
            for (int d = 0; d < ND; ++d) put(A.advdt, d, acc.s[d]);
            put(A.adrhodt, 0, acc.s[NSUM > ND ? ND : 0]);
        } else {
#pragma unroll
            for (int d = 0; d < ND; ++d) put(A.asr, d, m(d, d));
            put(A.asr, ND == 3 ? 3 : NS == 4 ? 3 : 2, 0.5 * (m(0, 1) + m(1, 0)));
            if (ZZ && acc.zz != 0.0) put(A.asr, 2, acc.zz);
            if (ND == 3) {
                put(A.asr, 4, 0.5 * (m(0, 2) + m(2, 0)));
                put(A.asr, 5, 0.5 * (m(1, 2) + m(2, 1)));
            }
            if (VORT) {
                put(A.avort, 0, 0.5 * (m(0, 1) - m(1, 0)));
                if (ND == 3) {
                    put(A.avort, 1, 0.5 * (m(0, 2) - m(2, 0)));
                    put(A.avort, 2, 0.5 * (m(1, 2) - m(2, 1)));
                }
            }
        }
    }

    // One candidate: the reference's exact test, then the functor's term
    // (returns 1 when accepted).  exact(): the candidate lies in this lane's
    // own strip; asked next to the cutoff only, as one further off is two
    // cells away otherwise.
    template <int BTK, bool, class Q, class Exact>
    static __device__ __forceinline__ int pair(const Par& p, const GridInst& G, const PfnInst& P, const Rec& o,
                                               double da, const Q& quad, const Exact& exact, float& nearest,
                                               Acc& acc) {
        const int bt = BTK >= 0 ? BTK : p.bt;
        Rec b;
        if (bt == BT_DYNAMIC) pos_read(quad, b);
        else rec_read(quad, b);
        double d[ND];
#pragma unroll
        for (int q = 0; q < ND; ++q) d[q] = o.x[q] - b.x[q];
        const double rr = dot_exact<ND>(d, d);
        nearest = fminf(nearest, __int_as_float(__double2hiint(rr)));
        bool in = rr < p.cut;
        if (in && rr > p.sure) in = exact();
        if (in) term<BTK>(p, G, P, o, da, b, d, rr, acc);
        return in ? 1 : 0;
    }
    static __device__ __forceinline__ void walked(const Par& p, const GridInst& G, const PfnInst& P, const Rec& o,
                                                  double da, Rec& b, const double* y, double r2, Acc& acc) {
        term<-1>(p, G, P, o, da, b, y, r2, acc);
        if (r2 == 0.0) spoil(p, acc);
    }

    template <int BTK>
    static __device__ __forceinline__ void term(const Par& p, const GridInst& G, const PfnInst& P, const Rec& o,
                                                double da, Rec& b, const double* d, double rr, Acc& acc) {
        const int bt = BTK >= 0 ? BTK : p.bt;
        if (bt == BT_DYNAMIC) {
            // src/PairwiseFunctors.jl:53,111,222,334: mirrored velocity, own density and stress
            double t = da;
#pragma unroll
            for (int q = 0; q < ND; ++q) t = fma(-d[q], G.normal[q], t);
            const double m = -jmin(G.beta, fabs(t / da));
#pragma unroll
            for (int q = 0; q < ND; ++q) b.v[q] = m * o.v[q];
            b.aux = o.aux;
            b.irho = o.irho;
            b.rho = o.rho;
            b.p = o.p;
#pragma unroll
            for (int q = 0; q < NSA; ++q) b.a[q] = o.a[q];
        }
        const double g = kgrad(p, rr, rsqrt_newton(rr));
        double dv[ND];
#pragma unroll
        for (int q = 0; q < ND; ++q) dv[q] = o.v[q] - b.v[q];
        if constexpr (!FLUID && !CAUCHY) {
            // strain rate and vorticity: f·(v_j − v_i)⊗∇W, f = m_j/ρ_j
            const double f = -g * b.aux;
            if (ZZ) acc.zz = fma(f, 0.0, acc.zz);  // NaN beside a neighbour of no finite volume
#pragma unroll
            for (int c = 0; c < ND; ++c) {
                const double w = f * d[c];
#pragma unroll
                for (int q = 0; q < ND; ++q) acc.s[(q * ND + c) % NSUM] = fma(dv[q], w, acc.s[(q * ND + c) % NSUM]);
            }
        } else {
            // dv·∇W = g·(dv·dx); artificial viscosity src/PairwisePhysics.jl:29-34
            const double vr = dot(d, dv);
            // (a comparison that leaves NaN as it is, like Julia's min)
            const double mu = (vr > 0.0 ? 0.0 : vr) * rcp_newton(rr + p.eps);
            const double pj = fma(p.beta, mu, -p.am) * mu * (2.0 * o.irho);  // π·ρ_j
            if (bt == BT_STATIC) {
                // Lennard-Jones wall, src/PairwiseFunctors.jl:210-219 (kq with system_b's mass)
                const double s = lennard_jones<ND>(d, rr, G.ljcut, p.c) - p.kq * g * pj * b.irho;
#pragma unroll
                for (int q = 0; q < ND; ++q) acc.s[q] = fma(s, d[q], acc.s[q]);
                return;
            }
            // the diffusion's ψ/ρ_j with ψ = 0: NaN when ρ_j is 0 or NaN, else vr
            double q = fma(0.0, b.irho, vr);
            // density diffusion (the plain fluid and the specialised self form are without it)
            if (PFN != GC_PFN_FLUID && BTK != BT_SELF && p.dd != 0.0) q = fma(p.dd * (o.rho - b.rho), b.irho, q);
            double* dr = &acc.s[NSUM > ND ? ND : 0];
            if constexpr (FLUID) {
                double e = fma(-pj, b.irho, b.aux) + o.aux;  // −p_i/ρ_i² − p_j/ρ_j² − π
                if (PFN == PFN_FLUID2) {
                    const double rij = o.irho * b.irho;
                    if (P.fs) {  // the fluid's pressure on both sides
                        const double pf = G.side_b ? b.p : o.p;
                        e = P.S == 1 ? -(pf + pf) * rij
                            : G.side_b ? b.aux - pf * (o.irho * o.irho) : o.aux - pf * (b.irho * b.irho);
                        e -= pj * b.irho;
                    } else if (P.S == 1) {
                        e = -(o.p + b.p) * rij - pj * b.irho;
                    }
                    // artificial surface tension ε·(−(|p_i| + |p_j|)/(ρ_i ρ_j))
                    if (P.two && P.has_eps) e -= P.eps * ((fabs(o.p) + fabs(b.p)) * rij);
                    if (P.S == 1) q = fma(vr, o.rho * b.irho, q - vr);
                }
                const double s = g * e;
#pragma unroll
                for (int c = 0; c < ND; ++c) acc.s[c] = fma(s, d[c], acc.s[c]);
                *dr = fma(g, q, *dr);
            } else {
                // (σ'_i + σ'_j − π·I)·∇W
                const double pi = pj * b.irho;
                double a[NSA], w[ND];
#pragma unroll
                for (int c = 0; c < NSA; ++c) a[c] = o.a[c] + b.a[c];
#pragma unroll
                for (int c = 0; c < ND; ++c) w[c] = g * d[c];
                if constexpr (ND == 2) {
                    acc.s[0] = fma(a[0] - pi, w[0], fma(a[NSA - 1], w[1], acc.s[0]));
                    acc.s[1] = fma(a[NSA - 1], w[0], fma(a[NSA > 1 ? 1 : 0] - pi, w[1], acc.s[1]));
                } else {
                    // xx yy zz xy xz yz
                    constexpr int Y = NSA > 1 ? 1 : 0, Z = NSA > 2 ? 2 : 0, XY = NSA > 3 ? 3 : 0, XZ = NSA > 4 ? 4 : 0,
                                  YZ = NSA > 5 ? 5 : 0;
                    // (a term is rounded to the sum's precision once, not product by product)
                    acc.s[0] += fma(a[0] - pi, w[0], fma(a[XY], w[1], a[XZ] * w[ND - 1]));
                    acc.s[1] += fma(a[XY], w[0], fma(a[Y] - pi, w[1], a[YZ] * w[ND - 1]));
                    acc.s[ND - 1] += fma(a[XZ], w[0], fma(a[YZ], w[1], (a[Z] - pi) * w[ND - 1]));
                }
                *dr = fma(g, q, *dr);
            }
        }
    }
};

// One translation unit per dimension: defines launch_force_<ND>d_f64.
template <int ND, int KK>
static int launch_f64_nd(const ForceArgs& A, bool count_only, cudaStream_t s) {
    if (count_only || A.pfn == GC_PFN_COUNT || A.pfn == GC_PFN_INTERPOLATE || A.pfn == GC_PFN_XSPH)
        return launch_nd<ND, KK>(A, count_only, s);
    return launch_win_nd<PhysF64, ND, KK>(A, s);
}
#define GC_DEFINE_FORCE_F64_TU(NDIM, NAME)                                                                          \
    int NAME(const ForceArgs& A, bool count_only, cudaStream_t s) {                                                 \
        if (A.kk == GC_KERNEL_CUBIC_SPLINE) return launch_f64_nd<NDIM, GC_KERNEL_CUBIC_SPLINE>(A, count_only, s);   \
        return launch_f64_nd<NDIM, GC_KERNEL_WENDLAND_C2>(A, count_only, s);                                        \
    }

}  // namespace gc
