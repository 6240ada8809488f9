// k_force_impl.cuh — the buffered sweep of the counting, interpolation and
// velocity-adjust (XSPH) functors in FP64, and what it shares with the window
// sweep of the others (k_sweep_win.cuh).
//
// Gather formulation of src/Interaction.jl:393-732: one thread owns one
// system_a particle and sums its side of every accepted pair of every
// interaction of the current stage, in registers, then writes once.  The
// reference's coloured half-shell writes both endpoints; the functors here are
// exactly antisymmetric (or symmetric) under i↔j and their terms the
// reference's own expressions, so each side's term is bit-identical to the one
// the reference adds — only the order of the additions differs.
//
// Candidate enumeration walks the same 3-cell strips of the CSR grid as the
// reference (3 strips in 2-D, 9 in 3-D) and applies the same acceptance
// test r² < (2h)² on the same FP64 dx, so the neighbour sets are
// bit-identical.  Accepted neighbour indices are staged in a per-thread
// column of shared memory and processed in batches, so that the pair terms
// run with every lane busy instead of diverging on rejections.
//
// The arithmetic relies on -fmad=false.
#pragma once
#include <type_traits>
#include <cstdio>
#include <cuda_pipeline.h>

#include "gc_device.cuh"
#include "gc_force.h"
#include "gc_kernels.h"

namespace gc {

template <int ND>
struct OwnState {
    double x[ND], v[ND];
    double rho;
};

// ------------------------------------------------------- pair physics
template <int ND, int NS>
struct Acc {
    double dv[ND];
    double dr;
    double sr[NS > 0 ? NS : 1];
    double w[ND == 2 ? 1 : 3];
};

// Neighbour j's FP64 state, read from system_b's planar arrays.
struct NbGlobal {
    const InterRef& r;
    int64_t j;
    __device__ __forceinline__ double x(int d) const { return r.bx[d * r.bN + j]; }
    __device__ __forceinline__ double v(int d) const { return r.bv[d * r.bN + j]; }
    __device__ __forceinline__ double rho() const { return r.brho[j]; }
    __device__ __forceinline__ double stress(int q) const { return r.bstress[q * r.bN + j]; }
};

// One candidate j (source nb) of reference r for owned particle i: the
// exact reference test r² < (2h)² (src/Interaction.jl:546-548) on the FP64
// positions, then the functor's i-side term.  Returns 1 when accepted.
template <int ND, int NS, int PFN, int KK>
__device__ __forceinline__ int process_pair(const ForceArgs& A, const InterRef& r, const GridInst& G,
                                            const PfnInst& P, int k, const OwnState<ND>& o, const NbGlobal& nb,
                                            Acc<ND, NS>& acc) {
    double dx[ND];
#pragma unroll
    for (int d = 0; d < ND; ++d) dx[d] = o.x[d] - nb.x(d);
    double rr = dotv<ND>(dx, dx);
    if (!(rr < G.cutoff_sq)) return 0;
    if (PFN == GC_PFN_COUNT) {
        acc.dv[0] += 1.0;
        acc.dr += 1.0;
        return 1;
    }
    if (PFN == GC_PFN_INTERPOLATE) {
        // InterpolateFieldFn(ps_a, ps_b::VirtualParticleSystem)
        // src/PairwiseFunctors.jl:424-428 from the virtual particle's side:
        // kw = w·(m_a/ρ_a[i]); f[j] += kw·f_a[i]; w_sum[j] += kw
        const double q = sqrt(rr) / G.H;
        const double kw = kernel_w<KK>(G.knorm, q) * (G.bmass / nb.rho());
        if (A.imask & (1 << GC_FIELD_V)) {
#pragma unroll
            for (int d = 0; d < ND; ++d) acc.dv[d] = acc.dv[d] + kw * nb.v(d);
        }
        if (A.imask & (1 << GC_FIELD_RHO)) acc.dr = acc.dr + kw * nb.rho();
        if (A.imask & (1 << GC_FIELD_STRESS)) {
#pragma unroll
            for (int q2 = 0; q2 < NS; ++q2) acc.sr[q2] = acc.sr[q2] + kw * nb.stress(q2);
        }
        if (A.iwsum) acc.w[0] = acc.w[0] + (A.iwsum == 2 ? 1.0 : kw);  // 2: NeighborCountFn's count
        return 1;
    }
    if (PFN == GC_PFN_XSPH) {
        // XSPHPfn src/PairwiseFunctors.jl:364-389, xsph_veladjust
        // src/PairwisePhysics.jl:268-270: du = ((-ε·dv)·w)/(ρ_i + ρ_j),
        // v_adjustment_i += du·m_j.  Every system_b kind contributes its stored
        // velocity and density (a boundary wrapper forwards to its system);
        // the system_b side is this same term with the roles swapped.
        const double q = sqrt(rr) / G.H;
        const double wk = kernel_w<KK>(G.knorm, q);
        const double den = o.rho + nb.rho();
        const double mj = r.btype == BT_SELF ? A.a_mass[k] : G.bmass;
#pragma unroll
        for (int d = 0; d < ND; ++d) {
            const double du = (((-P.alpha) * (o.v[d] - nb.v(d))) * wk) / den;
            acc.dv[d] = acc.dv[d] + du * mj;
        }
        return 1;
    }
    return 0;
}

// ------------------------------------------------------------ policy
// The gather policy of the counting, interpolation and velocity-adjust functors.
template <int ND, int NS, int PFN, int KK>
struct PhysGather {
    struct Own {
        OwnState<ND> o;
    };
    using AccT = Acc<ND, NS>;
    static __device__ __forceinline__ void load(const ForceArgs& A, int64_t gi, Own& w) {
        const int64_t N = A.aN;
#pragma unroll
        for (int d = 0; d < ND; ++d) {
            w.o.x[d] = A.ax[d * N + gi];
            w.o.v[d] = A.av[d * N + gi];
        }
        w.o.rho = A.arho[gi];
    }
    static __device__ __forceinline__ const double* xpos(const Own& w) { return w.o.x; }
    static __device__ __forceinline__ void init(const ForceArgs& A, int64_t gi, AccT& acc, bool from_memory) {
        const int64_t N = A.aN;
#pragma unroll
        for (int d = 0; d < ND; ++d) acc.dv[d] = 0.0;
        acc.dr = 0.0;
        if (!from_memory) return;
        if (PFN == GC_PFN_INTERPOLATE) {
            // targets: v (advdt), rho (adrhodt), stress (asr), w_sum (avort)
            if (A.imask & (1 << GC_FIELD_V)) {
#pragma unroll
                for (int d = 0; d < ND; ++d) acc.dv[d] = A.advdt[d * N + gi];
            }
            if (A.imask & (1 << GC_FIELD_RHO)) acc.dr = A.adrhodt[gi];
            if (A.imask & (1 << GC_FIELD_STRESS)) {
#pragma unroll
                for (int q = 0; q < NS; ++q) acc.sr[q] = A.asr[q * N + gi];
            }
            acc.w[0] = A.iwsum ? A.avort[gi] : 0.0;
        } else {  // XSPH (advdt is the v_adjustment array here) or counting
#pragma unroll
            for (int d = 0; d < ND; ++d) acc.dv[d] = A.advdt[d * N + gi];
            if (PFN == GC_PFN_COUNT) acc.dr = A.adrhodt[gi];
        }
    }
    static __device__ __forceinline__ void store(const ForceArgs& A, int64_t gi, const AccT& acc) {
        const int64_t N = A.aN;
        if (PFN == GC_PFN_INTERPOLATE) {
            if (A.imask & (1 << GC_FIELD_V)) {
#pragma unroll
                for (int d = 0; d < ND; ++d) A.advdt[d * N + gi] = acc.dv[d];
            }
            if (A.imask & (1 << GC_FIELD_RHO)) A.adrhodt[gi] = acc.dr;
            if (A.imask & (1 << GC_FIELD_STRESS)) {
#pragma unroll
                for (int q = 0; q < NS; ++q) A.asr[q * N + gi] = acc.sr[q];
            }
            if (A.iwsum) A.avort[gi] = acc.w[0];
        } else {
#pragma unroll
            for (int d = 0; d < ND; ++d) A.advdt[d * N + gi] = acc.dv[d];
            if (PFN == GC_PFN_COUNT) A.adrhodt[gi] = acc.dr;
        }
    }
    template <int P2>
    static __device__ __forceinline__ int pair(const ForceArgs& A, const InterRef& r, const GridInst& G,
                                               const PfnInst& P, int k, const Own& w, int32_t j, AccT& acc) {
        return process_pair<ND, NS, P2, KK>(A, r, G, P, k, w.o, NbGlobal{r, j}, acc);
    }
};

// ------------------------------------------------ shared sweep pieces
// The divisions of cells_of, out of line (rarely needed).
template <int ND>
static __device__ __noinline__ bool cells_divided(const GridInst& G, const double* x, int32_t* c) {
    bool ok = true;
    for (int d = 0; d < ND; ++d) {
        int64_t cd;
        const bool in = floor_i64(__dsub_rn(x[d], G.ming[d]) / G.cell, &cd) && cd >= 1 && cd < G.ng[d] - 1;
        c[d] = in ? (int32_t)cd : 1;
        ok = ok && in;
    }
    return ok;
}

// Cell coordinates floor((x − ming)/cell), and whether all lie inside the
// grid's border cells (1 where not).  The quotients come from the stored
// reciprocal, within a few ulps of the divided ones; only where that leaves
// a floor in doubt (next to an integer, or out of range) are the divisions
// made (src/Interaction.jl:197-206).
template <int ND>
__device__ __forceinline__ bool cells_of(const GridInst& G, const double* x, int32_t* c) {
    double q[ND];
    int64_t n[ND];
#pragma unroll
    for (int d = 0; d < ND; ++d) {
        q[d] = __dsub_rn(x[d], G.ming[d]) * G.inv_cell;
        n[d] = G.ng[d];
    }
    bool ok = true, sure = true;
#pragma unroll
    for (int d = 0; d < ND; ++d) {
        c[d] = __double2int_rd(q[d]);
        const double frac = q[d] - (double)c[d];
        sure = sure && frac > 1e-9 && frac < 1.0 - 1e-9 && q[d] < 1048576.0;
        ok = ok && c[d] >= 1 && c[d] < n[d] - 1;
    }
    if (sure && ok) return true;
    double xs[ND];
    int32_t cs[ND];
#pragma unroll
    for (int d = 0; d < ND; ++d) xs[d] = x[d];
    ok = cells_divided<ND>(G, xs, cs);
#pragma unroll
    for (int d = 0; d < ND; ++d) c[d] = cs[d];
    return ok;
}

// Per (warp, interaction) set-up of both sweeps.  Returns false when the
// warp has nothing to do with this interaction: system_b's box is out of
// reach of every lane (the box test has a 0.1% margin, so no pair is lost)
// or the instance's grid did not fit its buffer (flagged, nothing read).
// Otherwise c holds each lane's cell coordinates (ok: inside the grid, with
// a flagged error when not), c0/c1 lane 0's first two, and coop whether all
// active lanes share lane 0's grid column.
template <int ND>
__device__ __forceinline__ bool ref_cells(const ForceArgs& A, const InterRef& r, const GridInst& G, int k,
                                          const double* ox, bool active, int lane, int32_t gi, int32_t* c,
                                          bool& ok, int32_t& c0, int32_t& c1, bool& coop) {
    const unsigned FULL = 0xffffffffu;
    if (r.bbox) {
        const SysInst& B = r.bbox[k];
        bool near = B.n > 0;
        const double m = 1.001 * G.cell;
#pragma unroll
        for (int d = 0; d < ND; ++d) near = near && ox[d] >= B.bbmin[d] - m && ox[d] <= B.bbmax[d] + m;
        if (!__any_sync(FULL, active && near)) {
            if (active && r.counts) r.counts[gi] = 0;
            return false;
        }
    }
    if (G.cellbase + G.ncells > r.cs_cells) {
        if (lane == 0) atomicOr(A.err, ERR_CAPACITY);
        if (active && r.counts) r.counts[gi] = 0;
        return false;
    }
    // cell coordinates (a grid has < 2^31 cells, so they fit int32)
    ok = cells_of<ND>(G, ox, c);
    if (active && !ok) atomicOr(A.err, ERR_CAPACITY);
    c0 = __shfl_sync(FULL, c[0], 0);
    c1 = ND == 3 ? __shfl_sync(FULL, c[1], 0) : 0;
    const bool same = ok && c[0] == c0 && (ND == 2 || c[1] == c1);
    coop = __all_sync(FULL, !active || same);
    return true;
}

// The warp's range [zlo, zhi] of last-dimension cells over its active lanes.
template <int ND>
__device__ __forceinline__ void warp_zrange(const int32_t* c, bool active, int32_t& zlo, int32_t& zhi) {
    const unsigned FULL = 0xffffffffu;
    zlo = active ? c[ND - 1] : INT32_MAX;
    zhi = active ? c[ND - 1] : INT32_MIN;
#pragma unroll
    for (int o2 = 16; o2 > 0; o2 >>= 1) {
        const int32_t a2 = __shfl_xor_sync(FULL, zlo, o2), b2 = __shfl_xor_sync(FULL, zhi, o2);
        zlo = a2 < zlo ? a2 : zlo;
        zhi = b2 > zhi ? b2 : zhi;
    }
}

// Conservative FP32 prefilter of a batch of mb <= 32 candidates against this
// lane (coordinates relative to lane 0; rows of the batch `stride` floats
// apart, entries past mb far away): bit t set when candidate t may be within
// the cutoff.  Two candidates per packed FP32x2 instruction.  The chain
// starts from −cut, so it ends at r² − cut and its sign bit is the hit: one
// funnel shift per candidate moves it into the mask (candidates pushed from
// last to first).  A NaN result is not guaranteed a clear sign bit, so the
// callers mask out inactive lanes.
template <int ND>
__device__ __forceinline__ unsigned batch_hits(const float* cb, int stride, int mb, const float* xi, float cut_f) {
    const float2 neg1 = make_float2(-1.0f, -1.0f);
    const float2 ncut = make_float2(-cut_f, -cut_f);
    unsigned hits = 0;
#pragma unroll
    for (int t0 = 0; t0 < 32; t0 += 8) {
        if (t0 >= mb) break;  // warp-uniform
        unsigned h8 = 0;
#pragma unroll
        for (int t = 4; t >= 0; t -= 4) {
            float2 ra = ncut, rb = ncut;  // candidates t, t+1 and t+2, t+3
#pragma unroll
            for (int d = 0; d < ND; ++d) {
                const float* row = cb + d * stride + t0 + t;
                const float2 xa = *reinterpret_cast<const float2*>(row), xb = *reinterpret_cast<const float2*>(row + 2);
                const float2 xo = make_float2(xi[d], xi[d]);
                const float2 da = __ffma2_rn(xa, neg1, xo), db = __ffma2_rn(xb, neg1, xo);
                ra = __ffma2_rn(da, da, ra);
                rb = __ffma2_rn(db, db, rb);
            }
            h8 = __funnelshift_l(__float_as_uint(rb.y), h8, 1);
            h8 = __funnelshift_l(__float_as_uint(rb.x), h8, 1);
            h8 = __funnelshift_l(__float_as_uint(ra.y), h8, 1);
            h8 = __funnelshift_l(__float_as_uint(ra.x), h8, 1);
        }
        hits |= h8 << t0;
    }
    return hits;
}

// This lane's own strip range [lo, hi) and the self pair as a mask over the
// batch of 32 candidates starting at index jb.
__device__ __forceinline__ unsigned own_allow(int32_t lo, int32_t hi, int32_t jb, bool self, int32_t gi) {
    const int32_t tlo = lo - jb, thi = hi - jb;
    unsigned allow = tlo <= 0 ? 0xffffffffu : (tlo >= 32 ? 0u : 0xffffffffu << tlo);
    allow &= thi >= 32 ? 0xffffffffu : (thi <= 0 ? 0u : 0xffffffffu >> (32 - thi));
    if (self) {
        const int32_t ts = gi - jb;
        if (ts >= 0 && ts < 32) allow &= ~(1u << ts);
    }
    return allow;
}

// Per-warp copies of an interaction's grid and functor parameters (the pair
// loops read these: loop-invariant values the register budget would
// otherwise re-load from global memory for every pair).
constexpr int SWEEP_GI_BYTES = ((int)sizeof(GridInst) + 15) / 16 * 16;
constexpr int SWEEP_PI_BYTES = ((int)sizeof(PfnInst) + 15) / 16 * 16;
constexpr int SWEEP_PARAM_BYTES = SWEEP_GI_BYTES + SWEEP_PI_BYTES;

// Copy of a parameter block into a warp's shared memory, 4 bytes per lane.
template <class T>
__device__ __forceinline__ void warp_copy(T* dst, const T& src, int lane) {
    static_assert(sizeof(T) % 4 == 0, "4-byte words");
    const int* s = reinterpret_cast<const int*>(&src);
    int* d = reinterpret_cast<int*>(dst);
    for (int i = lane; i < (int)(sizeof(T) / 4); i += 32) d[i] = s[i];
}

// Shared memory of one block of k_sweep: the staged-neighbour columns, the
// per-warp candidate coordinates (ND rows of 32, then lane 0's position) and
// the per-warp parameter copies.
template <int ND>
__host__ __device__ constexpr int sweep_smem_bytes(int buf) {
    return (buf * FORCE_TPB * 4 + (FORCE_TPB / 32) * ND * 34 * 4 + 15) / 16 * 16 + (FORCE_TPB / 32) * SWEEP_PARAM_BYTES;
}

// ---------------------------------------------------------------- kernel
// One warp owns one group: up to 32 consecutive (sorted) system_a particles
// of one grid column (all cell coordinates but the last equal).  For each
// 3-cell strip of the reference stencil the warp walks the union of its
// lanes' candidate ranges — contiguous in the CSR because cells along the
// last dimension are consecutive — loading 32 candidates at a time with one
// coalesced load and broadcasting them by shuffles.  A lane keeps a
// candidate only inside its own strip range [cs[z-1], cs[z+2]) and when a
// conservative FP32 distance test passes; the policy's pair() then applies
// the exact reference test r² < (2h)² on FP64 positions.  Staged indices go
// to the lane's shared-memory column; when any column is nearly full the
// whole warp evaluates its staged pairs, so the pair physics runs on
// converged warps.
template <class Phys, bool COUNT_ONLY, int PFN>
__device__ __forceinline__ int flush_all(const ForceArgs& A, const InterRef& r, const GridInst& G,
                                         const PfnInst& P, int k, const typename Phys::Own& w, int nbuf,
                                         const int32_t* col, int BT, typename Phys::AccT& acc) {
    constexpr int P2 = COUNT_ONLY ? GC_PFN_COUNT : PFN;
    int acc_n = 0;
    for (int t = 0; t < nbuf; ++t) acc_n += Phys::template pair<P2>(A, r, G, P, k, w, col[t * BT], acc);
    return acc_n;
}

template <class Phys, int ND, int PFN, bool COUNT_ONLY>
__global__ void __launch_bounds__(FORCE_TPB, 4) k_sweep(ForceArgs A) {
    pdl_enter();
    extern __shared__ int32_t sbuf[];
    constexpr int BUF = FORCE_BUF;
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const int tid = threadIdx.x;
    const int BT = blockDim.x;
    int32_t* col = sbuf + tid;
    // per-warp candidate coordinates, ND rows of 32 floats, after the columns
    // per warp: ND rows of 32 candidate coordinates, then ND doubles (lane 0's position)
    float* cand = reinterpret_cast<float*>(sbuf + BUF * FORCE_TPB) + (tid >> 5) * (ND * 34);
    char* pbase = reinterpret_cast<char*>(sbuf) + (BUF * FORCE_TPB * 4 + (FORCE_TPB / 32) * ND * 34 * 4 + 15) / 16 * 16 +
                  (tid >> 5) * SWEEP_PARAM_BYTES;
    GridInst* gsm = reinterpret_cast<GridInst*>(pbase);
    PfnInst* psm = reinterpret_cast<PfnInst*>(pbase + SWEEP_GI_BYTES);
    const int64_t ngroups = *A.ngroups;
    const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t wg = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; wg < ngroups; wg += nwarps) {
        const int2 grp = A.groups[wg];
        const bool active = lane < group_count(grp);
        const int32_t gi = grp.x + (active ? lane : 0);  // packed indices fit int32
        const int k = group_inst(grp);
        typename Phys::Own w;
        Phys::load(A, gi, w);
        const double* ox = Phys::xpos(w);
        typename Phys::AccT acc;
        Phys::init(A, gi, acc, !COUNT_ONLY);

        for (int ri = 0; ri < A.nref; ++ri) {
            const InterRef& r = A.ref[ri];
            const GridInst& G = r.gi[k];
            const PfnInst& P = r.pi[k];
            int32_t c[ND], c0, c1;
            bool ok, coop;
            if (!ref_cells<ND>(A, r, G, k, ox, active, lane, gi, c, ok, c0, c1, coop)) continue;
            warp_copy(gsm, G, lane);
            warp_copy(psm, P, lane);
            __syncwarp();
            const GridInst& Gs = *gsm;
            const PfnInst& Ps = *psm;
            const int64_t Nb = r.bN;
            const bool self = r.btype == BT_SELF;
            int nbuf = 0;
            int32_t accepted = 0;
            if (coop) {
                constexpr int L = ND - 1;  // last dimension
                int32_t zlo, zhi;
                warp_zrange<ND>(c, active, zlo, zhi);
                // Conservative FP32 prefilter in coordinates relative to lane 0:
                // |rel| spans a few cells, so single-precision rounding moves r²
                // by < 1e-5 relative; the 1e-3 margin keeps every true pair.
                // Inactive lanes have an empty own range and accept nothing.
                // lane 0's position, the origin of the relative coordinates,
                // kept in the warp's shared memory rather than in registers
                double* xref = reinterpret_cast<double*>(cand + ND * 32);
                float xi[ND];
                if (lane == 0) {
#pragma unroll
                    for (int d = 0; d < ND; ++d) xref[d] = ox[d];
                }
                __syncwarp();
#pragma unroll
                for (int d = 0; d < ND; ++d) xi[d] = active ? (float)(ox[d] - xref[d]) : 0.f;
                const float cut_f = (float)(G.cutoff_sq * 1.001);
                const int64_t ngl = G.ng[L];
                const int nstrips = ND == 2 ? 3 : 9;
                for (int sidx = 0; sidx < nstrips; ++sidx) {
                    int64_t colflat;
                    if (ND == 2) colflat = c0 + sidx - 1;
                    else colflat = (c0 + sidx / 3 - 1) * G.ng[1] + (c1 + sidx % 3 - 1);
                    const int64_t base = G.cellbase + colflat * ngl;
                    const int32_t u0 = r.cs[base + zlo - 1], u1 = r.cs[base + zhi + 2];
                    const int32_t lo = active ? r.cs[base + c[L] - 1] : 0, hi = active ? r.cs[base + c[L] + 2] : 0;
                    for (int32_t ch = u0; ch < u1; ch += 32) {
                        if (__any_sync(FULL, nbuf > BUF - 32)) {
                            accepted += flush_all<Phys, COUNT_ONLY, PFN>(A, r, Gs, Ps, k, w, nbuf, col, BT, acc);
                            nbuf = 0;
                            __syncwarp();
                        }
                        // 32 candidates, coordinates relative to lane 0, staged in
                        // shared memory (beyond the range: far away)
                        const int32_t jl = ch + lane;
#pragma unroll
                        for (int d = 0; d < ND; ++d)
                            cand[d * 32 + lane] = jl < u1 ? (float)(r.bx[d * Nb + jl] - xref[d]) : 1e30f;
                        __syncwarp();
                        const int m = u1 - ch < 32 ? (int)(u1 - ch) : 32;
                        unsigned hits = batch_hits<ND>(cand, 32, m, xi, cut_f) & own_allow(lo, hi, ch, self, gi);
                        while (hits) {
                            const int t = __ffs(hits) - 1;
                            hits &= hits - 1;
                            col[(nbuf++) * BT] = ch + t;
                        }
                        __syncwarp();
                    }
                }
                accepted += flush_all<Phys, COUNT_ONLY, PFN>(A, r, Gs, Ps, k, w, nbuf, col, BT, acc);
                nbuf = 0;
                __syncwarp();
            } else if (active && ok) {
                // rare: lanes disagree on the column in this grid; walk own strips
                const int nstrips = ND == 2 ? 3 : 9;
                for (int sidx = 0; sidx < nstrips; ++sidx) {
                    int64_t base;
                    if (ND == 2) base = G.cellbase + (c[0] + sidx - 1) * G.ng[1] + (c[1] - 1);
                    else base = G.cellbase + ((c[0] + sidx / 3 - 1) * G.ng[1] + (c[1] + sidx % 3 - 1)) * G.ng[2] + (c[2] - 1);
                    const int32_t s0 = r.cs[base], e0 = r.cs[base + 3];
                    for (int32_t j = s0; j < e0; ++j) {
                        if (self && j == gi) continue;
                        col[(nbuf++) * BT] = j;
                        if (nbuf == BUF) {
                            accepted += flush_all<Phys, COUNT_ONLY, PFN>(A, r, Gs, Ps, k, w, nbuf, col, BT, acc);
                            nbuf = 0;
                        }
                    }
                }
                accepted += flush_all<Phys, COUNT_ONLY, PFN>(A, r, Gs, Ps, k, w, nbuf, col, BT, acc);
                nbuf = 0;
            }
            __syncwarp();
            if (active && r.counts) r.counts[gi] = accepted;
        }
        if (!COUNT_ONLY && active) Phys::store(A, gi, acc);
        __syncwarp();
    }
}

// ------------------------------------------------------------ dispatch
template <int ND, int NS, int PFN, int KK>
static void launch_t(const ForceArgs& A, cudaStream_t s) {
    constexpr bool COUNT_ONLY = PFN == GC_PFN_NONE;  // counting without sums
    constexpr int P2 = COUNT_ONLY ? GC_PFN_COUNT : PFN;
    int64_t blocks = (A.aN * 32 + FORCE_TPB - 1) / FORCE_TPB;
    if (blocks > (int64_t)A.num_sms * 16) blocks = (int64_t)A.num_sms * 16;
    if (blocks < 1) blocks = 1;
    const size_t smem = (size_t)sweep_smem_bytes<ND>(FORCE_BUF);
    k_sweep<PhysGather<ND, NS, P2, KK>, ND, P2, COUNT_ONLY><<<(int)blocks, FORCE_TPB, smem, s>>>(A);
    g_launches.fetch_add(1, std::memory_order_relaxed);
}

// The buffered sweep: neighbour counts, InterpolateFieldFn (and
// NeighborCountFn) and XSPHPfn.
template <int ND, int KK>
static int launch_nd(const ForceArgs& A, bool count_only, cudaStream_t s) {
    if (count_only) {
        launch_t<ND, 0, GC_PFN_NONE, KK>(A, s);
        return 0;
    }
    if (A.pfn == GC_PFN_COUNT) {
        launch_t<ND, 0, GC_PFN_COUNT, KK>(A, s);
        return 0;
    }
    if (A.pfn == GC_PFN_XSPH) {
        launch_t<ND, 0, GC_PFN_XSPH, KK>(A, s);
        return 0;
    }
    if (A.pfn != GC_PFN_INTERPOLATE) return GC_ERR_UNSUPPORTED;
    if (!(A.imask & (1 << GC_FIELD_STRESS))) launch_t<ND, 0, GC_PFN_INTERPOLATE, KK>(A, s);
    else if (ND == 2 && A.ns == 3) launch_t<ND, 3, GC_PFN_INTERPOLATE, KK>(A, s);
    else if (ND == 2 && A.ns == 4) launch_t<ND, 4, GC_PFN_INTERPOLATE, KK>(A, s);
    else if (ND == 3 && A.ns == 6) launch_t<ND, 6, GC_PFN_INTERPOLATE, KK>(A, s);
    else return GC_ERR_UNSUPPORTED;
    return 0;
}

}  // namespace gc
