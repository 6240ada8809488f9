// k_sweep_win.cuh — the pair sweep of the fluid and stress functors, over a
// policy of their arithmetic (PhysF32 in k_sweep_f32.cuh, PhysF64 in
// k_sweep_f64.cuh).
//
// The walk is k_force_impl.cuh's (one warp per group of up to 32 consecutive
// particles of one grid column, the union of its lanes' candidates), but a
// warp takes the strips of a whole window at once: the three strips of one
// row of the 3-D stencil, or the whole 2-D stencil.  It copies a chunk of the
// window's candidates (records, gc_force.h) into shared memory, tests their
// FP32 positions against every lane, and then each lane evaluates its
// accepted candidates from the copies.  A lane alone accepts different
// numbers of a single strip's candidates, and a warp's pair loop runs as long
// as its busiest lane: on a jittered 3-D lattice at h = 1.2 spacings 119
// rounds a group strip by strip, 88 by windows, 55 if all lanes were busy.
// The interactions in reach of a group are found by one lane each, and the
// next group's state is prefetched.
#pragma once
#include <cfloat>
#include <math_constants.h>

#include "k_force_impl.cuh"

namespace gc {

template <int ND>
__device__ __forceinline__ double dot_exact(const double* a, const double* b) {
    double s = __dmul_rn(a[0], b[0]);
#pragma unroll
    for (int d = 1; d < ND; ++d) s = __dadd_rn(s, __dmul_rn(a[d], b[d]));
    return s;
}

// Conservative FP32 test of a batch of mb <= 32 candidates (batch_hits of
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

// A candidate two cells away from a lane's own is out of its reach but for
// the rounding of the two cell coordinates (their quotients run up to the
// grid's cells per dimension): the relative band below (2h)² in which the
// lane's own strip range decides about it.
template <int ND>
__device__ __forceinline__ double strip_doubt(const GridInst& G) {
    int64_t n = G.ng[0];
#pragma unroll
    for (int d = 1; d < ND; ++d) n = G.ng[d] > n ? G.ng[d] : n;
    return 1e-9 + 1e-14 * (double)n;
}

// Loads from a shared-memory address (32 bits, so the pair loop's address
// arithmetic stays narrow).
__device__ __forceinline__ float4 lds128(uint32_t a) {
    return *reinterpret_cast<const float4*>(__cvta_shared_to_generic(a));
}
__device__ __forceinline__ unsigned lds32(uint32_t a) {
    return *reinterpret_cast<const unsigned*>(__cvta_shared_to_generic(a));
}

__device__ __forceinline__ void sts32(uint32_t a, unsigned x) {
    *reinterpret_cast<unsigned*>(__cvta_shared_to_generic(a)) = x;
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
// with the empty one that ends them (LIST: and a word before them).
template <int ND, int NQ, int CH, bool LIST>
__host__ __device__ constexpr int win_warp_bytes() {
    return NQ * CH * 16 + ND * CH * 4 + (CH / 32 + 1 + LIST) * 128;
}

template <class Phys, int ND, int PFN, int MINB, int CH, bool LIST>
__global__ void __launch_bounds__(WIN_TPB, MINB) k_sweep_win(ForceArgs A) {
    pdl_enter();
    static_assert(CH % 32 == 0 && CH / 32 <= 8, "a lane's masks are numbered by batch, four bits each in a word");
    constexpr int NQ = Phys::NQ;
    constexpr int NSTR = 3, NWIN = ND == 2 ? 1 : 3;  // strips per window, windows
    constexpr int WB = win_warp_bytes<ND, NQ, CH, LIST>();
    constexpr int L = ND - 1;
    extern __shared__ float4 sstg[];
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    char* wbase = reinterpret_cast<char*>(sstg) + (threadIdx.x >> 5) * WB;
    float4* slots = reinterpret_cast<float4*>(wbase);
    float* cand = reinterpret_cast<float*>(wbase + NQ * CH * 16);
    unsigned* masks = reinterpret_cast<unsigned*>(wbase + NQ * CH * 16 + ND * CH * 4 + LIST * 128) + lane;
    const uint32_t slots_s = (uint32_t)__cvta_generic_to_shared(slots);
    const uint32_t masks_s = (uint32_t)__cvta_generic_to_shared(masks);
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
            const float4* rec = A.arec + (int64_t)gi * Phys::RQ;
            Phys::rec_read([&](int q) { return rec[q]; }, o);
        }
        float xi[ND], xmax = 0.f;
#pragma unroll
        for (int d = 0; d < ND; ++d) xi[d] = Phys::h(o, d);
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
                for (int d = 0; d < ND; ++d) {
                    const double x0 = Phys::EXACT ? 0.0 : A.origin[k * MAXD + d];
                    reach = reach & (x0 + (double)ghi[d] >= B.bbmin[d] - m) & (x0 + (double)glo[d] <= B.bbmax[d] + m);
                }
            }
            visit = __ballot_sync(FULL, reach);
        }
        // the next group's state on its way to this SM
        {
            const int64_t gn = next.x + (lane < group_count(next) ? lane : 0);
            asm volatile("prefetch.global.L1 [%0];" ::"l"(A.arec + gn * Phys::RQ));
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
                typename Phys::Real da = 0;  // own distance to a dynamic boundary's plane
                if (r.btype == BT_DYNAMIC) {
                    double t = (x[0] - G.point[0]) * G.normal[0];
#pragma unroll
                    for (int d = 1; d < ND; ++d) t += (x[d] - G.point[d]) * G.normal[d];
                    da = (typename Phys::Real)t;
                }
                if (active && !ok) atomicOr(A.err, ERR_CAPACITY);
                const int32_t c0 = __shfl_sync(FULL, c[0], 0), c1 = ND == 3 ? __shfl_sync(FULL, c[1], 0) : 0;
                const bool same = ok && c[0] == c0 && (ND == 2 || c[1] == c1);
                // positions over 2^20 cells from their instance's point, of which an FP32
                // pair would lose more than FP32 arithmetic does, take FP64 differences
                const bool far = !Phys::EXACT && xmax * (float)G.inv_cell > 1048576.f;
                const bool coop = !far && __all_sync(FULL, !active || same);
                const bool self = r.btype == BT_SELF;
                typename Phys::Acc acc;
                Phys::zero(acc);
                const typename Phys::Par par = Phys::params(A, r, G, P, k, xmax + 2.f * (float)G.cell);
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
                    const int nq = r.btype == BT_DYNAMIC ? Phys::NQP : NQ;  // quads staged per candidate
                    // conservative cutoff of the candidate test: the coordinates' rounding, and
                    // 1e-5 for the arithmetic's, below 1e-6
                    const float ce = (float)G.cell + 4.8e-7f * (xmax + 2.f * (float)G.cell);
                    const float cut_f = 1.00001f * ce * ce;
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
                    auto exact_slot = [&](int wi, int32_t ch, int32_t t, double& r2) {
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
                        double y[ND];
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
                        // LIST: the candidates that were not counted.  In 2-D (few) the last four
                        // of the chunk, their slots' numbers + 1 a byte each; in 3-D those of the
                        // current mask, which take its place when the next one comes.
                        constexpr bool BYTES = LIST && ND == 2, MASKS = LIST && ND == 3;
                        unsigned left = 0;
                        const int32_t before = accepted;
                        auto pairs = [&](auto btk) {
                            uint32_t mp = masks_s, batch = slots_s;
                            unsigned cur = 0, nxt = lds32(mp), bq = bn;
                            while (cur | nxt) {
                                if (Phys::EXACT) {
                                    if (cur == 0) {
                                        cur = nxt;
                                        batch = slots_s + (bq & 15u) * (32 * 16);
                                        bq >>= 4;
                                        mp += 128;
                                        nxt = lds32(mp);
                                    }
                                } else {
                                    // selects: a branch here splits the warp nearly every round,
                                    // which the FP32 terms do not hide (699 against 690 us on the
                                    // million-particle dam break; FP64 prefers the branch)
                                    const bool pop = cur == 0;
                                    if (MASKS) {
                                        if (pop) sts32(mp - 128, left);
                                        left = pop ? 0u : left;
                                    }
                                    cur = pop ? nxt : cur;
                                    batch = pop ? slots_s + (bq & 15u) * (32 * 16) : batch;
                                    bq = pop ? bq >> 4 : bq;
                                    mp += pop ? 128 : 0;
                                    nxt = lds32(mp);
                                }
                                const int t = __clz(cur);
                                cur ^= 0x80000000u >> t;
                                const uint32_t slot = batch + t * 16;
                                const int in = Phys::template pair<decltype(btk)::value, LIST>(
                                    par, G, P, o, da, [&](int q) { return lds128(slot + q * CH * 16); },
                                    [&]() {
                                        double r2;
                                        return exact_slot(wc, cc, (int)(slot - slots_s) >> 4, r2);
                                    },
                                    nearest, acc);
                                accepted += in;
                                if (BYTES) left = in ? left : __byte_perm(left, ((slot - slots_s) >> 4) + 1, 0x2104);
                                if (MASKS) left = in ? left : left | 0x80000000u >> t;
                            }
                            if (MASKS) sts32(mp - 128, left);
                        };
                        if (self && !Phys::diffuses(par)) pairs(std::integral_constant<int, BT_SELF>{});
                        else pairs(std::integral_constant<int, -1>{});
                        // rare, but for particles at rest on a lattice with 2h a multiple of
                        // its spacing: candidates so near the cutoff that FP64 decides (counts
                        // them).  The masks are cut down to these first, so that the lanes wait
                        // for their FP64 positions together: the resting 80 k column's sweep
                        // 61 -> 40 us, the others unchanged.  And pairs at no distance, for
                        // which the reference's kernel gradient is 0/0: by their FP64 r², as
                        // FP32 pairs are equal an ulp apart too (709 us at 1 M particles with
                        // and without; decided in the first of the two loops, 724).  LIST: FP64 decides about
                        // all that was not counted, two candidates at a time for the latency.
                        if constexpr (LIST) {
                            int32_t u2[NSTR], e2[NSTR + 1];
                            window(wc, u2, e2);
                            // (the strip's range matters along its own direction alone)
                            const double edge = G.cell * (1.0 - strip_doubt<ND>(G)), cut = G.cutoff_sq;
                            double xo[ND];
#pragma unroll
                            for (int d = 0; d < ND; ++d) xo[d] = A.ax[d * A.aN + gi];
                            auto decide = [&](int t0, int t1) {  // (t1 < 0: none)
                                int t[2] = {t0, t1 < 0 ? t0 : t1};
                                double y[2][ND], r2[2];
                                bool in[2];
#pragma unroll
                                for (int q = 0; q < 2; ++q) {
                                    const int32_t tt = cc + t[q];
                                    const int32_t j = tt + (tt < e2[1] ? u2[0] : tt < e2[2] ? u2[1] : u2[2]);
#pragma unroll
                                    for (int d = 0; d < ND; ++d) y[q][d] = __dsub_rn(xo[d], r.bx[d * r.bN + j]);
                                    r2[q] = dot_exact<ND>(y[q], y[q]);
                                    in[q] = r2[q] < cut;
                                }
                                in[1] = in[1] && t1 >= 0;
#pragma unroll
                                for (int q = 0; q < 2; ++q) {
                                    if (in[q] && fabs(y[q][L]) > edge) in[q] = exact_slot(wc, cc, t[q], r2[q]);
                                    accepted += in[q];
                                    if (in[q] && (float)r2[q] == 0.f) Phys::spoil(par, acc);
                                }
                            };
                            const bool some = !Phys::lj_wall(r.btype) && (MASKS || left);
                            bool listed = BYTES;
                            if (BYTES && some && left >> 24) {
                                // four are all of them if the others were counted
                                int32_t others = before - accepted;
                                for (int mi = 0; mi < nm; ++mi) others += __popc(masks[mi * 32]);
                                listed = others == 4;
                            }
                            if (some && listed) {
                                for (; left; left >>= 16) decide((int)(left & 255u) - 1, (int)(left >> 8 & 255u) - 1);
                            } else if (some) {
                                for (int mi = 0; mi < nm; ++mi) {
                                    const int b = (bn >> (4 * mi) & 15u) * 32;
                                    for (unsigned cur = masks[mi * 32]; cur;) {
                                        const int t0 = __clz(cur);
                                        cur ^= 0x80000000u >> t0;
                                        int t1 = -1;
                                        if (MASKS && cur) {
                                            t1 = __clz(cur);
                                            cur ^= 0x80000000u >> t1;
                                            t1 += b;
                                        }
                                        // (2-D: all the accepted candidates, of which some were counted)
                                        if (MASKS || Phys::not_counted(par, o, [&](int c) { return slots[c * CH + b + t0]; }))
                                            decide(b + t0, t1);
                                    }
                                }
                            }
                        } else if (nearest <= Phys::band(par)) {
                            for (int mi = 0; mi < nm; ++mi) {
                                const int b = (bn >> (4 * mi) & 15u) * 32;
                                unsigned near = 0;
                                for (unsigned cur = masks[mi * 32]; cur;) {
                                    const int t = __clz(cur);
                                    cur ^= 0x80000000u >> t;
                                    auto quad = [&](int q) { return slots[q * CH + b + t]; };
                                    if (Phys::left_over(par, o, quad, acc)) near |= 0x80000000u >> t;
                                }
                                masks[mi * 32] = near;
                            }
                            if (!Phys::EXACT) {
                                unsigned near = 0;
                                for (int mi = -1;;) {
                                    while (!near && ++mi < nm) near = masks[mi * 32];
                                    if (!near) break;
                                    const int t = __clz(near);
                                    near ^= 0x80000000u >> t;
                                    double r2;
                                    if (!exact_slot(wc, cc, (int)(bn >> (4 * mi) & 15u) * 32 + t, r2)) continue;
                                    // (at no distance: counted already)
                                    if (r2 > 1e-9 * G.cutoff_sq) ++accepted;
                                    else if ((float)r2 == 0.f) Phys::spoil(par, acc);
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
                            if (r.btype != BT_DYNAMIC) Phys::rec_read([&](int q) { return rec[q]; }, b);
                            Phys::walked(par, G, P, o, da, b, y, r2, acc);
                            ++accepted;
                        }
                    }
                }
                if (active) Phys::store(A, r, G, k, par, gi, acc);
            }
            __syncwarp();
            if (active && r.counts) r.counts[gi] = accepted;
        }
        __syncwarp();
    }
}

// Shared memory of a block of which an SM holds `blocks` (228 KB, of which 1 KB
// a block is the system's; 1 KB to spare).
constexpr size_t sm_share(int blocks) { return (size_t)(228 * 1024 / (blocks < 2 ? 2 : blocks) - 2048); }

template <class Phys, int ND, int PFN, int C>
static int launch_win(const ForceArgs& A, cudaStream_t s) {
    constexpr WinCfg cf = Phys::EXACT ? WIN_CFGS64[C] : WIN_CFGS32[C];
    int64_t blocks = (A.aN * 32 + WIN_TPB - 1) / WIN_TPB;
    if (blocks > (int64_t)A.num_sms * cf.minb * 4) blocks = (int64_t)A.num_sms * cf.minb * 4;
    if (blocks < 1) blocks = 1;
    constexpr size_t need = (size_t)(WIN_TPB / 32) * win_warp_bytes<ND, Phys::NQ, cf.chunk, cf.list>();
    auto kern = k_sweep_win<Phys, ND, PFN, cf.minb, cf.chunk, cf.list>;
    // Few groups: a sweep launched while the kernel before it still runs
    // (programmatic dependent launch) finds free the SMs that finished first
    // and piles its blocks on those; with shared memory asked for beyond what
    // it needs no SM takes more than its even share.  18135 particles of 3-D
    // water, 8 blocks an SM at most: step 107 us; 5, 4 or 3: 93; 2: 96.
    size_t smem = need;
    if (A.sm_blocks && A.sm_blocks < cf.minb) smem = std::max(need, sm_share(A.sm_blocks));
    // Beyond 48 KB a block asks for it.  The attribute belongs to the current
    // device, and a process may have contexts on several: set at every such
    // launch (captured steps launch once), always to the most of this kernel.
    if (smem > 48 * 1024 &&
        cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)std::max(need, sm_share(2))) !=
            cudaSuccess)
        return GC_ERR_CUDA;
    kern<<<(int)blocks, WIN_TPB, smem, s>>>(A);
    g_launches.fetch_add(1, std::memory_order_relaxed);
    return 0;
}

template <template <int, int, int, int> class Phys, int ND, int NS, int PFN, int KK>
static int launch_win_cfg(const ForceArgs& A, cudaStream_t s) {
    using P = Phys<ND, NS, PFN, KK>;
    switch (A.cfg) {
        case 1: return launch_win<P, ND, PFN, 1>(A, s);
        case 2: return launch_win<P, ND, PFN, 2>(A, s);
        case 3: return launch_win<P, ND, PFN, 3>(A, s);
        default: return launch_win<P, ND, PFN, 0>(A, s);
    }
}

// The window sweep of A.pfn; GC_ERR_UNSUPPORTED for any other functor or
// shape of stress.
template <template <int, int, int, int> class Phys, int ND, int KK>
static int launch_win_nd(const ForceArgs& A, cudaStream_t s) {
    if (A.pfn == GC_PFN_FLUID) return launch_win_cfg<Phys, ND, 0, GC_PFN_FLUID, KK>(A, s);
    if (A.pfn == PFN_FLUID2) return launch_win_cfg<Phys, ND, 0, PFN_FLUID2, KK>(A, s);
    auto stress = [&](auto ns) -> int {
        constexpr int NS = decltype(ns)::value;
        if (A.pfn == GC_PFN_CAUCHY_FLUID) return launch_win_cfg<Phys, ND, NS, GC_PFN_CAUCHY_FLUID, KK>(A, s);
        if (A.pfn == GC_PFN_STRAIN_RATE) return launch_win_cfg<Phys, ND, NS, GC_PFN_STRAIN_RATE, KK>(A, s);
        if (A.pfn == GC_PFN_STRAIN_RATE_VORTICITY)
            return launch_win_cfg<Phys, ND, NS, GC_PFN_STRAIN_RATE_VORTICITY, KK>(A, s);
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

}  // namespace gc
