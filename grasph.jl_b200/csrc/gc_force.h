// gc_force.h — arguments of the fused pair-sweep kernels.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "gc_internal.h"

namespace gc {

constexpr int FORCE_TPB = 128;  // threads per block of the sweep
constexpr int WIN_TPB = 64;     // threads per block of the window sweep
constexpr int FORCE_BUF = 64;   // staged-neighbour column of the counting sweep (shared memory)

// Launch configurations of the window sweep: resident blocks per SM, candidates
// per chunk and, FP32-compensated, whether the pair loop lists the candidates
// that it does not add (for particles at rest on a lattice with pairs at the
// cutoff), chosen per (system, stage) by the tuner in gc_context.cu.  Every one
// gives the same bits.
struct WinCfg {
    int minb, chunk;
    bool list;
};
constexpr int NUM_FORCE_CFG = GC_NUM_SWEEP_CONFIGS;
constexpr WinCfg WIN_CFGS32[NUM_FORCE_CFG] = {{8, 192, false}, {8, 192, true}, {6, 224, false}, {10, 160, false}};
constexpr WinCfg WIN_CFGS64[NUM_FORCE_CFG] = {{6, 192, false}, {5, 192, false}, {7, 160, false}, {8, 128, false}};
constexpr int WIN_SM_BLOCKS = 10;  // no configuration holds more blocks on an SM
constexpr int MAX_REFS = 8;     // interactions fused into one launch

// system_b kinds as seen by a functor (src/PairwiseFunctors.jl dispatch)
enum { BT_SELF = 0, BT_DYNAMIC = 1, BT_STATIC = 2, BT_GHOST = 3, BT_SYSTEM = 4 };

// what a functor's records carry (refreshed before each sweep)
enum { AUX_P_OVER_RHO2 = 0, AUX_INV_RHO2 = 1, AUX_MASS_OVER_RHO = 2 };

// Device-side functor code: FluidPfn with its two-sided (multiphase),
// fluid-solid and surface-tension forms enabled; the plain GC_PFN_FLUID code
// compiles them out of the pair loop.
constexpr int PFN_FLUID2 = 16;
template <int P>
__host__ __device__ constexpr bool fluid_pfn() {
    return P == GC_PFN_FLUID || P == PFN_FLUID2;
}

struct InterRef {
    int btype;
    const SysInst* bbox;  // per-instance bounding box of system_b (nullptr: never skip)
    const GridInst* gi;   // per instance
    const PfnInst* pi;    // per instance, this stage
    const int32_t* cs;    // packed CSR over system_b (global b indices)
    int64_t cs_cells;     // cells of cs that are valid (an instance beyond them is skipped)
    const double *bx, *bv, *brho, *bstress;
    const float4* brec;   // sweep records of system_b (position-only ones of a dynamic boundary), or nullptr
    int brq;              // their stride in 16-byte quads
    const float* bh;      // FP32 positions, planar (stride bN), or nullptr
    int64_t bN;           // planar stride of system_b's arrays
    int32_t* counts;      // optional per-particle accepted-pair counts
};

struct ForceArgs {
    int nd, ns, pfn, kk;
    int64_t aN;
    const int32_t* a_inst_of;
    const double *ax, *av, *arho;
    double *advdt, *adrhodt, *asr, *avort;
    const double* a_c;     // per-instance sound speed
    const double* a_mass;  // per-instance particle mass
    const float* a_cf;     // FP32 copy of the sound speed
    const float4* arec;    // sweep records of system_a
    const double* origin;  // per instance, the point that FP32 positions count from
    int prec;              // GC_PRECISION_*
    int* err;
    const int2* groups;        // warp groups of system_a particles (group_of)
    const int64_t* ngroups;    // device count of groups
    int num_sms;
    int sm_blocks;             // most blocks of the window sweep on an SM, 0: as many as fit
    int cfg;                   // index into WIN_CFGS32 / WIN_CFGS64
    int imask, iwsum;          // InterpolateFieldFn: fields (1<<GC_FIELD_*), accumulate w_sum into avort
    int nref;
    InterRef ref[MAX_REFS];
};

// A warp group: up to 32 consecutive particles of one instance.
__host__ __device__ inline int2 group_of(int32_t start, int count, int inst) {
    int2 g;
    g.x = start;
    g.y = inst << 6 | count;
    return g;
}
__host__ __device__ inline int group_count(int2 g) { return g.y & 63; }
__host__ __device__ inline int group_inst(int2 g) { return g.y >> 6; }

int launch_force_f64(const ForceArgs& A, bool count_only, cudaStream_t s);
// Warp groups of the columns of a grid into groups[0, *ngroups).  scratch: two
// words, zero between launches.
void launch_groups(const GridInst* gi, int ninst, int nd, const int32_t* cs, int64_t ncols_cap, int64_t cells_cap,
                   int2* groups, int64_t* ngroups, unsigned long long* scratch, cudaStream_t s);
// Mode of a functor's records.
__host__ __device__ constexpr int aux_mode(int pfn) {
    return pfn == GC_PFN_FLUID || pfn == PFN_FLUID2 ? AUX_P_OVER_RHO2
           : pfn == GC_PFN_CAUCHY_FLUID             ? AUX_INV_RHO2
                                                    : AUX_MASS_OVER_RHO;
}
// Per-particle records of the window sweep, in 16-byte quads, so a neighbour
// costs a few wide loads.  σ' is the stress over ρ².  FP32-compensated: a
// position is an FP32 pair x = h + l (h the nearest float, l the rest), whose
// differences are as good as the FP64 difference rounded to FP32.
//   2-D: [hx hy lx ly] then
//     fluid       [vx vy -p/ρ² 1/ρ] [ρ 0 0 0]
//     strain rate [vx vy m/ρ 0]
//     Cauchy      [vx vy 1/ρ ρ] [σ'xx σ'yy σ'xy 0]
//   3-D: [hx hy hz w0] [lx ly lz w1] [vx vy vz w2], w being
//     fluid       -p/ρ², 1/ρ, ρ
//     strain rate m/ρ, 0, 0
//     Cauchy      1/ρ, ρ, σ'xx, then [σ'yy σ'zz σ'xy σ'xz] [σ'yz 0 0 0]
// FP64, two doubles a quad: x.. v.. then
//     fluid -p/ρ², 1/ρ, ρ, p; strain rate m/ρ, 0; Cauchy 1/ρ, ρ, σ'.. (0)
//   (2-D σ': xx yy xy).
// A dynamic boundary lends only positions: its records are the position
// quads alone (FP32 3-D with w = 0, FP64 3-D [x y] [z 0]).
__host__ __device__ constexpr int rec_quads(int nd, int mode, bool fp32) {
    return fp32 ? (mode == AUX_INV_RHO2 ? (nd == 2 ? 3 : 5) : mode == AUX_MASS_OVER_RHO ? (nd == 2 ? 2 : 3) : 3)
                : nd + (mode == AUX_INV_RHO2 ? (nd == 2 ? 3 : 4) : mode == AUX_MASS_OVER_RHO ? 1 : 2);
}
__host__ __device__ constexpr int pos_quads(int nd, bool) { return nd == 2 ? 1 : 2; }
// The FP32-compensated sweep's positions (h, l and hpos) count from a point of
// their instance, origin[instance·MAXD + d] (launch_plan_all): FP32 is as good
// in a domain far from the origin as next to it.  FP64 records and their hpos
// hold the positions themselves.
// hpos: the positions rounded to FP32, planar (the candidate test reads
// these).  Nothing is written without pos or rec, either of which may be
// nullptr; p and stress may be nullptr (zeros).
void launch_pack(bool fp32, int mode, int64_t N, const int64_t* count, int nd, int ns, const double* x,
                 const double* v, const double* rho, const double* p, const double* stress, const int32_t* inst_of,
                 const double* mass, const double* origin, float* hpos, float4* pos, float4* rec, cudaStream_t s);

}  // namespace gc
