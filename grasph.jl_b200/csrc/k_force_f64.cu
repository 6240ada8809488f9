// k_force_f64.cu — dispatch of the fused pair sweep, warp-group lists and
// sweep records.  Compiled with -fmad=false.
#include <cstdio>

#include "gc_device.cuh"
#include "gc_force.h"
#include "gc_kernels.h"
#include "gc_pack.cuh"

namespace gc {

int launch_force_2d_f64(const ForceArgs& A, bool count_only, cudaStream_t s);
int launch_force_3d_f64(const ForceArgs& A, bool count_only, cudaStream_t s);
int launch_force_2d_f32(const ForceArgs& A, cudaStream_t s);
int launch_force_3d_f32(const ForceArgs& A, cudaStream_t s);

int launch_force_f64(const ForceArgs& A, bool count_only, cudaStream_t s) {
    if (A.aN <= 0 || A.nref == 0) return 0;
    const bool f32 = A.prec == GC_PRECISION_FP32_COMPENSATED && !count_only && A.pfn != GC_PFN_COUNT;
    if (A.nd == 2) return f32 ? launch_force_2d_f32(A, s) : launch_force_2d_f64(A, count_only, s);
    return f32 ? launch_force_3d_f32(A, s) : launch_force_3d_f64(A, count_only, s);
}

// --------------------------------------------------------------- groups
// Columns of the primary grid → warp groups of ≤ 32 consecutive particles.
__device__ __forceinline__ int find_inst(const GridInst* gi, int ninst, int64_t col) {
    int lo = 0, hi = ninst - 1;
    while (lo < hi) {
        int mid = (lo + hi + 1) >> 1;
        if (gi[mid].colbase <= col) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

// `cells_cap`: cells of `cs` that are valid (cs holds cells_cap + 1
// entries); an instance whose grid reaches beyond them contributes nothing
// (the grid build has flagged the overflow).  A warp takes 32 columns, adds up
// their groups, and reserves them with one add on scratch[0]; the groups'
// order does not matter (each is swept by itself), so no scan over the
// columns is needed: one launch in place of four.  The last block
// (scratch[1] counts them) writes the total and clears the scratch.
__global__ void k_groups(const GridInst* __restrict__ gi, int ninst, int nd, const int32_t* __restrict__ cs,
                         int64_t ncols_cap, int64_t cells_cap, int2* __restrict__ groups, int64_t* ngroups,
                         unsigned long long* scratch) {
    pdl_enter();
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const int64_t all = gi[ninst - 1].colbase + gi[ninst - 1].ncols;
    const int64_t T = all < ncols_cap ? all : ncols_cap;
    const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t c0 = (((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5) * 32; c0 < T; c0 += nwarps * 32) {
        const int64_t c = c0 + lane;
        int k = 0;
        int32_t s0 = 0, n = 0;
        if (c < T) {
            k = find_inst(gi, ninst, c);
            const GridInst& G = gi[k];
            if (G.cellbase + G.ncells <= cells_cap) {
                const int64_t ngl = G.ng[nd - 1];
                const int64_t b = G.cellbase + (c - G.colbase) * ngl;
                s0 = cs[b];
                n = cs[b + ngl] - s0;
            }
        }
        const int32_t m = (n + 31) / 32;
        int32_t at = m;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int32_t y = __shfl_up_sync(FULL, at, o);
            if (lane >= o) at += y;
        }
        const int32_t total = __shfl_sync(FULL, at, 31);
        unsigned long long base = 0;
        if (lane == 0 && total > 0) base = atomicAdd(&scratch[0], (unsigned long long)total);
        const int64_t first = (int64_t)__shfl_sync(FULL, base, 0) + at - m;
        for (unsigned left = __ballot_sync(FULL, m > 0); left; left &= left - 1) {
            const int l = __ffs(left) - 1;
            const int64_t o = __shfl_sync(FULL, first, l);
            const int32_t sl = __shfl_sync(FULL, s0, l), nl = __shfl_sync(FULL, n, l), ml = __shfl_sync(FULL, m, l);
            const int kl = __shfl_sync(FULL, k, l);
            for (int32_t q = lane; q < ml; q += 32)
                groups[o + q] = group_of(sl + 32 * q, nl - 32 * q < 32 ? nl - 32 * q : 32, kl);
        }
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        if (atomicAdd(&scratch[1], 1ull) == gridDim.x - 1) {
            *ngroups = (int64_t)atomicExch(&scratch[0], 0ull);
            scratch[1] = 0ull;
        }
    }
}

void launch_groups(const GridInst* gi, int ninst, int nd, const int32_t* cs, int64_t ncols_cap, int64_t cells_cap,
                   int2* groups, int64_t* ngroups, unsigned long long* scratch, cudaStream_t s) {
    int64_t b = (ncols_cap + 255) / 256;
    b = b < 1 ? 1 : b > 2 * 148 ? 2 * 148 : b;
    k_groups<<<(int)b, 256, 0, s>>>(gi, ninst, nd, cs, ncols_cap, cells_cap, groups, ngroups, scratch);
    g_launches.fetch_add(1, std::memory_order_relaxed);
}

__global__ void k_pack(PackArgs a, const int64_t* count) {
    pdl_enter();
    const int64_t n = count ? *count : a.N;
    for (int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; g < n; g += (int64_t)gridDim.x * blockDim.x)
        pack_one(a, g);
}

void launch_pack(bool fp32, int mode, int64_t N, const int64_t* count, int nd, int ns, const double* x, const double* v,
                   const double* rho, const double* p, const double* stress, const int32_t* inst_of,
                   const double* mass, const double* origin, float* hpos, float4* pos, float4* rec, cudaStream_t s) {
    if (N <= 0 || (!pos && !rec)) return;
    int64_t blocks = (N + 255) / 256;
    if (blocks > 148 * 64) blocks = 148 * 64;
    PackArgs a{fp32, mode, nd, ns, N, x, v, rho, p, stress, inst_of, mass, origin, hpos, pos, rec};
    k_pack<<<(int)blocks, 256, 0, s>>>(a, count);
    g_launches.fetch_add(1, std::memory_order_relaxed);
}

}  // namespace gc
