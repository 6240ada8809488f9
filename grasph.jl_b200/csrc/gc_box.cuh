// gc_box.cuh — per-instance bounding boxes reduced inside a kernel that visits
// the positions: the bounding-box kernel and the full step.
#pragma once

#include <algorithm>

#include "gc_device.cuh"

namespace gc {

// Each block takes a contiguous run of tiles of blockDim particles, so it
// makes 2·nd atomics and not 2·nd per tile; `wave` blocks at most, those that
// are resident at once.
inline int64_t box_tiles_per_block(int64_t N, int tpb, int wave) {
    return std::max<int64_t>((std::max<int64_t>((N + tpb - 1) / tpb, 1) + wave - 1) / wave, 1);
}
inline int box_blocks(int64_t N, int tpb, int wave) {
    const int64_t tiles = std::max<int64_t>((N + tpb - 1) / tpb, 1), per = box_tiles_per_block(N, tpb, wave);
    return (int)((tiles + per - 1) / per);
}

// A thread's running min/max of its particles while they belong to one
// instance, flushed with atomics when the instance changes; the block reduces
// them once at the end (ordered keys: min/max is exact in any order).
// scratch: ninst·2·MAXD + 1 words in their reset state, and left so.
struct BoxRun {
    int krun = -1;
    unsigned long long mn[MAXD] = {~0ull, ~0ull, ~0ull}, mx[MAXD] = {0ull, 0ull, 0ull};

    __device__ __forceinline__ void flush(unsigned long long* scratch, int k, int nd) const {
#pragma unroll
        for (int d = 0; d < MAXD; ++d) {
            if (d >= nd) break;
            atomicMin(&scratch[(k * 2 + 0) * MAXD + d], mn[d]);
            atomicMax(&scratch[(k * 2 + 1) * MAXD + d], mx[d]);
        }
    }
    __device__ __forceinline__ void add(unsigned long long* scratch, int k, const double* x, int nd) {
        if (k != krun) {
            if (krun >= 0) flush(scratch, krun, nd);
            krun = k;
#pragma unroll
            for (int d = 0; d < MAXD; ++d) {
                mn[d] = ~0ull;
                mx[d] = 0ull;
            }
        }
#pragma unroll
        for (int d = 0; d < MAXD; ++d) {
            if (d >= nd) break;
            const unsigned long long key = ord_key(x[d]);
            mn[d] = key < mn[d] ? key : mn[d];
            mx[d] = key > mx[d] ? key : mx[d];
        }
    }
    // every thread of every block, once; the last block to finish writes the
    // boxes (blocks of at most 1024 threads)
    __device__ __forceinline__ void finish(unsigned long long* scratch, SysInst* inst, int ninst, int nd) {
        // thread 0 holds the block's first particle, so its instance is the
        // block's whenever the block has any
        __shared__ int k0;
        if (threadIdx.x == 0) k0 = krun;
        __syncthreads();
        const int uniform = __syncthreads_and(krun < 0 || krun == k0);
        if (uniform && k0 >= 0) {
            __shared__ unsigned long long smn[32][MAXD], smx[32][MAXD];
            const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
            for (int d = 0; d < MAXD; ++d) {
                if (d >= nd) break;
                unsigned long long a = mn[d], b = mx[d];
                for (int o = 16; o > 0; o >>= 1) {
                    const unsigned long long a2 = __shfl_down_sync(0xffffffffu, a, o);
                    const unsigned long long b2 = __shfl_down_sync(0xffffffffu, b, o);
                    a = a2 < a ? a2 : a;
                    b = b2 > b ? b2 : b;
                }
                if (lane == 0) {
                    smn[wid][d] = a;
                    smx[wid][d] = b;
                }
            }
            __syncthreads();
            if (threadIdx.x < nd) {
                const int d = threadIdx.x;
                unsigned long long a = ~0ull, b = 0ull;
                for (int w = 0; w < (int)(blockDim.x / 32); ++w) {
                    a = smn[w][d] < a ? smn[w][d] : a;
                    b = smx[w][d] > b ? smx[w][d] : b;
                }
                atomicMin(&scratch[(k0 * 2 + 0) * MAXD + d], a);
                atomicMax(&scratch[(k0 * 2 + 1) * MAXD + d], b);
            }
        } else if (krun >= 0) {
            flush(scratch, krun, nd);
        }
        unsigned long long* counter = scratch + (size_t)ninst * 2 * MAXD;
        __shared__ bool last;
        __threadfence();
        __syncthreads();
        if (threadIdx.x == 0) last = atomicAdd(counter, 1ull) == gridDim.x - 1;
        __syncthreads();
        if (!last) return;
        __threadfence();
        for (int k = threadIdx.x; k < ninst; k += blockDim.x) {
#pragma unroll
            for (int d = 0; d < MAXD; ++d) {
                if (d >= nd) break;
                const unsigned long long a = atomicExch(&scratch[(k * 2 + 0) * MAXD + d], ~0ull);
                const unsigned long long b = atomicExch(&scratch[(k * 2 + 1) * MAXD + d], 0ull);
                inst[k].bbmin[d] = a == ~0ull ? 0.0 : ord_val(a);
                inst[k].bbmax[d] = b == 0ull ? 0.0 : ord_val(b);
            }
        }
        if (threadIdx.x == 0) atomicExch(counter, 0ull);
    }
};

}  // namespace gc
