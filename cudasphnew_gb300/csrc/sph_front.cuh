// The front of a step (hash, cell offsets, scatter, rank, gather) as device code
// that a cooperative kernel runs phase by phase: k_front (sph_sort.cu), and
// k_steps (sph_step.cu), which takes whole steps in one launch.
#pragma once

#include <algorithm>
#include <atomic>

#include <cuda/atomic>

#include "sph_device.cuh"

namespace sph {

// words of SortBuffers::front: barrier arrivals, blocks gone, a wait gave up, then the blocks' sums
enum : int { FRONT_ARRIVED = 0, FRONT_GONE = 1, FRONT_FAILED = 2, FRONT_SUMS = 8 };

struct FrontArgs {
    int n;
    const float4* pos;
    const float4* vel;
    GridDev g;
    SortBuffers sb;
    float4* posS;
    float4* velS;
    unsigned int* status;
    NeighbourLists L;
    int lists;
    int phases;
    int waitLimit;
};

__device__ __forceinline__ unsigned int ordered_bits(float x) {
    unsigned int u = __float_as_uint(x);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

// Whether a launch of waiting blocks goes on: false while a wait that gave up
// is still to be reported.  Another block of the launch may be setting the
// word meanwhile, so one thread reads it for its block: a block whose warps
// saw it before and after would come apart at its own barriers.
__device__ __forceinline__ bool block_goes_on(const unsigned int* status) {
    return !__syncthreads_or(threadIdx.x == 0 &&
                             (*(volatile const unsigned int*)status & STATUS_DEVICE_WAIT) != 0u);
}

// Waits until every block of the grid has arrived `round` times.
__device__ __forceinline__ bool grid_barrier(unsigned int* front, unsigned int round, int waitLimit, unsigned int* status) {
    __shared__ int ok;
    __syncthreads();
    if (threadIdx.x == 0) {
        cuda::atomic_ref<unsigned int, cuda::thread_scope_device> arrived(front[FRONT_ARRIVED]);
        arrived.fetch_add(1u, cuda::memory_order_acq_rel);
        const unsigned int all = round * gridDim.x;
        int spins = 0;
        ok = 1;
        while (arrived.load(cuda::memory_order_acquire) < all || waitLimit < 0) {
            if (++spins > waitLimit) {
                ok = 0;
                atomicOr(status, STATUS_DEVICE_WAIT);
                atomicExch(front + FRONT_FAILED, 1u);
                break;
            }
            __nanosleep(20);
        }
    }
    __syncthreads();
    return ok != 0;
}

template <int THREADS>
__device__ __forceinline__ int front_block_sum(int v, int* warps) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) warps[threadIdx.x >> 5] = v;
    __syncthreads();
    int t = 0;
#pragma unroll
    for (int w = 0; w < THREADS / 32; w++) t += warps[w];
    return t;
}

// What kind of step a scene takes: VL_BUILDS on request or when a particle
// has moved farther than the skin allows since the last build (or the
// displacement is not finite), VL_SEARCHES in place of a build that the last
// step's own displacement would have outrun.
__device__ __forceinline__ unsigned int list_kind(const NeighbourLists& L, const SceneDev* __restrict__ scenes, int k) {
    const int S = L.numScenes;
    const unsigned int* f = L.flags;
    float lim2 = L.dispLimit2;
    if (scenes) {
        const float lim = 0.45f * L.skinFrac * scenes[k].ph.h;
        lim2 = lim * lim;
    }
    if (f[VL_BUILD * S + k]) return VL_BUILDS;
    const unsigned int last = f[VL_LAST * S + k];
    if (!(__uint_as_float(f[VL_DISP * S + k]) <= lim2)) return last == VL_REUSES ? VL_BUILDS : VL_SEARCHES;
    return last == VL_SEARCHES ? VL_BUILDS : VL_REUSES;
}

template <bool BATCH, int THREADS, bool FRESH>
__device__ __forceinline__ void front_gather(const FrontArgs& A) {
    for (int k = blockIdx.x * THREADS + threadIdx.x; k < A.n; k += gridDim.x * THREADS) {
        const int w = A.sb.workIds[k];
        const float4 p = load<FRESH>(A.pos + w), v = load<FRESH>(A.vel + w);
        A.posS[k] = p;
        A.velS[k] = v;
        const GridDev& g = BATCH ? A.sb.scenes[A.L.slotScene[k]].g : A.g;
        if (!(isfinite(p.x) && isfinite(p.y) && isfinite(p.z))) {
            atomicOr(A.status, STATUS_NON_FINITE);
        } else {
            bool outside = false;
            particle_hash(p, g, &outside);
            if (outside) atomicOr(A.status, STATUS_OUT_OF_DOMAIN);
        }
    }
}

// BATCH: the particle's scene (pos.w) supplies its grid, whose cells start at
// that scene's cellBase in the concatenated cell space.  REL: the position is
// cell-relative and the hash comes from its packed cell coordinates.
template <bool BATCH, bool REL, int THREADS>
__device__ __forceinline__ void front_hash(const FrontArgs& A) {
    for (int i = blockIdx.x * THREADS + threadIdx.x; i < A.n; i += gridDim.x * THREADS) {
        float4 p = A.pos[i];
        const GridDev& g = BATCH ? A.sb.scenes[__float_as_int(p.w)].g : A.g;
        bool outside = false;
        const bool finite = isfinite(p.x) && isfinite(p.y) && isfinite(p.z);
        if (!finite) {
            atomicOr(A.status, STATUS_NON_FINITE);
            p = make_float4(g.origin[0], g.origin[1], g.origin[2], 0.f);
        }
        int h;
        if (REL) {
            const int3 c = finite ? rel_cell(p) : make_int3(0, 0, 0);
            h = g.cellBase + g.dim[0] * (g.dim[1] * c.z + c.y) + c.x;
        } else {
            h = particle_hash(p, g, &outside);
        }
        if (outside) atomicOr(A.status, STATUS_OUT_OF_DOMAIN);
        A.sb.keySlot[i] = make_int2(h, atomicAdd(A.sb.cnt + h, 1));
    }
}

template <bool BATCH, bool REL, int THREADS, bool FRESH>
__device__ __forceinline__ void front_rank(const FrontArgs& A) {
    // (plain loads: what earlier phases of this launch wrote)
    for (int k = blockIdx.x * THREADS + threadIdx.x; k < A.n; k += gridDim.x * THREADS) {
        const int c = A.sb.sortedHash[k];
        const int s = A.sb.cellOffset[c], e = A.sb.cellOffset[c + 1];
        const int my = A.sb.tmpIds[k];
        if (A.lists && A.L.flags[VL_BUILD_NOW * A.L.numScenes + (BATCH ? A.L.slotScene[k] : 0)] == VL_REUSES) {
            int rId = 0;
            for (int t = s; t < e; t++) rId += A.sb.tmpIds[t] < my;
            A.sb.sortedIds[s + rId] = my;
            const int w = A.sb.workIds[k];
            A.posS[k] = load<FRESH>(A.pos + w);
            A.velS[k] = load<FRESH>(A.vel + w);
            continue;
        }
        const float4 p = load<FRESH>(A.pos + my);
        const GridDev& g = BATCH ? A.sb.scenes[__float_as_int(p.w)].g : A.g;
        const unsigned int key = ordered_bits(p.x);
        // the cell's mid-plane, in the frame its members' x is stored in
        const float mid = REL ? 0.5f * g.spacing
                              : g.origin[0] + ((float)((c - g.cellBase) % g.dim[0]) + 0.5f) * g.spacing;
        int rId = 0, rX = 0, below = 0;
        for (int t = s; t < e; t++) {
            const int o = A.sb.tmpIds[t];
            const float xo = load<FRESH>(&A.pos[o].x);
            const unsigned int ko = ordered_bits(xo);
            rId += o < my;
            rX += (ko < key) || (ko == key && o < my);
            below += xo < mid;
        }
        A.sb.sortedIds[s + rId] = my;
        A.sb.workIds[s + rX] = my;
        A.posS[s + rX] = p;
        A.velS[s + rX] = load<FRESH>(A.vel + my);
        if (rX == 0) A.sb.halfOffset[c] = s + below;
    }
}

// The phases of A.phases for the state at hand.  `round` counts the launch's
// barriers; `ok` turns false when one gave up (and the block shall leave).
template <bool BATCH, bool REL, int THREADS, bool FRESH>
__device__ __forceinline__ void front_phases(const FrontArgs& A, unsigned int& round, bool& ok) {
    __shared__ int warps[THREADS / 32];
    __shared__ int parts[THREADS / 32];  // each warp's counts, from the sums to the scan
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    unsigned int* front = A.sb.front;
    unsigned int* f = A.L.flags;
    const int S = A.L.numScenes;
    if (ok && A.lists) {
        // The decision, or (a launch of later phases alone) what it was.  What
        // it is taken from changes with the rank phase, when every block has
        // decided (where nothing sorts, to what gives the same decision again).
        bool sorts = false;
        if (A.phases & FRONT_HASH) {
            for (int k = t; k < S; k += THREADS) {
                const unsigned int kind = list_kind(A.L, A.sb.scenes, k);
                sorts |= kind != VL_REUSES;
                if (blockIdx.x == 0) f[VL_BUILD_NOW * S + k] = kind;
            }
            sorts = __syncthreads_or(sorts);
            if (blockIdx.x == 0 && t == 0) {
                f[VL_FLAGS * S + VL_SORT] = sorts ? 1u : 0u;
                f[VL_FLAGS * S + VL_STALE] = sorts ? 0u : 1u;
            }
        } else {
            sorts = f[VL_FLAGS * S + VL_SORT] != 0u;
        }
        if (!sorts) {
            if (!(A.phases & FRONT_RANK)) return;
            if (blockIdx.x == 0)
                for (int k = t; k < S; k += THREADS) f[VL_LAST * S + k] = VL_REUSES;
            front_gather<BATCH, THREADS, FRESH>(A);
            return;
        }
    }
    auto barrier = [&]() { ok = grid_barrier(front, ++round, A.waitLimit, A.status); };
    if (ok && (A.phases & FRONT_HASH)) {
        front_hash<BATCH, REL, THREADS>(A);
        if (A.phases & FRONT_SCAN) barrier();
    }
    // This block's stretch of cells and this warp's part of it, in vectors of
    // four counts (numCells + 1 of them; the buffers are padded).  A warp scans
    // its part on its own, SCAN_UNROLL vectors a lane in flight: few particles
    // in a grid of many cells (4,096 in 13.8 million) are a step of 91 us so, 353 when
    // every 2,048 cells took the block three barriers.
    constexpr int WARPS = THREADS / 32, SCAN_UNROLL = 2;
    const int4* cnt = reinterpret_cast<const int4*>(A.sb.cnt);
    const long long quads = ((long long)A.g.numCells + 4) / 4;
    const long long blockQuads = (quads + gridDim.x - 1) / gridDim.x, warpQuads = (blockQuads + WARPS - 1) / WARPS;
    const long long blockEnd = min(blockQuads * (blockIdx.x + 1), quads);
    const long long q0 = min(blockQuads * blockIdx.x + warpQuads * warp, blockEnd), q1 = min(q0 + warpQuads, blockEnd);
    if (ok && (A.phases & FRONT_SUM)) {
        int sum = 0;
#pragma unroll 4
        for (long long q = q0 + lane; q < q1; q += 32) {
            const int4 v = cnt[q];
            sum += v.x + v.y + v.z + v.w;
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
        if (lane == 0) parts[warp] = sum;
        __syncthreads();
        if (t == 0) {
            int all = 0;
            for (int w = 0; w < WARPS; w++) all += parts[w];
            front[FRONT_SUMS + blockIdx.x] = (unsigned int)all;
        }
        barrier();
    }
    if (ok && (A.phases & FRONT_SCAN)) {
        int run = 0;
        for (int b = t; b < (int)blockIdx.x; b += THREADS) run += (int)front[FRONT_SUMS + b];
        run = front_block_sum<THREADS>(run, warps);
        for (int w = 0; w < warp; w++) run += parts[w];
        for (long long base = q0; base < q1; base += 32 * SCAN_UNROLL) {
            int4 v[SCAN_UNROLL];
#pragma unroll
            for (int u = 0; u < SCAN_UNROLL; u++) {
                const long long q = base + 32 * u + lane;
                v[u] = q < q1 ? cnt[q] : make_int4(0, 0, 0, 0);
            }
#pragma unroll
            for (int u = 0; u < SCAN_UNROLL; u++) {
                const long long q = base + 32 * u + lane;
                const int local = v[u].x + v[u].y + v[u].z + v[u].w;
                int incl = local;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int x = __shfl_up_sync(0xffffffffu, incl, o);
                    if (lane >= o) incl += x;
                }
                int4 o;
                o.x = run + incl - local;
                o.y = o.x + v[u].x;
                o.z = o.y + v[u].y;
                o.w = o.z + v[u].z;
                if (q < q1) {
                    if (local) reinterpret_cast<int4*>(A.sb.cnt)[q] = make_int4(0, 0, 0, 0);
                    reinterpret_cast<int4*>(A.sb.cellOffset)[q] = o;
                    if (A.sb.halfOffset) reinterpret_cast<int4*>(A.sb.halfOffset)[q] = o;
                }
                run += __shfl_sync(0xffffffffu, incl, 31);
            }
        }
        if (A.phases & FRONT_SCATTER) barrier();
    }
    if (ok && (A.phases & FRONT_SCATTER)) {
        for (int i = blockIdx.x * THREADS + t; i < A.n; i += gridDim.x * THREADS) {
            const int2 ks = A.sb.keySlot[i];
            const int dst = A.sb.cellOffset[ks.x] + ks.y;
            A.sb.tmpIds[dst] = i;
            A.sb.sortedHash[dst] = ks.x;
        }
        if (A.phases & FRONT_RANK) barrier();
    }
    if (ok && (A.phases & FRONT_RANK)) {
        if (A.lists && blockIdx.x == 0) {
            for (int k = t; k < S; k += THREADS) {
                const unsigned int kind = f[VL_BUILD_NOW * S + k];
                f[VL_LAST * S + k] = kind;
                f[VL_BUILD * S + k] = 0u;
                if (kind != VL_REUSES) {
                    f[VL_DISP * S + k] = 0u;
                    if (kind == VL_BUILDS) f[VL_COUNT * S + k] += 1u;
                }
            }
        }
        front_rank<BATCH, REL, THREADS, FRESH>(A);
    }
}

// At the end of a launch: the last block to leave readies the words for the
// next one.
template <int THREADS>
__device__ __forceinline__ void front_leave(const FrontArgs& A) {
    __shared__ int last;
    const int t = threadIdx.x;
    unsigned int* front = A.sb.front;
    __syncthreads();
    if (t == 0) {
        __threadfence();
        last = atomicAdd(front + FRONT_GONE, 1u) == gridDim.x - 1u;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    const unsigned int failed = *(volatile unsigned int*)(front + FRONT_FAILED);
    const unsigned int latched = *(volatile unsigned int*)A.status & STATUS_DEVICE_WAIT;
    if (A.lists && latched)
        for (int k = t; k < A.L.numScenes; k += THREADS) {
            A.L.flags[VL_BUILD * A.L.numScenes + k] = 1u;
            A.L.flags[VL_BUILD_NOW * A.L.numScenes + k] = VL_NOTHING;
        }
    if (failed) {
        // (offsets of two different steps side by side: an empty grid instead)
        for (long long c = t; c < (((long long)A.g.numCells + 4) & ~3ll); c += THREADS) {
            A.sb.cnt[c] = 0;
            A.sb.cellOffset[c] = 0;
            if (A.sb.halfOffset) A.sb.halfOffset[c] = 0;
        }
    }
    __syncthreads();
    if (t < FRONT_SUMS) front[t] = 0u;
}

// `perSm` blocks of cooperative kernel K an SM, as far as the current device
// holds them at once (and front's words are enough).
template <auto K>
inline int resident_blocks(int threads, int perSm) {
    static std::atomic<int> known[64];  // blocks an SM times 4096, plus SMs
    int dev = 0;
    cudaGetDevice(&dev);
    int k = dev < 64 ? known[dev].load() : 0;
    if (k == 0) {
        int fit = 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&fit, K, threads, 0) != cudaSuccess || fit < 1) fit = 1;
        k = fit * 4096 + std::min(device_sms(), 4095);
        if (dev < 64) known[dev].store(k);
    }
    return std::min(std::min(perSm, k / 4096) * (k % 4096), FRONT_MAX_BLOCKS);
}

}  // namespace sph
