// Sorting stages of the GB300 SPH step and read-back helpers.
//
// Data layout in HBM (one handle, n particles, C cells):
//   pos, vel           float4[n]  particle-index order (the state; pos.w: the
//                                 scene of a batched handle, or the packed cell of
//                                 a cell-relative one)
//   posS, velS         float4[n]  copies in sorted (cell, id) order, per step
//   rho4S              float4[n]  (rho, p, p/rho^2, 1/rho) in sorted order
//   accS               float4[n]  acceleration in sorted order
//   cnt, cellOffset    int[C+1]   per-cell counts / their exclusive scan
// The sort is a counting sort: every particle takes an arrival slot in its
// cell with one atomic, a scan turns counts into cell offsets, and a rank pass
// orders each cell's members by particle id.  The result is the permutation of
// a stable sort by hash -- the order thrust::sort_by_key produces in the
// reference (particle_simulation.cu:2340).
#include <algorithm>
#include <cstdlib>

#include "sph_front.cuh"

namespace sph {

// ---------------------------------------------------------------------------
// AoS <-> float4 conversion (VD/SD layouts of particle_simulation.h:17-41)
// ---------------------------------------------------------------------------
__global__ void k_set_scene(float4* __restrict__ pos, int count, int sid) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < count) pos[i].w = __int_as_float(sid);
}

void launch_set_scene(float4* pos, int count, int sid, cudaStream_t s) {
    if (count > 0) k_set_scene<<<(count + 255) / 256, 256, 0, s>>>(pos, count, sid);
}

__global__ void k_unpack_aos(const float* __restrict__ aos, int stride, int offset, int n,
                             float4* __restrict__ out) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float* p = aos + (size_t)i * stride + offset;
    out[i] = make_float4(p[0], p[1], p[2], 0.0f);
}

__global__ void k_pack_aos(const float4* __restrict__ in, int n, float* __restrict__ aos, int stride,
                           int offset) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    float4 v = in[i];
    float* p = aos + (size_t)i * stride + offset;
    p[0] = v.x;
    p[1] = v.y;
    p[2] = v.z;
}

// Cell-relative state <-> absolute positions (sph_options.cellRelative).
__global__ void k_abs_to_rel(int n, float4* __restrict__ pos, GridDev g) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float4 p = pos[i];
    float3 rel;
    int3 c;
    rel_from_abs(make_float3(p.x, p.y, p.z), g, rel, c);
    pos[i] = make_float4(rel.x, rel.y, rel.z, rel_pack(c.x, c.y, c.z));
}

__global__ void k_rel_to_abs(int n, const float4* __restrict__ in, GridDev g, float* __restrict__ aos, int stride,
                             float4* __restrict__ out4) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float4 p = in[i];
    const float4 a = rel_abs(p, rel_cell(p), g);
    if (aos) {
        float* p = aos + (size_t)i * stride;
        p[0] = a.x;
        p[1] = a.y;
        p[2] = a.z;
    }
    if (out4) out4[i] = make_float4(a.x, a.y, a.z, 0.f);
}

void launch_abs_to_rel(int n, float4* pos, GridDev g, cudaStream_t s) {
    if (n > 0) k_abs_to_rel<<<(n + 255) / 256, 256, 0, s>>>(n, pos, g);
}

void launch_rel_to_abs(int n, const float4* pos, GridDev g, float* aos, int stride, float4* out4, cudaStream_t s) {
    if (n > 0) k_rel_to_abs<<<(n + 255) / 256, 256, 0, s>>>(n, pos, g, aos, stride, out4);
}

void launch_unpack_aos(const float* aos, int stride, int offset, int n, float4* out, cudaStream_t s) {
    if (n <= 0) return;
    k_unpack_aos<<<(n + 255) / 256, 256, 0, s>>>(aos, stride, offset, n, out);
}

// VD / velocity layout (three floats per particle) into a 16-byte aligned
// destination: each block stages its 256 particles' 768 floats in shared
// memory and stores them as 16-byte vectors, the trailing 0-3 floats singly.
// Into page-locked host memory this runs at the host link's rate (12 MB in
// ~68 us on GB300), where single-float stores and a pack followed by a DMA
// copy take ~80 us.
__global__ void __launch_bounds__(256) k_pack3_vec(const float4* __restrict__ in, int n, float* __restrict__ aos) {
    __shared__ __align__(16) float sm[768];
    const int base = blockIdx.x * 256;
    const int cnt = min(256, n - base);
    const int nf = cnt * 3, nv = nf >> 2;
    const int t = threadIdx.x;
    if (t < cnt) {
        const float4 v = in[base + t];
        sm[3 * t] = v.x;
        sm[3 * t + 1] = v.y;
        sm[3 * t + 2] = v.z;
    }
    __syncthreads();
    float* dst = aos + (size_t)base * 3;  // 3072-byte steps from an aligned start
    for (int k = t; k < nv; k += 256) reinterpret_cast<float4*>(dst)[k] = reinterpret_cast<const float4*>(sm)[k];
    for (int k = nv * 4 + t; k < nf; k += 256) dst[k] = sm[k];
}

void launch_pack_aos(const float4* in, int n, float* aos, int stride, int offset, cudaStream_t s) {
    if (n <= 0) return;
    if (stride == 3 && offset == 0 && (reinterpret_cast<uintptr_t>(aos) & 15) == 0)
        k_pack3_vec<<<(n + 255) / 256, 256, 0, s>>>(in, n, aos);
    else
        k_pack_aos<<<(n + 255) / 256, 256, 0, s>>>(in, n, aos, stride, offset);
}

// The poll limit of a wait: SPIN_LIMIT, or the integer in the environment
// variable SPH_SCAN_WAIT_LIMIT (read at each launch; a captured step graph
// keeps the value it was captured with).  Tests set it to exercise the
// give-up path; -1 abandons every wait at once.
int scan_wait_limit() {
    constexpr int SPIN_LIMIT = 1 << 22;
    const char* e = getenv("SPH_SCAN_WAIT_LIMIT");
    if (!e || !*e) return SPIN_LIMIT;
    return (int)strtol(e, nullptr, 10);
}

// ---------------------------------------------------------------------------
// The front of a step: hash, cell offsets, scatter, rank and gather, in one
// cooperative launch whose phases are set apart by grid barriers.  As separate
// kernels (six, with a memset and those that returned at once) a step spent
// more on their launches than on their work: a searching step of 131,071
// particles 77 -> 64 us, one of 16,384 that reuses its lists 29 -> 19 us.
//
//   hash     every particle takes an arrival slot in its cell with one atomic;
//   scan     the C+1 counts into cell offsets: every block sums its stretch of
//            cells, then adds the sums of the stretches before it and scans
//            its own; the counts are cleared as they are read;
//   scatter  ids to their cell's segment, in arrival order;
//   rank     orders each cell's members and gathers the state.  Two orders
//            come out of one pass over the cell segment:
//              by particle id -> sortedIds, the reference's permutation
//                 (stable sort by hash, particle_simulation.cu:2340), for the API;
//              by (x, id)     -> workIds, the order the neighbour kernels use:
//                 a cell's members sorted by x, so the lower and upper x-halves
//                 of a cell are two contiguous ranges (halfOffset: the first
//                 index with x >= the cell's mid-plane; an empty cell's is
//                 where the cell starts).
//            Ranks count the smaller keys in the segment; x is compared
//            through its order-preserving integer image so the order is total
//            (NaN included).
//
// The grid is small on purpose: a cooperative grid waits until all of it fits
// on the GPU, which the kernels of other handles (streams) then leave idle.
// One block an SM, two above FRONT_WIDE particles.  Three handles stepped in
// turn, us a step with 1 / 2 / 3 blocks an SM / five ordinary launches, and in
// brackets one handle alone: 262,144 particles searching 75 / 82 / 96 / 83
// [119 / 116 / 117 / 120]; reusing lists 56 / 59 / 67 / 64 [74 / 73 / 74 / 86];
// 1,048,576 reusing lists 198 / 201 / 208 / 210 [248 / 238 / 236 / 249].
//
// With reused neighbour lists each scene's kind of step (VL_REUSES ...) is
// decided first, by every block from the same flags.  Where no scene sorts
// there is nothing but a gather of the state into the kept order (workIds),
// with the hash's checks of each position; in a step that sorts, a scene that
// reuses its lists has its ids ranked and its state gathered into its kept order.
//
// Every wait is bounded.  A block whose wait gives up latches
// STATUS_DEVICE_WAIT and leaves; the rest follow (no block passes the barrier
// after one that a block has left), and the last to leave empties the counts
// and the cell tables, whose offsets may be of two steps, and asks for new
// lists.  Every id left behind is of this step or an earlier one.  The stages
// that follow find the condition (gave_up, VL_NOTHING) and leave the state as
// it was, and until it has been reported further steps do nothing.
// ---------------------------------------------------------------------------
constexpr int FRONT_THREADS = 512;
constexpr int FRONT_WIDE = 1 << 19;

template <bool BATCH, bool REL>
__global__ void __launch_bounds__(FRONT_THREADS, 3) k_front(FrontArgs A) {
    if (A.sb.skip && *A.sb.skip) return;
    unsigned int round = 0;
    bool ok = block_goes_on(A.status);
    front_phases<BATCH, REL, FRONT_THREADS, false>(A, round, ok);
    if (round || !ok) front_leave<FRONT_THREADS>(A);
}

template <bool BATCH, bool REL>
static void front_launch(FrontArgs A, cudaStream_t s) {
    // one particle a thread and sixteen cells, as far as the blocks may be
    const long long want = std::max(((long long)A.n + FRONT_THREADS - 1) / FRONT_THREADS,
                                    ((long long)A.g.numCells + 16 * FRONT_THREADS) / (16 * FRONT_THREADS));
    const int most = resident_blocks<k_front<BATCH, REL>>(FRONT_THREADS, A.n > FRONT_WIDE ? 2 : 1);
    // no more blocks than the last of their passes over the particles fills:
    // the SMs they leave are other handles' (six, searching, in turn: 131,072
    // particles 40.1 -> 39.2 us a step, 98,304 31.8 -> 29.3; one alone the same)
    const long long passes = (want + most - 1) / most;
    const int grid = (int)std::max(1ll, (want + passes - 1) / passes);
    void* args[] = {&A};
    cudaLaunchCooperativeKernel((const void*)k_front<BATCH, REL>, dim3(grid), dim3(FRONT_THREADS), args, 0, s);
}

void launch_front(int n, const float4* pos, const float4* vel, GridDev g, SortBuffers sb, float4* posS, float4* velS,
                  unsigned int* status, cudaStream_t s, const NeighbourLists* L, int phases) {
    if (n <= 0) return;
    FrontArgs A{n, pos, vel, g, sb, posS, velS, status, L ? *L : NeighbourLists{}, L ? 1 : 0, phases, scan_wait_limit()};
    if (sb.scenes) front_launch<true, false>(A, s);
    else if (g.rel) front_launch<false, true>(A, s);
    else front_launch<false, false>(A, s);
}

// ---------------------------------------------------------------------------
// Cell tables after a step that skipped them (reused lists, no build): the
// step's positions are those of its sorted copies (in the kept working
// order), so the tables are rebuilt from them -- the hash, scan and scatter
// over the positions put back in particle order, then the rank by id within
// each cell -- exactly as the step would have built them.
// ---------------------------------------------------------------------------
__global__ void k_unsort_positions(int n, const float4* __restrict__ posS, const int* __restrict__ workIds,
                                   const int* __restrict__ slotScene, float4* __restrict__ out) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    const float4 p = posS[k];  // (its fourth lane holds p/rho^2: the scene, for a batch, from the slot)
    out[workIds[k]] = make_float4(p.x, p.y, p.z, slotScene ? __int_as_float(slotScene[k]) : 0.f);
}

__global__ void k_rank_ids(int n, const int* __restrict__ sortedHash, const int* __restrict__ cellOffset,
                           const int* __restrict__ tmpIds, int* __restrict__ sortedIds) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    const int c = sortedHash[k];
    const int s = __ldg(cellOffset + c), e = __ldg(cellOffset + c + 1);
    const int my = tmpIds[k];
    int rId = 0;
    for (int t = s; t < e; t++) rId += __ldg(tmpIds + t) < my;
    sortedIds[s + rId] = my;
}

void launch_rebuild_tables(int n, const float4* posS, const int* workIds, const int* slotScene, GridDev g,
                           SortBuffers sb, float4* scratch, unsigned int* status, cudaStream_t s) {
    if (n <= 0) return;
    sb.skip = nullptr;
    sb.halfOffset = nullptr;  // stays the working order's
    k_unsort_positions<<<(n + 255) / 256, 256, 0, s>>>(n, posS, workIds, slotScene, scratch);
    launch_front(n, scratch, nullptr, g, sb, nullptr, nullptr, status, s, nullptr,
                 FRONT_HASH | FRONT_SUM | FRONT_SCAN | FRONT_SCATTER);
    k_rank_ids<<<(n + 255) / 256, 256, 0, s>>>(n, sb.sortedHash, sb.cellOffset, sb.tmpIds, sb.sortedIds);
}

// ---------------------------------------------------------------------------
// Read-back helpers
// ---------------------------------------------------------------------------
__global__ void k_unpermute(int n, const int* __restrict__ ids, const float4* __restrict__ src, int comp,
                            float* __restrict__ dst, int stride, int offset) {
    int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    float4 v = src[k];
    float* o = dst + (size_t)ids[k] * stride + offset;
    if (comp < 0) {
        o[0] = v.x;
        o[1] = v.y;
        o[2] = v.z;
    } else {
        o[0] = comp == 0 ? v.x : comp == 1 ? v.y : comp == 2 ? v.z : v.w;
    }
}

void launch_unpermute(int n, const int* sortedIds, const float4* srcS, int comp, float* dst, int stride,
                      int offset, cudaStream_t s) {
    if (n <= 0) return;
    k_unpermute<<<(n + 255) / 256, 256, 0, s>>>(n, sortedIds, srcS, comp, dst, stride, offset);
}

// Reference cell tables from the offsets: EMPTY (0xFFFFFFFF) for empty cells.
__global__ void k_cell_tables(int numCells, const int* __restrict__ off, int* start, int* end) {
    int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= numCells) return;
    int s = off[c], e = off[c + 1];
    bool occ = e > s;
    if (start) start[c] = occ ? s : -1;
    if (end) end[c] = occ ? e : -1;
}

void launch_cell_tables(int numCells, const int* cellOffset, int* start, int* end, cudaStream_t s) {
    if (numCells <= 0) return;
    k_cell_tables<<<(numCells + 255) / 256, 256, 0, s>>>(numCells, cellOffset, start, end);
}

}  // namespace sph
