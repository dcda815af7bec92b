// Density and force stages of the GB300 SPH step.
//
// Both run one thread per particle in the working order (cell, x, id) and
// walk the nine rows of the 27-cell stencil (sph_device.cuh), each cut to its
// candidate window.  Each row's terms are summed in plain FP32 (a row holds a
// handful of neighbours) and the row sums are added with Kahan compensation;
// a row that contributes exactly nothing is not added, so the window cut
// (which drops only zero terms) changes no result bit.
//
// The force stage comes in three forms that sum the same terms in the same
// order:
//   direct    -- distance test and pair interaction in one loop (the
//                reference's structure); a warp runs the interaction whenever
//                any lane's candidate is a neighbour;
//   mask      -- a row is tested in chunks of up to 32 candidates into a
//                register bit mask first, then only the set bits interact;
//   pretested -- the density stage, which tests every candidate anyway,
//                records each row's window start and a 32-bit neighbour mask;
//                the force stage runs the interactions of the set bits only
//                (rows longer than 32 candidates fall back to testing).
#include <algorithm>
#include <climits>

#include "sph_front.cuh"
#include "sph_mlp_tile.cuh"

namespace sph {

// ---------------------------------------------------------------------------
// Density + pressure (compute_particle_density_pressure,
// particle_simulation.cu:196-256; compute_particle_density_cell :1385-1419).
// Branch-free poly6 accumulation: max(h^2 - r^2, 0)^3.  Writes
// (rho, p, p/rho^2, 1/rho) for the force stage.
// ---------------------------------------------------------------------------
__device__ __forceinline__ bool within_r2(float r2, float R2) {  // r2 >= 0 or NaN
    return __float_as_uint(r2) <= __float_as_uint(R2);
}

// Up to 32 candidates of a row from slot `base`: their density terms added to
// rs one after the other, and the bits of those within h (bit k: candidate
// base + k), with SKIN also of those within R.  Four at a time, their loads
// in flight together and their bits put together from constants (230 against
// 254 us for the list build of a million particles, 21 against 27 at 16,384).
// REL: positions are cell-relative and moved into particle i's frame.
template <bool REL, bool SKIN, bool FRESH>
__device__ __forceinline__ void row_tests(const float4* posS, int base, int c, float4 xi, float h2,
                                          float R2, int cx, float dyo, float dzo, float spacing, float& rs,
                                          unsigned int& mR, unsigned int& mh) {
    mR = mh = 0u;
    auto at = [&](const float4* p) {
        const float4 x = load<FRESH>(p);
        return REL ? rel_in_frame(x, cx, dyo, dzo, spacing) : x;
    };
    const float4* p = posS + base;
    int k = 0;
#pragma unroll 1
    for (; k + 4 <= c; k += 4, p += 4) {
        const float4 x0 = at(p), x1 = at(p + 1), x2 = at(p + 2), x3 = at(p + 3);
        const float r0 = dist2(xi, x0), r1 = dist2(xi, x1), r2 = dist2(xi, x2), r3 = dist2(xi, x3);
        const float w0 = fmaxf(h2 - r0, 0.f), w1 = fmaxf(h2 - r1, 0.f);
        const float w2 = fmaxf(h2 - r2, 0.f), w3 = fmaxf(h2 - r3, 0.f);
        rs = fmaf(w0 * w0, w0, rs);
        rs = fmaf(w1 * w1, w1, rs);
        rs = fmaf(w2 * w2, w2, rs);
        rs = fmaf(w3 * w3, w3, rs);
        unsigned int a = 0u, b = 0u;
        if (SKIN) {
            if (within_r2(r0, R2)) a = 1u;
            if (within_r2(r1, R2)) a |= 2u;
            if (within_r2(r2, R2)) a |= 4u;
            if (within_r2(r3, R2)) a |= 8u;
            mR |= a << k;
        }
        if (neighbour_r2(r0, h2)) b = 1u;
        if (neighbour_r2(r1, h2)) b |= 2u;
        if (neighbour_r2(r2, h2)) b |= 4u;
        if (neighbour_r2(r3, h2)) b |= 8u;
        mh |= b << k;
    }
#pragma unroll 1
    for (; k < c; k++, p++) {
        const float r2 = dist2(xi, at(p));
        const float w = fmaxf(h2 - r2, 0.f);
        rs = fmaf(w * w, w, rs);
        if (SKIN) mR |= (within_r2(r2, R2) ? 1u : 0u) << k;
        mh |= (neighbour_r2(r2, h2) ? 1u : 0u) << k;
    }
}


// With REL the positions are cell-relative: every neighbour is moved into
// particle i's cell frame before its distance is taken.
// Occupancy: 40 registers (six 256-thread blocks per SM) cost no spills
// outside the batched form's setup, and the stage runs ~1 % faster than at
// 48; the cell-relative forms keep 48.
template <bool KAHAN, bool EMIT, bool BATCH, bool REL>
__global__ void __launch_bounds__(256, REL ? 5 : 6)
k_density(int n, const float4* __restrict__ posS, RowTables T, GridDev g_, PhysDev ph_, MapDev map_, int window,
          float4* __restrict__ rho4S, RowMasks M) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float4 xi = posS[i];
    const bool off = gave_up(T.status);
    if ((T.skip && *T.skip) || off) return;
    // batched handles: the particle's own scene supplies grid, constants and maps
    const SceneDev* S = BATCH ? T.scenes + __float_as_int(xi.w) : nullptr;
    const GridDev& g = BATCH ? S->g : g_;
    const PhysDev& ph = BATCH ? S->ph : ph_;
    const MapDev& map = BATCH ? S->map : map_;
    const int3 ci = REL ? rel_cell(xi) : make_int3(0, 0, 0);
    const Stencil st = REL ? stencil_rel(xi, ci, ph.h, g) : stencil(xi, ph.h, g);
    const float h2 = ph.h2;
    float sum = 0.f, comp = 0.f;
#pragma unroll 1
    for (int r = 0; r < 9; r++) {
        int s, e;
        float dyo = 0.f, dzo = 0.f;
        if (REL) row_range_rel(xi, ci, st, ph.h, g, T, window != 0, r, s, e, dyo, dzo);
        else row_range(xi, st, ph.h, g, T, window != 0, r, s, e);
        float rs = 0.f;
        unsigned int m = 0u, mR;
        for (int base = s; base < e; base += 32)
            row_tests<REL, false, false>(posS, base, min(32, e - base), xi, h2, 0.f, ci.x, dyo, dzo, g.spacing, rs, mR, m);
        if (KAHAN) {
            if (rs > 0.f) kahan_add(sum, comp, rs);
        } else {
            sum += rs;
        }
        if (EMIT) {
            const bool fits = e - s <= 32;  // bit k: candidate s + k
            M.start[(size_t)r * n + i] = fits ? s : (s | (int)0x80000000);
            M.mask[(size_t)r * n + i] = fits ? m : (unsigned int)e;
        }
    }
    float rho = (KAHAN ? __fsub_rn(sum, comp) : sum) * ph.poly6m;
    if (map.present) {
        float uvw[3];
        map_uvw(map, REL ? rel_abs(xi, ci, g) : xi, uvw);
        rho += tri_vec(map, uvw[0], uvw[1], uvw[2]).y;  // wall density, :242-248
    }
    const float p = ph.stiffness * (rho - ph.restDensity);
    const float inv = 1.0f / rho;
    rho4S[i] = make_float4(rho, p, p * inv * inv, inv);
}

// ---------------------------------------------------------------------------
// Density over reused neighbour lists (sph_options.neighbourSkin).
//
// Build form (steps that build the lists): every row that the skin sphere of
// radius R reaches, in the reference's order, its window at R walked in the
// working order.  The reference's own 3 x 3 rows give the density terms,
// summed as in k_density (candidates beyond h add exactly nothing, so the row
// sums are the same), and this step's neighbours by row for the force stage;
// every row gives its candidates within R to the particle's list.  A step that searches without
// building (VL_SEARCHES) takes windows at h and records those.
//
// A row is tested 32 candidates at a time into two bit masks (within R,
// within h), and only the set bits are appended: an append costs as much as a
// test and a quarter of the candidates pass.
// ---------------------------------------------------------------------------
// A group of a list.  The lists are read once a launch and are most of what
// misses L1 (184 of 302 sectors a warp in the density stage), so they leave no
// lines there (1,048,576 particles: density 61.6 -> 58.8 us; a batch of 16
// scenes: density 41.0 -> 39.0, force 74.0 -> 67.7).
template <bool FRESH>
__device__ __forceinline__ int4 load_group(const int4* p) {
    if (FRESH) return *p;
    int4 c;
    asm("ld.global.nc.L1::no_allocate.v4.s32 {%0, %1, %2, %3}, [%4];"
        : "=r"(c.x), "=r"(c.y), "=r"(c.z), "=r"(c.w)
        : "l"(p));
    return c;
}

// BATCH: the slot's scene supplies grid, constants, maps and R.
template <bool KAHAN, bool BATCH, bool FRESH>
__device__ __forceinline__ void density_build_one(int i, int n, bool lists, int scene, float4* posS, float4* velS,
                                                  const RowTables& T,
                                                  const GridDev& g_, const PhysDev& ph_, const MapDev& map_,
                                                  float4* rho4S, const NeighbourLists& L, const RowMasks& M) {
    const float4 xi = posS[i];
    const SceneDev* S = BATCH ? T.scenes + scene : nullptr;
    const GridDev& g = BATCH ? S->g : g_;
    const PhysDev& ph = BATCH ? S->ph : ph_;
    const MapDev& map = BATCH ? S->map : map_;
    const Stencil st = stencil(xi, ph.h, g);
    const float R = !lists ? ph.h : BATCH ? (1.0f + L.skinFrac) * ph.h : L.radius;
    const float h2 = ph.h2, R2 = BATCH ? R * R : L.radius2, eps = 1e-3f * ph.h;
    float sum = 0.f, comp = 0.f;
    int count = 0;
    int4 group = make_int4(n, n, n, n);
    auto append = [&](int t) {
        group = make_int4(group.y, group.z, group.w, t);
        count++;
        if ((count & 3) == 0 && count <= 4 * L.capacity) L.list[(size_t)((count >> 2) - 1) * n + i] = group;
    };
    // every row the sphere reaches, in the reference's order (k outer, j inner)
    const int y1 = min(st.y1, st.y0 + 2), z1 = min(st.z1, st.z0 + 2);
    int ya, yb, za, zb;
    cell_span(xi.y, R + eps, g, 1, ya, yb);
    cell_span(xi.z, R + eps, g, 2, za, zb);
    const float reach2 = R * R;
    auto rows = [&](auto&& row) {
#pragma unroll 1
        for (int z = za; z <= zb; z++) {
            const float gz = cell_gap(xi.z, z, g.origin[2], g.spacing, eps);
#pragma unroll 1
            for (int y = ya; y <= yb; y++) {
                const float gy = cell_gap(xi.y, y, g.origin[1], g.spacing, eps);
                int s, e;
                if (row_window<FRESH>(xi, y, z, reach2, gy * gy + gz * gz, eps, g, T, s, e)) row(y, z, s, e);
            }
        }
    };
    unsigned int seen = 0u;  // the reference's rows that were walked
    rows([&](int y, int z, int s0, int e0) {
        const bool inner = z >= st.z0 && z <= z1 && y >= st.y0 && y <= y1;
        float rs = 0.f;
        int first = -1, last = -1;
        unsigned long long m = 0ull;  // neighbours within h, bit t - first
        for (int base = s0; base < e0; base += 32) {
            unsigned int mR, mh;
            row_tests<false, true, FRESH>(posS, base, min(32, e0 - base), xi, h2, R2, 0, 0.f, 0.f, 0.f, rs, mR, mh);
            if (mh) {
                if (first < 0) {
                    const int k = __ffs(mh) - 1;
                    first = base + k;
                    m = mh >> k;
                } else if (base - first < 64) {
                    m |= (unsigned long long)mh << (base - first);
                }
                last = base + 31 - __clz(mh);
            }
            if (!lists) mR = 0u;
            while (mR) {
                const int k = __ffs(mR) - 1;
                mR &= mR - 1u;
                append(base + k);
            }
        }
        if (!inner) return;
        if (KAHAN) {
            if (rs > 0.f) kahan_add(sum, comp, rs);
        } else {
            sum += rs;
        }
        const int places = last - first + 1;
        const int slot = 3 * (z - st.z0) + y - st.y0;
        const size_t at = (size_t)slot * n + i;
        seen |= 1u << slot;
        M.start[at] = first < 0 ? 0 : places <= 32 ? first : first | (places <= 64 ? ROW_TWO_WORDS : (int)0x80000000);
        M.mask[at] = places <= 64 ? (unsigned int)m : (unsigned int)(last + 1);
        if (places > 32 && places <= 64) L.rowMask2[at] = (unsigned int)(m >> 32);
    });
    for (unsigned int none = ~seen & 0x1ffu; none; none &= none - 1u) {
        const size_t at = (size_t)(__ffs(none) - 1) * n + i;
        M.start[at] = 0;
        M.mask[at] = 0u;
    }
    if (lists && count <= 4 * L.capacity) {
        L.groups[i] = (unsigned char)((count + 3) >> 2);
        while (count & 3) append(n);
    } else {
        // too many for the list, or no list to build: the rows' windows
        int w = 0;
        rows([&](int, int, int s0, int e0) {
            if (w < VL_ROWS) {
                reinterpret_cast<int2*>(L.list + (size_t)(w >> 1) * n + i)[w & 1] = make_int2(s0, e0);
                w++;
            }
        });
        L.groups[i] = (unsigned char)(VL_WINDOWS + w);
    }
    L.posB[i] = xi;
    float rho = (KAHAN ? __fsub_rn(sum, comp) : sum) * ph.poly6m;
    if (map.present) {
        float uvw[3];
        map_uvw(map, xi, uvw);
        rho += tri_vec(map, uvw[0], uvw[1], uvw[2]).y;  // wall density, :242-248
    }
    const float p = ph.stiffness * (rho - ph.restDensity);
    const float inv = 1.0f / rho;
    rho4S[i] = make_float4(rho, p, p * inv * inv, inv);
    // what the force stage needs of a neighbour besides its position and
    // velocity rides in their unused fourth lanes: two loads per pair, not three
    posS[i].w = p * inv * inv;
    velS[i].w = inv;
}

constexpr int DENSITY_LIST_BLOCKS = 4;
// The density stage of a list step: the build form above where the scene's
// step does not reuse its lists.
// List form: the candidates within R, four at a time; each group's terms are
// summed in plain FP32 (as a row's few terms are) and the group sums are
// added with compensation.  The next group's slots are loaded before the
// current group's positions are used.
template <bool KAHAN, bool BATCH, bool MASKS, bool FRESH>
__device__ __forceinline__ void density_list_one(int i, int n, float4* posS, float4* velS, const RowTables& T,
                                                 const GridDev& g, const PhysDev& ph_, const MapDev& map_,
                                                 float4* rho4S, const NeighbourLists& L, const RowMasks& M) {
    const int scene = BATCH ? L.slotScene[i] : 0;
    const unsigned int kind = L.flags[VL_BUILD_NOW * L.numScenes + scene];
    if (kind != VL_REUSES) {
        if (!FRESH && kind == VL_NOTHING) return;
        density_build_one<KAHAN, BATCH, FRESH>(i, n, kind == VL_BUILDS, scene, posS, velS, T, g, ph_, map_, rho4S, L, M);
        return;
    }
    const float4 xi = posS[i];
    const PhysDev& ph = BATCH ? T.scenes[scene].ph : ph_;
    const MapDev& map = BATCH ? T.scenes[scene].map : map_;
    const float h2 = ph.h2;
    const unsigned int groups = L.groups[i];
    float sum = 0.f, comp = 0.f;
    auto total = [&](float rs) {
        if (KAHAN) kahan_add(sum, comp, rs);
        else sum += rs;
    };
    if (!(groups & VL_WINDOWS)) {
        const int4* lp = L.list + i;
        int4 c = groups ? load_group<FRESH>(lp) : make_int4(0, 0, 0, 0);
        unsigned int m = 0u;
#pragma unroll 1
        for (unsigned int k = 0; k < groups; k++) {
            const float4 x0 = load<FRESH>(posS + c.x), x1 = load<FRESH>(posS + c.y), x2 = load<FRESH>(posS + c.z),
                         x3 = load<FRESH>(posS + c.w);
            lp += n;
            if (k + 1 < groups) c = load_group<FRESH>(lp);
            const float r0 = dist2(xi, x0), r1 = dist2(xi, x1), r2 = dist2(xi, x2), r3 = dist2(xi, x3);
            if (MASKS) {
                unsigned int b = 0u;
                if (neighbour_r2(r0, h2)) b = 1u;
                if (neighbour_r2(r1, h2)) b |= 2u;
                if (neighbour_r2(r2, h2)) b |= 4u;
                if (neighbour_r2(r3, h2)) b |= 8u;
                m |= b << (4 * (k & 7u));
                if ((k & 7u) == 7u || k + 1 == groups) {
                    L.masks[(size_t)(k >> 3) * n + i] = m;
                    m = 0u;
                }
            }
            const float w0 = fmaxf(h2 - r0, 0.f), w1 = fmaxf(h2 - r1, 0.f);
            const float w2 = fmaxf(h2 - r2, 0.f), w3 = fmaxf(h2 - r3, 0.f);
            total(fmaf(w3 * w3, w3, fmaf(w2 * w2, w2, fmaf(w1 * w1, w1, w0 * w0 * w0))));
        }
    } else {
#pragma unroll 1
        for (unsigned int w = 0; w < groups - VL_WINDOWS; w++) {
            const int2 se = list_window(L, n, i, (int)w);
            float rs = 0.f;
#pragma unroll 4
            for (int t = se.x; t < se.y; t++) {
                const float d = fmaxf(h2 - dist2(xi, load<FRESH>(posS + t)), 0.f);
                rs = fmaf(d * d, d, rs);
            }
            total(rs);
        }
    }
    float rho = (KAHAN ? __fsub_rn(sum, comp) : sum) * ph.poly6m;
    if (map.present) {
        float uvw[3];
        map_uvw(map, xi, uvw);
        rho += tri_vec(map, uvw[0], uvw[1], uvw[2]).y;  // wall density, :242-248
    }
    const float p = ph.stiffness * (rho - ph.restDensity);
    const float inv = 1.0f / rho;
    rho4S[i] = make_float4(rho, p, p * inv * inv, inv);
    // what the force stage needs of a neighbour besides its position and
    // velocity rides in their unused fourth lanes: two loads per pair, not three
    posS[i].w = p * inv * inv;
    velS[i].w = inv;
}

template <bool KAHAN, bool BATCH, bool MASKS>
__global__ void __launch_bounds__(256, DENSITY_LIST_BLOCKS)
k_density_lists(int n, float4* posS, float4* velS, RowTables T, GridDev g, PhysDev ph, MapDev map,
                float4* __restrict__ rho4S, NeighbourLists L, RowMasks M) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) density_list_one<KAHAN, BATCH, MASKS, false>(i, n, posS, velS, T, g, ph, map, rho4S, L, M);
}

// The far record: r^2 of any particle to it is ~3e36, beyond every support
// and finite.
__global__ void k_list_far_record(int n, float4* posS, float4* velS) {
    posS[n] = make_float4(1e18f, 1e18f, 1e18f, 0.f);
    velS[n] = make_float4(0.f, 0.f, 0.f, 0.f);
}

void launch_list_far_record(int n, float4* posS, float4* velS, cudaStream_t s) {
    k_list_far_record<<<1, 1, 0, s>>>(n, posS, velS);
}

// ---------------------------------------------------------------------------
// Pair interaction (compute_viscosity_pressure_forces_and_ifsurf_cell,
// :1459-1556), per-row partial sums, compensated totals.
// ---------------------------------------------------------------------------
// The quantities of one pair (i, j) both the force sums and the feature
// sums use: offset, r^2, 1/r, h - r and the velocity difference v_j - v_i.
struct Pair {
    float dx, dy, dz, r2, rinv, hr, ux, uy, uz;
    __device__ __forceinline__ Pair(const PhysDev& ph, float4 xi, float4 vi, float4 xj, float4 vj) {
        dx = __fsub_rn(xi.x, xj.x);
        dy = __fsub_rn(xi.y, xj.y);
        dz = __fsub_rn(xi.z, xj.z);
        r2 = dist2(xi, xj);
        rinv = rsqrtf(r2);
        hr = ph.h - r2 * rinv;
        ux = vj.x - vi.x;
        uy = vj.y - vi.y;
        uz = vj.z - vi.z;
    }
};

// (sums of two products are spelled as fmaf here and in force_finish: which
// of the two the compiler fuses may differ between kernels, and every form of
// the stage gives the same bits)
template <bool TENSION>
struct RowSums {
    float fp[3], fv[3], cg[3], cl;
    int hits;
    __device__ __forceinline__ void clear() {
#pragma unroll
        for (int a = 0; a < 3; a++) fp[a] = fv[a] = cg[a] = 0.f;
        cl = 0.f;
        hits = 0;
    }
    // COUNT: count the pair here (a caller walking a neighbour mask adds the
    // mask's population once instead)
    template <bool COUNT = true>
    __device__ __forceinline__ void add(const PhysDev& ph, const Pair& p, float qi, float4 rj) {
        const float sp = (qi + rj.z) * p.hr * p.hr * p.rinv;  // (p_i/rho_i^2 + p_j/rho_j^2)(h-r)^2/r
        const float sv = rj.w * p.hr;                         // (h-r)/rho_j
        fp[0] = fmaf(sp, p.dx, fp[0]);
        fp[1] = fmaf(sp, p.dy, fp[1]);
        fp[2] = fmaf(sp, p.dz, fp[2]);
        fv[0] = fmaf(sv, p.ux, fv[0]);
        fv[1] = fmaf(sv, p.uy, fv[1]);
        fv[2] = fmaf(sv, p.uz, fv[2]);
        if (TENSION) {
            const float d2 = ph.h2 - p.r2;
            const float sc = rj.w * d2 * d2;
            cg[0] = fmaf(sc, p.dx, cg[0]);
            cg[1] = fmaf(sc, p.dy, cg[1]);
            cg[2] = fmaf(sc, p.dz, cg[2]);
            cl = fmaf(rj.w * d2, fmaf(-7.f, p.r2, 3.f * ph.h2), cl);
        }
        if (COUNT) hits++;
    }
    __device__ __forceinline__ void add(const PhysDev& ph, float4 xi, float4 vi, float qi, float4 xj, float4 vj,
                                        float4 rj) {
        add(ph, Pair(ph, xi, vi, xj, vj), qi, rj);
    }
};

// Neighbour sums of the learned corrector's input features (FEAT forms
// only; the scale factors poly6*m and m*gradSpiky are applied once at the
// end).  The neighbour count is the force sums' hit count.
struct FeatSums {
    float shep = 0.f, m1[3] = {0.f, 0.f, 0.f}, div = 0.f, curl[3] = {0.f, 0.f, 0.f}, cg[3] = {0.f, 0.f, 0.f};
    int cnt = 0;
    __device__ __forceinline__ void add(const PhysDev& ph, const Pair& p, float4 rj) {
        const float q = ph.h2 - p.r2;
        const float w = q * q * q * rj.w;              // W_ij / (poly6 m) * m/rho_j
        const float gs = p.hr * p.hr * p.rinv * rj.w;  // |gradW_ij| / (m gradSpiky) * m/rho_j / r
        shep += w;
        m1[0] = fmaf(w, p.ux, m1[0]);
        m1[1] = fmaf(w, p.uy, m1[1]);
        m1[2] = fmaf(w, p.uz, m1[2]);
        cg[0] = fmaf(gs, p.dx, cg[0]);
        cg[1] = fmaf(gs, p.dy, cg[1]);
        cg[2] = fmaf(gs, p.dz, cg[2]);
        div = fmaf(gs, p.ux * p.dx + p.uy * p.dy + p.uz * p.dz, div);   // u . d
        curl[0] = fmaf(gs, p.uy * p.dz - p.uz * p.dy, curl[0]);        // u x d
        curl[1] = fmaf(gs, p.uz * p.dx - p.ux * p.dz, curl[1]);
        curl[2] = fmaf(gs, p.ux * p.dy - p.uy * p.dx, curl[2]);
    }
};

// Where the force stage writes the features: feat[(byId ? workIds[i] : i) * 24].
struct FeatOut {
    float* feat;
    int byId;
    int boxWalls;
    float dtL;
};

template <bool KAHAN, bool TENSION>
struct ForceTotals {
    float fp[3] = {0.f, 0.f, 0.f}, cp[3] = {0.f, 0.f, 0.f};
    float fv[3] = {0.f, 0.f, 0.f}, cv[3] = {0.f, 0.f, 0.f};
    float cg[3] = {0.f, 0.f, 0.f}, cl = 0.f;
    __device__ __forceinline__ void add(const RowSums<TENSION>& r) {
        if (r.hits == 0) return;
        add_all(r);
    }
    __device__ __forceinline__ void add_all(const RowSums<TENSION>& r) {
#pragma unroll
        for (int a = 0; a < 3; a++) {
            if (KAHAN) {
                kahan_add(fp[a], cp[a], r.fp[a]);
                kahan_add(fv[a], cv[a], r.fv[a]);
            } else {
                fp[a] += r.fp[a];
                fv[a] += r.fv[a];
            }
            if (TENSION) cg[a] += r.cg[a];
        }
        if (TENSION) cl += r.cl;
    }
};

// The 24 input features of the learned step corrector:
//   0 rho/rho0 - 1;  1 Shepard sum sum_j (m/rho_j) W_ij;  2-4 v;  5-7 a/g;
//   8-10 sum_j (m/rho_j) W_ij (v_j - v_i);  11 dtL sum_j (m/rho_j)(v_j - v_i).gradW_ij;
//   12-14 dtL sum_j (m/rho_j)(v_j - v_i) x gradW_ij;  15-17 h sum_j (m/rho_j) gradW_ij;
//   18 neighbours/32;  19 wall distance/h (box walls and boundary map, capped at 4);
//   20-22 unit wall normal into the fluid;  23 |v| dtL/h.
// W is poly6, gradW the spiky gradient, sums over neighbours within h of
// the pre-step state.  No reference counterpart.
__device__ __forceinline__ void feature_values(const FeatSums& fs, int boxWalls, float dtL, float4 xi, float4 vi,
                                               float4 ri, const float* acc, float mapDist, const float* mapN,
                                               const PhysDev& ph, float* f) {
    const float h = ph.h;
    float dw = 4.f * h, nx = 0.f, ny = 0.f, nz = 0.f;
    if (boxWalls) {
        const float c[3] = {xi.x - ph.boxCen[0], xi.y - ph.boxCen[1], xi.z - ph.boxCen[2]};
#pragma unroll
        for (int a = 0; a < 3; a++) {
            const float da = ph.boxDim[a] - fabsf(c[a]);
            if (da < dw) {
                dw = da;
                const float sg = c[a] > 0.f ? -1.f : 1.f;
                nx = a == 0 ? sg : 0.f;
                ny = a == 1 ? sg : 0.f;
                nz = a == 2 ? sg : 0.f;
            }
        }
    }
    if (mapDist < dw) {
        dw = mapDist;
        nx = mapN[0];
        ny = mapN[1];
        nz = mapN[2];
    }
    dw = fminf(fmaxf(dw, 0.f), 4.f * h);
    const float gInv = ph.gravity != 0.f ? 1.f / ph.gravity : 1.f;
    const float gw = -ph.pressCoef;  // m gradSpiky
    const float kd = gw * dtL;
    const float vn = sqrtf(vi.x * vi.x + vi.y * vi.y + vi.z * vi.z);
    f[0] = ri.x / ph.restDensity - 1.f;
    f[1] = ph.poly6m * fs.shep;
    f[2] = vi.x;
    f[3] = vi.y;
    f[4] = vi.z;
    f[5] = acc[0] * gInv;
    f[6] = acc[1] * gInv;
    f[7] = acc[2] * gInv;
    f[8] = ph.poly6m * fs.m1[0];
    f[9] = ph.poly6m * fs.m1[1];
    f[10] = ph.poly6m * fs.m1[2];
    f[11] = kd * fs.div;
    f[12] = kd * fs.curl[0];
    f[13] = kd * fs.curl[1];
    f[14] = kd * fs.curl[2];
    f[15] = gw * h * fs.cg[0];
    f[16] = gw * h * fs.cg[1];
    f[17] = gw * h * fs.cg[2];
    f[18] = (float)fs.cnt * (1.f / 32.f);
    f[19] = dw / h;
    f[20] = nx;
    f[21] = ny;
    f[22] = nz;
    f[23] = vn * dtL / h;
}

__device__ __forceinline__ void store_features(float* feat, size_t row, const float* f) {
    float4* dst = reinterpret_cast<float4*>(feat + row * 24);
#pragma unroll
    for (int c = 0; c < 6; c++) dst[c] = make_float4(f[4 * c], f[4 * c + 1], f[4 * c + 2], f[4 * c + 3]);
}

// Wall terms, surface tension, a = F/rho - g, symplectic Euler, box
// collision, and the write-back (compute_particle_acceleration_ifsurf
// :407-473, integrate_euler :632-665, collision_handling :742-834).  The wall
// terms follow the reference's operation order exactly.
// Returns the new state (x, v) and the acceleration; the FEAT forms also
// return the boundary map's wall distance and unit normal (mapDist stays as
// given where the map is absent, mapN where the particle is beyond the
// map's rest distance).  xm is the absolute position the boundary map is
// read at (xi itself unless positions are cell-relative).
template <bool KAHAN, bool TENSION, bool FEAT>
__device__ __forceinline__ void force_finish(const ForceTotals<KAHAN, TENSION>& A, float4 xi, float4 vi, float4 ri,
                                             const PhysDev& ph, const MapDev& map, int collideFlag, float3& x,
                                             float3& v, float* acc, float& mapDist, float* mapN, float4 xm) {
    const float rho = ri.x;
    const float pc = ph.pressCoef * rho;
    float force[3];
#pragma unroll
    for (int a = 0; a < 3; a++) {
        const float P = KAHAN ? __fsub_rn(A.fp[a], A.cp[a]) : A.fp[a];
        const float V = KAHAN ? __fsub_rn(A.fv[a], A.cv[a]) : A.fv[a];
        force[a] = fmaf(pc, P, ph.viscCoef * V);
    }
    bool tension = TENSION;
    if (map.present) {
        float uvw[3];
        map_uvw(map, xm, uvw);
        const float4 s = tri_vec(map, uvw[0], uvw[1], uvw[2]);
        const float distWall = -s.x;
        if (FEAT) mapDist = distWall;
        if (distWall < map.restDistance) {
            tension = false;
            const float coeff = rho / (ph.dtCollide * ph.dtCollide) * (map.restDistance - distWall);
            float gN[3];
#pragma unroll
            for (int a = 0; a < 3; a++) {
                float up[3] = {uvw[0], uvw[1], uvw[2]}, dn[3] = {uvw[0], uvw[1], uvw[2]};
                up[a] = __fadd_rn(uvw[a], map.du[a]);
                dn[a] = __fsub_rn(uvw[a], map.du[a]);
                gN[a] = __fdiv_rn(__fsub_rn(tri_scalar(map, map.dist, up[0], up[1], up[2]),
                                            tri_scalar(map, map.dist, dn[0], dn[1], dn[2])),
                                  __fmul_rn(2.f, map.du[a]));
            }
            force[0] -= coeff * gN[0];
            force[1] -= coeff * gN[1];
            force[2] -= coeff * gN[2];
            if (FEAT) {
                const float gn = sqrtf(gN[0] * gN[0] + gN[1] * gN[1] + gN[2] * gN[2]);
                if (gn > 0.f) {
                    mapN[0] = -gN[0] / gn;
                    mapN[1] = -gN[1] / gn;
                    mapN[2] = -gN[2] / gn;
                }
            }
            force[0] -= vi.x * s.z;
            force[1] -= vi.y * s.z;
            force[2] -= vi.z * s.z;
        }
    }
    if (TENSION && tension) {
        const float cgx = ph.cgCoef * A.cg[0], cgy = ph.cgCoef * A.cg[1], cgz = ph.cgCoef * A.cg[2];
        const float norm = sqrtf(fmaf(cgz, cgz, fmaf(cgy, cgy, cgx * cgx)));
        if (norm > ph.normThresh) {
            const float fc = ph.tension * (ph.clCoef * A.cl) / norm;
            force[0] -= fc * cgx;
            force[1] -= fc * cgy;
            force[2] -= fc * cgz;
        }
    }
    acc[0] = force[0] / rho;
    acc[1] = force[1] / rho;
    acc[2] = force[2] / rho;
    acc[0] -= ph.gravityAxis == 0 ? ph.gravity : 0.f;
    acc[1] -= ph.gravityAxis == 1 ? ph.gravity : 0.f;
    acc[2] -= ph.gravityAxis == 2 ? ph.gravity : 0.f;
    v = make_float3(vi.x + ph.dt * acc[0], vi.y + ph.dt * acc[1], vi.z + ph.dt * acc[2]);
    x = make_float3(xi.x + ph.dt * v.x, xi.y + ph.dt * v.y, xi.z + ph.dt * v.z);
    if (collideFlag) collide(ph, x, v);
}

template <bool KAHAN, bool TENSION, bool FEAT>
__device__ __forceinline__ void force_epilogue(const ForceTotals<KAHAN, TENSION>& A, int i, float4 xi,
                                               float4 vi, float4 ri, const PhysDev& ph, const MapDev& map,
                                               int collideFlag, const int* __restrict__ workIds,
                                               float4* __restrict__ pos, float4* __restrict__ vel,
                                               float4* __restrict__ accS, const FeatSums& fs,
                                               const FeatOut& fo) {
    float mapDist = 1e30f, mapN[3] = {0.f, 0.f, 0.f};  // learned features only
    float3 x, v;
    float acc[3];
    force_finish<KAHAN, TENSION, FEAT>(A, xi, vi, ri, ph, map, collideFlag, x, v, acc, mapDist, mapN, xi);
    const int id = workIds[i];
    pos[id] = make_float4(x.x, x.y, x.z, xi.w);  // .w: the scene index of batched handles
    vel[id] = make_float4(v.x, v.y, v.z, 0.f);
    accS[i] = make_float4(acc[0], acc[1], acc[2], 0.f);
    if (FEAT) {
        float f[24];
        feature_values(fs, fo.boxWalls, fo.dtL, xi, vi, ri, acc, mapDist, mapN, ph, f);
        store_features(fo.feat, (size_t)(fo.byId ? id : i), f);
    }
}

// The cell-relative form's epilogue: the step is integrated in the
// particle's cell frame, then the position moves to the cell it now lies in
// (whole-cell steps, clamped to the grid).  The wall box collision works in
// that cell's frame too, and a particle it moves is re-binned again.
__device__ __forceinline__ void rel_rebin(float3& x, int3& c, const GridDev& g) {
    const float inv = 1.0f / g.spacing;
    float* xs[3] = {&x.x, &x.y, &x.z};
    int* cs[3] = {&c.x, &c.y, &c.z};
#pragma unroll
    for (int a = 0; a < 3; a++) {
        const float k = floorf(*xs[a] * inv);
        if (k != 0.f) {
            const int cn = min(max(*cs[a] + (int)k, 0), g.dim[a] - 1);
            *xs[a] = fmaf(-(float)(cn - *cs[a]), g.spacing, *xs[a]);
            *cs[a] = cn;
        }
    }
}

template <bool KAHAN, bool TENSION>
__device__ __forceinline__ void force_epilogue_rel(const ForceTotals<KAHAN, TENSION>& A, int i, float4 xi, int3 ci,
                                                   float4 vi, float4 ri, const PhysDev& ph, const GridDev& g,
                                                   const MapDev& map, int collideFlag, const int* __restrict__ workIds,
                                                   float4* __restrict__ pos, float4* __restrict__ vel,
                                                   float4* __restrict__ accS) {
    float mapDist = 1e30f, mapN[3] = {0.f, 0.f, 0.f};
    float3 x, v;
    float acc[3];
    force_finish<KAHAN, TENSION, false>(A, xi, vi, ri, ph, map, 0, x, v, acc, mapDist, mapN, rel_abs(xi, ci, g));
    int3 c = ci;
    rel_rebin(x, c, g);
    if (collideFlag) {
        // the wall box in this cell's frame: the collision keeps the offset's resolution
        const int cc[3] = {c.x, c.y, c.z};
        float cen[3];
#pragma unroll
        for (int a = 0; a < 3; a++)
            cen[a] = (float)((double)ph.boxCen[a] - ((double)g.origin[a] + (double)cc[a] * (double)g.spacing));
        const float3 before = x;
        collide_box(cen, ph, x, v);
        if (x.x != before.x || x.y != before.y || x.z != before.z) rel_rebin(x, c, g);
    }
    const int id = workIds[i];
    pos[id] = make_float4(x.x, x.y, x.z, rel_pack(c.x, c.y, c.z));
    vel[id] = make_float4(v.x, v.y, v.z, 0.f);
    accS[i] = make_float4(acc[0], acc[1], acc[2], 0.f);
}

struct ForceArgs {
    int n;
    const float4* posS;
    const float4* velS;
    const float4* rho4S;
    const int* workIds;
    RowTables T;
    GridDev g;
    PhysDev ph;
    MapDev map;
    int collide;
    int window;
    RowMasks M;
    float4* pos;
    float4* vel;
    float4* accS;
    FeatOut fo;
};

// Occupancy: the force stage is latency bound, so it runs as many warps as
// fit without heavy spilling.  The pretested form without surface tension
// fits 48 registers with a few spilled bytes outside the pair loop: five
// 256-thread blocks per SM (145 -> 140 us per million particles against
// four).  The other plain forms and the batched forms fit 64 registers, four
// blocks (210 -> 150 us against two; the 64-scene batch 1.55 -> 1.44 ms per
// step against three); the feature form takes up to 80, three blocks.
// REL: cell-relative positions (plain forms only): neighbours are moved into
// particle i's cell frame, the step is integrated there and re-binned.
template <bool KAHAN, bool TENSION, int FORM, bool FEAT, bool BATCH, bool REL = false>
__global__ void __launch_bounds__(256, FEAT ? 3 : (BATCH || TENSION || REL || FORM != FORCE_PRETESTED ? 4 : 5)) k_force(ForceArgs F) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= F.n) return;
    const float4 xi = F.posS[i];
    const float4 vi = F.velS[i];
    const float4 ri = F.rho4S[i];
    if (gave_up(F.T.status)) return;
    const SceneDev* S = BATCH ? F.T.scenes + __float_as_int(xi.w) : nullptr;
    const GridDev& g = BATCH ? S->g : F.g;
    const PhysDev& ph = BATCH ? S->ph : F.ph;
    const MapDev& map = BATCH ? S->map : F.map;
    const float h2 = ph.h2;
    const int3 ci = REL ? rel_cell(xi) : make_int3(0, 0, 0);
    Stencil st;
    if (REL) st = stencil_rel(xi, ci, ph.h, g);
    else if (FORM != FORCE_PRETESTED) st = stencil(xi, ph.h, g);
    float dyo = 0.f, dzo = 0.f;  // REL: the current row's y and z cell offsets (times spacing)
    auto neighbour = [&](int t) {
        float4 xj = __ldg(F.posS + t);
        if (REL) xj = rel_in_frame(xj, ci.x, dyo, dzo, g.spacing);
        return xj;
    };
    ForceTotals<KAHAN, TENSION> A;
    FeatSums fs;
    auto direct = [&](RowSums<TENSION>& R, int s, int e) {
        for (int t = s; t < e; t++) {
            const float4 xj = neighbour(t);
            const float r2 = dist2(xi, xj);
            if (neighbour_r2(r2, h2)) {
                const float4 vj = __ldg(F.velS + t), rj = __ldg(F.rho4S + t);
                const Pair p(ph, xi, vi, xj, vj);
                R.add(ph, p, ri.z, rj);
                if (FEAT) fs.add(ph, p, rj);
            }
        }
    };
    auto bits = [&](RowSums<TENSION>& R, int base, unsigned int m) {
        R.hits += __popc(m);
        while (m) {
            const int t = base + __ffs(m) - 1;
            m &= m - 1u;
            const float4 xj = neighbour(t), vj = __ldg(F.velS + t), rj = __ldg(F.rho4S + t);
            const Pair p(ph, xi, vi, xj, vj);
            R.template add<false>(ph, p, ri.z, rj);
            if (FEAT) fs.add(ph, p, rj);
        }
    };
#pragma unroll
    for (int r = 0; r < 9; r++) {
        RowSums<TENSION> R;
        R.clear();
        if (FORM == FORCE_PRETESTED) {
            if (REL) {
                dyo = (float)(st.y0 + r % 3 - ci.y) * g.spacing;
                dzo = (float)(st.z0 + r / 3 - ci.z) * g.spacing;
            }
            const int sv = __ldg(F.M.start + (size_t)r * F.n + i);
            const unsigned int m = __ldg(F.M.mask + (size_t)r * F.n + i);
            if (sv < 0) direct(R, sv & 0x7fffffff, (int)m);
            else bits(R, sv, m);
        } else {
            int s, e;
            if (REL) row_range_rel(xi, ci, st, ph.h, g, F.T, F.window != 0, r, s, e, dyo, dzo);
            else row_range(xi, st, ph.h, g, F.T, F.window != 0, r, s, e);
            if (FORM == FORCE_DIRECT) {
                direct(R, s, e);
            } else {
                for (int base = s; base < e; base += 32) {
                    const int cnt = min(32, e - base);
                    unsigned int m = 0u;
                    for (int k = 0; k < cnt; k++) {
                        const float r2 = dist2(xi, neighbour(base + k));
                        m |= neighbour_r2(r2, h2) ? (1u << k) : 0u;
                    }
                    bits(R, base, m);
                }
            }
        }
        A.add(R);
        if (FEAT) fs.cnt += R.hits;
    }
    if (REL)
        force_epilogue_rel<KAHAN, TENSION>(A, i, xi, ci, vi, ri, ph, g, map, F.collide, F.workIds, F.pos, F.vel,
                                           F.accS);
    else
        force_epilogue<KAHAN, TENSION, FEAT>(A, i, xi, vi, ri, ph, map, F.collide, F.workIds, F.pos, F.vel,
                                             F.accS, fs, F.fo);
}

// ---------------------------------------------------------------------------
// Force stage over reused neighbour lists, then wall terms, integration,
// collision and write-back as k_force.  A reusing step walks the lists: four
// candidates at a time, their eight records in flight together, those beyond
// h left out of the sums; a group's terms are summed in plain FP32 and the
// group sums added with compensation, as a row's are.  A building step takes
// the rows that the density stage recorded, so it adds exactly what k_force
// adds.  It also records, for the decision at the next step, the largest
// squared distance of a particle from where it was when the lists were built.
// ---------------------------------------------------------------------------
// Which of the c <= 32 candidates from slot `base` on lie within h: a bit each.
template <bool FRESH>
__device__ __forceinline__ unsigned int row_hits(const float4* posS, int base, int c, float4 xi, float h2) {
    unsigned int m = 0u;
    const float4* p = posS + base;
    int k = 0;
#pragma unroll 1
    for (; k + 4 <= c; k += 4, p += 4) {
        const float4 x0 = load<FRESH>(p), x1 = load<FRESH>(p + 1), x2 = load<FRESH>(p + 2), x3 = load<FRESH>(p + 3);
        unsigned int b = 0u;
        if (neighbour_r2(dist2(xi, x0), h2)) b = 1u;
        if (neighbour_r2(dist2(xi, x1), h2)) b |= 2u;
        if (neighbour_r2(dist2(xi, x2), h2)) b |= 4u;
        if (neighbour_r2(dist2(xi, x3), h2)) b |= 8u;
        m |= b << k;
    }
#pragma unroll 1
    for (; k < c; k++, p++) m |= (neighbour_r2(dist2(xi, load<FRESH>(p)), h2) ? 1u : 0u) << k;
    return m;
}

// The neighbours of a list step's particle: `pair` for each candidate (with
// `tested` when it is known to lie within h), `row` with the sums of each
// row's, window's or (group true) list group's pairs.  MASKS: the density
// stage has recorded which candidates lie within h, and only those are
// gathered, four at a time too.
template <bool TENSION, bool MASKS, bool FRESH, class PAIR, class ROW>
__device__ __forceinline__ void list_rows(int i, int n, unsigned int kind, const NeighbourLists& L, const RowMasks& M,
                                          const float4* posS, const float4* velS, float4 xi, float h2,
                                          PAIR&& pair, ROW&& row) {
    // the pairs of `places` places from `base` on, 32 at a time: m holds the
    // neighbours among the first, more(base, places) those of the next
    auto walk = [&](RowSums<TENSION>& R, int base, int places, unsigned int m, auto&& more) {
#pragma unroll 1
        for (;;) {
            while (m) {
                const int t = base + __ffs(m) - 1;
                m &= m - 1u;
                pair(R, load<FRESH>(posS + t), load<FRESH>(velS + t), true);
            }
            places -= 32;
            if (places <= 0) break;
            base += 32;
            m = more(base, min(32, places));
        }
    };
    // (tested first, so that only the neighbours' velocities are loaded)
    auto hits = [&](int base, int places) { return row_hits<FRESH>(posS, base, places, xi, h2); };
    if (kind != VL_REUSES) {
        int svN = load<FRESH>(M.start + i);
        unsigned int mN = load<FRESH>(M.mask + i);
#pragma unroll 1
        for (int r = 0; r < 9; r++) {
            const int sv = svN;
            const unsigned int m = mN;
            if (r + 1 < 9) {
                svN = load<FRESH>(M.start + (size_t)(r + 1) * n + i);
                mN = load<FRESH>(M.mask + (size_t)(r + 1) * n + i);
            }
            RowSums<TENSION> R;
            R.clear();
            if ((unsigned int)sv < (unsigned int)ROW_TWO_WORDS) {
                unsigned int b = m;
                while (b) {
                    const int t = sv + __ffs(b) - 1;
                    b &= b - 1u;
                    pair(R, load<FRESH>(posS + t), load<FRESH>(velS + t), true);
                }
            } else {
                const int base = sv & ~((int)0x80000000 | ROW_TWO_WORDS);
                const int places = sv < 0 ? (int)m - base : 64;
                walk(R, base, places, sv < 0 ? hits(base, 32) : m, [&](int b, int c) {
                    return sv < 0 ? hits(b, c) : load<FRESH>(L.rowMask2 + (size_t)r * n + i);
                });
            }
            row(R, false);
        }
        return;
    }
    const unsigned int groups = L.groups[i];
    if (groups & VL_WINDOWS) {
#pragma unroll 1
        for (unsigned int w = 0; w < groups - VL_WINDOWS; w++) {
            const int2 se = list_window(L, n, i, (int)w);
            RowSums<TENSION> R;
            R.clear();
            walk(R, se.x, se.y - se.x, hits(se.x, min(32, se.y - se.x)), hits);
            row(R, false);
        }
        return;
    }
    if (MASKS) {
#pragma unroll 1
        for (unsigned int w = 0; 8 * w < groups; w++) {
            unsigned int m = load<FRESH>(L.masks + (size_t)w * n + i);
            const int* word = reinterpret_cast<const int*>(L.list + (size_t)(8 * w) * n + i);
            auto next = [&]() {  // (past the last: the far record)
                if (!m) return n;
                const int k = __ffs(m) - 1;
                m &= m - 1u;
                return load<FRESH>(word + 4 * (size_t)(k >> 2) * n + (k & 3));
            };
            if (!m) continue;
            int4 c = make_int4(next(), next(), next(), next());
            while (c.x != n) {
                const float4 x0 = load<FRESH>(posS + c.x), x1 = load<FRESH>(posS + c.y), x2 = load<FRESH>(posS + c.z), x3 = load<FRESH>(posS + c.w);
                const float4 v0 = load<FRESH>(velS + c.x), v1 = load<FRESH>(velS + c.y), v2 = load<FRESH>(velS + c.z), v3 = load<FRESH>(velS + c.w);
                const int4 d = c;
                c.x = next();
                c.y = next();
                c.z = next();
                c.w = next();
                RowSums<TENSION> R;
                R.clear();
                pair(R, x0, v0, true);
                if (d.y != n) pair(R, x1, v1, true);
                if (d.z != n) pair(R, x2, v2, true);
                if (d.w != n) pair(R, x3, v3, true);
                row(R, true);
            }
        }
        return;
    }
    const int4* lp = L.list + i;
    int4 c = groups ? load_group<FRESH>(lp) : make_int4(0, 0, 0, 0);
#pragma unroll 1
    for (unsigned int k = 0; k < groups; k++) {
        const float4 x0 = load<FRESH>(posS + c.x), x1 = load<FRESH>(posS + c.y), x2 = load<FRESH>(posS + c.z), x3 = load<FRESH>(posS + c.w);
        const float4 v0 = load<FRESH>(velS + c.x), v1 = load<FRESH>(velS + c.y), v2 = load<FRESH>(velS + c.z), v3 = load<FRESH>(velS + c.w);
        lp += n;
        if (k + 1 < groups) c = load_group<FRESH>(lp);
        RowSums<TENSION> R;
        R.clear();
        pair(R, x0, v0, false);
        pair(R, x1, v1, false);
        pair(R, x2, v2, false);
        pair(R, x3, v3, false);
        row(R, true);
    }
}

// What bounds the reusing form at 1,048,576 particles: the L1 data pipe (78 %
// busy with two gathers of 16 bytes a pair), then issue (53 %).  Registers a
// thread, and what the stage takes: 64 (spills) 131 us, 72 109 us, 80 115 us.
constexpr int FORCE_REGS = 72;
// Displacement since the build into the scene's flag: one atomic per warp (or
// per scene a warp holds) that raises the recorded maximum.  Squared
// distances are non-negative, so their bits order as the values do; the
// maximum only grows, so a warp that does not exceed the value it reads
// (possibly an older, smaller one) has nothing to add.
template <bool BATCH>
__device__ __forceinline__ void record_displacement(const NeighbourLists& L, int scene, float d2) {
    const unsigned int v = __float_as_uint(d2);
    const unsigned int peers = BATCH ? __match_any_sync(0xffffffffu, scene) : 0xffffffffu;
    const unsigned int w = __reduce_max_sync(peers, v);
    unsigned int* f = L.flags + VL_DISP * L.numScenes + scene;
    if ((threadIdx.x & 31) == (unsigned int)(__ffs(peers) - 1) && w > 0u && w > *(volatile unsigned int*)f)
        atomicMax(f, w);
}

// (every thread of the warp calls it: i may lie beyond the particles)
template <bool KAHAN, bool TENSION, bool BATCH, bool MASKS, bool FRESH>
__device__ __forceinline__ void force_list_one(int i, int n, const float4* posS, const float4* velS,
                                               const float4* rho4S, const int* workIds, const PhysDev& ph_,
                                               const MapDev& map_, int collideFlag, const NeighbourLists& L,
                                               const RowMasks& M, float4* pos, float4* vel, float4* accS,
                                               const SceneDev* scenes) {
    float d2 = 0.f;
    int scene = 0;
    auto particle = [&]() {
        const float4 xi = posS[i];
        const float4 vi = velS[i];
        const float4 ri = rho4S[i];
        if (BATCH) scene = L.slotScene[i];
        const unsigned int kind = L.flags[VL_BUILD_NOW * L.numScenes + scene];
        if (!FRESH && kind == VL_NOTHING) return;
        const PhysDev& ph = BATCH ? scenes[scene].ph : ph_;
        const MapDev& map = BATCH ? scenes[scene].map : map_;
        const float h2 = ph.h2;
        ForceTotals<KAHAN, TENSION> A;
        // (a neighbour's p/rho^2 and 1/rho ride in the fourth lanes of its
        // sorted position and velocity, written by the density stage)
        list_rows<TENSION, MASKS, FRESH>(
            i, n, kind, L, M, posS, velS, xi, h2,
            [&](RowSums<TENSION>& R, float4 xj, float4 vj, bool tested) {
                Pair p(ph, xi, vi, xj, vj);
                const bool in = tested || neighbour_r2(p.r2, h2);
                if (FRESH) {  // (a pair out of reach adds zeros)
                    if (!in) {
                        p.r2 = h2;
                        p.hr = p.rinv = p.dx = p.dy = p.dz = p.ux = p.uy = p.uz = xj.w = vj.w = 0.f;
                    }
                    R.template add<false>(ph, p, ri.z, make_float4(0.f, 0.f, xj.w, vj.w));
                    R.hits += in;
                } else if (in) {
                    R.add(ph, p, ri.z, make_float4(0.f, 0.f, xj.w, vj.w));
                }
            },
            [&](const RowSums<TENSION>& R, bool group) {
                if (group) A.add_all(R);
                else A.add(R);
            });
        float mapDist = 1e30f, mapN[3] = {0.f, 0.f, 0.f};
        float3 x, v;
        float acc[3];
        force_finish<KAHAN, TENSION, false>(A, xi, vi, ri, ph, map, collideFlag, x, v, acc, mapDist, mapN, xi);
        const int id = workIds[i];
        // (the sorted copy's fourth lane holds p/rho^2; a batch keeps the scene there)
        pos[id] = make_float4(x.x, x.y, x.z, BATCH ? __int_as_float(scene) : 0.f);
        vel[id] = make_float4(v.x, v.y, v.z, 0.f);
        accS[i] = make_float4(acc[0], acc[1], acc[2], 0.f);
        const float4 b = load<FRESH>(L.posB + i);
        const float dx = x.x - b.x, dy = x.y - b.y, dz = x.z - b.z;
        d2 = dx * dx + dy * dy + dz * dz;
        if (!(d2 == d2)) d2 = __uint_as_float(0x7f800000u);  // NaN: as far as it gets
    };
    if (i < n) particle();
    record_displacement<BATCH>(L, scene, d2);
}

template <bool KAHAN, bool TENSION, bool BATCH, bool MASKS>
__global__ void __maxnreg__(FORCE_REGS)
k_force_lists(int n, const float4* __restrict__ posS, const float4* __restrict__ velS,
              const float4* __restrict__ rho4S, const int* __restrict__ workIds, PhysDev ph, MapDev map,
              int collideFlag, NeighbourLists L, RowMasks M, float4* __restrict__ pos, float4* __restrict__ vel,
              float4* __restrict__ accS, const SceneDev* __restrict__ scenes) {
    force_list_one<KAHAN, TENSION, BATCH, MASKS, false>(blockIdx.x * blockDim.x + threadIdx.x, n, posS, velS, rho4S, workIds,
                                                 ph, map, collideFlag, L, M, pos, vel, accS, scenes);
}

// ---------------------------------------------------------------------------
// Whole steps over the reused lists in one cooperative launch, for handles of
// few particles.  What bounds a step of 16,384 particles is no unit of the
// chip but the latency of what follows one another: three launches, and in
// each one wave of warps that walk their lists.  Here the phases of the front,
// the density stage and the force stage are set apart by grid barriers (1.0 to
// 1.5 us each, against 2 to 3 for a launch that waits for the one before), and
// a call of many steps takes up to STEPS_A_LAUNCH of them a launch.  A step
// alone on the chip, and with three handles in turn, in us, before and now:
//   4,096   24.8 -> 21.0    9.4 -> 7.4
//   16,384  25.5 -> 20.6   10.2 -> 8.4
//   24,576  26.6 -> 23.2   11.0 -> 9.7
//   32,768  27.5 -> 23.0   11.8 -> 14.5
// (three 32,768-particle grids no longer fit the chip side by side and wait
// for one another: the line is drawn below that).  More list groups in flight
// a thread (2 to 8, at 140 to 200 registers) gave nothing.
// A grid of more cells than STEPS_CELLS is left to k_front, whose blocks are
// four times as large: the scan of a building step walks every cell.
// The stages are the kernels' own functions and give the same bits; FRESH:
// what one phase writes another reads in the same launch, so no read goes
// through the read-only path, and the few warps that run evaluate every pair
// without a branch (4 % of a step: a group's four pairs overlap).
// ---------------------------------------------------------------------------
constexpr int STEPS_PARTICLES = 24576;
constexpr int STEPS_CELLS = 1 << 18;
constexpr int STEPS_BLOCKS = 4;  // blocks an SM (128 registers a thread: no spills)
constexpr int STEPS_THREADS = 128;
constexpr int STEPS_A_LAUNCH = 32;  // (a bound on a launch: 0.74 ms for 24,576 particles that reuse their lists)

struct StepsArgs {
    FrontArgs F;
    RowTables T;
    PhysDev ph;
    MapDev map;
    RowMasks M;
    float4* rho4S;
    float4* accS;
    float4* pos;
    float4* vel;
    int collide;
    int steps;
};

template <bool KAHAN, bool TENSION, bool MASKS>
__global__ void __launch_bounds__(STEPS_THREADS, STEPS_BLOCKS) k_steps(StepsArgs A) {
    const FrontArgs& F = A.F;
    unsigned int round = 0;
    bool ok = block_goes_on(F.status);
    auto barrier = [&]() { ok = grid_barrier(F.sb.front, ++round, F.waitLimit, F.status); };
    const int stride = gridDim.x * STEPS_THREADS;
    const int first = blockIdx.x * STEPS_THREADS + threadIdx.x;
    for (int s = 0; s < A.steps && ok; s++) {
        front_phases<false, false, STEPS_THREADS, true>(F, round, ok);
        if (!ok) break;
        barrier();
        if (!ok) break;
        for (int i = first; i < F.n; i += stride)
            density_list_one<KAHAN, false, MASKS, true>(i, F.n, F.posS, F.velS, A.T, F.g, A.ph, A.map, A.rho4S, F.L, A.M);
        barrier();
        if (!ok) break;
        for (int base = blockIdx.x * STEPS_THREADS; base < F.n; base += stride)
            force_list_one<KAHAN, TENSION, false, MASKS, true>(base + (int)threadIdx.x, F.n, F.posS, F.velS, A.rho4S,
                                                        F.sb.workIds, A.ph, A.map, A.collide, F.L, A.M, A.pos, A.vel,
                                                        A.accS, nullptr);
        if (s + 1 < A.steps) barrier();
    }
    front_leave<STEPS_THREADS>(F);
}

// ---------------------------------------------------------------------------
// The pretested force form with each warp's neighbour rows staged in shared
// memory by TMA (plain handles).  The 32 particles of a warp are consecutive
// in the working order, so their windows into one stencil row overlap: the
// warp takes the union of its lanes' windows and one lane copies it into
// shared memory with three bulk copies (sorted position, velocity and
// density records, cp.async.bulk completing on an mbarrier).  Rows are
// double-buffered: row r + 1's copies are issued before row r is processed.
// Every lane then reads its neighbours from shared memory instead of
// gathering them through L1.  A row whose union exceeds ST_ROW candidates (a
// warp across a cell-row boundary, or a window too long for a mask) is read
// from global memory as before.  The same pairs in the same order: results
// are bit-identical to the other forms.  Each wait is bounded; a wait that
// gives up latches STATUS_DEVICE_WAIT, the warp reads global memory from
// then on and waits once more, bounded, for its copies still in flight.
// ---------------------------------------------------------------------------
constexpr int ST_ROW = 72;     // staged candidates per warp, row and buffer
constexpr int ST_WARPS = 8;    // 256-thread blocks
constexpr int ST_SMEM = ST_WARPS * 2 * 3 * ST_ROW * 16 + ST_WARPS * 2 * 8;
constexpr uint32_t ST_WAIT_LIMIT = 1u << 22;

template <bool KAHAN, bool TENSION>
__global__ void __launch_bounds__(ST_WARPS * 32, 4) k_force_staged(ForceArgs F, unsigned int* status) {
    extern __shared__ __align__(128) unsigned char stsm[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    float4* buf = reinterpret_cast<float4*>(stsm) + warp * (2 * 3 * ST_ROW);  // [buffer][P, V, Q][ST_ROW]
    uint64_t* bars = reinterpret_cast<uint64_t*>(stsm + ST_WARPS * 2 * 3 * ST_ROW * 16) + 2 * warp;
    // the whole warp leaves or none (others may be latching the word)
    if (__any_sync(0xffffffffu, *(volatile const unsigned int*)status & STATUS_DEVICE_WAIT)) return;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const bool valid = i < F.n;  // no early return: the warp stages its rows together
    if (lane == 0) {
        tc::mbar_init(bars, 1);
        tc::mbar_init(bars + 1, 1);
    }
    __syncwarp();
    float4 xi = make_float4(0.f, 0.f, 0.f, 0.f), vi = xi, ri = xi;
    if (valid) {
        xi = F.posS[i];
        vi = F.velS[i];
        ri = F.rho4S[i];
    }
    const PhysDev& ph = F.ph;
    ForceTotals<KAHAN, TENSION> A;
    // a row: this lane's window (start, mask) and the warp's staged union [u0, u0 + len)
    auto row_info = [&](int r, int& sv, unsigned int& mk, int& u0, int& len) {
        sv = 0;
        mk = 0u;
        int lo = INT_MAX, hi = INT_MIN;
        if (valid) {
            sv = __ldg(F.M.start + (size_t)r * F.n + i);
            mk = __ldg(F.M.mask + (size_t)r * F.n + i);
            if (sv >= 0 && mk) {
                lo = sv + __ffs(mk) - 1;
                hi = sv + 32 - __clz(mk);
            }
        }
        u0 = __reduce_min_sync(0xffffffffu, lo);
        const int u1 = __reduce_max_sync(0xffffffffu, hi);
        len = u1 > u0 ? u1 - u0 : 0;
        if (len > ST_ROW) len = -1;  // not staged
    };
    unsigned int phase = 0u, pending = 0u;  // per buffer: wait parity, copy in flight
    bool broken = false;
    auto issue = [&](int b, int u0, int len) {
        if (lane == 0) {
            float4* d = buf + b * 3 * ST_ROW;
            const uint32_t bytes = (uint32_t)len * 16u;
            tc::fence_async_smem();  // this warp's reads of the buffer come first
            tc::mbar_arrive_expect_tx(bars + b, 3u * bytes);
            tc::bulk_g2s(d, F.posS + u0, bytes, bars + b);
            tc::bulk_g2s(d + ST_ROW, F.velS + u0, bytes, bars + b);
            tc::bulk_g2s(d + 2 * ST_ROW, F.rho4S + u0, bytes, bars + b);
        }
        pending |= 1u << b;
    };
    int sv, u0, len;
    unsigned int mk;
    row_info(0, sv, mk, u0, len);
    if (len > 0) issue(0, u0, len);
#pragma unroll 1
    for (int r = 0; r < 9; r++) {
        const int b = r & 1;
        int svN = 0, u0N = 0, lenN = 0;
        unsigned int mkN = 0u;
        if (r + 1 < 9) {
            row_info(r + 1, svN, mkN, u0N, lenN);
            if (lenN > 0 && !broken) issue(b ^ 1, u0N, lenN);
        }
        bool staged = len > 0 && (pending >> b & 1u);
        if (staged) {
            const bool ok = __all_sync(0xffffffffu, tc::mbar_wait(bars + b, phase >> b & 1u, ST_WAIT_LIMIT));
            if (ok) {
                phase ^= 1u << b;
                pending &= ~(1u << b);
            } else {
                if (lane == 0 && status) atomicOr(status, STATUS_DEVICE_WAIT);
                broken = true;
                staged = false;
            }
        }
        RowSums<TENSION> R;
        R.clear();
        if (valid) {
            if (sv < 0) {
                // a window too long for a mask: test and interact from global memory
                for (int t = sv & 0x7fffffff; t < (int)mk; t++) {
                    const float4 xj = __ldg(F.posS + t);
                    const float r2 = dist2(xi, xj);
                    if (neighbour_r2(r2, ph.h2)) {
                        const float4 vj = __ldg(F.velS + t), rj = __ldg(F.rho4S + t);
                        R.add(ph, Pair(ph, xi, vi, xj, vj), ri.z, rj);
                    }
                }
            } else {
                const float4* P = buf + b * 3 * ST_ROW;
                R.hits += __popc(mk);
                while (mk) {
                    const int t = sv + __ffs(mk) - 1;
                    mk &= mk - 1u;
                    float4 xj, vj, rj;
                    if (staged) {
                        xj = P[t - u0];
                        vj = P[ST_ROW + t - u0];
                        rj = P[2 * ST_ROW + t - u0];
                    } else {
                        xj = __ldg(F.posS + t);
                        vj = __ldg(F.velS + t);
                        rj = __ldg(F.rho4S + t);
                    }
                    R.template add<false>(ph, Pair(ph, xi, vi, xj, vj), ri.z, rj);
                }
            }
        }
        __syncwarp();  // the buffer is refilled two rows on
        A.add(R);
        sv = svN;
        mk = mkN;
        u0 = u0N;
        len = lenN;
    }
    if (broken && lane == 0)  // copies still in flight land before the block leaves
        for (int b = 0; b < 2; b++)
            if (pending >> b & 1u) tc::mbar_wait(bars + b, phase >> b & 1u, ST_WAIT_LIMIT);
    __syncwarp();
    if (valid) {
        FeatSums fs;
        force_epilogue<KAHAN, TENSION, false>(A, i, xi, vi, ri, ph, F.map, F.collide, F.workIds, F.pos, F.vel,
                                              F.accS, fs, F.fo);
    }
}

// ---------------------------------------------------------------------------
// The learned step's force stage with the corrector fused in.  The pretested
// pair loop, wall terms, integration and collision of k_force, then the
// 24 features of each particle go straight to shared memory as a BF16 MMA
// operand.  The block's two 128-particle tiles run the MLP together: each
// layer is two tcgen05.mma groups (one per tile, accumulators in TMEM
// columns 64 * tile) behind one commit, and every warp then reads its own
// tile's accumulator lanes.  Each particle's correction is added before its
// single write-back.  Three or four blocks share an SM, so one block's MMA
// round trips overlap the others' pair loops.  The raw features also go to
// `fo.feat` when it is set.
// ---------------------------------------------------------------------------
// Shared memory is kept small: the pair loop's neighbour gathers live on
// the L1 cache, which shares the SM's 256 KB with it.  The operand region
// holds the two feature tiles until layer 1's MMAs have read them, then the
// two hidden tiles of layer 1, then those of layer 2.
constexpr int L_W = 0;                        // W1, W2, W3 (mlp::IMG_FWD_BYTES)
constexpr int L_X = mlp::IMG_FWD_BYTES;       // operand region: two 128 x 32 feature tiles, ...
constexpr int L_H = L_X;                      // ... later two 128 x 64 hidden tiles
constexpr int L_BIAS = L_H + 2 * 16384;
constexpr int L_NORM = L_BIAS + 4 * mlp::NBIAS;
constexpr int L_BAR = L_NORM + 4 * mlp::NNORM;  // MMA barrier, TMEM slot, weight-copy barrier
constexpr int L_SMEM = L_BAR + 32;
constexpr int L_TMEM = 128;                   // 4 blocks x 128 = 512 columns
constexpr int L_THREADS = 256;
// Resident blocks per SM.  Over the lists three (80 registers): a group's
// gathers are in flight together, and four blocks' 64 registers spill them
// (524,288 particles 221 us a step with three, 249 with four, 235 with two;
// 60,000: 50, 57, 48).  With the per-step search four when the grid fills the
// GPU several times over, the pair loop being latency bound; three for small
// grids, where per-thread latency counts.
constexpr int L_BLOCKS_MAX = 4;
static_assert(L_X % 1024 == 0 && L_BIAS % 16 == 0 && L_NORM % 16 == 0 && L_BAR % 8 == 0, "layout");
static_assert(L_BLOCKS_MAX * (L_SMEM + 1024) <= 227 * 1024 && L_BLOCKS_MAX * L_TMEM <= 512,
              "resident blocks per SM");

// LISTS: the neighbours come from the reused lists, or in a building step
// from the rows the density stage recorded (as in k_force_lists; the same
// pairs in the same order as the per-step search there), their p/rho^2 and
// 1/rho from the fourth lanes of their sorted position and velocity, and the
// kernel records the largest squared distance of a corrected position from where
// the particle was when the lists were built.
template <bool KAHAN, bool TENSION, int BLOCKS, bool LISTS, bool MASKS>
__global__ void __launch_bounds__(L_THREADS, BLOCKS)
k_force_learned(ForceArgs F, MlpDev m, unsigned int* status, NeighbourLists L) {
    using namespace mlp;
    extern __shared__ __align__(1024) unsigned char sm[];
    __shared__ int sOk;
    const int t = threadIdx.x, warp = t >> 5, half = t >> 7, r = t & 127;
    uint64_t* bar = reinterpret_cast<uint64_t*>(sm + L_BAR);
    uint32_t* slot = reinterpret_cast<uint32_t*>(sm + L_BAR + 8);
    uint64_t* wbar = reinterpret_cast<uint64_t*>(sm + L_BAR + 16);
    float* sBias = reinterpret_cast<float*>(sm + L_BIAS);
    float* sNorm = reinterpret_cast<float*>(sm + L_NORM);
    for (int k = t; k < NBIAS; k += L_THREADS) sBias[k] = epilogue_bias(m.bias, k);
    for (int k = t; k < NNORM; k += L_THREADS) sNorm[k] = m.norm[k];
    if (t == 0) {
        tc::mbar_init(bar, 1);
        tc::mbar_init(wbar, 1);
        // one thread reads the latch for its block (others may be setting it)
        sOk = *(volatile unsigned int*)status & STATUS_DEVICE_WAIT ? 3 : 1;
        // the weight image arrives by one TMA bulk copy while the pair loop runs
        if (sOk == 1) {
            tc::mbar_arrive_expect_tx(wbar, IMG_FWD_BYTES);
            tc::bulk_g2s(sm + L_W, m.image, IMG_FWD_BYTES, wbar);
        }
    }
    if (warp == 0) tc::tmem_alloc(slot, L_TMEM);
    tc::cta_sync();
    const uint32_t tb = *slot;
    if (sOk == 3) {
        tc::cta_sync();
        if (warp == 0) tc::tmem_dealloc(tb, L_TMEM);
        return;
    }
    const int i = blockIdx.x * L_THREADS + t;
    const bool valid = i < F.n;
    float3 x = make_float3(0.f, 0.f, 0.f), v = x;
    float4 xi = make_float4(0.f, 0.f, 0.f, 0.f);
    int id = 0;
    {
        float f[IN];
        if (valid) {
            xi = F.posS[i];
            const float4 vi = F.velS[i];
            const float4 ri = F.rho4S[i];
            const PhysDev& ph = F.ph;
            ForceTotals<KAHAN, TENSION> A;
            FeatSums fs;
            if (LISTS) {
                list_rows<TENSION, MASKS, false>(
                    i, F.n, L.flags[VL_BUILD_NOW * L.numScenes], L, F.M, F.posS, F.velS, xi, ph.h2,
                    [&](RowSums<TENSION>& R, float4 xj, float4 vj, bool tested) {
                        const Pair p(ph, xi, vi, xj, vj);
                        if (tested || neighbour_r2(p.r2, ph.h2)) {
                            const float4 rj = make_float4(0.f, 0.f, xj.w, vj.w);
                            R.add(ph, p, ri.z, rj);
                            fs.add(ph, p, rj);
                        }
                    },
                    [&](const RowSums<TENSION>& R, bool group) {
                        if (group) A.add_all(R);
                        else A.add(R);
                        fs.cnt += R.hits;
                    });
            }
#pragma unroll
            for (int row = 0; row < (LISTS ? 0 : 9); row++) {
                RowSums<TENSION> R;
                R.clear();
                const int sv = __ldg(F.M.start + (size_t)row * F.n + i);
                unsigned int mk = __ldg(F.M.mask + (size_t)row * F.n + i);
                if (sv < 0) {
                    for (int tt = sv & 0x7fffffff; tt < (int)mk; tt++) {
                        const float4 xj = __ldg(F.posS + tt);
                        const float r2 = dist2(xi, xj);
                        if (neighbour_r2(r2, ph.h2)) {
                            const float4 vj = __ldg(F.velS + tt), rj = __ldg(F.rho4S + tt);
                            const Pair p(ph, xi, vi, xj, vj);
                            R.add(ph, p, ri.z, rj);
                            fs.add(ph, p, rj);
                        }
                    }
                } else {
                    R.hits += __popc(mk);
                    while (mk) {
                        const int tt = sv + __ffs(mk) - 1;
                        mk &= mk - 1u;
                        const float4 xj = __ldg(F.posS + tt), vj = __ldg(F.velS + tt), rj = __ldg(F.rho4S + tt);
                        const Pair p(ph, xi, vi, xj, vj);
                        R.template add<false>(ph, p, ri.z, rj);
                        fs.add(ph, p, rj);
                    }
                }
                A.add(R);
                fs.cnt += R.hits;
            }
            float acc[3], mapDist = 1e30f, mapN[3] = {0.f, 0.f, 0.f};
            force_finish<KAHAN, TENSION, true>(A, xi, vi, ri, ph, F.map, F.collide, x, v, acc, mapDist, mapN, xi);
            id = F.workIds[i];
            F.accS[i] = make_float4(acc[0], acc[1], acc[2], 0.f);
            feature_values(fs, F.fo.boxWalls, F.fo.dtL, xi, vi, ri, acc, mapDist, mapN, ph, f);
            if (F.fo.feat) store_features(F.fo.feat, (size_t)(F.fo.byId ? id : i), f);
        }
        store_feature_row(sm + L_X + half * 8192, r, f, valid, sNorm);
    }
    const uint32_t sW = tc::smem_u32(sm + L_W);
    const uint32_t sX = tc::smem_u32(sm + L_X), sH = tc::smem_u32(sm + L_H);
    unsigned char* myH = sm + L_H + half * 16384;
    const uint32_t tl = tc::tmem_at(tb, 32 * (warp & 3), 64 * half);  // this warp's lanes of its tile
    uint32_t phase = 0;
    // sOk: 1 running, 0 an MMA wait gave up, 2 the weight copy never landed (3, above: a wait of the sort gave up)
    if (t == 0 && !tc::mbar_wait(wbar, 0, WAIT_LIMIT)) {
        sOk = 2;
        atomicOr(status, STATUS_DEVICE_WAIT);
    }
    tc::cta_sync();
    if (sOk == 1) do {
        tc::cta_sync();
        if (t == 0) {
            tc::mma_chain(tb, sX, sW + IMG_W1, INP, HID, false);
            tc::mma_chain(tb + 64, sX + 8192, sW + IMG_W1, INP, HID, false);
        }
        if (!commit_and_wait(bar, phase, &sOk, t)) break;
        hidden_layer_out(tl, sBias, myH, r);
        tc::cta_sync();
        if (t == 0) {
            tc::mma_chain(tb, sH, sW + IMG_W2, HID, HID, false);
            tc::mma_chain(tb + 64, sH + 16384, sW + IMG_W2, HID, HID, false);
        }
        // once the wait returns the MMAs have read layer 1's tiles: layer 2
        // overwrites them
        if (!commit_and_wait(bar, phase, &sOk, t)) break;
        hidden_layer_out(tl, sBias + HID, myH, r);
        tc::cta_sync();
        if (t == 0) {
            tc::mma_chain(tb, sH, sW + IMG_W3, HID, OUTP, false);
            tc::mma_chain(tb + 64, sH + 16384, sW + IMG_W3, HID, OUTP, false);
        }
        if (!commit_and_wait(bar, phase, &sOk, t)) break;
        float y[16];
        tc::tmem_ld16(tl, y);
        if (valid) {
            float c[OUT];
            decode_correction(sNorm, sBias + 2 * HID, y, c);
            x = make_float3(x.x + c[0], x.y + c[1], x.z + c[2]);
            v = make_float3(v.x + c[3], v.y + c[4], v.z + c[5]);
            if (F.collide) collide(F.ph, x, v);
            F.pos[id] = make_float4(x.x, x.y, x.z, LISTS ? 0.f : xi.w);
            F.vel[id] = make_float4(v.x, v.y, v.z, 0.f);
        }
    } while (false);
    tc::cta_sync();
    if (sOk == 0) drain(bar, phase, t, status);
    if (sOk == 2 && t == 0) tc::mbar_wait(wbar, 0, WAIT_LIMIT);  // once more for the copy in flight
    tc::cta_sync();
    if (warp == 0) tc::tmem_dealloc(tb, L_TMEM);
    if (LISTS) {  // as in k_force_lists
        float d2 = 0.f;
        if (valid) {
            const float4 b = __ldg(L.posB + i);
            const float dx = x.x - b.x, dy = x.y - b.y, dz = x.z - b.z;
            d2 = dx * dx + dy * dy + dz * dz;
            if (!(d2 == d2)) d2 = __uint_as_float(0x7f800000u);
        }
        record_displacement<false>(L, 0, d2);
    }
}

// ---------------------------------------------------------------------------
// Launchers
// ---------------------------------------------------------------------------
void launch_density(int n, const float4* posS, RowTables T, GridDev g, PhysDev ph, MapDev map, float4* rho4S,
                    int* rowStart, unsigned int* rowMask, const StepConfig& cfg, cudaStream_t s) {
    if (n <= 0) return;
    const int bs = cfg.densityBlock > 0 ? cfg.densityBlock : 128;
    const int grid = (n + bs - 1) / bs;
    const RowMasks M{rowStart, rowMask};
    const bool emit = cfg.forceVariant >= FORCE_PRETESTED;  // the pretested and staged forms read masks
#define SPH_DENSITY(K, E, B) k_density<K, E, B, false><<<grid, bs, 0, s>>>(n, posS, T, g, ph, map, cfg.prune, rho4S, M)
#define SPH_DENSITY_REL(K, E) k_density<K, E, false, true><<<grid, bs, 0, s>>>(n, posS, T, g, ph, map, cfg.prune, rho4S, M)
    if (g.rel) {
        if (cfg.kahan) {
            if (emit) SPH_DENSITY_REL(true, true);
            else SPH_DENSITY_REL(true, false);
        } else {
            if (emit) SPH_DENSITY_REL(false, true);
            else SPH_DENSITY_REL(false, false);
        }
    } else if (T.scenes) {
        if (cfg.kahan) {
            if (emit) SPH_DENSITY(true, true, true);
            else SPH_DENSITY(true, false, true);
        } else {
            if (emit) SPH_DENSITY(false, true, true);
            else SPH_DENSITY(false, false, true);
        }
    } else {
        if (cfg.kahan) {
            if (emit) SPH_DENSITY(true, true, false);
            else SPH_DENSITY(true, false, false);
        } else {
            if (emit) SPH_DENSITY(false, true, false);
            else SPH_DENSITY(false, false, false);
        }
    }
#undef SPH_DENSITY
#undef SPH_DENSITY_REL
}

template <bool KAHAN, bool TENSION>
static void force_dispatch(const ForceArgs& F, const StepConfig& cfg, unsigned int* status, cudaStream_t s) {
    const int bs = cfg.forceBlock > 0 ? cfg.forceBlock : 128;
    const int grid = (F.n + bs - 1) / bs;
    if (F.T.scenes) {
        // batched scenes (plain steps only; no feature recording); the staged
        // form is the plain handles' only, the pretested one serves here
        if (cfg.forceVariant >= FORCE_PRETESTED)
            k_force<KAHAN, TENSION, FORCE_PRETESTED, false, true><<<grid, bs, 0, s>>>(F);
        else if (cfg.forceVariant == FORCE_MASK)
            k_force<KAHAN, TENSION, FORCE_MASK, false, true><<<grid, bs, 0, s>>>(F);
        else
            k_force<KAHAN, TENSION, FORCE_DIRECT, false, true><<<grid, bs, 0, s>>>(F);
    } else if (F.g.rel) {
        // cell-relative positions (plain steps only; the pretested form stands
        // in for the staged one)
        if (cfg.forceVariant >= FORCE_PRETESTED)
            k_force<KAHAN, TENSION, FORCE_PRETESTED, false, false, true><<<grid, bs, 0, s>>>(F);
        else if (cfg.forceVariant == FORCE_MASK)
            k_force<KAHAN, TENSION, FORCE_MASK, false, false, true><<<grid, bs, 0, s>>>(F);
        else
            k_force<KAHAN, TENSION, FORCE_DIRECT, false, false, true><<<grid, bs, 0, s>>>(F);
    } else if (F.fo.feat) {
        // the learned step's force stage records the corrector's features; the
        // density stage has recorded the neighbour masks (pretested form)
        k_force<KAHAN, TENSION, FORCE_PRETESTED, true, false><<<grid, bs, 0, s>>>(F);
    } else if (cfg.forceVariant == FORCE_STAGED) {
        ensure_dynamic_smem<k_force_staged<KAHAN, TENSION>>(ST_SMEM);
        k_force_staged<KAHAN, TENSION>
            <<<(F.n + ST_WARPS * 32 - 1) / (ST_WARPS * 32), ST_WARPS * 32, ST_SMEM, s>>>(F, status);
    } else if (cfg.forceVariant == FORCE_PRETESTED) {
        k_force<KAHAN, TENSION, FORCE_PRETESTED, false, false><<<grid, bs, 0, s>>>(F);
    } else if (cfg.forceVariant == FORCE_MASK) {
        k_force<KAHAN, TENSION, FORCE_MASK, false, false><<<grid, bs, 0, s>>>(F);
    } else {
        k_force<KAHAN, TENSION, FORCE_DIRECT, false, false><<<grid, bs, 0, s>>>(F);
    }
}

void launch_force(int n, const float4* posS, const float4* velS, const float4* rho4S, const int* workIds,
                  RowTables T, GridDev g, PhysDev ph, MapDev map, int collide, const int* rowStart,
                  const unsigned int* rowMask, float4* pos, float4* vel, float4* accS, const StepConfig& cfg,
                  cudaStream_t s, const FeatureOut* feat, unsigned int* status) {
    if (n <= 0) return;
    FeatOut fo{nullptr, 0, 0, 0.f};
    if (feat) fo = FeatOut{feat->feat, feat->byId, feat->boxWalls, feat->dtL};
    ForceArgs F{n,  posS, velS, rho4S, workIds, T, g, ph, map, collide, cfg.prune,
                RowMasks{const_cast<int*>(rowStart), const_cast<unsigned int*>(rowMask)}, pos, vel, accS, fo};
    const bool tension = ph.tension != 0.0f;
    if (cfg.kahan) {
        if (tension) force_dispatch<true, true>(F, cfg, status, s);
        else force_dispatch<true, false>(F, cfg, status, s);
    } else {
        if (tension) force_dispatch<false, true>(F, cfg, status, s);
        else force_dispatch<false, false>(F, cfg, status, s);
    }
}

template <bool KAHAN, bool TENSION, int BLOCKS, bool LISTS, bool MASKS = false>
static void force_learned_launch(const ForceArgs& F, MlpDev m, unsigned int* status, const NeighbourLists& L,
                                 cudaStream_t s) {
    ensure_dynamic_smem<k_force_learned<KAHAN, TENSION, BLOCKS, LISTS, MASKS>>(L_SMEM);
    k_force_learned<KAHAN, TENSION, BLOCKS, LISTS, MASKS>
        <<<(F.n + L_THREADS - 1) / L_THREADS, L_THREADS, L_SMEM, s>>>(F, m, status, L);
}

template <bool KAHAN, bool TENSION>
static void force_learned_dispatch(const ForceArgs& F, MlpDev m, unsigned int* status, const NeighbourLists* L,
                                   cudaStream_t s) {
    const long long blocks = (F.n + L_THREADS - 1) / L_THREADS;
    if (L && L->masks)
        force_learned_launch<KAHAN, TENSION, 3, true, true>(F, m, status, *L, s);
    else if (L)
        force_learned_launch<KAHAN, TENSION, 3, true>(F, m, status, *L, s);
    else if (blocks >= 2LL * L_BLOCKS_MAX * device_sms())
        force_learned_launch<KAHAN, TENSION, L_BLOCKS_MAX, false>(F, m, status, NeighbourLists{}, s);
    else
        force_learned_launch<KAHAN, TENSION, 3, false>(F, m, status, NeighbourLists{}, s);
}

void launch_force_learned(int n, const float4* posS, const float4* velS, const float4* rho4S, const int* workIds,
                          RowTables T, GridDev g, PhysDev ph, MapDev map, int collide, const int* rowStart,
                          const unsigned int* rowMask, float4* pos, float4* vel, float4* accS, const StepConfig& cfg,
                          const FeatureOut& feat, MlpDev m, unsigned int* status, cudaStream_t s,
                          const NeighbourLists* lists) {
    if (n <= 0) return;
    const FeatOut fo{feat.feat, feat.byId, feat.boxWalls, feat.dtL};
    ForceArgs F{n,  posS, velS, rho4S, workIds, T, g, ph, map, collide, cfg.prune,
                RowMasks{const_cast<int*>(rowStart), const_cast<unsigned int*>(rowMask)}, pos, vel, accS, fo};
    const bool tension = ph.tension != 0.0f;
    if (cfg.kahan) {
        if (tension) force_learned_dispatch<true, true>(F, m, status, lists, s);
        else force_learned_dispatch<true, false>(F, m, status, lists, s);
    } else {
        if (tension) force_learned_dispatch<false, true>(F, m, status, lists, s);
        else force_learned_dispatch<false, false>(F, m, status, lists, s);
    }
}

// After the positions were written: the largest squared distance of a
// particle from where it was when the lists were built, in place of the one
// the steps accumulated (the next step builds the lists again only if that
// exceeds the rebuild distance).  flags[VL_DISP] must be zero on entry.
template <bool BATCH>
__global__ void k_list_displacement(int n, const float4* __restrict__ pos, const int* __restrict__ workIds,
                                    NeighbourLists L) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    float d2 = 0.f;
    int scene = 0;
    if (k < n) {
        const float4 x = __ldg(pos + workIds[k]), b = __ldg(L.posB + k);
        if (BATCH) scene = L.slotScene[k];
        const float dx = x.x - b.x, dy = x.y - b.y, dz = x.z - b.z;
        d2 = dx * dx + dy * dy + dz * dz;
        if (!(d2 == d2)) d2 = __uint_as_float(0x7f800000u);
    }
    record_displacement<BATCH>(L, scene, d2);
}

void launch_list_displacement(int n, const float4* pos, const int* workIds, const NeighbourLists& L, cudaStream_t s) {
    if (n <= 0) return;
    cudaMemsetAsync(L.flags + VL_DISP * L.numScenes, 0, sizeof(unsigned int) * L.numScenes, s);
    if (L.numScenes > 1) k_list_displacement<true><<<(n + 255) / 256, 256, 0, s>>>(n, pos, workIds, L);
    else k_list_displacement<false><<<(n + 255) / 256, 256, 0, s>>>(n, pos, workIds, L);
}

void launch_density_lists(int n, float4* posS, float4* velS, RowTables T, GridDev g, PhysDev ph, MapDev map,
                          float4* rho4S, const NeighbourLists& L, RowMasks M, const StepConfig& cfg, cudaStream_t s) {
    if (n <= 0) return;
    const int bs = cfg.densityBlock > 0 ? cfg.densityBlock : 128;
    const int grid = (n + bs - 1) / bs;
#define SPH_DENSITY_LISTS(K, B, X) \
    k_density_lists<K, B, X><<<grid, bs, 0, s>>>(n, posS, velS, T, g, ph, map, rho4S, L, M)
#define SPH_DENSITY_LISTS_B(K)                                \
    do {                                                      \
        if (T.scenes && L.masks) SPH_DENSITY_LISTS(K, true, true); \
        else if (T.scenes) SPH_DENSITY_LISTS(K, true, false); \
        else if (L.masks) SPH_DENSITY_LISTS(K, false, true);  \
        else SPH_DENSITY_LISTS(K, false, false);              \
    } while (0)
    if (cfg.kahan) SPH_DENSITY_LISTS_B(true);
    else SPH_DENSITY_LISTS_B(false);
#undef SPH_DENSITY_LISTS_B
#undef SPH_DENSITY_LISTS
}

void launch_force_lists(int n, const float4* posS, const float4* velS, const float4* rho4S, const int* workIds,
                        PhysDev ph, MapDev map, int collide, const NeighbourLists& L, RowMasks M, float4* pos,
                        float4* vel, float4* accS, const StepConfig& cfg, cudaStream_t s, const SceneDev* scenes) {
    if (n <= 0) return;
    const int bs = cfg.forceBlock > 0 ? cfg.forceBlock : 128;
    const int grid = (n + bs - 1) / bs;
    // (a batch's tension coefficient is the largest of its scenes': it selects
    // whether the colour field is computed at all)
    const bool tension = ph.tension != 0.0f;
#define SPH_FORCE_LISTS(K, T, B, X)                                                                             \
    k_force_lists<K, T, B, X><<<grid, bs, 0, s>>>(n, posS, velS, rho4S, workIds, ph, map, collide, L, M, pos, vel, \
                                                  accS, scenes)
#define SPH_FORCE_LISTS_B(K, T)                                \
    do {                                                       \
        if (scenes && L.masks) SPH_FORCE_LISTS(K, T, true, true); \
        else if (scenes) SPH_FORCE_LISTS(K, T, true, false);   \
        else if (L.masks) SPH_FORCE_LISTS(K, T, false, true);  \
        else SPH_FORCE_LISTS(K, T, false, false);              \
    } while (0)
    if (cfg.kahan) {
        if (tension) SPH_FORCE_LISTS_B(true, true);
        else SPH_FORCE_LISTS_B(true, false);
    } else {
        if (tension) SPH_FORCE_LISTS_B(false, true);
        else SPH_FORCE_LISTS_B(false, false);
    }
#undef SPH_FORCE_LISTS_B
#undef SPH_FORCE_LISTS
}

template <bool KAHAN, bool TENSION, bool MASKS>
static void steps_launch(StepsArgs& A, cudaStream_t s) {
    const int want = std::max((A.F.n + STEPS_THREADS - 1) / STEPS_THREADS, A.F.g.numCells / (16 * STEPS_THREADS));
    const int grid = std::min(want, resident_blocks<k_steps<KAHAN, TENSION, MASKS>>(STEPS_THREADS, STEPS_BLOCKS));
    void* args[] = {&A};
    cudaLaunchCooperativeKernel((const void*)k_steps<KAHAN, TENSION, MASKS>, dim3(grid), dim3(STEPS_THREADS), args, 0, s);
}

bool takes_whole_steps(int n, int numCells) { return n <= STEPS_PARTICLES && numCells <= STEPS_CELLS; }

void launch_steps(int n, float4* pos, float4* vel, GridDev g, SortBuffers sb, RowTables T, float4* posS, float4* velS,
                  float4* rho4S, float4* accS, PhysDev ph, MapDev map, int collide, const NeighbourLists& L, RowMasks M,
                  const StepConfig& cfg, int steps, unsigned int* status, cudaStream_t s) {
    if (n <= 0) return;
    StepsArgs A{FrontArgs{n, pos, vel, g, sb, posS, velS, status, L, 1, FRONT_ALL, scan_wait_limit()},
                T, ph, map, M, rho4S, accS, pos, vel, collide, 0};
    const bool tension = ph.tension != 0.0f;
    for (; steps > 0; steps -= A.steps) {
        A.steps = std::min(steps, STEPS_A_LAUNCH);
#define SPH_STEPS(K, T)                          \
    do {                                         \
        if (L.masks) steps_launch<K, T, true>(A, s); \
        else steps_launch<K, T, false>(A, s);    \
    } while (0)
        if (cfg.kahan) {
            if (tension) SPH_STEPS(true, true);
            else SPH_STEPS(true, false);
        } else {
            if (tension) SPH_STEPS(false, true);
            else SPH_STEPS(false, false);
        }
#undef SPH_STEPS
    }
}

}  // namespace sph
