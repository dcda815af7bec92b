// Boundary maps of "SPH in complex shapes" (SphInComplexShapes.cpp:203-427),
// built on the GPU.
//
// The reference scatters each ghost particle's poly6 / viscosity-kernel value
// onto the grid nodes within its support (SetBox, :269-304).  Here every node
// gathers from the ghost lattice points within its support instead, visiting
// them in the same k, j, i lattice order the reference creates its ghosts in,
// so each node's sum is accumulated in the reference's order and needs no
// atomics.  This file is compiled with --fmad=false: node positions, signed
// distances and kernel values are formed one rounded operation at a time, as
// the reference's host code does.
//
// What bounds it: signed distances in FP64 (1/64 of the FP32 rate here) and
// FP64 kernel coefficients, once per node and ghost candidate, took 22.8 ms
// for a 128^3 map.  The lattice's ghosts are now found once, as one bit a
// lattice point, and the nodes walk the set bits; a distance is taken in FP64
// only where an FP32 one with a bound on its error cannot decide; the
// coefficients are formed on the host; the band's nodes are listed, so that the
// sums fill their warps.  22.8 -> 0.20 ms for that map (sphere and cone;
// lattice 9 us, distances 69, sums of the band's nodes 125).
#include <math.h>

#include <algorithm>

#include "sph_internal.h"

namespace sph {
namespace {

struct MapArgs {
    float start[3];
    float spacing;
    unsigned int dims[3];
    float restDistance, h, mass, restDensity, viscosity, ps;
    int numShapes;
    sph_shape shapes[8];
    int boxOnly;             // one box container: SetBox's ghost rule
    int boxIndex;
    float latStart[3];       // ghost lattice origin and last index per axis
    unsigned int latMax[3];
    const unsigned int* ghosts;  // a bit per lattice point, x rows of rowWords words; NULL: tested at each node
    unsigned int rowWords;
    float densityCoeff;      // evaluateDensityKernel's and evaluateViscosityKernel's coefficients
    double viscosityCoeff;
    float viscosityHi, viscosityLo;  // the same as a sum of two floats; hi 0: out of their range
    // SPH_SHAPE_MESH solids: the signed distance grid of shape slot i
    const float* grid[8];
    float gridOrigin[8][3];
    float gridDx[8];
    unsigned int gridDims[8][3];
};

// Trilinear signed distance of a grid solid (negative inside); no solid
// outside the grid's box.
__device__ double grid_sdf(const MapArgs& A, int s, const double* x) {
    double w[3];
    size_t i0[3];
    for (int a = 0; a < 3; a++) {
        const unsigned int n = A.gridDims[s][a];
        const double u = (x[a] - (double)A.gridOrigin[s][a]) / (double)A.gridDx[s];
        if (!(u >= 0.0) || u > (double)(n - 1)) return 1e30;
        const double f = n > 1 ? fmin(floor(u), (double)(n - 2)) : 0.0;
        i0[a] = (size_t)f;
        w[a] = n > 1 ? u - f : 0.0;
    }
    const unsigned int* d = A.gridDims[s];
    auto at = [&](int di, int dj, int dk) {
        const size_t ii = i0[0] + (d[0] > 1 ? di : 0), jj = i0[1] + (d[1] > 1 ? dj : 0),
                     kk = i0[2] + (d[2] > 1 ? dk : 0);
        return (double)A.grid[s][ii + (size_t)d[0] * (jj + (size_t)d[1] * kk)];
    };
    const double c00 = at(0, 0, 0) + w[0] * (at(1, 0, 0) - at(0, 0, 0));
    const double c10 = at(0, 1, 0) + w[0] * (at(1, 1, 0) - at(0, 1, 0));
    const double c01 = at(0, 0, 1) + w[0] * (at(1, 0, 1) - at(0, 0, 1));
    const double c11 = at(0, 1, 1) + w[0] * (at(1, 1, 1) - at(0, 1, 1));
    const double c0 = c00 + w[1] * (c10 - c00), c1 = c01 + w[1] * (c11 - c01);
    return c0 + w[2] * (c1 - c0);
}

// computeSignedDistancePoint3Box3 (SphInComplexShapes.cpp:714-747), axis-aligned.
__device__ float box_signed_distance(const float* pos, const float* c, const float* e) {
    float t[3] = {pos[0] - c[0], pos[1] - c[1], pos[2] - c[2]};
    float a = fabsf(t[0]) - e[0];
    float b = fabsf(t[1]) - e[1];
    float cc = fabsf(t[2]) - e[2];
    float distance = fabsf(a) < fabsf(b) ? a : b;
    if (fabsf(distance) > fabsf(cc)) distance = cc;
    if (a > 0.0f || b > 0.0f || cc > 0.0f) {
        float sq = 0.0f;
        for (int k = 0; k < 3; k++) {
            float d = 0.0f;
            if (t[k] < -e[k]) d = t[k] + e[k];
            else if (t[k] > e[k]) d = t[k] - e[k];
            sq += d * d;
        }
        distance = sqrtf(sq);
    }
    return distance;
}

__device__ bool inside_box(const float* pos, const float* c, const float* e) {
    for (int k = 0; k < 3; k++)
        if (fabsf(pos[k] - c[k]) >= e[k]) return false;
    return true;
}

// Solid cone on its base disc: distance to the triangle (0,0)-(R,0)-(0,H) in
// the (radial, axial) half-plane, negative inside.
__device__ double cone_sdf(const double* x, const float* p) {
    double q = sqrt((x[0] - p[0]) * (x[0] - p[0]) + (x[1] - p[1]) * (x[1] - p[1]));
    double z = x[2] - p[2];
    double R = p[3], H = p[4];
    double bq = fmin(fmax(q, 0.0), R);
    double d2 = (q - bq) * (q - bq) + z * z;
    double ex = -R, ez = H;
    double t = ((q - R) * ex + z * ez) / (ex * ex + ez * ez);
    t = fmin(fmax(t, 0.0), 1.0);
    double sx = q - (R + t * ex), sz = z - t * ez;
    d2 = fmin(d2, sx * sx + sz * sz);
    bool inside = z >= 0.0 && z <= H && q <= R * (1.0 - z / H);
    double d = sqrt(d2);
    return inside ? -d : d;
}

// Distance to the solid, positive in the fluid.
__device__ float solid_distance(const MapArgs& A, const float* xf) {
    double x[3] = {xf[0], xf[1], xf[2]};
    double s = 1e30;
    for (int i = 0; i < A.numShapes; i++) {
        const sph_shape& S = A.shapes[i];
        double d;
        if (S.kind == SPH_SHAPE_SPHERE) {
            double dx = x[0] - S.p[0], dy = x[1] - S.p[1], dz = x[2] - S.p[2];
            d = sqrt(dx * dx + dy * dy + dz * dz) - S.p[3];
        } else if (S.kind == SPH_SHAPE_CONE) {
            d = cone_sdf(x, S.p);
        } else if (S.kind == SPH_SHAPE_MESH) {
            d = grid_sdf(A, i, x);
        } else {
            d = -(double)box_signed_distance(xf, S.p, S.p + 3);
        }
        s = fmin(s, d);
    }
    return (float)s;
}

// The distance to the solids in FP32 and a bound on its error: `margin` is
// many times what the roundings of the few operations on numbers up to the
// coordinates' own size can add up to.  (A mesh's grid ends abruptly: no
// estimate, an infinite margin.)
__device__ float solid_estimate(const MapArgs& A, const float* x, float& margin) {
    float s = 1e30f, scale = fabsf(x[0]) + fabsf(x[1]) + fabsf(x[2]);
    for (int i = 0; i < A.numShapes; i++) {
        const sph_shape& S = A.shapes[i];
        float d;
        if (S.kind == SPH_SHAPE_SPHERE) {
            const float dx = x[0] - S.p[0], dy = x[1] - S.p[1], dz = x[2] - S.p[2];
            d = sqrtf(dx * dx + dy * dy + dz * dz) - S.p[3];
        } else if (S.kind == SPH_SHAPE_CONE) {
            const float dx = x[0] - S.p[0], dy = x[1] - S.p[1], z = x[2] - S.p[2], R = S.p[3], H = S.p[4];
            const float q = sqrtf(dx * dx + dy * dy);
            const float b = q - fminf(q, R);
            const float t = fminf(fmaxf(((q - R) * -R + z * H) / (R * R + H * H), 0.0f), 1.0f);
            const float sx = q - (R - t * R), sz = z - t * H;
            d = sqrtf(fminf(b * b + z * z, sx * sx + sz * sz));
            if (z >= 0.0f && z <= H && q <= R * (1.0f - z / H)) d = -d;
        } else if (S.kind == SPH_SHAPE_BOX) {
            d = -box_signed_distance(x, S.p, S.p + 3);
        } else {
            margin = INFINITY;
            return 0.0f;
        }
        for (int k = 0; k < 6; k++) scale += fabsf(S.p[k]);
        s = fminf(s, d);
    }
    // (lengths whose squares leave FP32's range have no estimate either)
    margin = scale > 1e-15f && scale < 1e15f ? 128.0f / 16777216.0f * scale : INFINITY;
    return s;
}

// evaluateDensityKernel / evaluateViscosityKernel (SphInComplexShapes.cpp:666-690).
__device__ float eval_density_kernel(const MapArgs& A, float sqDist) {
    float sqh = A.h * A.h;
    float diff = sqh - sqDist;
    if (diff < 0.0f) return 0.0f;
    return A.densityCoeff * diff * diff * diff;
}

__device__ float eval_viscosity_kernel(const MapArgs& A, float sqDist) {
    float dist = sqrtf(sqDist);
    if (dist > A.h) return 0.0f;
    const float x = A.h - dist;
    if (A.viscosityHi == 0.0f) return (float)(A.viscosityCoeff * x);
    // the FP64 product rounded to FP32, from FP32 operations (the FP64 pipe and
    // its conversions held the sums: 315 -> 125 us for a 128^3 map).  The two
    // products are within 2^-46 of the exact one, the FP64 product within
    // 2^-53: where all numbers within 2^-44 of theirs round alike, so does it.
    const float p = A.viscosityHi * x;
    const float low = __fmaf_rn(A.viscosityLo, x, __fmaf_rn(A.viscosityHi, x, -p));
    const float s = p + low;
    const float rest = low - (s - p), slack = s * 5.6843419e-14f;
    if (s + (rest - slack) == s && s + (rest + slack) == s) return s;
    return (float)(A.viscosityCoeff * x);
}

__device__ void node_pos(const MapArgs& A, int i, int j, int k, float* p) {
    p[0] = A.start[0] + A.spacing * (float)i;
    p[1] = A.start[1] + A.spacing * (float)j;
    p[2] = A.start[2] + A.spacing * (float)k;
}

__device__ bool is_ghost(const MapArgs& A, const float* g) {
    const sph_shape& B = A.shapes[A.boxIndex];
    if (A.boxOnly) return !inside_box(g, B.p, B.p + 3);
    float margin;
    const float d = solid_estimate(A, g, margin);
    if (fabsf(d) > margin) return d < 0.0f;
    return solid_distance(A, g) <= 0.0f;
}

// The ghosts of the lattice: word w of row (j, k) by one warp, a lane a point.
__global__ void k_ghost_bits(MapArgs A, unsigned int* __restrict__ bits, size_t words) {
    const size_t w = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (w >= words) return;  // the whole warp
    const unsigned int i = 32u * (unsigned int)(w % A.rowWords) + (threadIdx.x & 31u);
    const size_t row = w / A.rowWords;
    const unsigned int j = (unsigned int)(row % (A.latMax[1] + 1u)), k = (unsigned int)(row / (A.latMax[1] + 1u));
    const float g[3] = {A.latStart[0] + (float)(int)i * A.ps, A.latStart[1] + (float)(int)j * A.ps,
                        A.latStart[2] + (float)(int)k * A.ps};
    const unsigned int m = __ballot_sync(0xffffffffu, i <= A.latMax[0] && is_ghost(A, g));
    if ((threadIdx.x & 31u) == 0u) bits[w] = m;
}

// The density and viscosity of node n in the band (position np).
__device__ void splat_node(const MapArgs& A, const float* np, float& outRho, float& outVis) {
    // ghost lattice points that can lie within h of this node
    int lo[3], hi[3];
    for (int a = 0; a < 3; a++) {
        float f0 = floorf((np[a] - A.h - A.latStart[a]) / A.ps) - 1.0f;
        float f1 = floorf((np[a] + A.h - A.latStart[a]) / A.ps) + 1.0f;
        f0 = fmaxf(f0, 0.0f);
        f1 = fminf(f1, (float)A.latMax[a]);
        lo[a] = (int)f0;
        hi[a] = (int)f1;
    }
    outRho = outVis = 0.0f;
    auto add = [&](int ii, float gy, float gz) {
        const float dx = A.latStart[0] + (float)ii * A.ps - np[0], dy = gy - np[1], dz = gz - np[2];
        const float sq = dx * dx + dy * dy + dz * dz;
        outRho += eval_density_kernel(A, sq);
        outVis += eval_viscosity_kernel(A, sq);
    };
    for (int kk = lo[2]; kk <= hi[2]; kk++)
        for (int jj = lo[1]; jj <= hi[1]; jj++) {
            const float gy = A.latStart[1] + (float)jj * A.ps, gz = A.latStart[2] + (float)kk * A.ps;
            if (!A.ghosts) {
                for (int ii = lo[0]; ii <= hi[0]; ii++) {
                    const float g[3] = {A.latStart[0] + (float)ii * A.ps, gy, gz};
                    if (is_ghost(A, g)) add(ii, gy, gz);
                }
                continue;
            }
            const unsigned int* row = A.ghosts + ((size_t)kk * (A.latMax[1] + 1u) + (size_t)jj) * A.rowWords;
            for (int w = lo[0] >> 5; w <= hi[0] >> 5; w++) {
                unsigned int m = __ldg(row + w);
                if (w == lo[0] >> 5) m &= 0xffffffffu << (lo[0] & 31);
                if (w == hi[0] >> 5) m &= 0xffffffffu >> (31 - (hi[0] & 31));
                while (m) {
                    const int b = __ffs(m) - 1;
                    m &= m - 1u;
                    add(32 * w + b, gy, gz);
                }
            }
        }
    outRho *= A.mass;
    outVis *= A.viscosity * A.mass / A.restDensity;
}

struct MapOut {
    float *dist, *dens, *visc;
    float4* map4;
    __device__ void store(size_t n, float d, float rho, float vis) const {
        if (dist) dist[n] = d;
        if (dens) dens[n] = rho;
        if (visc) visc[n] = vis;
        if (map4) map4[n] = make_float4(d, rho, vis, 0.0f);
    }
};

__device__ void node_of(const MapArgs& A, size_t n, float* np) {
    const int i = (int)(n % A.dims[0]);
    const int j = (int)((n / A.dims[0]) % A.dims[1]);
    const int k = (int)(n / ((size_t)A.dims[0] * A.dims[1]));
    node_pos(A, i, j, k, np);
}

// Every node's distance.  The nodes in the band (one in twenty, scattered
// over the warps) are listed for k_splat_band, which fills its warps with
// them; without room for the list each thread takes its own node's sums.
__global__ void k_build_maps(MapArgs A, MapOut out, unsigned int* band, unsigned int* bandCount) {
    const size_t n = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    const bool valid = n < (size_t)A.dims[0] * A.dims[1] * A.dims[2];
    float np[3] = {0.0f, 0.0f, 0.0f};
    float outD = -A.restDistance, outRho = 0.0f, outVis = 0.0f;
    bool inBand = false;
    if (valid) {
        node_of(A, n, np);
        float margin;
        const float est = solid_estimate(A, np, margin);
        // a node certainly beyond the band needs no distance
        float d = fabsf(est) - margin > A.h ? A.h : -solid_distance(A, np);
        inBand = fabsf(d) < A.h;
        if (inBand) {
            if (fabsf(d) > A.restDistance) d = d / fabsf(d) * A.restDistance;
            outD = d;
        }
    }
    if (band) {
        const unsigned int peers = __ballot_sync(0xffffffffu, inBand), lane = threadIdx.x & 31u;
        unsigned int at = 0u;
        if (lane == 0u && peers) at = atomicAdd(bandCount, (unsigned int)__popc(peers));
        at = __shfl_sync(0xffffffffu, at, 0) + __popc(peers & ((1u << lane) - 1u));
        if (inBand) band[at] = (unsigned int)n;
    } else if (inBand) {
        splat_node(A, np, outRho, outVis);
    }
    if (valid) out.store(n, outD, outRho, outVis);
}

__global__ void __launch_bounds__(128) k_splat_band(MapArgs A, MapOut out, const unsigned int* __restrict__ band,
                                                    const unsigned int* __restrict__ bandCount) {
    const unsigned int count = *bandCount;
    for (unsigned int k = blockIdx.x * blockDim.x + threadIdx.x; k < count; k += gridDim.x * blockDim.x) {
        const size_t n = band[k];
        float np[3], rho, vis;
        node_of(A, n, np);
        splat_node(A, np, rho, vis);
        if (out.dens) out.dens[n] = rho;
        if (out.visc) out.visc[n] = vis;
        if (out.map4) {
            out.map4[n].y = rho;
            out.map4[n].z = vis;
        }
    }
}

// Lattices of up to 2^26 words (256 MB of bits) have their ghosts found once.
constexpr double GHOST_WORDS_MAX = 67108864.0;

}  // namespace

cudaError_t launch_build_maps(const sph_boundary_desc& D, const unsigned int dims[3], float* dist, float* dens,
                              float* visc, float4* map4, cudaStream_t s) {
    MapArgs A{};
    for (int a = 0; a < 3; a++) {
        A.start[a] = D.gridStart[a];
        A.dims[a] = dims[a];
    }
    A.spacing = D.gridSpacing;
    A.restDistance = D.restDistance;
    A.h = D.compactSupport;
    A.mass = D.particleMass;
    A.restDensity = D.restDensity;
    A.viscosity = D.viscosity;
    A.ps = D.particleSpacing;
    A.numShapes = D.numShapes;
    A.boxIndex = 0;
    int boxes = 0;
    for (int i = 0; i < D.numShapes && i < 8; i++) {
        A.shapes[i] = D.shapes[i];
        if (D.shapes[i].kind == SPH_SHAPE_BOX) {
            if (boxes == 0) A.boxIndex = i;
            boxes++;
        }
    }
    A.boxOnly = (boxes == 1 && D.numShapes == 1) ? 1 : 0;
    // Ghost lattice: SetBox's (SphInComplexShapes.cpp:233-244) around a box
    // container, else the map grid grown by compactSupport + particleSpacing.
    float margin = D.compactSupport + D.particleSpacing;
    for (int a = 0; a < 3; a++) {
        if (boxes > 0) {
            const sph_shape& B = D.shapes[A.boxIndex];
            float ext = B.p[3 + a] + margin;
            A.latStart[a] = B.p[a] - ext;
            A.latMax[a] = (unsigned int)(2 * ext / D.particleSpacing);
        } else {
            float len = (float)(dims[a] - 1) * D.gridSpacing + 2 * margin;
            A.latStart[a] = D.gridStart[a] - margin;
            A.latMax[a] = (unsigned int)(len / D.particleSpacing);
        }
    }
    size_t total = (size_t)dims[0] * dims[1] * dims[2];
    if (total == 0) return cudaSuccess;
    const float h = A.h;
    A.densityCoeff = (float)(315.0f / (64.0f * 3.14159265358979323846 * h * h * h * h * h * h * h * h * h));
    A.viscosityCoeff = 45.0f / (3.14159265358979323846 * h * h * h * h * h * h);
    if (A.viscosityCoeff > 1e-20 && A.viscosityCoeff < 1e20) {
        A.viscosityHi = (float)A.viscosityCoeff;
        A.viscosityLo = (float)(A.viscosityCoeff - (double)A.viscosityHi);
    }
    // grid solids: device copies of their distances for the build
    float* devGrid[8] = {};
    cudaError_t e = cudaSuccess;
    for (int i = 0; i < D.numShapes && i < 8 && e == cudaSuccess; i++) {
        if (D.shapes[i].kind != SPH_SHAPE_MESH) continue;
        const sph_sdf_grid& G = D.sdfGrids[(int)D.shapes[i].p[0]];
        const size_t nodes = (size_t)G.dims[0] * G.dims[1] * G.dims[2];
        e = cudaMalloc((void**)&devGrid[i], sizeof(float) * nodes);
        if (e == cudaSuccess) e = cudaMemcpyAsync(devGrid[i], G.distance, sizeof(float) * nodes, cudaMemcpyHostToDevice, s);
        A.grid[i] = devGrid[i];
        A.gridDx[i] = G.dx;
        for (int a = 0; a < 3; a++) {
            A.gridOrigin[i][a] = G.origin[a];
            A.gridDims[i][a] = G.dims[a];
        }
    }
    // scratch of the build: the band's count and node list, the lattice's bits
    A.rowWords = A.latMax[0] / 32u + 1u;
    const double wanted = (double)A.rowWords * ((double)A.latMax[1] + 1.0) * ((double)A.latMax[2] + 1.0);
    const size_t words = wanted <= GHOST_WORDS_MAX ? (size_t)wanted : 0;
    const MapOut out{dist, dens, visc, map4};
    unsigned int* scratch = nullptr;
    if (e == cudaSuccess && cudaMallocAsync((void**)&scratch, sizeof(unsigned int) * (4 + total + words), s) != cudaSuccess) {
        cudaGetLastError();  // no room: the nodes test the lattice and take their sums themselves
        scratch = nullptr;
    }
    unsigned int *count = scratch, *band = scratch ? scratch + 4 : nullptr;
    if (scratch) e = cudaMemsetAsync(count, 0, sizeof(unsigned int), s);
    if (scratch && words && e == cudaSuccess) {
        unsigned int* bits = band + total;
        k_ghost_bits<<<(unsigned int)((words + 3) / 4), 128, 0, s>>>(A, bits, words);
        e = cudaGetLastError();
        A.ghosts = bits;
    }
    if (e == cudaSuccess) {
        k_build_maps<<<(unsigned int)((total + 127) / 128), 128, 0, s>>>(A, out, band, count);
        e = cudaGetLastError();
    }
    if (band && e == cudaSuccess) {
        const size_t full = (size_t)device_sms() * 12;
        k_splat_band<<<(unsigned int)std::min((total + 127) / 128, full), 128, 0, s>>>(A, out, band, count);
        e = cudaGetLastError();
    }
    if (scratch) {
        const cudaError_t f = cudaFreeAsync(scratch, s);
        if (e == cudaSuccess) e = f;
    }
    bool any = false;
    for (float* g : devGrid) any = any || g;
    if (any) {
        const cudaError_t w = cudaStreamSynchronize(s);  // the grids are freed after the build
        if (e == cudaSuccess) e = w;
        for (float* g : devGrid)
            if (g) cudaFree(g);
    }
    return e;
}

}  // namespace sph
