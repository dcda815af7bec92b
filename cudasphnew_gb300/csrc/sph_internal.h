// Internal declarations shared by the kernels (sph_kernels.cu) and the host
// orchestration (sph_api.cu).  Not part of the public ABI.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/sph.h"

namespace sph {

// Device-side status bits, latched per handle and mapped to sph_status.
enum : unsigned int {
    STATUS_OUT_OF_DOMAIN = 1u,
    STATUS_DEVICE_WAIT = 2u,
    STATUS_NON_FINITE = 4u,
};

// Uniform cell grid (gridOrigin/gridSpacing/gridDim of SimulationParameters).
struct GridDev {
    float origin[3];
    float spacing;
    float inv;     // 1 / spacing
    int dim[3];
    int numCells;
    int cellBase;  // first global cell index of this grid (batched scenes; else 0)
    int rel;       // positions are cell-relative (sph_options.cellRelative)
};

// Largest grid of a cell-relative handle: cell coordinates pack 11:11:10 bits.
constexpr int REL_MAX_X = 2048, REL_MAX_Y = 2048, REL_MAX_Z = 1024;

// Trilinear boundary maps: map4 = (signed distance, wall density, wall
// viscosity, 0) per node, dist = signed distance alone (gradient samples).
struct MapDev {
    const float4* map4;
    const float* dist;
    float origin[3];
    float length[3];   // (dims-1)*spacing, particle_simulation.cu:2628-2631
    float dimsf[3];
    int dims[3];
    float du[3];       // spacing/length: the gradient step, :429-431
    float restDistance;
    int present;
};

// Per-level physical constants, pre-combined.
struct PhysDev {
    float h, h2;
    float poly6m;      // poly6 * mass
    float mass;
    float stiffness, restDensity;
    float pressCoef;   // -mass * gradSpiky (times rho_i per particle)
    float viscCoef;    // mu * mass * laplVisc
    float cgCoef;      // mass * gradPoly6
    float clCoef;      // mass * laplPoly6
    float tension, normThresh;
    float dt;          // integration step of this level
    float dtCollide;   // gSimParamsDev.timeStep (collision restitution term)
    float gravity;
    int gravityAxis;
    float boxCen[3], boxDim[3], restitution;
};

// One scene of a batched handle: its own cell grid (at cellBase in the
// concatenated cell space), physical constants, walls and boundary maps.  A
// particle's scene index travels in the .w lane of its position.
struct SceneDev {
    GridDev g;
    PhysDev ph;
    MapDev map;
};

// Scratch of the counting sort + cell scan.
struct SortBuffers {
    int* cnt;                 // [C+1] per-cell counters (kept zero between steps)
    int* cellOffset;          // [C+1] exclusive scan of cnt: first sorted index of each cell
    int2* keySlot;            // [n]   (hash, arrival slot in its cell)
    int* tmpIds;              // [n]   ids scattered to their cell segment, unordered
    int* sortedHash;          // [n]
    int* sortedIds;           // [n]   the reference's permutation (cell, id)
    int* workIds;             // [n]   the working order (cell, x, id) of the sorted arrays
    int* halfOffset;          // [C+1] first working index of each cell's upper x-half
    unsigned int* front;      // [FRONT_WORDS] a cooperative launch's barrier and block sums, zero between launches
    const SceneDev* scenes;   // batched handles: per-scene grids (else NULL)
    const int* skip;          // when non-NULL and set on the device, the sorted copies and
                              // tables already hold the current state: the sort stages return
};

// Two-scale state (AdvanceTwoScale): particle states, the three-way lists,
// persistent child slots 8*parent + k, and the fine level's sort.
struct TwoScaleDev {
    unsigned char* state;       // [n rounded up to 4] 2-bit history per particle
    int* blockCounts;           // [3 * blocks] per-block class counts
    int* counts;                // [5] split, boundary, default, children (device side); [4]: length
                                //     of markList, zero between steps
    int* markList;              // [n] working-order indices of split particles, any order
    int* splitIds;              // [n]
    int* boundaryIds;           // [n]
    int* defaultIds;            // [n]
    int* subIds;                // [8n] child list: split children, then boundary children
    float4* subPos;             // [8n] slots
    float4* subVel;
    float4* subAcc;
    float2* subRho;             // (density, pressure)
    int* subCnt;                // [Cs+1] fine-level counters (kept zero between steps)
    int* subOffset;             // [Cs+1] fine-level cell offsets
    int2* subKeySlot;           // [8n]
    int* subTmp;                // [8n]
    int* subSortedHash;         // [8n]
    int* subSortedIds;          // [8n] slots in (fine cell, list position) order
    float4* subPosS;            // [8n] child positions in that order
    float4* subVelS;            // [8n] child velocities in that order
    float splitMin[3], splitMax[3];
    int childMode;              // sph_options.childMode
    const unsigned int* status; // as RowTables::status
};

// Per-row lookup tables of the neighbour search.
struct RowTables {
    const int* cellOffset;  // [C+1]
    const int* halfOffset;  // [C+1]
    const SceneDev* scenes; // batched handles: per-scene grids, constants, maps (else NULL)
    const int* skip;        // as SortBuffers::skip, read by the density stage only
    const unsigned int* status;  // with STATUS_DEVICE_WAIT latched there is no sorted step to work on
                                 // (the list kernels know from VL_NOTHING)
};

// Reused neighbour lists (sph_options.neighbourSkin).  When the lists are
// built, every particle records the sorted slots of the particles within its
// skin sphere (radius R = (1 + skin) h), itself among them, row by row of the
// stencil in the working order, four to a group (the last group filled up
// with slot n, a record far from everything that the sorted copies keep there).
// Later steps keep that working order (the state is gathered into it) and
// visit only those candidates, until some particle has moved farther than
// 0.45 skin h from where it was at the build.  A particle with more
// candidates than the lists have room for records its rows' windows
// [start, end) instead, two to a group, and tests every particle in them: two
// to three times the candidates.  The fluid is soft and its lower layers
// compress, a particle there has three to eight times the candidates of one at
// rest (44 at the default skin), so the lists take all the room there is
// (alloc_lists).  With room for 96 a step of the 1,048,576-particle obstacle
// scene took 235 us after 500 steps, 636 after 2,000 and 2,131 after 4,000,
// now 236, 451 and 1,708; with one bit mask per row, below, 290, 509 and 1,710
// (there every tenth particle of the fluid has 355 candidates or more).
//
// Why flat lists: with one bit mask per stencil row the lanes of a warp wait
// at every row for the one with most neighbours there (21 of 32 lanes active,
// ~55 gathers for 30 neighbours, each waited for alone); over a flat list
// they wait once, and a group's four gathers are in flight together.
// Batched handles keep one set of flags per scene (field-major: field f of
// scene k at flags[f * numScenes + k]); each scene decides its builds from
// its own particles' displacement and its own h, so a scene in a batch
// builds exactly when it would alone.  The list kernels take a slot's scene
// from slotScene (the .w lane of the sorted position, which carries the
// scene in the batch's other kernels, holds p/rho^2 once a list density
// kernel has run).
constexpr int VL_GROUPS_MIN = 24;        // list groups of a particle: at least (96 candidates) ...
constexpr int VL_GROUPS_MAX = 120;       // ... and at most; alloc_lists chooses
constexpr int VL_GROUPS_SHORT = 8;       // the fewest it falls back to where memory is short
// Above this skin the density stage of a reusing step records which candidates
// lie within h.  1,048,576 particles, force us without and with the masks: skin
// 0.1 105 | 134, 0.2 154 | 137, 0.3 195 | 154, 0.4 202 | 154; with a packing of
// h/2.6 0.1 257 | 302, 0.2 326 | 331.  (Only every second candidate is a
// neighbour from 0.25 on, and a gather that is not made is worth the list
// entries read one by one.)
constexpr float VL_MASK_SKIN = 0.25f;
constexpr int VL_ROWS = 16;              // rows within R <= 1.4 gridSpacing: at most 4 x 4
constexpr unsigned int VL_WINDOWS = 0x80u;  // `groups` of a particle that records windows: this plus their number
static_assert(VL_ROWS <= 2 * VL_GROUPS_SHORT && VL_GROUPS_MAX < (int)VL_WINDOWS, "windows fit the groups");
enum : int {
    VL_BUILD = 0,      // a build is requested (state written, another kind of step ran)
    VL_BUILD_NOW = 1,  // this step's kind, a VL_REUSES ... (decided at the start of the step)
    VL_DISP = 2,       // largest squared displacement since the build (float bits)
    VL_COUNT = 3,      // builds so far
    VL_LAST = 4,       // the kind of the step before, until this step's front is done
    VL_FLAGS = 5,
};
// A step reuses the lists, builds them, or searches without building: when a
// step has moved some particle past the rebuild distance by itself, lists
// built for it were never used, and the steps that follow search as a handle
// without lists does (recording windows of radius h) until one stays within
// the distance again.  VL_NOTHING: a wait of the step's sort gave up (or an
// earlier one's did, still to be reported), and the list kernels do nothing.
enum : unsigned int { VL_REUSES = 0, VL_BUILDS = 1, VL_SEARCHES = 2, VL_NOTHING = 3 };
// Two words after the per-scene flags: whether this step sorts (some scene
// builds; a step that builds nothing keeps the working order and skips the
// hash, scan and scatter), and whether the cell tables on the device are
// older than the last step (it skipped them; sph_read_cells rebuilds them
// from that step's sorted copies).
enum : int { VL_SORT = 0, VL_STALE = 1, VL_GLOBAL = 2 };
struct NeighbourLists {
    int4* list;            // [capacity][n] candidates within R, or two windows [start, end) a group
    int capacity;          // groups allocated
    unsigned char* groups; // [n] groups in use, or VL_WINDOWS + windows in use
    unsigned int* rowMask2; // [9][n] of RowMasks' rows with 33 to 64 places: the bits of the upper half
    unsigned int* masks;   // [(capacity + 7) / 8][n] a reusing step's candidates within h, a bit each, eight
                           //   groups a word; NULL: the force stage tests the candidates itself
    float4* posB;          // [n] positions at the build, working order
    unsigned int* flags;   // [VL_FLAGS][numScenes], then [VL_GLOBAL]
    float radius, radius2; // R and R^2 (single-scene handles; a batch's kernels take each scene's h)
    float dispLimit2;      // (0.45 skin h)^2 (likewise)
    float skinFrac;        // sph_options.neighbourSkin
    int numScenes;         // 1, or the batch's scene count
    int* slotScene;        // batched handles: [n] the scene of each sorted slot (a scene's particles
                           // always fill the same slot range: its cells follow the previous scene's)
};

// What the density stage records for the force stage of the per-step search,
// and of a step that builds the lists (there also rows of 33 to 64 places,
// ROW_TWO_WORDS set in their start: NeighbourLists::rowMask2).
struct RowMasks {
    int* start;          // [9][n] window start, bit 31 set when the row was not masked
    unsigned int* mask;  // [9][n] neighbour bits relative to start, or the window end
};
constexpr int ROW_TWO_WORDS = 0x40000000;  // (a handle's particles are fewer: 2^30 would take 400 GB)

// Launch configuration of the step (chosen per handle; see the autotuner).
enum ForceVariant { FORCE_DIRECT = 0, FORCE_MASK = 1, FORCE_PRETESTED = 2, FORCE_STAGED = 3 };

struct StepConfig {
    int densityBlock = 128;
    int forceBlock = 128;
    int forceVariant = FORCE_PRETESTED;
    int prune = 1;   // row / half-cell window cut (sph_device.cuh)
    int kahan = 1;
};

// Raises a kernel's dynamic shared memory limit once per device (the
// attribute belongs to the current device); K is the kernel itself, so each
// kernel keeps its own record.
template <auto K>
inline void ensure_dynamic_smem(int bytes) {
    static unsigned long long done = 0ull;  // one bit per device ordinal below 64
    int dev = 0;
    cudaGetDevice(&dev);
    const unsigned long long bit = dev < 64 ? 1ull << dev : 0ull;
    if (bit && (done & bit)) return;
    if (cudaFuncSetAttribute(K, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) == cudaSuccess) done |= bit;
}

// The current device's multiprocessor count.
inline int device_sms() {
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return sms > 0 ? sms : 1;
}

// The cell tables are padded: the scan reads and writes whole vectors.
constexpr int SCAN_TILE = 8192;

// ---------------------------------------------------------------------------
// Launch wrappers (sph_kernels.cu)
// ---------------------------------------------------------------------------
void launch_unpack_aos(const float* aos, int stride, int offset, int n, float4* out, cudaStream_t s);
// pos[i].w = scene index `sid` (as integer bits) for i < count.
void launch_set_scene(float4* pos, int count, int sid, cudaStream_t s);
void launch_pack_aos(const float4* in, int n, float* aos, int stride, int offset, cudaStream_t s);
// Cell-relative positions: absolute -> (offset, packed cell) in place, and
// back to absolute (AoS with `stride` floats per particle and/or float4s).
void launch_abs_to_rel(int n, float4* pos, GridDev g, cudaStream_t s);
void launch_rel_to_abs(int n, const float4* pos, GridDev g, float* aos, int stride, float4* out4, cudaStream_t s);
// The front of a step (k_front): hash, scan, scatter, rank and gather of the
// state (pos, vel) into the sorted copies, the permutations and the cell
// tables.  With `lists` the kind of step is decided first, and one that sorts
// nothing only gathers.  Parts of it: `phases`, in this order.
enum : int { FRONT_HASH = 1, FRONT_SUM = 2, FRONT_SCAN = 4, FRONT_SCATTER = 8, FRONT_RANK = 16, FRONT_ALL = 31 };
constexpr int FRONT_MAX_BLOCKS = 4088;
constexpr int FRONT_WORDS = FRONT_MAX_BLOCKS + 8;
void launch_front(int n, const float4* pos, const float4* vel, GridDev g, SortBuffers sb, float4* posS, float4* velS,
                  unsigned int* status, cudaStream_t s, const NeighbourLists* lists = nullptr, int phases = FRONT_ALL);
// The poll limit of device-side waits (a test may shorten it).
int scan_wait_limit();
// `steps` whole plain steps over the reused lists (single scene, absolute
// positions): in one launch after another of several steps each.
bool takes_whole_steps(int n, int numCells);
void launch_steps(int n, float4* pos, float4* vel, GridDev g, SortBuffers sb, RowTables T, float4* posS, float4* velS,
                  float4* rho4S, float4* accS, PhysDev ph, MapDev map, int collide, const NeighbourLists& L, RowMasks M,
                  const StepConfig& cfg, int steps, unsigned int* status, cudaStream_t s);
// The cell tables of the sorted copies' positions (sortedHash, sortedIds,
// cellOffset) after a step that skipped them; the working order, the sorted
// copies and the lists stay as they are.  `scratch`: n float4.
void launch_rebuild_tables(int n, const float4* posS, const int* workIds, const int* slotScene, GridDev g,
                           SortBuffers sb, float4* scratch, unsigned int* status, cudaStream_t s);
// Density stage over reused neighbour lists: the build form (the reference's
// rows and the skin rows, recording the lists, and in M this step's
// neighbours by row) or the list form, as each scene's kind of step asks.
// Besides rho4S, each particle's p/rho^2 and 1/rho go to the fourth lanes of
// its sorted position and velocity, where the list force stage reads them.
void launch_density_lists(int n, float4* posS, float4* velS, RowTables T, GridDev g, PhysDev ph, MapDev map,
                          float4* rho4S, const NeighbourLists& L, RowMasks M, const StepConfig& cfg,
                          cudaStream_t s);
// After a write of the positions: the largest distance from the build
// positions, measured afresh (the lists stay if it is within the limit).
// (Batched handles: each particle's scene from the .w lane of its position.)
void launch_list_displacement(int n, const float4* pos, const int* workIds, const NeighbourLists& L,
                              cudaStream_t s);
// Force stage over the lists, or over M's rows in a step that builds them;
// also records the largest displacement since the build.  With `scenes` (batched handles) each
// particle's constants and maps come from its scene's record.
void launch_force_lists(int n, const float4* posS, const float4* velS, const float4* rho4S, const int* workIds,
                        PhysDev ph, MapDev map, int collide, const NeighbourLists& L, RowMasks M, float4* pos,
                        float4* vel, float4* accS, const StepConfig& cfg, cudaStream_t s,
                        const SceneDev* scenes = nullptr);
// The far record that a list's unused entries name: posS[n], velS[n].
void launch_list_far_record(int n, float4* posS, float4* velS, cudaStream_t s);
void launch_density(int n, const float4* posS, RowTables T, GridDev g, PhysDev ph, MapDev map,
                    float4* rho4S, int* rowStart, unsigned int* rowMask, const StepConfig& cfg,
                    cudaStream_t s);
// Learned-step features recorded by the force stage (24 floats per particle
// at index workIds[i] when byId, else i; see feature_values in sph_step.cu).
struct FeatureOut {
    float* feat;
    int byId;
    int boxWalls;
    float dtL;
};
void launch_force(int n, const float4* posS, const float4* velS, const float4* rho4S,
                  const int* workIds, RowTables T, GridDev g, PhysDev ph, MapDev map, int collide,
                  const int* rowStart, const unsigned int* rowMask, float4* pos, float4* vel,
                  float4* accS, const StepConfig& cfg, cudaStream_t s, const FeatureOut* feat = nullptr,
                  unsigned int* status = nullptr);
void launch_unpermute(int n, const int* sortedIds, const float4* srcS, int comp, float* dst,
                      int stride, int offset, cudaStream_t s);
void launch_cell_tables(int numCells, const int* cellOffset, int* start, int* end, cudaStream_t s);

// Two-scale pass (sph_twoscale.cu).
void launch_ts_states(int n, const float4* posS, const int* workIds, const int* cellOffset, GridDev g, float h,
                      const TwoScaleDev& T, cudaStream_t s);
void launch_ts_children(int n, float4* posS, float4* velS, const float4* accS, const float4* rho4S,
                        const int* workIds, float mass, PhysDev ph, int collide, float4* pos, float4* vel,
                        const TwoScaleDev& T, cudaStream_t s);
void launch_ts_project(const float4* coarsePos, const int* workIds, int byId, const float4* rho4S,
                       const int* cellOffset, GridDev g, float hs, const TwoScaleDev& T, int capacity,
                       cudaStream_t s);
void launch_ts_sub_sort(GridDev sg, const TwoScaleDev& T, SortBuffers subSb, int capacity, unsigned int* status,
                        cudaStream_t s);
void launch_ts_sub_density(GridDev sg, PhysDev sph, const TwoScaleDev& T, int capacity, cudaStream_t s);
void launch_ts_sub_force(GridDev sg, PhysDev sph, const TwoScaleDev& T, int capacity, cudaStream_t s);
void launch_ts_pack_sd(const TwoScaleDev& T, int slots, float* dst, cudaStream_t s);

// FP64 diagnostics (sph_diag.cu): out[DIAG_TERMS] in this order; the maximum
// relative density error is the last term.
enum { DIAG_MASS = 0, DIAG_MOM_X, DIAG_MOM_Y, DIAG_MOM_Z, DIAG_KINETIC, DIAG_POTENTIAL, DIAG_RHO_SUM,
       DIAG_RHO_MAXERR, DIAG_TERMS };
int diag_partial_rows();
void launch_diagnostics(int n, const float4* pos, const float4* vel, const float4* rho4S, int haveRho,
                        double mass, double gravity, double rest0, int axis, double* partial, double* out,
                        cudaStream_t s);

// Boundary maps.
// Builds the maps of `d` (grid solids are uploaded for the build and freed
// after it, synchronising `s`).
cudaError_t launch_build_maps(const sph_boundary_desc& d, const unsigned int dims[3], float* dist,
                              float* dens, float* visc, float4* map4, cudaStream_t s);

}  // namespace sph
