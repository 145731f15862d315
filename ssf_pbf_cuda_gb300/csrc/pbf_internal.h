// Internal interfaces between the host runtime (pbf_engine.cu) and the
// device kernels (pbf_kernels.cu).  Not part of the C ABI.
#pragma once
#include <cstdint>
#include <cstddef>
#include <cuda_runtime.h>
#include <nvtx3/nvToolsExt.h>

namespace pbf103 {

// A named NVTX range on the calling host thread for the life of the object
// (the host runtime's stages show up on a profiler's timeline; with no
// profiler attached a range costs a function-pointer test).
struct NvtxRange {
    explicit NvtxRange(const char *name) { nvtxRangePushA(name); }
    ~NvtxRange() { nvtxRangePop(); }
    NvtxRange(const NvtxRange &) = delete;
    NvtxRange &operator=(const NvtxRange &) = delete;
};

// Per-scene constants, one 240-byte record per scene slot in device memory.
// Derived once on the host from pbf_params (the reference keeps these in
// __constant__ symbols and a function-static, pbf_position_update.cu:14-17,
// pbf_solve.cpp:92; here they are per scene so scenes never share state).
struct SceneDesc {
    uint32_t p_off;      // first particle slot of the scene in the flat arrays
    uint32_t capacity;   // particle slots owned by the scene
    uint32_t c_off;      // first cell of the scene in the flat cell arrays
    uint32_t ncell;      // Gx*Gy*Gz; cell ncell (local) is the deleted bucket
    uint32_t gx, gy, gz; // power-of-two hash grid
    uint32_t cap;        // neighbour slots usable (max_pair - 1)
    float cw;            // cell width
    float h2;            // h*h, neighbour acceptance
    float inv_h;         // 1/h
    float alpha;         // poly6 factor 1.56668147065 / h^3
    float beta;          // spiky-derivative factor -14.3239448745 / h^4
    float m;             // particle mass
    float inv_rho0;      // 1 / rest density
    float m2rho2;        // m^2 / rho0^2
    float relax;         // CFM epsilon
    float dt;
    float inv_dt;
    float inv_k;         // reference s_corr: 1 / W(0.4h)^4
    float inv_wdq;       // textbook s_corr: 1 / W(dq h)
    float scorr_k;
    int32_t scorr_n;
    int32_t tensile_mode;
    int32_t xsph_mode;
    int32_t vort_mode;
    float xsph_c;
    float vort_eps;
    float alpha6;        // 1.56668147065 * inv_h * inv_h * inv_h (Wpoly6 order)
    float h;
    float g[3];
    uint32_t max_coll;
    float amin[3];
    uint32_t b_off;      // first float4 of the scene's boundary primitives
    float amax[3];
    uint32_t n_inner;
    uint32_t n_outer;
    uint32_t n_planes;
    uint32_t builtin_sphere;
    float ih2;           // 1/h^2 (poly6 from r^2)
    // the pair passes sum W / alpha = t^3 and grad W / beta = s' d (t = 1 -
    // r^2/h^2, s' = (1 - r/h)^2 / r) and apply alpha and beta once per
    // particle, through these products (each computed in double):
    float tens_c;        // reference s_corr: 10 alpha^4 / W(0.4h)^4, the factor of (t^3)^4
    float scorr_c;       // textbook s_corr: k alpha^n / W(dq h)^n, the factor of (t^3)^n
    uint32_t list16;     // the neighbour list holds u16 scene-local indices (capacity <= 65,536)
    // clear_box: the boundary is planes with unit-axis normals only; a
    // projected position p with box_lo <= p <= box_hi hits none of them
    uint32_t clear_box;
    float box_lo[3], box_hi[3];
    float lam_c;         // alpha m / rho0: C = lam_c sum t^3 - 1
    float lam_k;         // m^2 beta^2 / rho0^2: the factor of |sum s' d|^2 + sum (s' r)^2
    float dp_k;          // m beta / rho0: delta-p = dp_k sum coef s' d
    uint32_t pad_[1];
};
static_assert(sizeof(SceneDesc) % 16 == 0, "SceneDesc must stay 16-byte sized");

// Device-resident launch control; lets a captured graph run on a scene set
// that changes between launches.
struct Ctrl {
    uint32_t n_tiles;       // particle tiles at the front of tile_scene/tile_start
    uint32_t n_cells;       // cell entries to scan (high-water mark of cell ranges)
    uint32_t n_scenes;
    uint32_t n_cell_tiles;  // cell tiles after them: LaunchShape::cell_tile cells of one scene each
};

// Device-resident pointers to a step's packed AoS float3 input
// (pbf_batch_step_packed): set by a one-thread kernel before each such step,
// so a captured graph reads whichever buffers the call names.
struct PackedIn {
    const float *x, *v;  // v may be null (zero velocities)
};

struct StepArgs {
    const SceneDesc *scenes;
    const uint32_t *tile_scene;   // tile -> scene
    const uint32_t *tile_start;   // tile -> first local particle index (cell tiles: first local cell)
    const Ctrl *ctrl;
    uint32_t *scene_num;          // particles per scene at step start
    uint32_t *flags;              // per-scene PBF_FLAG_* words
    float4 *x, *v;                // particle phase (sorted after each step)
    float4 *xs;                   // predicted positions, input order
    uint32_t *key, *slot, *tmp, *perm;
    uint32_t *count, *offsets, *bsum;
    // working slots: sorted slots, with a bucket of several alias classes grouped by class
    float4 *xa, *xb, *xold;       // working positions, (position, lambda), old x (.w = sorted slot)
    uint32_t *nbr;                // neighbour lists, in rows of 16 bytes per working slot
    uint8_t *nnb;                 // list entries stored (the particle itself is not stored)
    uint8_t *selfat;              // position of the particle itself in its walk-order list, kNotListed if cut
    float4 *w;                    // vorticity
    float4 *pa;                   // (x, y, z, vx) and (vy, vz) between the list-form post passes, working slots
    float2 *pb;
    float4 *vs;                   // velocity between the walk-form post passes, sorted slots
    const float4 *bnd;            // boundary primitives
    uint32_t *id, *id_tmp;        // particle ids (phase order) and their copy in working order
    uint8_t *cls;                 // alias class of each particle (input order)
    uint32_t *wpos;               // sorted slot -> working slot
    uint32_t *dense;              // [0] count, then (cell, scene) pairs of buckets for k_dense_sort
    uint32_t *mid;                // the same for buckets of kMidMin+1 .. kDenseMin members
    uint64_t *chist;              // per cell: 8 x 8-bit class ends of its bucket, or kClassWhole
    uint32_t *next_id;            // per scene: id of the next particle added
    uint64_t nbr_stride;
    uint32_t nbr_rows;            // 16-byte rows a list has
    uint4 *tile_hdr;              // small steps: the tiles' headers (SMALL_LOOP_BEGIN)
    const PackedIn *pin;          // packed-input steps: the input buffers
    const uint32_t *pack_off;     // packed-input steps: first packed particle of each scene
};

struct LaunchShape {
    uint32_t tile;        // particles per tile = threads per block
    uint32_t grid;        // persistent grid (blocks) for the light tile kernels
    uint32_t scan_grid;   // grid for the three scan kernels; 0 = one kernel
    uint32_t scan_cluster; // one kernel: blocks of its cluster, 0 = one block
    uint32_t scan_rounds; // one kernel: rounds of 1024 cells a block holds in registers
    uint32_t chunk;       // neighbours per chunk in the large steps' lambda pass (4 or 8)
    // persistent grids of the heavy kernels, each from its own occupancy
    uint32_t grid_nb, grid_lambda, grid_dp;
    uint32_t grid_omega[2], grid_apply[2], grid_xsph[2];  // list-form post passes: u32 lists, u16 lists
    uint32_t grid_cells;  // grid of k_rank_cells: a block of cell_tile threads per cell tile
    uint32_t cell_tile;   // cells per cell tile = threads per k_rank_cells block (autotuned)
    uint32_t rank_each;   // few particle slots (at most kSmallStep): per-particle rank
    uint32_t small;       // latency-bound step (as few): walk by shared ranges, wide list reads
    uint32_t front;       // small steps: k_front's rounds of 1024 cells a block, 0 = a kernel per phase
    uint32_t front_cluster; // blocks of its cluster
    uint32_t tile_shift;  // log2 of tile
    uint32_t small_split; // small steps: their walk takes kSplit lanes a particle (k_neighbors_split)
    uint32_t small_lanes; // small steps: their list passes take kLanes lanes a particle
    uint32_t small_tiles; // small steps: tiles rounded up to a power of two, for which headers are written
    uint32_t nb_smem;     // the walk's bytes of shared memory for the block's lists (large steps: 0 = stored directly)
    bool operator==(const LaunchShape &o) const
    {
        return tile == o.tile && grid == o.grid && scan_grid == o.scan_grid && scan_rounds == o.scan_rounds && scan_cluster == o.scan_cluster &&
               chunk == o.chunk &&
               grid_cells == o.grid_cells && cell_tile == o.cell_tile && rank_each == o.rank_each && small == o.small && small_tiles == o.small_tiles && small_split == o.small_split && small_lanes == o.small_lanes && nb_smem == o.nb_smem &&
               front == o.front && front_cluster == o.front_cluster &&
               grid_nb == o.grid_nb && grid_lambda == o.grid_lambda && grid_dp == o.grid_dp &&
               grid_omega[0] == o.grid_omega[0] && grid_omega[1] == o.grid_omega[1] && grid_apply[0] == o.grid_apply[0] &&
               grid_apply[1] == o.grid_apply[1] && grid_xsph[0] == o.grid_xsph[0] && grid_xsph[1] == o.grid_xsph[1];
    }
};

// Resident blocks per SM of each kernel class at a tile size / chunk.
struct Occupancy {
    uint32_t light, nb, lambda, dp, cells;
    uint32_t omega[2], apply[2], xsph[2];
};
Occupancy occupancy(uint32_t tile, uint32_t chunk);
uint32_t scan_cluster_limit();  // blocks the scan's cluster may have on the current device

// Called after every kernel launch of a step (per-kernel event timing).
struct StepHook {
    virtual void launched(const char *kernel_name) = 0;
    virtual ~StepHook() = default;
};

// Post-solve passes a step runs (bit set: some active scene needs that form).
enum : uint32_t {
    kPostXsphWalk = 1,       // XSPH, the reference's uncapped 27-cell walk
    kPostXsphList = 2,       // XSPH over the step's neighbour list
    kPostVortReference = 4,  // vorticity, the reference's walk and kernel scaling
    kPostVortTextbook = 8,   // vorticity, textbook form over the neighbour list
    kPostList32 = 16,        // some scene keeps a u32 neighbour list (list forms launch per list format)
    kPostList16 = 32,        // some scene keeps a u16 neighbour list
};

// Enqueue one full solver step for every scene in the tile list.
// Returns the number of kernels launched.
// packed: the step reads its input positions and velocities from the packed
// AoS float3 buffers named in *a.pin (scene s from a.pack_off[s]) instead of
// the particle phase, and numbers the particles afresh, as an upload does.
uint32_t enqueue_step(const StepArgs &a, const LaunchShape &s, int iters, uint32_t post_modes,
                      cudaStream_t stream, StepHook *hook = nullptr, bool packed = false);
void launch_set_packed_in(PackedIn *dst, const float *x, const float *v, cudaStream_t st);

// Edge conversions between the ABI's AoS float3 and the internal float4.
void launch_aos3_to_f4(const float *src, float4 *dst, uint32_t n, cudaStream_t st);
// A scene's upload: n particles widened at x, v and numbered (append: from
// *next_id on, which the caller then bumps), *scene_num = total.
void launch_load_phase(const float *sx, const float *sv, float4 *x, float4 *v, uint32_t *id, uint32_t *next_id,
                       uint32_t *scene_num, uint32_t n, uint32_t total, bool append, cudaStream_t st);
void launch_store_phase(const float4 *x, const float4 *v, float *dx, float *dv, uint32_t n, cudaStream_t st,
                        const uint32_t *num = nullptr, uint32_t *num_out = nullptr);
void launch_set_u32(uint32_t *dst, uint32_t value, cudaStream_t st);
// pack_off[active[k]] = sum of the live counts of active[0..k), counts[k] =
// the live count of active[k], computed on the device (one block)
void launch_pack_offsets(const uint32_t *active, uint32_t n_active, const uint32_t *scene_num, uint32_t *pack_off,
                         uint32_t *counts, cudaStream_t st);
// *next_id += n (an append's ids are handed out)
void launch_bump_next_id(uint32_t *next_id, uint32_t n, cudaStream_t st);
// Whole-batch moves between a packed AoS float3 buffer (active scenes in
// slot order, pack_off[s] = first packed particle of scene s) and the
// scene-sliced float4 phase arrays.  unpack uses the tile list (counts must
// already be in scene_num); pack writes the scene_num[s] first particles.
void launch_unpack(const StepArgs &a, const LaunchShape &sh, const uint32_t *pack_off, const float *src_x,
                   const float *src_v, cudaStream_t st);
void launch_pack(const StepArgs &a, const LaunchShape &sh, const uint32_t *pack_off, float *dst_x, float *dst_v,
                 cudaStream_t st);

// chist value of a bucket in plain sorted order, walked whole (more than 254
// members, or a table of fewer than 4 cells on an axis)
constexpr uint64_t kClassWhole = ~0ull;

constexpr uint32_t kScanItemsPerWarp = 512;   // 32 lanes x 16
constexpr uint32_t kScanWarps = 8;
constexpr uint32_t kScanTile = kScanItemsPerWarp * kScanWarps;  // 4096 cells per scan tile
constexpr uint32_t kBlockScanMax = 8192;      // cells up to which one block scans the whole table
constexpr uint32_t kScanClusterMax = 16;      // blocks of the scan's cluster (1024 threads each)
constexpr uint32_t kScanRoundsMax = 18;       // cells a thread of it may hold: tables are 2^k + 1 cells, up to 2^18 + 1
constexpr uint32_t kNbSmemMax = 96 * 1024;  // shared-memory budget for a k_neighbors_lambda block's lists
// Particle slots up to which a step is bound by latency rather than throughput:
// the small steps' list passes fit one wave (8 blocks of 64 on 152 SMs).  At 65,000
// particles they take 114 us a step and the large steps' 138, at 80,000 (two
// waves) 158 and 145.
constexpr uint32_t kSmallStep = 77824;
constexpr uint32_t kSmallBlock = 64;        // particles of a block of the small steps' list passes
constexpr uint32_t kSmallTiles = 2048;      // tiles a small step may have, rounded up to a power of two
static_assert(kSmallTiles >= kSmallStep / 64, "a header per tile of a small step");
// shared memory of their walk beside the lists: per warp 27 ranges of up to 32 cells and the cells' coordinates
constexpr uint32_t kSmallWalkSmem = kSmallBlock / 32 * (32 * 27 * 8 + 96 * 4);
constexpr uint64_t kFrontSlots = 1u << 29;  // k_front: particle slots at most (indices beside an alias class)
constexpr uint32_t kFrontRounds = 4;        // k_front: rounds of 1024 cells a block at most (1, 2 or 4)
constexpr uint32_t kSplit = 4;              // lanes a particle in the smallest steps' walk
constexpr uint32_t kSplitBlock = kSplit * kSmallBlock;
// Particle slots up to which the walk is split: 15,000 particles 76 us a step
// against 78 with one lane a particle, 20,000 84 against 80 (10,648 at h = 1.4
// spacings 47 against 51).
constexpr uint32_t kSplitStep = 16384;
// Lanes a particle in the smallest steps' list passes: up to kLanesLong slots
// where lists are long (more than the 16 slots a lane takes at once, by the
// neighbours expected within h at rest density), and with short ones between
// more blocks of kSmallBlock particles than SMs and kLanesStep slots.  A step
// in us, two lanes against one:
//   h = 2 spacings    500: 52, 57  4,096: 58, 62  8,192: 60, 66  16,384: 70, 76  24,000: 80, 82  32,768: 105, 87
//   h = 1.4 spacings  500: 41, 40  4,096: 45, 45  8,192: 46, 45  10,648: 49.5, 51.5  16,384: 54, 56  20,000: 62, 60
// (four lanes: 55 at 4,096 and 70 at 12,000 against 66).
constexpr uint32_t kLanes = 2;
constexpr uint32_t kLanesStep = 16384, kLanesLong = 24576;
constexpr uint32_t kCellTile = 256;         // default cells per cell tile = threads per k_rank_cells block
constexpr uint32_t kCellTileMin = 64, kCellTileMax = 512;  // the autotuner's range
constexpr uint32_t kMidMin = 16;            // buckets with more members are queued (warp or block per bucket)
constexpr uint32_t kList16Max = 65536;      // scenes of at most this many slots keep u16 neighbour lists
constexpr uint8_t kNotListed = 0xFF;        // selfat of a particle the cap cut from its own list
constexpr uint32_t kWalkSpare = 8;          // spare float4 records after each per-particle array

}  // namespace pbf103
