// sph.cuh -- the gather kernels of one two-scale WCSPH step.
#pragma once
#include "grid.cuh"
#include "tss_device.cuh"

namespace tss {

// One scale's arrays.  "cur" arrays are in this step's (cell, id) order, "list"
// arrays (n*) hold the state the next step starts from, in that same order for
// existing particles, with newly created high-res children appended.
struct ScaleView {
    const float2* pos;
    // velocity (.xy, written by the grid build), p / rho^2 (.z) and rho (.w, both written
    // by the density pass): with pos, what a force pair needs of a neighbour, in one
    // 16-byte load.  As four arrays (and a state byte for every pair) the force kernels
    // waited on five loads a neighbour instead of two.
    float4* vq;
    const uint8_t* st;
    const int32_t* id;
    float* dens;
    float* pres;
    float* tr;       // low scale: each split parent's tether radius, written by the low-res force
    // low scale, one byte per cell: the low-res force sets a cell to the step counter
    // (mod 256) when the cell holds an entry in state 0 after the split marks.  Any
    // other value only makes the high-res force walk a row it could skip.
    uint8_t* cflag;
    // Neighbour lists the density pass records for the force pass of the same scale:
    // entry c of sorted particle i is
    // nbr[c * nbr_stride + i] = j - i for its c-th same-scale neighbour within the
    // density's support (itself left out), in window order; nnbr[i] is their count;
    // kNbrCrowd when there are more than kMaxNbr (the first kMaxNbr are listed); or
    // kNbrOverflow when an offset does not fit 16 bits (none are).
    int16_t* nbr;
    uint8_t* nnbr;
    long long nbr_stride;  // entries per list column: the scale's capacity
    float2* acc;     // the accelerations; until the force, a short list's wall terms (wall_scale)
    const int* off;  // dense cell offsets [C+1]
    int32_t* map;    // slot id -> index in the cur arrays
    float2* npos;
    float2* nvel;
    uint8_t* nst;
    int32_t* nid;
    float* ndens;    // carried densities/pressures (relaxation only; may be null)
    float* npres;
    // the next step's grid keys, written where the list entries are written
    unsigned* gcount;
    int* gkey;
    int* grank;
    unsigned* gtile;
};

struct StepView {
    ScaleView L, H;
    const float2* wpos;     // walls: each scene's in (low cell, id) order from its wall base
    const int* woff;        // wall cell offsets on the low grid
    const uint8_t* wnear;   // per low cell: 1 when a cell within two cells of it holds a wall particle
    Counters* cnt;
    uint8_t* split_flag;    // [n_low]
    int32_t* split_ids;     // [n_low] parents split this step (= next step's fresh list)
    unsigned* split_tile;   // [ceil(n_low / kSplitTile)] splits per tile: cleared by the low-res density, counted by the force
    float2* relax_pos;      // [capH] relaxation scratch
    float2* relax_vel;
    int nL;                 // low-res count (constant for a solver)
    int wallL, wallH;       // the low-res density's last blocks: the two lists' wall terms
    // batches only: per-scene parameters and each sorted particle's scene
    const Params* table;
    const uint16_t* scL;
    const uint16_t* scH;
};

// The longest list.  A split parent's four children end up close together, so high-res
// lists are 3 + 4 per neighbouring clump long: on a dam break of 1.0M high-res
// particles 0.27 % of them have more than 20 neighbours, but 8 % of the warps hold one
// and walk again (high-res density and force 93 and 151 us), and 0.005 % more than 24
// (82 and 138 us; 28: 78 and 133).  24 is what fits without the handle's memory
// growing: a grid build borrows the lists for its permutation (12 bytes an entry).
constexpr int kMaxNbr = 24;
constexpr uint8_t kNbrOverflow = 255, kNbrCrowd = 254;

// Short lists: one particle per thread leaves most of the GPU idle and a step waits
// for each thread's chain of loads and pairs.  A list of at most so many particles is
// taken by groups of 8 or 4 lanes a particle (gather.cuh), whatever its capacity: the
// kernels choose by the count on the device.  Stage times in us (n low-res and about
// as many high-res particles; exact arithmetic; one thread / 4 / 8 / 16 lanes):
//   n          1,500              10,000             22,000             48,000
//   low force  24 / 16 / 14 / 12  24 / 17 / 14 / 14  24 / 18 / 16 / 20  24 / 18 / 24 / 30
//   high force 31 / 21 / 16 / 15  28 / 20 / 17 / 18  28 / 21 / 19 / 25  33 / 26 / 29 / 38
//   low dens.  11 / 11 / 11 / 9   11 / 13 / 11 / 11  12 / 13 / 14 / 17  13 / 17 / 21 / 25
//   high dens. 12 / 11 / 10 / 8   12 / 12 / 10 / 12  12 / 13 / 14 / 16  17 / 17 / 20 / 26
// A density search is short and its groups do more work than its threads (the two run
// as parallel branches), so it returns to one thread earlier than a force does.  The limits
// lie inside that sweep, which has no size between those shown and was taken in the exact
// arithmetic alone: 8 lanes are still a little ahead of 4 at 22,000, and 4 lanes ahead of
// one thread at 48,000, its last size.
constexpr int kDensity8Max = 12000;
constexpr int kForce8Max = 20000, kForce4Max = 48000;

constexpr int kSplitThreads = 256;
constexpr int kSplitItems = 16;
constexpr int kSplitTile = kSplitThreads * kSplitItems;

// B = false: one scene, parameters P0 (kernel constants).  B = true: a batch of
// scenes; each particle's parameters are V.table[scene of the particle], and each
// scene's grids sit at its cell bases in one global cell space.  The gathers
// (densities, forces) are further templated on how a particle's window is walked
// (gather.cuh) and launched through the launchers below.
template <bool B> __global__ void k_split(Params P0, StepView V);
template <bool B> __global__ void k_relax_density(Params P0, StepView V);
template <bool B> __global__ void k_relax_force(Params P0, StepView V);
__global__ void k_relax_apply(Params P0, StepView V);
__global__ void k_step_finish(Counters* c);

// host launchers (batched selects B; warp: one particle per warp instead of per
// thread; fast: FastArith instead of ExactArith, arith.cuh).  Gather g: 0 high-res
// density, 1 low-res density, 2 low-res force, 3 high-res force.
void launch_gather(int g, bool batched, bool warp, bool fast, int blocks, int threads, cudaStream_t s,
                   const Params& P, const StepView& V);
void launch_k_split(bool batched, int blocks, int threads, cudaStream_t s, const Params& P, const StepView& V);
// one relaxation sub-step: density, force, apply
cudaError_t launch_relax(bool batched, int blocks, int threads, cudaStream_t s, const Params& P, const StepView& V);
// resident blocks per SM of gather g at `threads` threads per block; 0 on error
int gather_occupancy(int g, bool batched, bool warp, bool fast, int threads);
// wnear of one scene's dimx x dimy low grid from its wall cell offsets (both
// pointers at the scene's first cell), after its wall grid is built
void launch_wall_near(const int* woff, uint8_t* wnear, int dimx, int dimy, cudaStream_t s);

}  // namespace tss
