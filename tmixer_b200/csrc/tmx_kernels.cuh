// tmx_kernels.cuh -- launch declarations of the kernels in tmx_kernels.cu
// (FP64 form, reductions) and tmx_kernels_lp.cu (FP32 / FP16-storage forms).
// Population, density and inlet-profile buffers are typed by the form
// (double / float / __half storage; double / float arithmetic), hence void*.
#pragma once
#include "tmx_device.cuh"

namespace tmx {

// Buffers of one step (populations in/out, boundary densities previous/this
// step, macroscopic fields, FP16-form moments previous/this step, inlet
// profiles); the kernels cast to the form's types.
struct StepPtrs {
    const void* pin;
    void* pout;
    const void* rprev;
    void* rcur;
    double* mac;
    const float4* mprev;
    float4* mcur;
    const void* uin1;
    const void* uin2;
};

constexpr int kBoundaryThreadsHost = 128;  // block size of the boundary kernels
constexpr int kBoundaryLanesHost = 4;      // threads per boundary node (one per field)
// A batched boundary block takes kListAlign consecutive list entries at a
// time; the batch pads each mixer's part of a list to a multiple of it.
constexpr int kListAlign = kBoundaryThreadsHost / kBoundaryLanesHost;

#define TMX_DECLARE_INIT_KERNEL(NAME) __global__ void k_init_##NAME(StepPtrs X, Geom G, Phys P, double rho0);
#define TMX_DECLARE_STEP_KERNELS(NAME)                                                                          \
    TMX_DECLARE_INIT_KERNEL(NAME)                                                                               \
    __global__ void k_bulk_##NAME(StepPtrs X, Geom G, Phys P, int write_macro);
#define TMX_DECLARE_BOUNDARY_KERNELS(NAME)                                                                      \
    __global__ void k_bfaces_##NAME(StepPtrs X, const int* bnode, const unsigned char* bcls, int nb, Geom G,    \
                                    Phys P, int write_macro);                                                   \
    __global__ void k_bedges_##NAME(StepPtrs X, const int* bnode, const unsigned char* bcls, int nb, Geom G,    \
                                    Phys P, int write_macro);

TMX_DECLARE_INIT_KERNEL(f64)
TMX_DECLARE_INIT_KERNEL(f32)
TMX_DECLARE_STEP_KERNELS(f16)
TMX_DECLARE_BOUNDARY_KERNELS(f16)

// Runs of the FP64 and FP32 steps (tmx_run64.cuh, tmx_run32.cuh): {first node, nodes | kind << 9 |
// box << 12 | iface << 13, x of the first node, mixer}, up to
// NT consecutive nodes of one plane of a box, NT the kernel's threads (128 or
// 256; run_threads in tmx_host.h).  iface: the row whose ey = 1 (1) or ey = -1
// (2) sources lie in the other box.
enum RunKind { kRunRows = 0, kRunZ1, kRunZT, kRunYT, kRunY1 };
constexpr int run32_smem_host(int nt) { return 19 * (nt + 2) * 16 + nt / 32 * 400 + 544; }  // RunShared32
constexpr int run_smem_host(int nt) { return 2 * 19 * (nt + 4) * 8 + nt / 32 * 800 + 400; }  // RunShared
// The runs, and the edge and corner nodes enode[0..ne); counters[parity] hands
// out the runs, counters[1 - parity] is cleared for the next step.
#define TMX_DECLARE_RUN(NT, NAME)                                                                               \
    __global__ void k_run##NT##_##NAME(const __grid_constant__ StepPtrs X, const __grid_constant__ Geom G,         \
                                    const __grid_constant__ Phys P, int write_macro, const int4* runs,          \
                                    int nruns, const int* enode, const unsigned char* ecls, int ne,             \
                                    int* counters, int parity, int* error);
TMX_DECLARE_RUN(128, f64)
TMX_DECLARE_RUN(256, f64)
TMX_DECLARE_RUN(128, f32)

// Mixers that a batch can hold: a tile's entry has 22 bits for the mixer's slot
// (the boundary lists' mixer * 256 + class 23, a run's 31).  As many of the
// smallest mixers that the FP16 form can have take 247 GB.
constexpr int kMaxMixers = 1 << 22;

// One mixer of a batch: its buffers for either parity of the batch's step
// counter, its geometry and its physics constants (device memory, read by
// the batched kernels).
struct MixerDesc {
    StepPtrs X[2];
    Geom G;
    Phys P;
};

// Batched step kernels: one launch covers every mixer of a batch.
//   bulk    a persistent grid walks a list of cell blocks {mixer, first
//           node, node count, 0}; NT threads per block (128, 256 or 512).
//   faces / edges   boundary-node lists of {node, mixer * 256 + class}, 
//           four threads per node, persistent grid; each mixer's part
//           starts at a multiple of kListAlign, padded with node -1.
// counts[0..4] = number of cell blocks, face nodes, edge nodes, sweep tiles,
// runs (device memory, so that captured graphs stay valid when the batch
// changes); counts[5..6] hand out the runs or tiles of a step of either parity,
// each cleared by the step before.
#define TMX_DECLARE_BATCH_KERNELS(NAME)                                                                           \
    __global__ void k_bulk_batch128_##NAME(const MixerDesc* D, const int4* blocks, const int* counts, int parity, \
                                           int write_macro);                                                      \
    __global__ void k_bulk_batch256_##NAME(const MixerDesc* D, const int4* blocks, const int* counts, int parity, \
                                           int write_macro);                                                      \
    __global__ void k_bulk_batch512_##NAME(const MixerDesc* D, const int4* blocks, const int* counts, int parity, \
                                           int write_macro);                                                      \
    __global__ void k_bfaces_batch_##NAME(const MixerDesc* D, const int2* list, const int* counts, int parity,    \
                                          int write_macro);                                                       \
    __global__ void k_bedges_batch_##NAME(const MixerDesc* D, const int2* list, const int* counts, int parity,    \
                                          int write_macro);

constexpr int kCounts = 7;
// The FP64 and FP32 forms' batched steps (runs as k_run128_*'s, of every mixer).
constexpr int kRunBatchThreads = 128;
__global__ void k_run_batch_f64(const MixerDesc* D, const int4* runs, const int2* edges, int* counts, int parity,
                                int write_macro, int what, int* error);
__global__ void k_run_batch_f32(const MixerDesc* D, const int4* runs, const int2* edges, int* counts, int parity,
                                int write_macro, int what, int* error);
TMX_DECLARE_BATCH_KERNELS(f16)

// The FP16 form's interior by tiles of 32 TY nodes of a plane swept through z
// (tmx_engine.cuh sweep_tile): tiles[t] = {mixer * 2 + box | planes << 23, x0,
// y0 | s << 29, z0}; the single-mixer kernels take mixer 0, the batched ones read
// the tile count from counts[3] and hand the tiles out by counts[5 + parity].
// Dynamic shared memory: sweep_smem_host.
// A tile is w = 32 >> s columns wide.  In tiles with groups (s = 0, 1 or 2) a warp's
// lanes are 1 << s groups of w, group c TY rows above group c - 1, side by side in
// shared memory with a halo each (rows of sweep_pitch records), so that boxes narrower
// than 32 columns, and what is left of wider ones, fill the lanes.  Their code costs
// every tile a little: a batch takes them where they save a tenth of its tiles or
// more (8 mixers of 544,000 nodes in boxes 16 to 192 columns wide, 13% fewer: 86.7 ->
// 79.8 us; 64 of 41M nodes, 3% fewer: 3.56 -> 3.58 ms), a single mixer never
// (221,184 nodes, 14% fewer: 27.8 -> 28.6 us; 4.2M, none: 318 -> 336 us).
__host__ __device__ constexpr int sweep_pitch(bool groups) { return groups ? 40 : 34; }
// The end of a tile's columns: w on, but never the box's last column alone (an
// x wall's species come from its neighbour in the same group).
__host__ __device__ constexpr int sweep_end(int x0, int nx, int w)
{
    return x0 + w >= nx ? nx : (x0 + w == nx - 1 ? x0 + w - 1 : x0 + w);
}
// A lane's place in its warp's row of a tile: column and row from the tile's
// first, and its record's column in shared memory, less the halo's one.
struct SweepLane {
    int x, y, col;
};
__host__ __device__ constexpr SweepLane sweep_lane(int s, int lane, int warp, int ty)
{
    const int c = lane >> (5 - s);
    return SweepLane{lane & ((32 >> s) - 1), warp + c * ty, lane + 2 * c};
}
// The place of record column col of a row of shared memory: column from the tile's
// first, and group (1 << s or more: unused).
__host__ __device__ constexpr int sweep_group(int s, int col)
{
    const int p = (32 >> s) + 2;
    return (col >= p) + (col >= 2 * p) + (col >= 3 * p);
}
__host__ __device__ constexpr int sweep_column(int s, int col) { return col - sweep_group(s, col) * ((32 >> s) + 2) - 1; }
constexpr int kSweepWalls = 256;  // wall row entries that a batch's block takes at a time
#define TMX_DECLARE_SWEEP(SUFFIX)                                                                               \
    __global__ void k_sweep##SUFFIX##_f16(StepPtrs X, Geom G, Phys P, int write_macro, const int4* tiles,     \
                                          int ntiles);                                                         \
    __global__ void k_sweepw##SUFFIX##_f16(const __grid_constant__ StepPtrs X, const __grid_constant__ Geom G, \
                                          const __grid_constant__ Phys P, int write_macro, const int4* tiles,  \
                                          int ntiles, const int* bnode, const unsigned char* bcls, int nw,     \
                                          int e0, int ne);
#define TMX_DECLARE_SWEEP_BATCH(SUFFIX)                                                                       \
    __global__ void k_sweep_batch##SUFFIX##_f16(const MixerDesc* D, const int4* tiles, const int2* walls,     \
                                                int* counts, int parity, int write_macro);
TMX_DECLARE_SWEEP(8)
TMX_DECLARE_SWEEP_BATCH(8)
TMX_DECLARE_SWEEP_BATCH(4)
TMX_DECLARE_SWEEP_BATCH(8g)
TMX_DECLARE_SWEEP_BATCH(4g)
TMX_DECLARE_SWEEP(4)
constexpr int sweep_smem_host(int ty, bool groups) { return 2 * 4 * (ty + 2) * sweep_pitch(groups) * 16; }

// Threads per species of the row kernels (blocks of 3 kRowPart; the pressure and
// power kernel has kRowPart).
constexpr int kRowPart = 128;

// Outlet mixing quality of batch mixers: for entry e, mixer slots[e], the
// I_A, I_B, I_C of mixing row 1 (the first row of tmx_mixing) into
// out[3e..3e+2], with the arithmetic of k_mixing_rows and its finish.
__global__ void k_outlet_im_batch(const MixerDesc* D, const int* slots, int n, double* out);

// Health of batch mixers: flags[m] |= 1 for every mixer m with a non-finite
// macroscopic value (density, velocity or concentration) in the last fields
// written, over the batch's cell-block list (counts[0] blocks).
__global__ void k_nonfinite_batch(const MixerDesc* D, const int4* blocks, const int* counts, int* flags);

// One field of a box (src: its first node, x fastest) in [i][j][k] order.
__global__ void k_box_ijk(const double* src, int nx, int ny, int nz, double* dst);

__global__ void k_mixing_rows(const double* __restrict__ Mac, Geom G, double* __restrict__ stats);
__global__ void k_sums(const double* __restrict__ Mac, Geom G, double* __restrict__ partial);
// The inlet duct series of the reduced-precision forms, computed on the device.
__global__ void k_inlet_series(int iny, int nz, double* __restrict__ raw);
// Pressure and specific power of one mixer (layout of out: tmx_kernels.cu).
__global__ void k_pressure_power(const double* __restrict__ Mac, Geom G, double tau, double* __restrict__ out);

// Fixed scratch of tmx_mixing_static: kMixStaticRows rows of 9 statistics
// followed by kMixStaticRows finished rows of 7 numbers (512 KiB per device).
constexpr int kMixStaticRows = 4096;
__global__ void k_mixing_finish(const double* __restrict__ stats, Geom G, double* __restrict__ rows);
// Device address of that scratch on the current device.
cudaError_t mixing_static_scratch(double** ptr);

}  // namespace tmx
