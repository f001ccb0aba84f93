// tmx_host.h -- host-side pieces shared by the single-mixer handle
// (tmx_api.cu) and the batched engine (tmx_batch.cu): error reporting, the
// kernel table of each precision form, and the translation of a tmx_case
// into device geometry, physics constants, boundary lists and inlet
// profiles.
#pragma once
#include <cuda_runtime.h>

#include <algorithm>
#include <vector>

#include "../../include/tmx.h"
#include "tmx_kernels.cuh"

namespace tmx_host {

using tmx::Geom;
using tmx::Phys;

// Record the error text of the calling thread (returned by tmx_last_error)
// and return code.
int fail(int code, const char* fmt, ...);
const char* last_error();

#define TMX_CK(call)                                                                                    \
    do {                                                                                                \
        cudaError_t e_ = (call);                                                                        \
        if (e_ != cudaSuccess)                                                                          \
            return ::tmx_host::fail(TMX_E_CUDA, "%s: %s (%s:%d)", #call, cudaGetErrorString(e_), __FILE__, \
                                    __LINE__);                                                          \
    } while (0)

// the step kernels of one form
struct StepKernels {
    void (*init)(tmx::StepPtrs, Geom, Phys, double);
    void (*bulk)(tmx::StepPtrs, Geom, Phys, int);
    // the face and edge lists as two launches (forms whose bulk runs beside them)
    void (*faces)(tmx::StepPtrs, const int*, const unsigned char*, int, Geom, Phys, int);
    void (*edges)(tmx::StepPtrs, const int*, const unsigned char*, int, Geom, Phys, int);
    // the whole step in one launch, by runs of up to 128 or 256 nodes (FP64 and
    // FP32; the pointers above are null)
    void (*run[2])(tmx::StepPtrs, Geom, Phys, int, const int4*, int, const int*, const unsigned char*, int, int*, int, int*);
    int (*run_smem)(int nt);  // its dynamic shared memory
    int sbytes, tbytes;
    bool moments;  // the form stores per-node FP32 moments next to the populations
};
extern const StepKernels kForms[3];

constexpr int kSumBlocks = 592;

// Validation of a case (the body of tmx_case_check).
int check_case(const tmx_case& c);
void geometry_of(const tmx_case& c, Geom& G);
void physics_of(const tmx_case& c, Phys& P);
// Device bytes of one single-mixer handle.
long long footprint(const Geom& G, long long nb, int precision);
long long boundary_count(const Geom& G);
// Class of a boundary node (tmx_classes.h), -1 for a node no case covers.
int classify(const Geom& G, int b, int i, int j, int k);
// Boundary nodes sorted faces first, then by class, then by node index; the
// first nface entries are face classes.  With nswept the faces that the sweep
// kernels update come last among them and *nswept counts them: the ends of the
// interior rows (the inlets, the mixing box's x walls) and the z wall faces
// (K_FACE_Z1, K_FACE_ZT), of which each lies above or below an interior node
// and each interior node of planes 2 and nz - 1 has one (checked; an internal
// error otherwise).  Without interior nodes (nz < 3) they stay in place and
// *nswept is 0.  Returns TMX_OK or a failure code.
int boundary_list(const Geom& G, std::vector<int>& nodes, std::vector<unsigned char>& cls, int& nface,
                  std::vector<int>* class_count, int* nswept);
// Inlet profiles Uin1, Uin2 ((iny+3) x (nz+3)) as the reference computes them:
// the duct series (which depends on iny and nz only) and its mean, then the
// scaling to umean and the shifts.
void inlet_profile(const tmx_case& c, std::vector<double>& U1, std::vector<double>& U2);
void inlet_series(int iny, int nz, std::vector<double>& raw, double& average);
// The same series computed on the current device (k_inlet_series) with the
// host's summation of the mean; for the reduced-precision forms.
int inlet_series_device(int iny, int nz, cudaStream_t stream, std::vector<double>& raw, double& average);
// The inlet profiles of a case in its form: the host series for FP64 (the
// reference's bits), the device series otherwise.
int inlet_profile_form(const tmx_case& c, cudaStream_t stream, std::vector<double>& U1, std::vector<double>& U2);
void inlet_scale(const tmx_case& c, const std::vector<double>& raw, double average, std::vector<double>& U1,
                 std::vector<double>& U2);

// The FP16 form's sweep kernels by shape (include/tmx.h TMX_SHAPE_SWEEP*):
// tile height, the single-mixer and batched kernels and their dynamic shared
// memory.
struct SweepShape {
    int kind, ty;
    void (*tiles)(tmx::StepPtrs, Geom, Phys, int, const int4*, int);
    void (*single)(tmx::StepPtrs, Geom, Phys, int, const int4*, int, const int*, const unsigned char*, int, int, int);
    void (*batch[2])(const tmx::MixerDesc*, const int4*, const int2*, int*, int, int);  // [1]: tiles with groups
    int threads() const { return 32 * ty; }
    int smem(bool groups) const { return tmx::sweep_smem_host(ty, groups); }
};
inline const SweepShape* sweep_shape(int kind)
{
    static const SweepShape shapes[] = {
        {TMX_SHAPE_SWEEP8, 8, tmx::k_sweep8_f16, tmx::k_sweepw8_f16, {tmx::k_sweep_batch8_f16, tmx::k_sweep_batch8g_f16}},
        {TMX_SHAPE_SWEEP4, 4, tmx::k_sweep4_f16, tmx::k_sweepw4_f16, {tmx::k_sweep_batch4_f16, tmx::k_sweep_batch4g_f16}},
    };
    for (const SweepShape& e : shapes)
        if (e.kind == kind) return &e;
    return nullptr;
}
// Allow each sweep kernel its dynamic shared memory on the current device
// (idempotent); returns the first error.
inline cudaError_t sweep_allow_smem()
{
    for (int kind = TMX_SHAPE_SWEEP8; kind <= TMX_SHAPE_SWEEP4; kind++) {
        const SweepShape* sh = sweep_shape(kind);
        cudaError_t e = cudaFuncSetAttribute((const void*)sh->single, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             sh->smem(false));
        if (e == cudaSuccess)
            e = cudaFuncSetAttribute((const void*)sh->tiles, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     sh->smem(false));
        for (int g = 0; g < 2 && e == cudaSuccess; g++)
            e = cudaFuncSetAttribute((const void*)sh->batch[g], cudaFuncAttributeMaxDynamicSharedMemorySize, sh->smem(g));
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

// Tiles of the sweep kernels (tmx_engine.cuh sweep_tile) for one mixer:
// {mixer * 2 + box | planes << 23, x0, y0 | s << 29, z0}, the columns from x0
// (sweep_end) by ty << s rows of a box (0-based x0, y0; the rows of interior nodes)
// over zchunk interior planes from z0 (250 at most), z-chunks outermost.  groups: the widths
// are those that cover the box with the fewest tiles, the wider of equals
// (24, 40 and 48 columns by 47, 79 and 95 rows of 4: 9, 25 and 36 tiles a plane where
// 32 columns each take 24, 40 and 48); else s = 0.
inline void sweep_tiles(const Geom& G, int mixer, int ty, int zchunk, bool groups, std::vector<int4>& out)
{
    zchunk = zchunk < 250 ? zchunk : 250;
    std::vector<int> wide[2];  // per box: the s of a tile from column x
    for (int b = 0; b < 2; b++) {
        const int nx = G.nx[b], rows = G.ny[b] - 1;
        std::vector<int> least(nx + 1, 0);
        wide[b].assign(nx, 0);
        for (int x = nx - 1; x >= 0; x--)
            for (int s = 0; s < (groups ? 3 : 1); s++) {
                const int n = (rows + (ty << s) - 1) / (ty << s) + least[tmx::sweep_end(x, nx, 32 >> s)];
                if (s == 0 || n < least[x]) {
                    least[x] = n;
                    wide[b][x] = s;
                }
            }
    }
    for (int z0 = 2; z0 <= G.nz - 1; z0 += zchunk)
        for (int b = 0; b < 2; b++)
            // rows 0 .. ny-2 of box 0 (the opening's included), 1 .. ny-1 of box 1
            for (int r = 0; r < G.ny[b] - 1; r += ty)
                for (int x0 = 0; x0 < G.nx[b]; x0 = tmx::sweep_end(x0, G.nx[b], 32 >> wide[b][x0])) {
                    const int s = wide[b][x0];
                    if (r % (ty << s) == 0)
                        out.push_back(make_int4((mixer * 2 + b) | std::min(zchunk, G.nz - z0) << 23, x0,
                                                (r + b) | s << 29, z0));
                }
}

// Steps of one captured graph where many are asked for (an even number: the
// buffers are back in place).  A graph of its own per step costs a small mixer a
// microsecond or two between steps.
constexpr int kGraphSteps = 16;
// The next launch's steps where `left` are asked for: building such a graph costs
// what 50 to 150 steps save by it (W=32, the first 20 steps of a handle: FP64 123 us a
// step by a new graph of 16, 117 one by one, 113 by one that is there), so one by
// one until kGraphWorth steps have gone that way or are asked for.
constexpr int kGraphWorth = 64;
inline int graph_length(int left, bool built, int singles)
{
    return left > kGraphSteps && (built || left + singles > kGraphWorth) ? kGraphSteps : 1;
}

// Launch a step's kernel; overlap: as soon as the step before it in the stream
// leaves room, which the kernel waits for by itself (step_wait).
template <class... P, class... A>
cudaError_t launch_step(void (*kernel)(P...), int blocks, int threads, int smem, cudaStream_t stream, bool overlap,
                        A... args)
{
    cudaLaunchConfig_t c{};
    c.gridDim = dim3((unsigned)blocks);
    c.blockDim = dim3((unsigned)threads);
    c.dynamicSmemBytes = (size_t)smem;
    c.stream = stream;
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    c.attrs = &at;
    c.numAttrs = overlap ? 1 : 0;
    return cudaLaunchKernelEx(&c, kernel, P(args)...);
}

// Threads per block, and so nodes per run, of the FP64 step (FP32: 128): 256, whose 2 KB
// copies get the most from DRAM, or 128 where the finer runs fill the SMs more
// evenly (step by 128 / 256: 65,536 nodes 23.7 / 30.5 us, 524,288 nodes 116.4 /
// 118.4 us, 1.8M nodes 358.7 / 357.7 us, 4.9M nodes 969 / 956 us).
inline int run_threads(int precision, long long nodes)
{
    return precision != TMX_FP64 || nodes < 2000000 ? 128 : 256;
}
// Runs of the FP64 and FP32 steps (tmx_kernels.cuh) for one mixer, of up to nt nodes:
// every node but the edges and corners, plane by plane; the long runs first,
// then the short ones (which even out the end of the launch).
inline void step_runs(const Geom& G, int mixer, int nt, std::vector<int4>& out)
{
    std::vector<int4> rest;
    for (int k = 1; k <= G.nz; k++)
        for (int b = 0; b < 2; b++) {
            // columns i0..i1 of row j0 through row j1 (whole rows between)
            auto add = [&](int kind, int iface, int i0, int j0, int i1, int j1) {
                if (j1 < j0 || (j1 == j0 && i1 < i0)) return;
                int g = tmx::node_index(G, b, i0, j0, k), i = i0;
                const int end = tmx::node_index(G, b, i1, j1, k) + 1;
                while (g < end) {
                    // (ends at multiples of 32 nodes: whole 256-byte stores)
                    const int n = std::min(end - g, nt - g % 32);
                    (n > nt / 2 ? out : rest)
                        .push_back(make_int4(g, n | kind << 9 | b << 12 | iface << 13, i, mixer));
                    g += n;
                    i = (i - 1 + n) % G.nx[b] + 1;
                }
            };
            const bool wall = k == 1 || k == G.nz;
            const int rows = k == 1 ? tmx::kRunZ1 : (k == G.nz ? tmx::kRunZT : tmx::kRunRows);
            const int nx = G.nx[b], ny = G.ny[b];
            if (b == 0) {
                add(rows, 0, 1, 2, nx, ny - 1);
                add(rows, 1, G.ia + 1, 1, G.ib - 1, 1);
                if (!wall) {
                    add(tmx::kRunYT, 0, 2, ny, nx - 1, ny);
                    add(tmx::kRunY1, 0, 2, 1, G.ia - 1, 1);
                    add(tmx::kRunY1, 0, G.ib + 1, 1, nx - 1, 1);
                }
            } else {
                add(rows, 0, 1, 2, nx, ny - 1);
                add(rows, 2, 1, ny, nx, ny);
                if (!wall) add(tmx::kRunY1, 0, 2, 1, nx - 1, 1);
            }
        }
    out.insert(out.end(), rest.begin(), rest.end());
}

// One field of a box from the device (first node dev, x fastest) to the host in
// the reference's [i][j][k] order, by way of scratch: device memory of
// a box's doubles that nothing else uses meanwhile (the population buffer that
// the next step writes).  Waits for the stream.
int box_to_host(const Geom& G, int box, const double* dev, double* scratch, cudaStream_t stream, double* host_out);

// An int that kernels set when they give up (mapped host memory, 0 to begin
// with), and its return; null when there is no memory.
int* error_flag_take();
void error_flag_give(int* flag);

// Planes per 32 x 4 tile of a new FP16 handle: the fewest from 3 whose tiles the
// GPU holds at once (slots blocks), 8 where none does.  A tile goes through its
// planes one after another, so a small mixer wants short tiles (221,184 nodes 27.7
// us by 4 planes, 35.8 by 8), and a second, partly filled wave costs a whole one
// (221,184 nodes 31.8 us by 3 planes).  1 or 2 planes, whose tiles read most records
// twice or three times, only where half of the GPU holds them with the boundary's
// blocks (rest): 1,024 nodes 12.2 / 14.0 us by 1 / 3 planes, 8,192 nodes 13.0 / 14.5,
// 27,648 nodes 13.9 / 16.7 by 2 / 3; but 43,904 nodes 18.6 / 15.8.
inline int sweep_planes(const Geom& G, int slots, int rest)
{
    for (int z = 1; z < 8; z++) {
        std::vector<int4> t;
        sweep_tiles(G, 0, 4, z, false, t);
        const int n = (int)t.size();
        if (z < 3 ? 2 * (n + rest) <= slots : n <= slots) return z;
    }
    return 8;
}
// ... and of an FP16 batch that no shape was set for: 4, or 8 where those make
// kBatchRounds rounds of tiles or more.  Up to two rounds the end of the last one
// decides, either way (by 4 / 8 planes: 8 mixers of 544,000 nodes, one round, 81 /
// 90 us; 3 of 415,000, 0.9 rounds, 63.4 / 55.6; 3 of 1.1M, 2.0 rounds, 125.8 / 127.2);
// then fewer records read twice count for more with the size (2.6 rounds 163.5 /
// 161.6, 4.7 rounds 257.4 / 256.1, 7.2 rounds 381 / 377, 12 rounds 625 / 605, 23
// rounds 1,228 / 1,186, 64 mixers of 41M nodes, 68 rounds, 3.71 / 3.58 ms).
constexpr int kBatchPlanes = 4, kBatchRounds = 4;

// Checkpoint layout (tmx_checkpoint, tmx_batch_checkpoint): this header, then
// the sections in the order of `bytes`: the population buffer the next step
// reads (76 planes of ps values of the storage type), the previous step's
// densities (4 planes, arithmetic type), the FP16 form's moment records
// (2 float4 per node, or nothing), the macroscopic fields (7 FP64 planes) and
// the two inlet profiles ((iny+3)(nz+3) FP64 values each).
// "TMXCKPT2": FP16 records {(rho, cA, cB, cC), (ux, uy, uz, omt)};
// "TMXCKPT1" (refused) had {(rho, ux, uy, uz), (cA, cB, cC, omt)}
constexpr char kCheckpointMagic[9] = "TMXCKPT2";
struct CheckpointHeader {
    char magic[8];  // kCheckpointMagic
    int abi;
    int precision;
    tmx_case c;
    long long steps;
    long long ps;
    long long bytes[5];
};
inline void checkpoint_sections(const Geom& G, int precision, long long bytes[5])
{
    const StepKernels& K = kForms[precision];
    bytes[0] = 76LL * G.ps * K.sbytes;
    bytes[1] = 4LL * G.ps * K.tbytes;
    bytes[2] = K.moments ? 2LL * G.ps * 16 : 0;
    bytes[3] = 7LL * G.ps * 8;
    bytes[4] = 2LL * (G.iny + 3) * (G.nz + 3) * 8;
}
inline long long checkpoint_total(const long long bytes[5])
{
    return (long long)sizeof(CheckpointHeader) + bytes[0] + bytes[1] + bytes[2] + bytes[3] + bytes[4];
}
// Check a checkpoint against a case; TMX_OK or TMX_E_INVALID with a message.
int checkpoint_check(const void* buf, long long size, const tmx_case& c, const Geom& G);

}  // namespace tmx_host
