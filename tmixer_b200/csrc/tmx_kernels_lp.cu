// tmx_kernels_lp.cu -- sm_100a kernels of the reduced-precision forms: FP32
// arithmetic with FP32 storage, and FP32 arithmetic with populations stored in
// FP16 as f_q - feq_q of the node that wrote them.  Both keep the four fields
// of a (direction, node) pair side by side, one vector access each.  Compiled
// with multiply-add contraction (the default); results are compared with the
// FP64 form within stated tolerances, not bit for bit.
#include "tmx_engine.cuh"
#include "tmx_run32.cuh"

namespace tmx {

TMX_DEFINE_INIT_KERNEL(F32, f32)

// The FP32 step (tmx_run32.cuh): the runs, and the edge and corner nodes, a warp
// each, which the warps take while their block's first run is on its way (the
// blocks without a run first).
__global__ void __launch_bounds__(128, 4) k_run128_f32(
    const __grid_constant__ StepPtrs X, const __grid_constant__ Geom G, const __grid_constant__ Phys P,
    int write_macro, const int4* __restrict__ runs, int nruns, const int* __restrict__ enode,
    const unsigned char* __restrict__ ecls, int ne, int* __restrict__ counters, int parity, int* error)
{
    constexpr int NT = 128;
    extern __shared__ __align__(16) unsigned char run_smem[];
    RunShared32<NT>& S = *(RunShared32<NT>*)run_smem;
    const int warp = threadIdx.x >> 5, nb = gridDim.x;
    const auto ready = [&] {
        step_wait();
        if (blockIdx.x == 0 && threadIdx.x == 0) counters[1 - parity] = 0;  // the next step's
    };
    step_begin();
    run32_loop<NT>([&](const int4&) { return RunView32{&X, &G, &P}; }, runs, nruns, blockIdx.x, nb, counters + parity,
                   write_macro, S, error, ready, [&] {
                       const int at = (int)(blockIdx.x + nb - nruns % nb) % nb;
                       for (int e = at * (NT / 32) + warp; e < ne; e += nb * (NT / 32))
                           run32_edge(X, G, P, write_macro, enode[e], ecls[e], S.edge[warp]);
                   });
}

// The same over the mixers of a batch, as k_run_batch_f64.
__global__ void __launch_bounds__(kRunBatchThreads, 512 / kRunBatchThreads) k_run_batch_f32(
    const MixerDesc* __restrict__ D, const int4* __restrict__ runs, const int2* __restrict__ edges,
    int* __restrict__ counts, int parity, int write_macro, int what, int* error)
{
    constexpr int NT = kRunBatchThreads;
    extern __shared__ __align__(16) unsigned char run_smem[];
    RunShared32<NT>& S = *(RunShared32<NT>*)run_smem;
    const int warp = threadIdx.x >> 5, nb = gridDim.x;
    const int nruns = what & 1 ? counts[4] : 0, ne = what & 2 ? counts[2] : 0;
    const auto ready = [&] {
        step_wait();
        if (blockIdx.x == 0 && threadIdx.x == 0) counts[5 + (1 - parity)] = 0;  // the next step's
    };
    step_begin();
    run32_loop<NT>(
        [&](const int4& t) {
            const MixerDesc& d = D[run_mixer(t)];
            return RunView32{&d.X[parity], &d.G, &d.P};
        },
        runs, nruns, blockIdx.x, nb, counts + 5 + parity, write_macro, S, error, ready, [&] {
            const int at = (int)(blockIdx.x + nb - nruns % nb) % nb;
            for (int e = at * (NT / 32) + warp; e < ne; e += nb * (NT / 32)) {
                const int2 t = edges[e];
                if (t.x < 0) continue;
                const MixerDesc& d = D[t.y >> 8];
                run32_edge(d.X[parity], d.G, d.P, write_macro, t.x, t.y & 255, S.edge[warp]);
            }
        });
}

TMX_DEFINE_STEP_KERNELS(F16, f16)
TMX_DEFINE_BOUNDARY_KERNELS(F16, f16)
TMX_DEFINE_BATCH_KERNELS(F16, f16)
TMX_DEFINE_SWEEP_KERNELS(F16, f16)

}  // namespace tmx
