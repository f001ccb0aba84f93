// tmx_run32.cuh -- the step of the FP32 form: one kernel over every node but the
// edges and corners, runs (tmx_run.cuh) fed through shared memory by bulk copies
// of 16 NT bytes, the four fields of a node side by side.
//
// One slot of 19 x (NT + 2) nodes holds a run.  It is read into registers (76
// values a thread) and filled again at once, by the last warp to read it, so
// that the next run is on its way while this one collides and stores.  A run of
// a wall takes two fillings: the flow's sources, then the species', those of
// the node that they are copied from.
#pragma once
#include "tmx_run.cuh"

namespace tmx {

// Shared memory of a block of NT threads.
template <int NT>
struct __align__(16) RunShared32 {
    float4 slot[19 * (NT + 2)];  // rows of a window of up to NT + 2 nodes
    int4 run[3];                 // by the run's ordinal in the block, mod 3; n = 0: none
    int off[3][2][20];           // ... its offsets by direction, of the flow and of the species
    unsigned long long full;
    int done;                    // warps that have read the slot
    float edge[NT / 32][kEdgeBuf];
};
static_assert(sizeof(RunShared32<128>) == run32_smem_host(128), "host copy of the size");

// What the step reads and writes of one mixer.
struct RunView32 {
    const StepPtrs* X;
    const Geom* G;
    const Phys* P;
};

// The window of a direction in its plane: the run's sources and one more node at
// either end, for the x walls' neighbours; the last stop at the end of the buffer.
__host__ __device__ inline void run32_window(int g0, int n, int off, int q, long long ps, int& first, int& count)
{
    first = g0 + off - 1;
    count = n + 2;
    const long long left = (19 - q) * ps - first;
    if (count > left) count = (int)left;
}

template <int NT>
__device__ __forceinline__ void run32_prepare(RunShared32<NT>& S, int ord, const Geom& G)
{
    const int lane = threadIdx.x & 31, q = lane < 19 ? lane : 18;
    const Run R = run_of(G, S.run[ord]);
    int ex, ey, ez, opp;
    dir_of(q, ex, ey, ez, opp);
#pragma unroll
    for (int c = 0; c < 2; c++)
        if (lane < 19) S.off[ord][c][q] = run_pulls(R, c, ey, ez) ? run_offset(R, c, ex, ey, ez) : kRunNone;
}

// Fill the slot with the flow's (c = 0) or the species' (1) sources of run
// number ord (one warp; lane q copies direction q).
template <int NT>
__device__ __forceinline__ void run32_fill(RunShared32<NT>& S, int ord, const RunView32& M, int c)
{
    const int q = threadIdx.x & 31;
    const unsigned bar = smem_addr(&S.full);
    const int off = q < 19 ? S.off[ord][c][q] : kRunNone;
    const long long ps = M.G->ps;
    int first = 0, count = 0;
    if (off != kRunNone) run32_window(S.run[ord].x, S.run[ord].y & 511, off, q, ps, first, count);
    const unsigned bytes = __reduce_add_sync(0xffffffffu, (unsigned)count) * 16u;
    if (q == 0) mbar_expect(bar, bytes);
    __syncwarp();
    if (count)
        bulk_load(smem_addr(&S.slot[q * (NT + 2)]), (const float4*)M.X->pin + q * ps + first, (unsigned)count * 16u,
                  bar);
}

// This warp has read the slot; true for the last warp, which fills it again.
template <int NT>
__device__ __forceinline__ bool run32_release(RunShared32<NT>& S)
{
    __syncwarp();
    int last = 0;
    if ((threadIdx.x & 31) == 0) {
        asm volatile("atom.acq_rel.cta.shared::cta.add.u32 %0, [%1], 1;"
                     : "=r"(last)
                     : "r"(smem_addr(&S.done))
                     : "memory");
        if (last == NT / 32 - 1) S.done = 0;
    }
    return __shfl_sync(0xffffffffu, last, 0) == NT / 32 - 1;
}

// An edge or corner node, out of line: its registers are not the runs' concern.
__device__ __noinline__ void run32_edge(const StepPtrs& X, const Geom& G, const Phys& P, int write_macro, int node,
                                        int cls, float* buf)
{
    edge_node<F32>(X, G, P, write_macro, node, cls, buf);
}

// (out of line: W=24 27.6 us a step, 28.0 with it in the loop's code)
__device__ __noinline__ void run32_give_up(int* error, unsigned bar) { mbar_give_up(error, bar); }

// The runs of one block: two by its number, then by the launch's counter.
// get(t) gives the buffers, geometry and constants of run t's mixer.  error: set
// when a copy does not arrive.  ready(): waits for the step before; meanwhile():
// what the warps do while the first run's copies are on their way.
template <int NT, class Get, class Ready, class Mean>
__device__ __forceinline__ void run32_loop(const Get& get, const int4* __restrict__ runs, int nruns, int first,
                                           int nblocks, int* __restrict__ counter, int write_macro,
                                           RunShared32<NT>& S, int* error, const Ready& ready, const Mean& meanwhile)
{
    const int t = threadIdx.x, warp = t >> 5;
    constexpr int kWarps = NT / 32;
    if (first >= nruns) {  // (the whole block)
        ready();
        meanwhile();
        return;
    }
    const int4 none = make_int4(0, 0, 1, 0);
    if (t == 0) {
        mbar_init(smem_addr(&S.full), 1);
        S.done = 0;
        S.run[0] = runs[first];
        S.run[1] = first + nblocks < nruns ? runs[first + nblocks] : none;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    if (warp == 0) run32_prepare(S, 0, *get(S.run[0]).G);
    if (warp == kWarps - 1 && (S.run[1].y & 511)) run32_prepare(S, 1, *get(S.run[1]).G);
    ready();
    if (warp == 0) {
        __syncwarp();
        run32_fill(S, 0, get(S.run[0]), 0);
    }
    meanwhile();
    unsigned phase = 0;
    int ord = 0;
    for (;;) {
        const int nxt = ord == 2 ? 0 : ord + 1, nn = nxt == 2 ? 0 : nxt + 1;
        if (!mbar_wait(smem_addr(&S.full), phase)) return run32_give_up(error, smem_addr(&S.full));
        phase ^= 1;
        const int4 tr = S.run[ord];
        if ((tr.y & 511) == 0) return;
        const RunView32 M = get(tr);
        const int g = tr.x + t;
        const RunNode N = run_node(*M.G, run_of(*M.G, tr), t);
        const bool wall = ((tr.y >> 9) & 7) != kRunRows;
        // the run after the next: its index now, its entry after the reads, its
        // offsets before this run ends
        int next = 0;
        if (t == NT - 1) next = 2 * nblocks + atomicAdd(counter, 1);

        float2 p01[19], p23[19];
        const float4* __restrict__ row = &S.slot[t + 1];
#pragma unroll
        for (int q = 0; q < 19; q++) {
            const float4 v = row[q * (NT + 2)];
            p01[q] = make_float2(v.x, v.y);
            p23[q] = make_float2(v.z, v.w);
        }
        if (wall) {
            if (run32_release(S)) run32_fill(S, ord, M, 1);
            if (!mbar_wait(smem_addr(&S.full), phase)) return run32_give_up(error, smem_addr(&S.full));
            phase ^= 1;
        }
        if (wall | (N.xs != 0)) {
            const float4* __restrict__ from = row + N.xs;
#pragma unroll
            for (int q = 0; q < 19; q++) {
                const float4 v = from[q * (NT + 2)];
                p01[q].y = v.y;
                p23[q] = make_float2(v.z, v.w);
            }
        }
        if (run32_release(S)) {
            if (S.run[nxt].y & 511) run32_fill(S, nxt, get(S.run[nxt]), 0);
            else if ((t & 31) == 0) mbar_expect(smem_addr(&S.full), 0);  // wakes the block to leave
        }
        if (t == NT - 1) {
            if (next < nruns) cp_async16(&S.run[nn], runs + next);
            else S.run[nn] = none;
        }
        if (N.act) {
            if (N.cls == K_INLET1 || N.cls == K_INLET2) {
                int b, i, j, k;
                decode(*M.G, g, b, i, j, k);
                xface_inlet<F32>(*M.X, *M.G, *M.P, N.cls, j, k, p01, p23);
            } else if (N.cls >= 0) {
                float v[19];
#pragma unroll
                for (int q = 0; q < 19; q++) v[q] = p01[q].x;
                wall_flow_closure(N.cls, (float)M.P->rho_out, v);
#pragma unroll
                for (int q = 0; q < 19; q++) p01[q].x = v[q];
            }
            // (the densities of the faces, and of the interior nodes beside the
            // junction edges, Tmixer.cpp:8609, :8851)
            lp_finish<F32>(*M.X, *M.G, *M.P, write_macro, g, p01, p23, N.cls == K_OUTLET, N.cls != -1);
        }
        if (warp == kWarps - 1) {
            cp_async_commit();
            cp_async_wait_all();
            __syncwarp();
            if (S.run[nn].y & 511) run32_prepare(S, nn, *get(S.run[nn]).G);
        }
        ord = nxt;
    }
}

}  // namespace tmx
