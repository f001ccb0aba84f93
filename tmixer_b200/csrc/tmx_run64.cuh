// tmx_run64.cuh -- the step of the plain FP64 form: one kernel over every node
// but the edges and corners, fed through shared memory (device code; the
// kernels that instantiate it are in tmx_kernels.cu).
//
// Runs (tmx_run.cuh) come as bulk copies of 8 NT bytes, 19 to a field.
// Two slots of 19 x (NT + 4) values hold one field each.  A field is read into
// registers and its slot filled again at once (by the last warp to read it),
// so that two fields are in flight while one is collided, past the end of the
// run into the next one.  B, whose sum the collision of A needs, is summed
// before and read when A is done.
//
// What bounds it: DRAM.  Moving these bytes in this way without arithmetic
// (bulk copies of 256 nodes, two slots, two blocks per SM, plain stores) runs
// at 5.9 to 6.3 TB/s; the same bytes by 8-byte cp.async in runs of 32 nodes at
// 4.7 TB/s, whatever the number in flight.
#pragma once
#include "tmx_run.cuh"

namespace tmx {

// What the step reads and writes of one mixer.
struct RunView {
    const double* pin;
    double *pout, *rcur, *mac;
    const double *uin1, *uin2;
    const Geom* G;
    const Phys* P;
};
__device__ __forceinline__ RunView run_view(const StepPtrs& X, const Geom& G, const Phys& P)
{
    return RunView{(const double*)X.pin, (double*)X.pout, (double*)X.rcur, X.mac, (const double*)X.uin1,
                   (const double*)X.uin2, &G, &P};
}

// The window of a direction in its plane (first value and number, both even: a
// bulk copy starts and ends at 16 bytes): the run's sources and one more at
// either end, for the x walls' neighbours.  Plane p of the 76; the last values
// stop at the end of the buffer.
__host__ __device__ inline void run_window(int g0, int n, int off, int p, long long ps, int& first, int& count)
{
    first = (g0 + off - 1) & ~1;
    count = (n + 5) & ~1;
    const long long left = (76 - p) * ps - first;
    if (count > left) count = (int)left;
}

// Shared memory of a block of NT threads: the two slots (rows of a window of up
// to NT + 4 values), the next runs, the barriers.
template <int NT>
struct __align__(16) RunShared {
    static constexpr int kRow = NT + 4;
    double slot[2][19 * kRow];
    int4 run[2];         // by the run's ordinal in the block; n = 0: none
    int off[2][2][20];   // ... its offsets by direction, of the flow and of the species
    unsigned par[2][2];  // ... and the parities that they begin with
    unsigned long long full[2];
    int done[2];  // warps that have read a slot
    double edge[NT / 32][kEdgeBuf];
};
static_assert(sizeof(RunShared<128>) == run_smem_host(128) && sizeof(RunShared<256>) == run_smem_host(256),
              "host copy of the size");

// What a block needs of its run number ord (in S.run): the offsets of the
// sources and their parities (one warp; lane q does direction q).
template <int NT>
__device__ __forceinline__ void run_prepare(RunShared<NT>& S, int ord, const Geom& G)
{
    const int lane = threadIdx.x & 31, q = lane < 19 ? lane : 18;
    const Run R = run_of(G, S.run[ord]);
    int ex, ey, ez, opp;
    dir_of(q, ex, ey, ez, opp);
#pragma unroll
    for (int c = 0; c < 2; c++) {
        const int off = run_offset(R, c, ex, ey, ez);
        const unsigned par = __ballot_sync(0xffffffffu, ((R.g0 + off - 1) & 1) && lane < 19);
        if (lane < 19) S.off[ord][c][q] = run_pulls(R, c, ey, ez) ? off : kRunNone;
        if (lane == 0) S.par[ord][c] = par;
    }
}

// Fill a slot with field fld of run number ord (one warp; lane q copies
// direction q).
template <int NT>
__device__ __forceinline__ void run_fill(RunShared<NT>& S, int slot, int ord, const RunView& M, int fld)
{
    const int q = threadIdx.x & 31, p = fld * 19 + q;
    const unsigned bar = smem_addr(&S.full[slot]);
    const int off = q < 19 ? S.off[ord][fld ? 1 : 0][q] : kRunNone;
    const long long ps = M.G->ps;
    int first = 0, count = 0;
    if (off != kRunNone) run_window(S.run[ord].x, S.run[ord].y & 511, off, p, ps, first, count);
    const unsigned bytes = __reduce_add_sync(0xffffffffu, (unsigned)count) * 8u;
    if (q == 0) mbar_expect(bar, bytes);
    __syncwarp();
    if (count)
        bulk_load(smem_addr(&S.slot[slot][q * (NT + 4)]), M.pin + p * ps + first, (unsigned)count * 8u, bar);
}

// Where a thread's values of a field lie: in row q of the slot one or two
// beyond the thread's number, by the parity of the source that the window
// begins with (bit q).  kRunEven: rows and planes of even length, where only
// the x component counts.
constexpr unsigned run_even()
{
    unsigned m = 0;
    for (int q = 0; q < 19; q++) m |= (EX(q) == 0 ? 1u : 0u) << q;
    return m;
}
constexpr unsigned kRunEven = run_even();
template <int NT>
__device__ __forceinline__ void run_read(const double* __restrict__ row, unsigned par, double (&v)[19])
{
    if (par == kRunEven) {
#pragma unroll
        for (int q = 0; q < 19; q++) v[q] = row[q * (NT + 4) + (EX(q) == 0 ? 2 : 1)];
    } else {
#pragma unroll
        for (int q = 0; q < 19; q++) v[q] = row[q * (NT + 4) + 1 + ((par >> q) & 1)];
    }
}
template <int NT>
__device__ __forceinline__ double run_sum(const double* __restrict__ row, unsigned par)
{
    double s = 0.0;
    if (par == kRunEven) {
#pragma unroll
        for (int q = 0; q < 19; q++) {
            const double x = row[q * (NT + 4) + (EX(q) == 0 ? 2 : 1)];
            s = q ? s + x : x;
        }
    } else {
#pragma unroll
        for (int q = 0; q < 19; q++) {
            const double x = row[q * (NT + 4) + 1 + ((par >> q) & 1)];
            s = q ? s + x : x;
        }
    }
    return s;
}

// The populations that an inlet node's closure sets, of a species in its slot
// (closure_face).
template <int NT>
__device__ __forceinline__ void run_inlet_species(double* row, unsigned par, int cls, double cin)
{
    const double w1 = 2.0 / 18.0 * cin, w2 = 2.0 / 36.0 * cin;
    auto at = [&](int q) -> double& { return row[q * (NT + 4) + 1 + ((par >> q) & 1)]; };
    const bool one = cls == K_INLET1;
    constexpr int in[5] = {1, 7, 10, 11, 14}, out[5] = {3, 9, 8, 13, 12};  // opposite pairs
#pragma unroll
    for (int e = 0; e < 5; e++) {
        const double w = e ? w2 : w1;
        if (one) at(in[e]) = -at(out[e]) + w;
        else at(out[e]) = -at(in[e]) + w;
    }
}

// Collide and store one field of a node: f * c1 + c2 * feq plus the
// reaction's w_q * rt * m (collide_store's operations; m is -1 for A and B and
// 2 for C, products that do not round; the flow adds -0.0, which changes no
// value).
__device__ __forceinline__ void run_collide(double* __restrict__ p, long long ps, const double (&v)[19], double r,
                                            const double (&poly)[19], double c1, double c2, double w0, double w1,
                                            double w2)
{
#pragma unroll
    for (int q = 0; q < 19; q++) {
        const double o = v[q] * c1 + c2 * feq_div(r * poly[q], q);
        *p = o + (q == 0 ? w0 : (q <= 6 ? w1 : w2));
        p += ps;
    }
}
// The same for a density so small that the equilibrium needs the IEEE division
// (rare): a loop over local memory.
__device__ __forceinline__ void run_collide_exact(double* __restrict__ p, long long ps, const double (&v)[19], double r,
                                                  const double (&poly)[19], double c1, double c2, double w0, double w1,
                                                  double w2)
{
    double pl[19], vl[19];
#pragma unroll
    for (int q = 0; q < 19; q++) {
        pl[q] = poly[q];
        vl[q] = v[q];
    }
#pragma unroll 1
    for (int q = 0; q < 19; q++) {
        const double o = vl[q] * c1 + c2 * __ddiv_rn(r * pl[q], q == 0 ? 3.0 : (q <= 6 ? 18.0 : 36.0));
        *p = o + (q == 0 ? w0 : (q <= 6 ? w1 : w2));
        p += ps;
    }
}

// An edge or corner node, out of line: its registers are not the runs' concern.
__device__ __noinline__ void run_edge(const StepPtrs& X, const Geom& G, const Phys& P, int write_macro, int node, int cls,
                                      double* buf)
{
    edge_node<F64>(X, G, P, write_macro, node, cls, buf);
}

// The runs of one block: the first by its number, then by the launch's counter.
// get(t) gives the buffers, geometry and constants of run t's mixer.  error: set
// when a copy does not arrive.  ready(): waits for the step before; meanwhile():
// what the warps do while the first run's copies are on their way.
template <int NT, class Get, class Ready, class Mean>
__device__ __forceinline__ void run_loop(const Get& get, const int4* __restrict__ runs, int nruns, int first,
                                         int nblocks, int* __restrict__ counter, int write_macro, RunShared<NT>& S,
                                         int* error, const Ready& ready, const Mean& meanwhile)
{
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    constexpr int kWarps = NT / 32;
    if (first >= nruns) {  // (the whole block)
        ready();
        meanwhile();
        return;
    }
    if (t == 0) {
        for (int s = 0; s < 2; s++) {
            mbar_init(smem_addr(&S.full[s]), 1);
            S.done[s] = 0;
        }
        S.run[0] = runs[first];
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    if (warp == 0) run_prepare(S, 0, *get(S.run[0]).G);
    ready();
    if (warp == 0) {
        const RunView M = get(S.run[0]);
        __syncwarp();
        run_fill(S, 0, 0, M, 0);
        run_fill(S, 1, 0, M, 1);
    }
    meanwhile();
    for (int ord = 0;; ord ^= 1) {
        // (each barrier goes through two phases a run: the parities repeat)
        if (!mbar_wait(smem_addr(&S.full[0]), 0)) goto gave_up;
        const int4 tr = S.run[ord];
        if ((tr.y & 511) == 0) return;
        const RunView M = get(tr);
        const Phys& P = *M.P;
        const long long ps = M.G->ps;
        const int g = tr.x + t;
        // the node's class, x shift and activity, in one register
        int what;
        {
            const RunNode N = run_node(*M.G, run_of(*M.G, tr), t);
            what = (N.cls << 3) | ((N.xs + 1) << 1) | (int)N.act;
        }
        const auto cls = [&] { return what >> 3; };
        const auto inlet = [&] { return cls() == K_INLET1 || cls() == K_INLET2; };
        const auto act = [&] { return (what & 1) != 0; };
        double* __restrict__ p = M.pout + g;
        // the next run: its index now, its entry after the flow, there for
        // all before the block has read B
        int next = 0;
        if (t == NT - 1) next = nblocks + atomicAdd(counter, 1);

        double poly[19], v[19];
        double r = 0.0, cb = 0.0, rt = 0.0;
#pragma unroll 1
        for (int f = 0; f < 4; f++) {
            const int s = f & 1;
            if (s && !mbar_wait(smem_addr(&S.full[1]), f >> 1)) goto gave_up;
            run_read<NT>(&S.slot[s][t + (f ? ((what >> 1) & 3) - 1 : 0)], S.par[ord][f ? 1 : 0], v);
            // the slot is free once every warp has read it; the last fills it
            // with the field after the next
            __syncwarp();
            int last = 0;
            if (lane == 0) {
                asm volatile("atom.acq_rel.cta.shared::cta.add.u32 %0, [%1], 1;"
                             : "=r"(last)
                             : "r"(smem_addr(&S.done[s]))
                             : "memory");
            }
            last = __shfl_sync(0xffffffffu, last, 0);
            if (last == kWarps - 1) {
                if (lane == 0) S.done[s] = 0;
                const int of = f < 2 ? ord : ord ^ 1;
                if (S.run[of].y & 511) {
                    run_fill(S, s, of, get(S.run[of]), f ^ 2);
                } else if (f == 2 && lane == 0) {
                    mbar_expect(smem_addr(&S.full[0]), 0);  // wakes the block to leave
                }
            }
            if (f == 0) {
                // the closure, the moments, the polynomial that the four fields share
                if (act()) {
                    if (inlet()) {
                        BCtx<F64> c{};
                        c.uin1 = M.uin1;
                        c.uin2 = M.uin2;
                        c.G = M.G;
                        c.P = M.P;
                        decode(*M.G, g, c.b, c.i, c.j, c.k);
                        closure_face<F64>(c, cls(), 0, v);
                    } else if (cls() >= 0) {
                        wall_flow_closure(cls(), P.rho_out, v);
                    }
                    r = sum19(v);
                    // the outlet row's density is pinned to rho_out (Tmixer.cpp:9575-9582)
                    if (cls() == K_OUTLET) r = P.rho_out;
                    double sxm, sym, szm;
                    momentum(v, sxm, sym, szm);
                    const double ux = sxm / r, uy = sym / r, uz = szm / r;
                    eq_poly(ux, uy, uz, poly);
                    if (write_macro) {
                        M.mac[ps + g] = ux;
                        M.mac[2 * ps + g] = uy;
                        M.mac[3 * ps + g] = uz;
                    }
                }
                if (t == NT - 1) {
                    if (next < nruns) cp_async16(&S.run[ord ^ 1], runs + next);
                    else S.run[ord ^ 1] = make_int4(0, 0, 1, 0);
                }
            } else if (f != 2) {
                if (inlet()) {
                    BCtx<F64> c{};
                    c.P = M.P;
                    closure_face<F64>(c, cls(), f, v);
                }
                r = sum19(v);
            }
            if (f == 1) {
                // B, of which the collision of A needs the sum
                if (warp == kWarps - 1) {
                    cp_async_commit();
                    cp_async_wait_all();
                    __syncwarp();
                    if (S.run[ord ^ 1].y & 511) run_prepare(S, ord ^ 1, *get(S.run[ord ^ 1]).G);
                }
                if (!mbar_wait(smem_addr(&S.full[0]), 1)) goto gave_up;
                double* __restrict__ rb = &S.slot[0][t + ((what >> 1) & 3) - 1];
                if (inlet()) {
                    run_inlet_species<NT>(rb, S.par[ord][1], cls(), P.cin[1][cls() == K_INLET2]);
                    // (written here, filled again by a bulk copy)
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                }
                cb = run_sum<NT>(rb, S.par[ord][1]);
                rt = P.rateconst * r * cb;
            } else if (f == 2) {
                r = cb;
            }
            if (act()) {
                // densities the closures read next step: the faces', and those
                // of the interior nodes beside the junction edges
                // (Tmixer.cpp:8609, :8851)
                if (cls() != -1) M.rcur[f * ps + g] = r;
                if (write_macro) M.mac[(f ? 3 + f : 0) * ps + g] = r;
                const double c1 = P.c1[f], c2 = P.c2[f];
                const double m = f == 0 ? -0.0 : (f == 3 ? 2.0 : -1.0);
                const double w0 = f ? (wq(0) * rt) * m : m, w1 = f ? (wq(1) * rt) * m : m, w2 = f ? (wq(7) * rt) * m : m;
                if (tiny_density(r))
                    run_collide_exact(p, ps, v, r, poly, c1, c2, w0, w1, w2);
                else
                    run_collide(p, ps, v, r, poly, c1, c2, w0, w1, w2);
                p += 19 * ps;
            }
        }
    }
gave_up:
    mbar_give_up(error, smem_addr(&S.full[0]));
    mbar_give_up(error, smem_addr(&S.full[1]));
}

}  // namespace tmx
