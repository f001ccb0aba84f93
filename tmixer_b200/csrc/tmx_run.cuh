// tmx_run.cuh -- runs: what the FP64 and FP32 steps (tmx_run64.cuh,
// tmx_run32.cuh) share.  A block of NT threads takes one run at a time: up to NT
// consecutive nodes of one plane, all interior rows (whose ends are the inlets
// or the mixing box's x walls), or a row of the y walls, the outlet or a z wall
// (step_runs in tmx_host.h).  A run's sources of one direction are consecutive
// too, so they come as one bulk copy into shared memory, and the wall faces cost
// what an interior node does: their closure, and another node to copy the
// species from.
#pragma once
#include "tmx_engine.cuh"

namespace tmx {

__device__ __forceinline__ unsigned smem_addr(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(unsigned bar, int count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect(unsigned bar, unsigned bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
// Wait for a phase of a barrier; false if it does not come within two seconds
// (a try that fails takes 4 us; the caller gives up and reports it).
__device__ __forceinline__ bool mbar_wait(unsigned bar, unsigned parity)
{
    for (int i = 0; i < (1 << 19); i++) {
        unsigned done;
        asm volatile(
            "{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}"
            : "=r"(done)
            : "r"(bar), "r"(parity)
            : "memory");
        if (done) return true;
    }
    return false;
}
// What a thread does that gave up waiting: it sets the error flag and waits once
// more for the copies of bar that are in flight (they write shared memory that the
// block leaves), whichever its phase is.
__device__ __forceinline__ void mbar_give_up(int* error, unsigned bar)
{
    *error = 1;
    mbar_wait(bar, 0);
    mbar_wait(bar, 1);
}
__device__ __forceinline__ void bulk_load(unsigned dst, const void* src, unsigned bytes, unsigned bar)
{
    asm volatile("cp.async.bulk.shared::cta.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
                 "l"(src), "r"(bytes), "r"(bar)
                 : "memory");
}

// A run, the same for the whole block: its first node, nodes, kind and box, and
// the strides of its sources.  Direction q of node h (the node itself for the
// flow, node + shift for the species) comes from h - ex - ez * sz, for ey = 1
// from h + op - ex - ez * szp, for ey = -1 from h + om - ex - ez * szm: the own
// box's strides, or on the two rows that meet at the opening the other box's
// (bulk_src).
struct Run {
    int g0, n, kind, b, i0, nx;
    int shift, op, om, ops, oms, sz, szp, szm;
};
__host__ __device__ inline int run_mixer(const int4& t) { return t.w; }
__host__ __device__ inline Run run_of(const Geom& G, const int4& t)
{
    Run R;
    R.g0 = t.x;
    R.n = t.y & 511;
    R.kind = (t.y >> 9) & 7;
    R.b = (t.y >> 12) & 1;
    const int iface = (t.y >> 13) & 3;
    R.i0 = t.z;
    R.nx = box_nx(G, R.b);
    R.sz = R.szp = R.szm = R.nx * box_ny(G, R.b);
    const int k0 = iface ? (R.g0 - box_base(G, R.b)) / R.sz : 0;
    R.op = -R.nx;
    R.om = R.nx;
    if (iface == 1) {
        R.szp = G.mnx * G.mny;
        R.op = G.base[1] + (k0 * G.mny + G.mny - 1) * G.mnx + 1 - G.ia - k0 * R.sz;
    } else if (iface == 2) {
        R.szm = G.inx * G.iny;
        R.om = k0 * R.szm + G.ia - 1 - G.base[1] - (k0 * G.mny + G.mny - 1) * G.mnx;
    }
    const int dk = R.kind == kRunZ1 ? 1 : (R.kind == kRunZT ? -1 : 0);
    R.shift = dk ? dk * R.sz : (R.kind == kRunYT ? -R.nx : (R.kind == kRunY1 ? R.nx : 0));
    R.ops = R.op + dk * (R.szp - R.sz);
    R.oms = R.om + dk * (R.szm - R.sz);
    return R;
}
// A thread's node of a run: active, x, face class (-1: interior, -2: interior
// beside a junction edge) and the x shift to the species' source node.
struct RunNode {
    bool act;
    int cls, xs;
};
__host__ __device__ inline RunNode run_node(const Geom& G, const Run& R, int t)
{
    RunNode N;
    N.act = t < R.n;
    N.cls = -1;
    N.xs = 0;
    const int i = (R.i0 - 1 + t) % R.nx + 1;  // the run may pass the end of a row
    const bool lo = i == 1, hi = i == R.nx;
    if (R.kind == kRunRows) {
        if (lo | hi) {
            N.cls = R.b ? (lo ? K_FACE_MX1 : K_FACE_MXT) : (lo ? K_INLET1 : K_INLET2);
            if (R.b) N.xs = lo ? 1 : -1;
        } else if (!R.b && (i == G.ia || i == G.ib) && (R.g0 + t) / R.nx % G.iny == 1) {
            N.cls = -2;
        }
    } else if (R.kind == kRunZ1 || R.kind == kRunZT) {
        N.act = N.act && !lo && !hi;  // the ends of the rows are edges
        N.cls = R.kind == kRunZ1 ? K_FACE_Z1 : K_FACE_ZT;
    } else {
        N.cls = R.kind == kRunYT ? K_FACE_YT : (R.b ? K_OUTLET : K_FACE_Y1);
    }
    return N;
}
// The offset of direction (ex, ey, ez)'s source of a field from the node.
__host__ __device__ inline int run_offset(const Run& R, int fld, int ex, int ey, int ez)
{
    const int o = ey > 0 ? (fld ? R.ops : R.op) : (ey < 0 ? (fld ? R.oms : R.om) : 0);
    return (fld ? R.shift : 0) + o - ex - ez * (ey > 0 ? R.szp : (ey < 0 ? R.szm : R.sz));
}
constexpr int kRunNone = -0x7fffffff;  // for an offset: no sources
// Whether a field's direction has sources at all (the flow of a wall row has
// none from beyond the wall; the closure sets those).
__host__ __device__ inline bool run_pulls(const Run& R, int fld, int ey, int ez)
{
    if (fld) return true;
    return !((R.kind == kRunZ1 && ez > 0) || (R.kind == kRunZT && ez < 0) || (R.kind == kRunYT && ey < 0) ||
             (R.kind == kRunY1 && ey > 0));
}
}  // namespace tmx
