// Checks the FP64 step's run lists on the host: every node that is no edge or
// corner lies in exactly one run, with the class of the general
// classification; every direction of every field is pulled from the source of
// the general rule (pull_src), the species of a copied face from the interior
// neighbour's, in the copied window's place that the kernel reads; and every
// window is aligned and inside the population buffer.  Arguments: inx iny nz mnx mny ia, repeated.
#include <cstdio>
#include <cstdlib>
#include <vector>

#include "../../tmixer_b200/csrc/tmx_host.h"
#include "../../tmixer_b200/csrc/tmx_run32.cuh"
#include "../../tmixer_b200/csrc/tmx_run64.cuh"

using namespace tmx;

static int check(const Geom& G, int nt)
{
    std::vector<int4> runs;
    tmx_host::step_runs(G, 5, nt, runs);
    std::vector<char> seen(G.nnodes, 0);
    for (const int4& t : runs) {
        if (run_mixer(t) != 5) return std::printf("mixer\n"), 1;
        const Run R = run_of(G, t);
        if (R.n < 1 || R.n > nt) return std::printf("run of %d\n", R.n), 1;
        int first[4][19], count[4][19];
        for (int fld = 0; fld < 4; fld++)
            for (int q = 0; q < 19; q++) {
                const int p = fld * 19 + q;
                first[fld][q] = count[fld][q] = 0;
                if (!run_pulls(R, fld, EY(q), EZ(q))) continue;
                run_window(R.g0, R.n, run_offset(R, fld, EX(q), EY(q), EZ(q)), p, G.ps, first[fld][q], count[fld][q]);
                const long long at = p * G.ps + first[fld][q];
                if (at < 0 || at % 2 || count[fld][q] % 2 || count[fld][q] > nt + 4 || at + count[fld][q] > 76 * G.ps)
                    return std::printf("window %lld + %d\n", at, count[fld][q]), 1;
            }
        // the FP32 form's windows: the value that thread e reads is at e + 1 (+ xs)
        for (int c = 0; c < 2; c++)
            for (int q = 0; q < 19; q++) {
                const int off = run_offset(R, c, EX(q), EY(q), EZ(q));
                int f = 0, n = 0;
                if (!run_pulls(R, c, EY(q), EZ(q))) continue;
                run32_window(R.g0, R.n, off, q, G.ps, f, n);
                const long long at = q * G.ps + f;
                if (at < 0 || n > nt + 2 || at + n > 19 * G.ps || f + 1 != R.g0 + off)
                    return std::printf("FP32 window %lld + %d\n", at, n), 1;
                for (int e = 0; e < R.n; e++) {
                    const RunNode N = run_node(G, R, e);
                    if (N.act && e + 1 + (c ? N.xs : 0) >= n) return std::printf("FP32 window too short\n"), 1;
                }
            }
        for (int e = 0; e < nt; e++) {
            const RunNode N = run_node(G, R, e);
            if (!N.act) continue;
            const int g = R.g0 + e;
            if (g < 0 || g >= G.nnodes || seen[g]++) return std::printf("node %d\n", g), 1;
            int b, i, j, k;
            decode(G, g, b, i, j, k);
            const int c = is_boundary(G, b, i, j, k) ? tmx_host::classify(G, b, i, j, k) : -1;
            const bool junction = c < 0 && b == 0 && j == 2 && (i == G.ia || i == G.ib);
            if (N.cls != (junction ? -2 : c)) return std::printf("class %d of node %d\n", N.cls, g), 1;
            int di = 0, dj = 0, dk = 0;
            switch (c) {
            case K_FACE_YT: dj = -1; break;
            case K_FACE_Y1:
            case K_OUTLET: dj = 1; break;
            case K_FACE_MX1: di = 1; break;
            case K_FACE_MXT: di = -1; break;
            case K_FACE_ZT: dk = -1; break;
            case K_FACE_Z1: dk = 1; break;
            default: break;
            }
            for (int fld = 0; fld < 4; fld++) {
                unsigned par = 0;
                for (int q = 0; q < 19; q++)
                    par |= ((unsigned)(R.g0 + run_offset(R, fld, EX(q), EY(q), EZ(q)) - 1) & 1u) << q;
                for (int q = 0; q < 19; q++) {
                    const int want = fld ? pull_src(G, b, i + di, j + dj, k + dk, q) : pull_src(G, b, i, j, k, q);
                    if (want < 0) {
                        if (fld && (di | dj | dk)) return std::printf("copied species without a source\n"), 1;
                        continue;
                    }
                    // the value that the thread reads from its slot's row
                    const int at = e + (fld ? N.xs : 0) + 1 + (par >> q & 1);
                    if (par == kRunEven && (int)(par >> q & 1) != (EX(q) == 0)) return std::printf("even\n"), 1;
                    if (at >= count[fld][q] || first[fld][q] + at != want)
                        return std::printf("field %d direction %d of node %d: %d, not %d\n", fld, q, g,
                                           first[fld][q] + at, want),
                               1;
                }
            }
        }
    }
    for (int g = 0; g < G.nnodes; g++) {
        int b, i, j, k;
        decode(G, g, b, i, j, k);
        const int c = is_boundary(G, b, i, j, k) ? tmx_host::classify(G, b, i, j, k) : -1;
        if (seen[g] != (c < 0 || is_face_class(c))) return std::printf("node %d covered %d times\n", g, seen[g]), 1;
    }
    return 0;
}

int main(int argc, char** argv)
{
    for (int a = 1; a + 5 < argc; a += 6) {
        tmx_case c{};
        c.inx = atoi(argv[a]);
        c.iny = atoi(argv[a + 1]);
        c.nz = atoi(argv[a + 2]);
        c.mnx = atoi(argv[a + 3]);
        c.mny = atoi(argv[a + 4]);
        c.ia = atoi(argv[a + 5]);
        Geom G;
        tmx_host::geometry_of(c, G);
        if (check(G, 128) || check(G, 256)) {
            std::printf("case %d %d %d %d %d %d\n", c.inx, c.iny, c.nz, c.mnx, c.mny, c.ia);
            return 1;
        }
    }
    std::printf("ok\n");
    return 0;
}
