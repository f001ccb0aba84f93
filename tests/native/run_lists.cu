// Checks the FP64 step's run lists on the host: every node that is no edge or
// corner lies in exactly one run, with the class of the general
// classification; every direction of every field is pulled from the source of
// the general rule (pull_src), the species of a copied face from the interior
// neighbour's, in the copied window's place that the kernel reads; and every
// window is aligned and inside the population buffer.  Also the FP16 form's tiles
// (check_tiles).  Arguments: inx iny nz mnx mny ia, repeated.
#include <cstdio>
#include <cstdlib>
#include <vector>

#include "../../tmixer_b200/csrc/tmx_host.h"
#include "../../tmixer_b200/csrc/tmx_run32.cuh"
#include "../../tmixer_b200/csrc/tmx_run64.cuh"

using namespace tmx;

static int check(const Geom& G, int nt, int mixer)
{
    std::vector<int4> runs;
    tmx_host::step_runs(G, mixer, nt, runs);
    std::vector<char> seen(G.nnodes, 0);
    for (const int4& t : runs) {
        if (run_mixer(t) != mixer) return std::printf("mixer\n"), 1;
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

// The tiles of the FP16 form: every node of the interior rows (the x faces
// among them, the opening's ends not) in exactly one, the species' source of an x wall
// in the same group of lanes, and every record of a node's sources staged in the
// place that the node reads.
static int check_tiles(const Geom& G, int ty, int planes, bool groups, int mixer)
{
    std::vector<int4> tiles;
    tmx_host::sweep_tiles(G, mixer, ty, planes, groups, tiles);
    std::vector<char> seen(G.nnodes, 0);
    const int pitch = sweep_pitch(groups);
    for (const int4& t : tiles) {
        const int b = t.x & 1, s = t.z >> 29, z1 = t.w + (t.x >> 23), w = 32 >> s;
        const int nx = box_nx(G, b), ny = box_ny(G, b), x1 = sweep_end(t.y, nx, w);
        if ((t.x & 0x7fffff) >> 1 != mixer || (!groups && s)) return std::printf("mixer or groups\n"), 1;
        if (x1 - t.y < 2 || x1 - t.y > w || t.w < 2 || z1 > G.nz) return std::printf("tile\n"), 1;
        for (int warp = 0; warp < ty; warp++)
            for (int lane = 0; lane < 32; lane++) {
                const SweepLane at = sweep_lane(s, lane, warp, ty);
                const int x = t.y + at.x, y = (t.z & 0x1fffffff) + at.y;
                if (x >= x1 || y >= ny || (b ? y < 1 : y >= ny - 1)) continue;
                if (b == 0 && y == 0 && (x < G.ia || x >= G.ib - 1)) continue;
                for (int k = t.w; k < z1; k++)
                    if (seen[box_base(G, b) + ((k - 1) * ny + y) * nx + x]++) return std::printf("twice\n"), 1;
                const int from = x == 0 ? lane + 1 : (x == nx - 1 ? lane - 1 : lane);
                if (from >> (5 - s) != lane >> (5 - s)) return std::printf("wall's neighbour\n"), 1;
                for (int dx = -1; dx <= 1; dx++)
                    for (int dy = -1; dy <= 1; dy++) {
                        const int col = at.col + 1 + dx, row = warp + 1 + dy, c = sweep_group(s, col);
                        if (col < 0 || col >= pitch || c != lane >> (5 - s) || sweep_column(s, col) != at.x + dx ||
                            c * ty + row - 1 != at.y + dy)
                            return std::printf("record\n"), 1;
                    }
            }
    }
    for (int b = 0; b < 2; b++)
        for (int k = 2; k < G.nz; k++)
            for (int y = 0; y < box_ny(G, b); y++)
                for (int x = 0; x < box_nx(G, b); x++) {
                    bool in = b ? y > 0 : y < G.iny - 1;
                    if (b == 0 && y == 0) in = x >= G.ia && x < G.ib - 1;
                    if (seen[box_base(G, b) + ((k - 1) * box_ny(G, b) + y) * box_nx(G, b) + x] != (in ? 1 : 0))
                        return std::printf("cover %d %d %d %d\n", b, x, y, k), 1;
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
        int bad = 0;
        // a mixer's slot as small batches have it, in the first two cases also large ones
        for (int m : {5, 65536, kMaxMixers - 1}) {
            if (bad || (m > 5 && a > 7)) break;
            bad = check(G, 128, m) || check(G, 256, m);
            for (int v = 0; v < 12 && !bad; v++)
                bad = check_tiles(G, v & 1 ? 8 : 4, v < 4 ? 1 : (v < 8 ? 3 : 1000), v & 2, m);
        }
        if (bad) {
            std::printf("case %d %d %d %d %d %d\n", c.inx, c.iny, c.nz, c.mnx, c.mny, c.ia);
            return 1;
        }
    }
    std::printf("ok\n");
    return 0;
}
