// tmx_kernels.cu -- sm_100a kernels of the plain FP64 form (bit-exact with
// the reference) and the FP64 reductions over the macroscopic fields.  This
// translation unit is compiled with --fmad=false: every multiply and add is
// rounded separately, as in the reference's x86-64 build; the only fused
// operations are the explicit __fma_rn of the correctly rounded constant
// divisions (tmx_device.cuh).  The step itself is in tmx_engine.cuh.
#include "tmx_engine.cuh"
#include "tmx_run64.cuh"

namespace tmx {

TMX_DEFINE_INIT_KERNEL(F64, f64)

// The FP64 step (tmx_run64.cuh): the runs, and the edge and corner nodes, a
// warp each, which the warps take while their block's first run is on its way
// (on a small mixer the blocks without a run take them).
template <int NT>
__device__ __forceinline__ void run_step(const StepPtrs& X, const Geom& G, const Phys& P, int write_macro,
                                         const int4* __restrict__ runs, int nruns, const int* __restrict__ enode,
                                         const unsigned char* __restrict__ ecls, int ne, int* __restrict__ counters,
                                         int parity, int* error, RunShared<NT>& S)
{
    const int warp = threadIdx.x >> 5, nb = gridDim.x;
    const auto ready = [&] {
        step_wait();
        if (blockIdx.x == 0 && threadIdx.x == 0) counters[1 - parity] = 0;  // the next step's
    };
    step_begin();
    run_loop<NT>([&](const int4&) { return run_view(X, G, P); }, runs, nruns, blockIdx.x, nb, counters + parity,
                 write_macro, S, error, ready, [&] {
                     // the blocks without a run first
                     const int at = (int)(blockIdx.x + nb - nruns % nb) % nb;
                     for (int e = at * (NT / 32) + warp; e < ne; e += nb * (NT / 32))
                         run_edge(X, G, P, write_macro, enode[e], ecls[e], S.edge[warp]);
                 });
}
#define TMX_DEFINE_RUN(NT)                                                                                      \
    __global__ void __launch_bounds__(NT, 512 / NT) k_run##NT##_f64(                                            \
        const __grid_constant__ StepPtrs X, const __grid_constant__ Geom G, const __grid_constant__ Phys P,     \
        int write_macro, const int4* __restrict__ runs, int nruns, const int* __restrict__ enode,               \
        const unsigned char* __restrict__ ecls, int ne, int* __restrict__ counters, int parity, int* error)     \
    {                                                                                                           \
        extern __shared__ __align__(16) unsigned char run_smem[];                                               \
        run_step<NT>(X, G, P, write_macro, runs, nruns, enode, ecls, ne, counters, parity, error,               \
                     *(RunShared<NT>*)run_smem);                                                                \
    }
TMX_DEFINE_RUN(128)
TMX_DEFINE_RUN(256)

// The FP64 step of a batch: the runs and edges of every mixer in one launch;
// counts[4] runs, counts[2] edge entries, counts[5 + parity] hands out the runs.
// what: 1 the runs, 2 the edges, 3 both.
__global__ void __launch_bounds__(kRunBatchThreads, 512 / kRunBatchThreads) k_run_batch_f64(
    const MixerDesc* __restrict__ D, const int4* __restrict__ runs, const int2* __restrict__ edges,
    int* __restrict__ counts, int parity, int write_macro, int what, int* error)
{
    constexpr int NT = kRunBatchThreads;
    extern __shared__ __align__(16) unsigned char run_smem[];
    RunShared<NT>& S = *(RunShared<NT>*)run_smem;
    const int warp = threadIdx.x >> 5, nb = gridDim.x;
    const int nruns = what & 1 ? counts[4] : 0, ne = what & 2 ? counts[2] : 0;
    const auto ready = [&] {
        step_wait();
        if (blockIdx.x == 0 && threadIdx.x == 0) counts[5 + (1 - parity)] = 0;  // the next step's
    };
    step_begin();
    run_loop<NT>(
        [&](const int4& t) {
            const MixerDesc& d = D[run_mixer(t)];
            return run_view(d.X[parity], d.G, d.P);
        },
        runs, nruns, blockIdx.x, nb, counts + 5 + parity, write_macro, S, error, ready, [&] {
            const int at = (int)(blockIdx.x + nb - nruns % nb) % nb;
            for (int e = at * (NT / 32) + warp; e < ne; e += nb * (NT / 32)) {
                const int2 t = edges[e];
                if (t.x < 0) continue;
                const MixerDesc& d = D[t.y >> 8];
                run_edge(d.X[parity], d.G, d.P, write_macro, t.x, t.y & 255, S.edge[warp]);
            }
        });
}

// ---------------------------------------------------------------------------
// mixing quality (Tmixer.cpp:10161-10409): per row, per species, the sums of
// the reference in its order (k inner, i outer), then per-row maxima.  Rows:
// mixing 1..mny, then inlet 1..iny over x = ia..ib.  One block per row, kRowPart
// threads per species: a thread sums a column over k, the part's first thread
// the columns in order.  (One thread per species took 130 us for the W=32
// mixer, waiting for a value at a time; now 12 us.)
// ---------------------------------------------------------------------------
struct RowShared {
    double col[3][kRowPart], mx[3][kRowPart], out[3][3];
};
// avg, var and max of the three species of a row in S.out[s] (for all threads)
__device__ __forceinline__ void row_stats(const double* __restrict__ Mac, const Geom& G, int row, RowShared& S)
{
    const int b = row < G.mny ? 1 : 0;
    const int j = b == 1 ? row + 1 : row - G.mny + 1;
    const int i0 = b == 1 ? 1 : G.ia, i1 = b == 1 ? G.mnx : G.ib;
    const int s = threadIdx.x / kRowPart, t = threadIdx.x % kRowPart;
    const double* cfield = Mac + (long long)(4 + s) * G.ps;
    const long long plane = (long long)box_nx(G, b) * box_ny(G, b);
    double mx = __longlong_as_double(0xfff0000000000000ULL);  // -inf
    double avg = 0.0;
#pragma unroll 1
    for (int pass = 0; pass < 2; pass++) {
        double sumx = 0.0;
        for (int c0 = i0; c0 <= i1; c0 += kRowPart) {
            const int i = c0 + t;
            if (i <= i1) {
                const double* c = cfield + node_index(G, b, i, j, 1);
                double sumz = 0.0;
                if (pass == 0) {
#pragma unroll 8
                    for (int k = 0; k < G.nz; k++) {
                        const double v = c[k * plane];
                        sumz += v;
                        mx = fmax(mx, v);
                    }
                } else {
#pragma unroll 8
                    for (int k = 0; k < G.nz; k++) {
                        const double d = c[k * plane] - avg;
                        sumz += d * d;
                    }
                }
                S.col[s][t] = sumz;
            }
            __syncthreads();
            if (t == 0) {
                const int n = min(kRowPart, i1 - c0 + 1);
#pragma unroll 8
                for (int c = 0; c < n; c++) sumx += S.col[s][c];
            }
            __syncthreads();
        }
        if (pass == 0) {
            S.mx[s][t] = mx;
            if (t == 0) S.out[s][0] = (sumx / (1.0 * G.nz * G.mnx));
        } else if (t == 0) {
            S.out[s][1] = (1.0 / (1.0 * G.nz * G.mnx)) * sumx;
        }
        __syncthreads();
        avg = S.out[s][0];
    }
    for (int o = kRowPart / 2; o > 0; o >>= 1) {
        if (t < o) S.mx[s][t] = fmax(S.mx[s][t], S.mx[s][t + o]);
        __syncthreads();
    }
    if (t == 0) S.out[s][2] = S.mx[s][0];
    __syncthreads();
}

__global__ void __launch_bounds__(3 * kRowPart) k_mixing_rows(const double* __restrict__ Mac, Geom G,
                                                              double* __restrict__ stats)
{
    __shared__ RowShared S;
    row_stats(Mac, G, blockIdx.x, S);
    if (threadIdx.x < 9) stats[blockIdx.x * 9 + threadIdx.x] = S.out[threadIdx.x % 3][threadIdx.x / 3];
}

// Outlet row (mixing row 1, the first row of the reference's order) of batch
// mixers: its running maximum is max(0, the row's maximum).  One block per
// entry.
__global__ void __launch_bounds__(3 * kRowPart) k_outlet_im_batch(const MixerDesc* __restrict__ D,
                                                                  const int* __restrict__ slots, int n,
                                                                  double* __restrict__ out)
{
    __shared__ RowShared S;
    const int e = blockIdx.x, s = threadIdx.x;
    if (e >= n) return;
    const MixerDesc& d = D[slots[e]];
    row_stats(d.X[0].mac, d.G, 0, S);
    if (s >= 3) return;
    const double avg = S.out[s][0], var = S.out[s][1], m = S.out[s][2];
    double mx = 0.0;
    if (mx < m) mx = m;
    const bool ok = S.out[0][0] > 0 && S.out[1][0] > 0 && S.out[2][0] > 0;
    out[3 * e + s] = ok ? 1.0 - sqrt(var / (avg * (mx - avg))) : 0.0;
}

__global__ void k_nonfinite_batch(const MixerDesc* __restrict__ D, const int4* __restrict__ blocks,
                                  const int* __restrict__ counts, int* __restrict__ flags)
{
    const int nblk = counts[0];
    for (int b = blockIdx.x; b < nblk; b += gridDim.x) {
        const int4 cb = blocks[b];
        const MixerDesc& d = D[cb.x];
        const double* mac = d.X[0].mac;
        const long long ps = d.G.ps;
        bool bad = false;
        for (int t = threadIdx.x; t < cb.z; t += blockDim.x)
            for (int f = 0; f < 7; f++) bad |= !isfinite(mac[f * ps + cb.y + t]);
        if (__syncthreads_or(bad) && threadIdx.x == 0) atomicOr(&flags[cb.x], 1);
    }
}

// ---------------------------------------------------------------------------
// The rectangular-duct series of GenerateInletVelocity (Tmixer.cpp:1426-1480)
// on the device, for the reduced-precision forms: raw[(j+1)*(nz+3) + k+1] =
// sum over m, n = 1..100 of (1 - cos m pi)(1 - cos n pi) sin(m pi j / (2 AR d))
// sin(n pi k / (2 d)) / (m n (m^2 + AR^2 n^2)), j < iny, k < nz.  The factors
// (1 - cos m pi) are exactly 0 for even m and 2 for odd m, so only odd m and n
// are summed, with sinpi for the sines.  Agrees with the host's libm series to
// about 1e-15 relative (the FP64 form keeps the host series, bit for bit).
// ---------------------------------------------------------------------------
__global__ void k_inlet_series(int iny, int nz, double* __restrict__ raw)
{
    const double d = ((nz - 1.0) / 2.0), w = ((iny - 1.0) / 2.0);
    const double AR = (1.0 * w / d), AR2 = AR * AR;
    const double den_m = 2.0 * AR * d, den_n = 2.0 * d;
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < iny * nz; t += gridDim.x * blockDim.x) {
        const int j = t / nz, k = t % nz;
        double nsum = 0.0;
        for (int n = 1; n <= 100; n += 2) {
            const double sn = sinpi((n * (double)k) / den_n);
            double msum = 0.0;
            for (int m = 1; m <= 100; m += 2) {
                const double N = 4.0 * sinpi((m * (double)j) / den_m) * sn;
                const double D = (double)(m * n) * ((double)(m * m) + (AR2 * n * n));
                msum += N / D;
            }
            nsum += msum;
        }
        raw[(j + 1) * (nz + 3) + (k + 1)] = nsum;
    }
}

// ---------------------------------------------------------------------------
// Fixed device scratch of tmx_mixing_static (no allocation in that call).
// Every word the call reads is written earlier in the same call, so nothing
// in it has to start at zero.
// ---------------------------------------------------------------------------
static __device__ __align__(256) double g_mix_scratch[kMixStaticRows * (9 + 7)];

cudaError_t mixing_static_scratch(double** ptr) { return cudaGetSymbolAddress((void**)ptr, g_mix_scratch); }

// Finish the rows of write_MixingQuality() (Tmixer.cpp:10161-10409) on the
// device, with the same arithmetic as the host finish of tmx_mixing: running
// maxima over the rows in the reference's order starting at 0, then
// I_s = 1 - sqrt(var / (avg * (max - avg))).  One warp per species; lane l
// takes a contiguous chunk of rows, and a shuffle scan of the chunk maxima
// gives each chunk its running maximum on entry.  The update "if (m < v)
// m = v" from 0 keeps m = max(+0, non-NaN values), whatever the grouping, so
// the chunked scan equals the sequential one bit for bit.
__global__ void k_mixing_finish(const double* __restrict__ stats, Geom G, double* __restrict__ rows)
{
    const int q = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (q >= 3) return;
    const int nrow = G.mny + G.iny;
    const int chunk = (nrow + 31) / 32;
    const int r0 = min(lane * chunk, nrow), r1 = min(r0 + chunk, nrow);
    double m = 0.0;
    for (int r = r0; r < r1; r++) {
        const double v = stats[r * 9 + 6 + q];
        if (m < v) m = v;
    }
    for (int o = 1; o < 32; o <<= 1) {
        const double y = __shfl_up_sync(0xffffffffu, m, o);
        if (lane >= o && m < y) m = y;
    }
    double mx = __shfl_up_sync(0xffffffffu, m, 1);
    if (lane == 0) mx = 0.0;
    for (int r = r0; r < r1; r++) {
        const double* s = stats + r * 9;
        double* o = rows + r * 7;
        const bool mixing_row = r < G.mny;
        if (q == 0) o[0] = mixing_row ? r + 1 : (r - G.mny + 1) + G.mny;
        if (mx < s[6 + q]) mx = s[6 + q];
        o[1 + q] = s[q];
        const bool ok = mixing_row ? (s[0] > 0 && s[1] > 0 && s[2] > 0) : (s[0] > 0);
        o[4 + q] = ok ? 1.0 - sqrt(s[3 + q] / (s[q] * (mx - s[q]))) : 0.0;
    }
}

// ---------------------------------------------------------------------------
// Pressure and specific power (the numbers of write_Pressure_Power,
// Tmixer.cpp:9866-10027), one block per output item, each a sum in the
// reference's order: a thread takes one turn of the outer loop with its inner
// loop, the first threads add up the turns.  (One thread per item took 2.1 ms
// for the W=32 mixer and 11 ms at W=64.)  out: [0] the pressure of inlet row iny
// over the opening (p_top), [1 .. nrow] the row pressures (mixing rows 1..mny,
// inlet rows 1..iny over x = ia..ib), then inx cross-section pressures of the
// inlet box, then for each mixing row j = 2..mny-1 four rates: cross-section and
// total as the reference computes them (its x loop assigns rather than adds,
// so only column mnx-1 enters the sums over k) and the same two summed over
// every column.  Pressures are mean density / 3; rates use
// vis = (2 tau - 1) / 6 and the central differences of the velocity.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(kRowPart) k_pressure_power(const double* __restrict__ Mac, Geom G, double tau,
                                                             double* __restrict__ out)
{
    __shared__ double part[4][kRowPart];
    const int nrow = G.mny + G.iny, t = threadIdx.x, item = blockIdx.x;
    const double* rho = Mac;
    const double *ux = Mac + G.ps, *uy = Mac + 2 * G.ps, *uz = Mac + 3 * G.ps;
    const long long plane[2] = {(long long)G.inx * G.iny, (long long)G.mnx * G.mny};
    double sum = 0.0;  // thread m < 4: the sum of part m
    if (item <= nrow + G.inx) {
        // mean density of a row over its columns, or of the inlet's cross-section
        // x = i over its rows
        const bool cross = item > nrow;
        const int r = item - 1, i = item - nrow;
        const int b = !cross && item > 0 && r < G.mny ? 1 : 0;
        const int j = item == 0 ? G.iny : (b ? r + 1 : r - G.mny + 1);
        const int o0 = cross ? 1 : (b ? 1 : G.ia), o1 = cross ? G.iny : (b ? G.mnx : G.ib);
        for (int c0 = o0; c0 <= o1; c0 += kRowPart) {
            const int o = c0 + t;
            if (o <= o1) {
                const double* c = rho + (cross ? node_index(G, 0, i, o, 1) : node_index(G, b, o, j, 1));
                double sumz = 0.0;
#pragma unroll 8
                for (int k = 0; k < G.nz; k++) sumz += c[k * plane[b]];
                part[0][t] = sumz;
            }
            __syncthreads();
            if (t == 0)
                for (int c = 0; c < min(kRowPart, o1 - c0 + 1); c++) sum += part[0][c];
            __syncthreads();
        }
        if (t == 0) out[item] = (sum / (1.0 * G.nz * (cross ? G.iny : G.mnx))) / 3.0;
        return;
    }
    const int j = item - nrow - G.inx + 1;  // 2 .. mny-1
    for (int k0 = 2; k0 < G.nz; k0 += kRowPart) {
        const int k = k0 + t;
        if (k < G.nz) {
            double sx = 0.0, stx = 0.0, allx = 0.0, alltx = 0.0;
            for (int i = 2; i < G.mnx; i++) {
#define TMX_M(a, ii, jj, kk) a[node_index(G, 1, ii, jj, kk)]
                const double delux = (TMX_M(ux, i + 1, j, k) - TMX_M(ux, i - 1, j, k)) / 2.0;
                const double delvy = (TMX_M(uy, i, j + 1, k) - TMX_M(uy, i, j - 1, k)) / 2.0;
                const double delwz = (TMX_M(uz, i, j, k + 1) - TMX_M(uz, i, j, k - 1)) / 2.0;
                const double deluy = (TMX_M(ux, i, j + 1, k) - TMX_M(ux, i, j - 1, k)) / 2.0;
                const double delvx = (TMX_M(uy, i + 1, j, k) - TMX_M(uy, i - 1, j, k)) / 2.0;
                const double deluz = (TMX_M(ux, i, j, k + 1) - TMX_M(ux, i, j, k - 1)) / 2.0;
                const double delwx = (TMX_M(uz, i + 1, j, k) - TMX_M(uz, i - 1, j, k)) / 2.0;
                const double delvz = (TMX_M(uy, i, j, k + 1) - TMX_M(uy, i, j, k - 1)) / 2.0;
                const double delwy = (TMX_M(uz, i, j + 1, k) - TMX_M(uz, i, j - 1, k)) / 2.0;
#undef TMX_M
                const double a = deluz + delwx, bxy = delvx + deluy, c = delvz + delwy;
                sx = delux * delux + delwz * delwz + 0.5 * (a * a);
                stx = delux * delux + delvy * delvy + delwz * delwz + 0.5 * (bxy * bxy) + 0.5 * (a * a) + 0.5 * (c * c);
                allx += sx;
                alltx += stx;
            }
            part[0][t] = sx;
            part[1][t] = stx;
            part[2][t] = allx;
            part[3][t] = alltx;
        }
        __syncthreads();
        if (t < 4)
            for (int c = 0; c < min(kRowPart, G.nz - k0); c++) sum += part[t][c];
        __syncthreads();
    }
    if (t < 4) {
        const double vis = ((2.0 * tau - 1.0) / 6.0) * (1.0 * 1.0 * 1.0);
        const double n = 1.0 * (G.nz - 2) * (G.mnx - 2);
        out[1 + nrow + G.inx + 4 * (j - 2) + t] = 2.0 * vis * (sum / n);
    }
}

// ---------------------------------------------------------------------------
// One field of a box (x fastest) in the reference's [i][j][k] order (z
// fastest), in 32 x 32 tiles of one row y through shared memory, for the copy to
// the host.  (Transposed by the host after the copy, a field of 4.2M nodes took
// 18 ms; here 20 us before the copy's 1.6 ms.)
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(256) k_box_ijk(const double* __restrict__ src, int nx, int ny, int nz,
                                                 double* __restrict__ dst)
{
    __shared__ double tile[32][33];
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5, tilesx = (nx + 31) / 32, tilesz = (nz + 31) / 32;
    const long long n = (long long)tilesx * tilesz * ny;
    for (long long t = blockIdx.x; t < n; t += gridDim.x) {
        const int i0 = (int)(t % tilesx) * 32, k0 = (int)(t / tilesx % tilesz) * 32, j = (int)(t / tilesx / tilesz);
        for (int k = ty; k < 32; k += 8)
            if (i0 + tx < nx && k0 + k < nz) tile[k][tx] = src[((long long)(k0 + k) * ny + j) * nx + i0 + tx];
        __syncthreads();
        for (int i = ty; i < 32; i += 8)
            if (i0 + i < nx && k0 + tx < nz) dst[((long long)(i0 + i) * ny + j) * nz + k0 + tx] = tile[tx][i];
        __syncthreads();
    }
}

// ---------------------------------------------------------------------------
// FP64 totals: warp-shuffle block reduction, one partial per block
// ---------------------------------------------------------------------------
__global__ void k_sums(const double* __restrict__ Mac, Geom G, double* __restrict__ partial)
{
    double acc[6] = {0, 0, 0, 0, 0, 0};
    for (int g = blockIdx.x * blockDim.x + threadIdx.x; g < G.nnodes; g += gridDim.x * blockDim.x) {
        const double r = Mac[g], a = Mac[4 * G.ps + g], b2 = Mac[5 * G.ps + g], c3 = Mac[6 * G.ps + g];
        acc[0] += r;
        acc[1] += a;
        acc[2] += b2;
        acc[3] += c3;
        int b, i, j, k;
        decode(G, g, b, i, j, k);
        if (b == 1 && j == 1) acc[4] += r * Mac[2 * G.ps + g];
        const double uxv = Mac[G.ps + g], uyv = Mac[2 * G.ps + g], uzv = Mac[3 * G.ps + g];
        if (!isfinite(r) || !isfinite(a) || !isfinite(b2) || !isfinite(c3) || !isfinite(uxv) || !isfinite(uyv) ||
            !isfinite(uzv))
            acc[5] += 1.0;
    }
    __shared__ double sh[6][32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
    for (int m = 0; m < 6; m++) {
        double v = acc[m];
        for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
        if (lane == 0) sh[m][w] = v;
    }
    __syncthreads();
    if (w == 0) {
        const int nw = blockDim.x >> 5;
#pragma unroll
        for (int m = 0; m < 6; m++) {
            double v = lane < nw ? sh[m][lane] : 0.0;
            for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
            if (lane == 0) partial[blockIdx.x * 6 + m] = v;
        }
    }
}

}  // namespace tmx
