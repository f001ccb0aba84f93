// tmx_api.cu -- host side of the C ABI declared in include/tmx.h.
//
// Owns the device state of one T-mixer solve: two population buffers (A-B
// pull), two density buffers (previous / current step, read by boundary
// closures), the macroscopic fields of the last step, the compact boundary
// node list and the inlet profiles.  Kernels are in tmx_kernels.cu.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <mutex>
#include <string>
#include <thread>
#include <vector>

#include "../../include/tmx.h"
#include "tmx_classes.h"
#include "tmx_host.h"
#include "tmx_kernels.cuh"

using tmx::Geom;
using tmx::Phys;
using namespace tmx_host;

namespace tmx_host {

thread_local std::string g_err;

const char* last_error() { return g_err.c_str(); }

int fail(int code, const char* fmt, ...)
{
    char buf[512];
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(buf, sizeof buf, fmt, ap);
    va_end(ap);
    g_err = buf;
    return code;
}

}  // namespace tmx_host

struct tmx_handle {
    tmx_case c;
    Geom G;
    Phys P;
    int device = 0;
    cudaStream_t stream = nullptr;
    // populations (storage type of the form) and densities (its arithmetic type)
    void* pop[2] = {nullptr, nullptr};
    void* rho[2] = {nullptr, nullptr};
    double* mac = nullptr;
    int* bnode = nullptr;
    unsigned char* bcls = nullptr;
    int nb = 0;
    void* uin_d[2] = {nullptr, nullptr};
    float4* mom[2] = {nullptr, nullptr};  // FP16 form: moments of the nodes that wrote pop[s]
    double* stats = nullptr;
    double* partial = nullptr;
    double* diag = nullptr;  // pressure / power outputs (allocated on first use)
    std::vector<double> uin1, uin2;
    std::vector<int> class_count;
    int cur = 0;   // population buffer holding the state
    int rcur = 0;  // density buffer holding the previous step's densities
    long long steps = 0;
    bool inited = false;
    long long bytes = 0;
    int bulk_blocks = 0;
    // FP16: the face and edge kernels run on these beside the interior kernel
    // (disjoint outputs, read-only shared inputs)
    cudaStream_t aux = nullptr, aux2 = nullptr;
    cudaEvent_t fork = nullptr, join = nullptr, join2 = nullptr;
    int nface = 0;  // the first nface boundary nodes are face classes
    // the last nswept faces are those that the sweep kernels update
    // (boundary_list)
    int nswept = 0;
    // FP64 and FP32 forms: the run list and grid of the run kernel, its two run
    // counters
    int4* runs = nullptr;
    int nruns = 0, run_slots = 0, run_nt = 256;
    int* counters = nullptr;
    int* error = nullptr;  // mapped host memory: set by a kernel whose copies did not arrive
    // one captured step per (state buffer, macroscopic output) combination
    cudaGraphExec_t graph[2][2] = {{nullptr, nullptr}, {nullptr, nullptr}};
    // ... and kGraphSteps of them by state buffer
    cudaGraphExec_t graph_many[2] = {nullptr, nullptr};
    int singles = 0;  // steps launched one by one (graph_length)
    int sbytes = 8, tbytes = 8;  // storage / arithmetic bytes per value of the form
    const struct StepKernels* K = nullptr;
    // interior kernel shape (tmx_set_shape): TMX_SHAPE_*, planes per tile,
    // and the sweep kernels' tile list and grid
    int shape = TMX_SHAPE_FLAT, zchunk = 8;
    int4* tiles = nullptr;
    int ntiles = 0, sweep_slots = 0;  // tiles, and blocks of their kernel that the GPU holds at once
};

const StepKernels tmx_host::kForms[3] = {
    {tmx::k_init_f64, nullptr, nullptr, nullptr, {tmx::k_run128_f64, tmx::k_run256_f64}, tmx::run_smem_host, 8, 8,
     false},
    {tmx::k_init_f32, nullptr, nullptr, nullptr, {tmx::k_run128_f32, tmx::k_run128_f32}, tmx::run32_smem_host, 4, 4,
     false},
    {tmx::k_init_f16, tmx::k_bulk_f16, tmx::k_bfaces_f16, tmx::k_bedges_f16, {nullptr, nullptr}, nullptr, 2, 4,
     true},
};

namespace tmx_host {

// The FP16 form's equilibrium polynomial (tmx_engine.cuh poly_q_rn), in host
// single precision with every operation rounded on its own.
float poly_q_host(int q, float ux, float uy, float uz, float omt)
{
    const int ex = tmx::EX(q), ey = tmx::EY(q), ez = tmx::EZ(q);
    if (q == 0) return omt;
    const float a = ex > 0 ? ux : -ux, b = ey > 0 ? uy : -uy, c = ez > 0 ? uz : -uz;
    const float eu = ex ? (ey ? a + b : (ez ? a + c : a)) : (ey ? (ez ? b + c : b) : c);
    return std::fmaf(eu, std::fmaf(4.5f, eu, 3.0f), omt);
}

// IEEE binary16 bits to float (host side of tmx_populations)
float half_bits_to_float(unsigned short h)
{
    const unsigned sign = (h >> 15) & 1u, exp = (h >> 10) & 31u, man = h & 1023u;
    float v;
    if (exp == 0) v = std::ldexp((float)man, -24);
    else if (exp == 31) v = man ? NAN : INFINITY;
    else v = std::ldexp((float)(man | 1024u), (int)exp - 25);
    return sign ? -v : v;
}

void geometry_of(const tmx_case& c, Geom& G)
{
    G.inx = c.inx;
    G.iny = c.iny;
    G.nz = c.nz;
    G.mnx = c.mnx;
    G.mny = c.mny;
    G.ia = c.ia;
    G.ib = c.ia + c.mnx - 1;
    G.nx[0] = c.inx;
    G.ny[0] = c.iny;
    G.nx[1] = c.mnx;
    G.ny[1] = c.mny;
    G.base[0] = 0;
    G.base[1] = c.inx * c.iny * c.nz;
    G.nnodes = G.base[1] + c.mnx * c.mny * c.nz;
    G.ps = ((long long)G.nnodes + 63) / 64 * 64;
}

void physics_of(const tmx_case& c, Phys& P)
{
    const double taus[4] = {c.tau, c.tau_a, c.tau_b, c.tau_c};
    for (int f = 0; f < 4; f++) {
        P.c1[f] = (1.0 - 1.0 / taus[f]);  // Tmixer.cpp:9677 "(1.0 - 1.0 / tau)"
        P.c2[f] = (1.0 / taus[f]);
    }
    P.rateconst = c.rateconst;
    P.rho_out = c.rho_out;
    for (int s = 0; s < 3; s++)
        for (int n = 0; n < 2; n++) P.cin[s][n] = c.c_in[s][n];
}

long long footprint(const Geom& G, long long nb, int precision)
{
    const StepKernels& K = kForms[precision];
    long long b = 0;
    b += 2LL * 76 * G.ps * K.sbytes;  // populations
    b += 2LL * 4 * G.ps * K.tbytes;   // densities
    if (K.moments) b += 2LL * 2 * G.ps * 16;  // FP16 form: moments
    b += 7LL * G.ps * 8;       // macroscopic fields
    b += nb * 5;               // boundary list
    b += 2LL * (G.iny + 3) * (G.nz + 3) * K.tbytes;
    b += (long long)(G.mny + G.iny) * 9 * 8 + kSumBlocks * 6 * 8;
    return b;
}

long long boundary_count(const Geom& G)
{
    long long n = 0;
    for (int b = 0; b < 2; b++)
        for (int i = 1; i <= G.nx[b]; i++)
            for (int j = 1; j <= G.ny[b]; j++)
                for (int k = 1; k <= G.nz; k++) n += tmx::is_boundary(G, b, i, j, k);
    return n;
}

// Class of a boundary node, following the node sets of the reference's cases
// (Tmixer.cpp:2023-9033).  Returns -1 for a node no case covers.
int classify(const Geom& G, int b, int i, int j, int k)
{
    using namespace tmx;
    const int nz = G.nz;
    const bool zlo = k == 1, zhi = k == nz, zmid = !zlo && !zhi;
    if (b == 0) {
        const int inx = G.inx, iny = G.iny, ia = G.ia, ib = G.ib;
        const bool ylo = j == 1, yhi = j == iny, ymid = !ylo && !yhi;
        if (i == 1 || i == inx) {
            const bool lo = i == 1;
            if (ylo) return zlo ? (lo ? K_CORNER_1 + 6 : K_CORNER_1 + 7) : zhi ? (lo ? K_CORNER_1 + 2 : K_CORNER_1 + 3)
                                                                              : (lo ? K_EDGE_X1_Y1 : K_EDGE_XT_Y1);
            if (yhi) return zlo ? (lo ? K_CORNER_1 + 4 : K_CORNER_1 + 5) : zhi ? (lo ? K_CORNER_1 + 0 : K_CORNER_1 + 1)
                                                                              : (lo ? K_EDGE_X1_YT : K_EDGE_XT_YT);
            return zlo ? (lo ? K_EDGE_X1_Z1 : K_EDGE_XT_Z1) : zhi ? (lo ? K_EDGE_X1_ZTOP : K_EDGE_XT_ZTOP)
                                                                 : (lo ? K_INLET1 : K_INLET2);
        }
        if (yhi) return zlo ? K_EDGE_YT_Z1 : zhi ? K_EDGE_YT_ZT : K_FACE_YT;
        if (ylo) {
            if (i < ia || i > ib) return zlo ? K_EDGE_Y1_Z1 : zhi ? K_EDGE_Y1_ZTOP : K_FACE_Y1;
            if (i == ia) return zlo ? K_CORNER_1 + 15 : zhi ? K_CORNER_1 + 12 : K_JUNC_DD;
            if (i == ib) return zlo ? K_CORNER_1 + 14 : zhi ? K_CORNER_1 + 13 : K_JUNC_CC;
            return zlo ? K_FACE_Z1 : zhi ? K_FACE_ZT : -1;  // opening nodes of Cases 19 / 17
        }
        (void)ymid;
        if (zlo) return K_FACE_Z1;
        if (zhi) return K_FACE_ZT;
        return -1;
    }
    const int mnx = G.mnx;
    const bool xlo = i == 1, xhi = i == mnx;
    if (j == 1) {
        if (xlo) return zlo ? K_CORNER_1 + 8 : zhi ? K_CORNER_1 + 10 : K_MEDGE_AAp;
        if (xhi) return zlo ? K_CORNER_1 + 9 : zhi ? K_CORNER_1 + 11 : K_MEDGE_BBp;
        return zlo ? K_MEDGE_AB : zhi ? K_MEDGE_ApBp : K_OUTLET;
    }
    if (xlo) return zlo ? K_MEDGE_AD : zhi ? K_MEDGE_ApDp : K_FACE_MX1;
    if (xhi) return zlo ? K_MEDGE_BC : zhi ? K_MEDGE_BpCp : K_FACE_MXT;
    if (zlo) return K_FACE_Z1;
    if (zhi) return K_FACE_ZT;
    (void)zmid;
    return -1;
}

// Inlet profiles exactly as GenerateInletVelocity() (Tmixer.cpp:1426-1539)
// computes them: a rectangular-duct series (100 x 100 terms, libm sin/cos,
// the same loop nesting and operation order), scaled to mean umean, then
// shifted one node down in z (Uin1) and, negated, one node up (Uin2), with
// Uin1[.][1] and Uin2[.][nz] zeroed.
void inlet_series(int iny, int nz, std::vector<double>& U1, double& average)
{
    const int W = nz + 3;
    U1.assign((size_t)(iny + 3) * W, 0.0);
    auto at = [W](std::vector<double>& a, int j, int k) -> double& { return a[(size_t)j * W + k]; };
    const double pi = 3.14159265358979323846;
    const double d = ((nz - 1.0) / 2.0);
    const double w = ((iny - 1.0) / 2.0);
    const double AR = (1.0 * w / d);
    const double den_m = 2.0 * AR * d, den_n = 2.0 * d, AR2 = AR * AR;
    // every (j, k) is an independent sum: rows are spread over host threads,
    // each value computed exactly as a single thread would
    auto rows = [&](int j0, int j1) {
        for (int j = j0; j < j1; j++)
            for (int k = 0; k < nz; k++) {
                double nsum = 0;
                for (int n = 1; n <= 100; n++) {
                    double msum = 0;
                    for (int m = 1; m <= 100; m++) {
                        const double N = (1.0 - std::cos(m * pi)) * (1.0 - std::cos(n * pi)) *
                                         std::sin(((m * pi) / den_m) * (j)) * std::sin(((n * pi) / den_n) * (k));
                        const double D = m * n * ((m * m) + (AR2 * n * n));
                        msum += (N / D);
                    }
                    nsum += msum;
                }
                at(U1, j + 1, k + 1) = nsum;
            }
    };
    const int nt = std::max(1, std::min((int)std::thread::hardware_concurrency(), iny));
    std::vector<std::thread> pool;
    for (int t = 1; t < nt; t++) pool.emplace_back(rows, iny * t / nt, iny * (t + 1) / nt);
    rows(0, iny / nt);
    for (auto& th : pool) th.join();
    double sum = 0;
    for (int i = 1; i <= iny; i++)
        for (int j = 1; j <= nz; j++) sum += at(U1, i, j);
    average = sum / ((iny) * (nz));
}

void inlet_scale(const tmx_case& c, const std::vector<double>& raw, double average, std::vector<double>& U1,
                 std::vector<double>& U2)
{
    const int iny = c.iny, nz = c.nz, W = nz + 3;
    U1 = raw;
    U2.assign((size_t)(iny + 3) * W, 0.0);
    auto at = [W](std::vector<double>& a, int j, int k) -> double& { return a[(size_t)j * W + k]; };
    for (int i = 1; i <= iny; i++)
        for (int j = 1; j <= nz; j++) at(U1, i, j) = at(U1, i, j) * (c.umean / average);
    for (int j = 0; j < iny; j++)
        for (int k = 0; k < nz; k++) {
            at(U1, j + 1, k) = at(U1, j + 1, k + 1);
            at(U2, j + 1, k + 2) = -at(U1, j + 1, k);
        }
    for (int i = 1; i <= iny; i++) {
        at(U1, i, 1) = 0;
        at(U2, i, nz) = 0;
    }
}

int inlet_series_device(int iny, int nz, cudaStream_t stream, std::vector<double>& raw, double& average)
{
    const size_t n = (size_t)(iny + 3) * (nz + 3);
    double* d = nullptr;
    TMX_CK(cudaMalloc((void**)&d, n * sizeof(double)));
    cudaError_t e = cudaMemsetAsync(d, 0, n * sizeof(double), stream);
    if (e == cudaSuccess) {
        tmx::k_inlet_series<<<std::max(1, std::min((iny * nz + 127) / 128, 1024)), 128, 0, stream>>>(iny, nz, d);
        e = cudaGetLastError();
    }
    raw.assign(n, 0.0);
    if (e == cudaSuccess) e = cudaMemcpyAsync(raw.data(), d, n * sizeof(double), cudaMemcpyDeviceToHost, stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(stream);
    cudaFree(d);
    TMX_CK(e);
    const int W = nz + 3;
    double sum = 0;
    for (int i = 1; i <= iny; i++)
        for (int j = 1; j <= nz; j++) sum += raw[(size_t)i * W + j];
    average = sum / ((iny) * (nz));
    return TMX_OK;
}

int inlet_profile_form(const tmx_case& c, cudaStream_t stream, std::vector<double>& U1, std::vector<double>& U2)
{
    if (c.precision == TMX_FP64) {
        inlet_profile(c, U1, U2);
        return TMX_OK;
    }
    std::vector<double> raw;
    double average;
    int rc = inlet_series_device(c.iny, c.nz, stream, raw, average);
    if (rc) return rc;
    inlet_scale(c, raw, average, U1, U2);
    return TMX_OK;
}

void inlet_profile(const tmx_case& c, std::vector<double>& U1, std::vector<double>& U2)
{
    std::vector<double> raw;
    double average;
    inlet_series(c.iny, c.nz, raw, average);
    inlet_scale(c, raw, average, U1, U2);
}

int boundary_list(const Geom& G, std::vector<int>& nodes, std::vector<unsigned char>& cls, int& nface,
                  std::vector<int>* class_count, int* nswept)
{
    struct Entry {
        int cls, node;
        bool swept;
    };
    std::vector<Entry> all;
    all.reserve((size_t)boundary_count(G));
    if (class_count) class_count->assign(tmx::K_NCLASSES, 0);
    bool zsep = nswept != nullptr;
    long long zcount = 0, interior2 = 0;
    for (int b = 0; b < 2; b++)
        for (int i = 1; i <= G.nx[b]; i++)
            for (int j = 1; j <= G.ny[b]; j++) {
                if (G.nz >= 3 && !tmx::is_boundary(G, b, i, j, 2)) interior2++;
                for (int k = 1; k <= G.nz; k++) {
                    if (!tmx::is_boundary(G, b, i, j, k)) continue;
                    const int c = classify(G, b, i, j, k);
                    if (c < 0)
                        return fail(TMX_E_INVALID, "internal: boundary node (%d,%d,%d,%d) has no class", b, i, j, k);
                    if (class_count) (*class_count)[c]++;
                    const bool zw = c == tmx::K_FACE_Z1 || c == tmx::K_FACE_ZT;
                    if (zw) {
                        // the interior node of the column the sweep kernels
                        // update this wall node with (zwall_node)
                        const int kw = c == tmx::K_FACE_Z1 ? 1 : G.nz, kn = c == tmx::K_FACE_Z1 ? 2 : G.nz - 1;
                        if (k != kw || G.nz < 3 || tmx::is_boundary(G, b, i, j, kn)) zsep = false;
                        zcount++;
                    }
                    const bool end = c == tmx::K_INLET1 || c == tmx::K_INLET2 || c == tmx::K_FACE_MX1 || c == tmx::K_FACE_MXT;
                    all.push_back({c, tmx::node_index(G, b, i, j, k), zw || end});
                }
            }
    // every z wall node above or below an interior node, and every interior
    // node of planes 2 and nz - 1 under or over one
    if (zcount != 2 * interior2) zsep = false;
    if (nswept && !zsep && interior2 > 0)
        return fail(TMX_E_INVALID, "internal: the z wall faces do not pair with the interior nodes of planes 2 and %d",
                    G.nz - 1);
    // faces first (with zsep the swept ones last among them), then edges
    // and corners; by class, then node
    std::vector<std::pair<int, int>> bl;
    bl.reserve(all.size());
    for (const Entry& e : all)
        bl.emplace_back((tmx::is_face_class(e.cls) ? (zsep && e.swept ? 128 : 0) : 256) + e.cls, e.node);
    std::sort(bl.begin(), bl.end());
    nodes.resize(bl.size());
    cls.resize(bl.size());
    nface = 0;
    int nzw = 0;
    for (size_t t = 0; t < bl.size(); t++) {
        nodes[t] = bl[t].second;
        cls[t] = (unsigned char)(bl[t].first & 127);
        if (bl[t].first < 256) nface++;
        if (bl[t].first >= 128 && bl[t].first < 256) nzw++;
    }
    if (nswept) *nswept = nzw;
    return TMX_OK;
}

int box_to_host(const Geom& G, int box, const double* dev, double* scratch, cudaStream_t stream, double* host_out)
{
    const int nx = G.nx[box], ny = G.ny[box], nz = G.nz;
    const long long tiles = (long long)((nx + 31) / 32) * ((nz + 31) / 32) * ny;
    tmx::k_box_ijk<<<(int)std::min(tiles, 148LL * 8), 256, 0, stream>>>(dev, nx, ny, nz, scratch);
    TMX_CK(cudaGetLastError());
    TMX_CK(cudaMemcpyAsync(host_out, scratch, (size_t)nx * ny * nz * sizeof(double), cudaMemcpyDeviceToHost, stream));
    TMX_CK(cudaStreamSynchronize(stream));
    return TMX_OK;
}

// The flags lie in one page of the process, mapped when the first is taken
// (mapping memory takes about a millisecond, a handle's creation two); beyond
// its 1024 a flag is mapped by itself.
namespace {
constexpr int kFlags = 1024;
std::mutex g_flag_mu;
int* g_flags = nullptr;
bool g_flag_used[kFlags];
}  // namespace

int* error_flag_take()
{
    std::lock_guard<std::mutex> lk(g_flag_mu);
    const unsigned how = cudaHostAllocMapped | cudaHostAllocPortable;
    if (!g_flags && cudaHostAlloc((void**)&g_flags, kFlags * sizeof(int), how) != cudaSuccess) {
        g_flags = nullptr;
        cudaGetLastError();
        return nullptr;
    }
    for (int i = 0; i < kFlags; i++)
        if (!g_flag_used[i]) {
            g_flag_used[i] = true;
            g_flags[i] = 0;
            return g_flags + i;
        }
    int* f = nullptr;
    if (cudaHostAlloc((void**)&f, sizeof(int), how) != cudaSuccess) {
        cudaGetLastError();
        return nullptr;
    }
    *f = 0;
    return f;
}

void error_flag_give(int* flag)
{
    if (!flag) return;
    std::lock_guard<std::mutex> lk(g_flag_mu);
    if (flag >= g_flags && flag < g_flags + kFlags) g_flag_used[flag - g_flags] = false;
    else cudaFreeHost(flag);
}

}  // namespace tmx_host

namespace {

// cudaMemcpy from pageable memory may return before the last of it has arrived, and
// a handle's stream does not wait for such copies: a call whose copies a step
// reads ends with this.
cudaError_t copies_arrived() { return cudaStreamSynchronize(cudaStreamLegacy); }

void drop_graphs(tmx_handle* h)
{
    cudaGraphExec_t* all[6] = {&h->graph[0][0], &h->graph[0][1],   &h->graph[1][0],
                               &h->graph[1][1], &h->graph_many[0], &h->graph_many[1]};
    for (cudaGraphExec_t* g : all)
        if (*g) {
            cudaGraphExecDestroy(*g);
            *g = nullptr;
        }
}

void free_all(tmx_handle* h)
{
    for (int s = 0; s < 2; s++) {
        cudaFree(h->pop[s]);
        cudaFree(h->rho[s]);
        cudaFree(h->uin_d[s]);
        cudaFree(h->mom[s]);
        h->pop[s] = h->rho[s] = h->uin_d[s] = nullptr;
        h->mom[s] = nullptr;
    }
    drop_graphs(h);
    if (h->fork) cudaEventDestroy(h->fork);
    if (h->join) cudaEventDestroy(h->join);
    if (h->join2) cudaEventDestroy(h->join2);
    h->fork = h->join = h->join2 = nullptr;
    if (h->aux) cudaStreamDestroy(h->aux);
    if (h->aux2) cudaStreamDestroy(h->aux2);
    h->aux = h->aux2 = nullptr;
    cudaFree(h->mac);
    cudaFree(h->bnode);
    cudaFree(h->bcls);
    cudaFree(h->stats);
    cudaFree(h->partial);
    cudaFree(h->tiles);
    h->tiles = nullptr;
    cudaFree(h->runs);
    cudaFree(h->counters);
    error_flag_give(h->error);
    h->error = nullptr;
    h->runs = nullptr;
    h->counters = nullptr;
    cudaFree(h->diag);
    h->diag = nullptr;
    h->mac = h->stats = h->partial = nullptr;
    h->bnode = nullptr;
    h->bcls = nullptr;
    if (h->stream) cudaStreamDestroy(h->stream);
    h->stream = nullptr;
}

// The FP64 or FP32 step from buffer `cur`: one launch.  With ev (4 events) the edges
// and the runs are launched one after the other, so that each event pair times
// its part alone.  overlap: launched behind another step of the same graph.
int enqueue_run(tmx_handle* h, const tmx::StepPtrs& X, int cur, int write_macro, cudaEvent_t* ev, bool overlap)
{
    const int ne = h->nb - h->nface, nr = h->nruns;
    auto launch = [&](int nruns, int nedges) -> cudaError_t {
        const int per = h->run_nt / 32;  // a warp per edge node
        const int blocks = std::max(1, std::min(h->run_slots, (nedges + per - 1) / per + nruns));
        return launch_step(h->K->run[h->run_nt > 128], blocks, h->run_nt, h->K->run_smem(h->run_nt), h->stream, overlap,
                           X, h->G, h->P, write_macro, h->runs, nruns, h->bnode + h->nface, h->bcls + h->nface, nedges,
                           h->counters, cur, h->error);
    };
    if (ev) {
        TMX_CK(cudaEventRecord(ev[2], h->stream));
        TMX_CK(launch(0, ne));
        TMX_CK(cudaEventRecord(ev[3], h->stream));
        TMX_CK(cudaEventRecord(ev[0], h->stream));
        TMX_CK(launch(nr, 0));
        TMX_CK(cudaEventRecord(ev[1], h->stream));
    } else {
        TMX_CK(launch(nr, ne));
    }
    TMX_CK(cudaGetLastError());
    return TMX_OK;
}

// The FP16 step with the wall rows in the tiles' launch.  Where its blocks with
// the edges' fill half of the GPU at most the edges are in it too (1,000 to 22,000
// nodes 13.1 to 16.7 us a step against 16.4 to 18.3 in three kernels); else the edge
// kernel runs beside it (edges by warps of the tile kernel hold up the tiles that
// share an SM with them; in it / beside: 43,904 nodes 20.6 / 15.6 us, 65,536 19.7 /
// 18.1, 221,184 33.3 / 27.4).
int enqueue_sweep(tmx_handle* h, const SweepShape* sh, const tmx::StepPtrs& X, int write_macro, bool overlap)
{
    // the wall rows are the faces that the tiles leave, the first of the list
    const int nw = h->nface - h->nswept, ne = h->nb - h->nface, nt = sh->threads();
    const int wb = (nw + nt - 1) / nt, eb = (ne + nt / 32 - 1) / (nt / 32);
    const bool one = 2 * (h->ntiles + wb + eb) <= h->sweep_slots;
    const bool beside = !one && ne > 0;
    if (beside) {
        const int bt = tmx::kBoundaryThreadsHost, nl = tmx::kBoundaryLanesHost;
        TMX_CK(cudaEventRecord(h->fork, h->stream));
        TMX_CK(cudaStreamWaitEvent(h->aux2, h->fork, 0));
        h->K->edges<<<(nl * ne + bt - 1) / bt, bt, 0, h->aux2>>>(X, h->bnode + h->nface, h->bcls + h->nface, ne, h->G,
                                                                 h->P, write_macro);
        TMX_CK(cudaEventRecord(h->join2, h->aux2));
    }
    TMX_CK(launch_step(sh->single, h->ntiles + wb + (one ? eb : 0), nt, sh->smem(false), h->stream, one && overlap, X, h->G,
                       h->P, write_macro, h->tiles, h->ntiles, h->bnode, h->bcls, nw, h->nface, one ? ne : 0));
    if (beside) TMX_CK(cudaStreamWaitEvent(h->stream, h->join2, 0));
    TMX_CK(cudaGetLastError());
    return TMX_OK;
}

// Queue one step from buffer `cur`: the face and the edge kernel on the two
// auxiliary streams, forked from and joined back into the main stream, and the
// interior kernel on the main stream (FP64 and FP32: enqueue_run).  With ev (4
// events) each part is bracketed by its own pair of events.  The state and density
// buffers flip together every step, so one parity index selects both.
int enqueue_step(tmx_handle* h, int cur, int write_macro, cudaEvent_t* ev, bool overlap = false)
{
    const Geom& G = h->G;
    tmx::StepPtrs X;
    X.pin = h->pop[cur];
    X.pout = h->pop[1 - cur];
    X.rprev = h->rho[cur];
    X.rcur = h->rho[1 - cur];
    X.mac = h->mac;
    X.mprev = h->mom[cur];
    X.mcur = h->mom[1 - cur];
    X.uin1 = h->uin_d[0];
    X.uin2 = h->uin_d[1];
    if (h->K->run[0]) return enqueue_run(h, X, cur, write_macro, ev, overlap);
    // FP16 by up to four rounds of tiles: the wall rows with them.  Beyond, and for
    // the timed parts, a face kernel: tiles without the walls' and edges' code spill
    // less (76 B loaded back a thread against 104), and the face kernel's share
    // falls with the size.  Together / apart (each repeats to 0.2%): 0.75M nodes 75.0 /
    // 80.2 us, 1.0M 97.9 / 94.7, 1.4M 117.2 / 120.9, 1.8M 146.5 / 148.4; beyond four
    // rounds 2.2M 186.6 / 187.4, 2.8M 225.6 / 226.9, 4.2M 311.7 / 311.7, the reference
    // case's 4.9M 420.5 / 415.3.
    const SweepShape* sh = sweep_shape(h->shape);
    if (sh && !ev && h->ntiles <= 4 * h->sweep_slots) return enqueue_sweep(h, sh, X, write_macro, overlap);
    TMX_CK(cudaEventRecord(h->fork, h->stream));
    TMX_CK(cudaStreamWaitEvent(h->aux, h->fork, 0));
    TMX_CK(cudaStreamWaitEvent(h->aux2, h->fork, 0));
    if (ev) TMX_CK(cudaEventRecord(ev[2], h->aux));
    const int nf = h->nface, ne = h->nb - h->nface;
    const int bt = tmx::kBoundaryThreadsHost, nl = tmx::kBoundaryLanesHost;  // nl threads per face
    const int nfk = sh ? nf - h->nswept : nf;  // a sweep shape's tiles update the last nswept faces
    if (nfk > 0)
        h->K->faces<<<(nl * nfk + bt - 1) / bt, bt, 0, h->aux>>>(X, h->bnode, h->bcls, nfk, G, h->P, write_macro);
    if (ne > 0)
        h->K->edges<<<(nl * ne + bt - 1) / bt, bt, 0, h->aux2>>>(X, h->bnode + nf, h->bcls + nf, ne, G, h->P,
                                                                 write_macro);
    TMX_CK(cudaEventRecord(h->join2, h->aux2));
    if (ev) {  // the boundary time spans both boundary kernels
        TMX_CK(cudaStreamWaitEvent(h->aux, h->join2, 0));
        TMX_CK(cudaEventRecord(ev[3], h->aux));
    }
    TMX_CK(cudaEventRecord(h->join, h->aux));
    // The boundary kernels (64 registers) run beside the bulk kernel (FP16
    // step 75 us side by side, 85 us in order); timed steps (ev given) run it
    // after them, so that each event pair times its kernels alone.
    if (ev) {
        TMX_CK(cudaStreamWaitEvent(h->stream, h->join, 0));
        TMX_CK(cudaStreamWaitEvent(h->stream, h->join2, 0));
    }
    if (ev) TMX_CK(cudaEventRecord(ev[0], h->stream));
    if (sh)
        sh->tiles<<<h->ntiles, sh->threads(), sh->smem(false), h->stream>>>(X, G, h->P, write_macro, h->tiles, h->ntiles);
    else
        h->K->bulk<<<h->bulk_blocks, 256, 0, h->stream>>>(X, G, h->P, write_macro);
    if (ev) TMX_CK(cudaEventRecord(ev[1], h->stream));
    if (!ev) {
        TMX_CK(cudaStreamWaitEvent(h->stream, h->join, 0));
        TMX_CK(cudaStreamWaitEvent(h->stream, h->join2, 0));
    }
    TMX_CK(cudaGetLastError());
    return TMX_OK;
}

// After the stream has been waited for: whether every step's copies arrived.
int settled(const tmx_handle* h)
{
    if (h->error && *(volatile int*)h->error)
        return fail(TMX_E_CUDA, "a step gave up waiting for its copies: the state is not valid");
    return TMX_OK;
}

int advance(tmx_handle* h, int steps = 1)
{
    if (steps & 1) h->cur = 1 - h->cur;
    h->rcur = h->cur;
    h->steps += steps;
    return TMX_OK;
}

// n steps (one, or kGraphSteps without macroscopic output) through a captured
// graph, built on first use for this parity.
int graph_steps(tmx_handle* h, int n, int write_macro)
{
    cudaGraphExec_t& ex = n > 1 ? h->graph_many[h->cur] : h->graph[h->cur][write_macro];
    if (!ex) {
        cudaGraph_t gr = nullptr;
        TMX_CK(cudaStreamBeginCapture(h->stream, cudaStreamCaptureModeThreadLocal));
        int rc = TMX_OK;
        for (int s = 0; s < n && rc == TMX_OK; s++) rc = enqueue_step(h, h->cur ^ (s & 1), write_macro, nullptr, s > 0);
        cudaError_t e = cudaStreamEndCapture(h->stream, &gr);
        if (rc) {
            if (gr) cudaGraphDestroy(gr);
            return rc;
        }
        TMX_CK(e);
        e = cudaGraphInstantiate(&ex, gr, 0);
        cudaGraphDestroy(gr);
        TMX_CK(e);
    }
    TMX_CK(cudaGraphLaunch(ex, h->stream));
    return advance(h, n);
}

int timed_step(tmx_handle* h, int write_macro, cudaEvent_t* ev)
{
    int rc = enqueue_step(h, h->cur, write_macro, ev);
    if (rc) return rc;
    return advance(h);
}

}  // namespace

namespace tmx_host {

int check_case(const tmx_case& cc)
{
    const tmx_case* c = &cc;
    if (c->inx < 3 || c->iny < 3 || c->nz < 3 || c->mnx < 3 || c->mny < 3)
        return fail(TMX_E_INVALID, "every box size must be >= 3 (inx=%d iny=%d nz=%d mnx=%d mny=%d)", c->inx, c->iny,
                    c->nz, c->mnx, c->mny);
    if (c->ia < 2 || c->ia + c->mnx - 1 > c->inx - 1)
        return fail(TMX_E_INVALID, "opening columns ia=%d..ib=%d must lie within 2..inx-1=%d", c->ia,
                    c->ia + c->mnx - 1, c->inx - 1);
    const double t[4] = {c->tau, c->tau_a, c->tau_b, c->tau_c};
    for (double v : t)
        if (!(v > 0.5) || !std::isfinite(v)) return fail(TMX_E_INVALID, "relaxation times must be finite and > 0.5");
    if (!std::isfinite(c->rho0) || !(c->rho0 > 0) || !std::isfinite(c->rho_out) || !(c->rho_out > 0))
        return fail(TMX_E_INVALID, "rho0 and rho_out must be finite and positive");
    if (!std::isfinite(c->umean) || !std::isfinite(c->rateconst)) return fail(TMX_E_INVALID, "non-finite parameter");
    if (c->precision < TMX_FP64 || c->precision > TMX_FP16)
        return fail(TMX_E_INVALID, "unsupported precision %d", c->precision);
    const long long n = (long long)c->inx * c->iny * c->nz + (long long)c->mnx * c->mny * c->nz;
    if (n > 2000000000LL) return fail(TMX_E_INVALID, "too many nodes (%lld)", n);
    return TMX_OK;
}

// Two cases are the same solve: every field equal (the struct's padding
// bytes are not compared, so a case filled member by member matches one
// cleared with memset first).  Doubles compare by their bits.
static bool same_case(const tmx_case& a, const tmx_case& b)
{
    auto same = [](double x, double y) { return std::memcmp(&x, &y, sizeof x) == 0; };
    bool eq = a.inx == b.inx && a.iny == b.iny && a.nz == b.nz && a.mnx == b.mnx && a.mny == b.mny && a.ia == b.ia &&
              a.precision == b.precision && same(a.tau, b.tau) && same(a.tau_a, b.tau_a) && same(a.tau_b, b.tau_b) &&
              same(a.tau_c, b.tau_c) && same(a.rho0, b.rho0) && same(a.rho_out, b.rho_out) &&
              same(a.rateconst, b.rateconst) && same(a.umean, b.umean);
    for (int s = 0; s < 3; s++)
        for (int n = 0; n < 2; n++) eq = eq && same(a.c_in[s][n], b.c_in[s][n]);
    return eq;
}

int checkpoint_check(const void* buf, long long size, const tmx_case& c, const Geom& G)
{
    if (size < (long long)sizeof(CheckpointHeader)) return fail(TMX_E_INVALID, "checkpoint too small");
    CheckpointHeader hd;
    std::memcpy(&hd, buf, sizeof hd);
    if (std::memcmp(hd.magic, "TMXCKPT1", 8) == 0)
        return fail(TMX_E_INVALID, "checkpoint of an earlier format (FP16 moment records ordered differently)");
    if (std::memcmp(hd.magic, kCheckpointMagic, 8) != 0) return fail(TMX_E_INVALID, "not a checkpoint");
    if (hd.abi != TMX_ABI_VERSION) return fail(TMX_E_INVALID, "checkpoint of ABI %d, library %d", hd.abi, TMX_ABI_VERSION);
    if (hd.precision != c.precision)
        return fail(TMX_E_INVALID, "checkpoint of precision %d, target %d", hd.precision, c.precision);
    if (!same_case(hd.c, c)) return fail(TMX_E_INVALID, "checkpoint of a different case");
    long long b[5];
    checkpoint_sections(G, c.precision, b);
    if (hd.ps != G.ps || std::memcmp(hd.bytes, b, sizeof b) != 0 || size != checkpoint_total(b))
        return fail(TMX_E_INVALID, "checkpoint sizes do not match the case");
    if (hd.steps < 0) return fail(TMX_E_INVALID, "checkpoint with a negative step count");
    return TMX_OK;
}

}  // namespace tmx_host

extern "C" {

int tmx_abi_version(void) { return TMX_ABI_VERSION; }

const char* tmx_last_error(void) { return last_error(); }

int tmx_case_reference(tmx_case* out)
{
    if (!out) return fail(TMX_E_INVALID, "tmx_case_reference: null output");
    std::memset(out, 0, sizeof *out);
    out->inx = 401;
    out->iny = 51;
    out->nz = 51;
    out->mnx = 101;
    out->mny = 800 - 50;
    out->ia = ((401 + 1) / 2) - ((101 - 1) / 2);
    out->tau = 0.6;
    const double tc = (0.5 * (((2.0 * 0.6 - 1.0) / 3.0) + 1.0));
    out->tau_a = out->tau_b = out->tau_c = tc;
    out->rho0 = 3.0;
    out->rho_out = 3.0;
    out->c_in[0][0] = 1.0;
    out->c_in[1][1] = 1.0;
    out->rateconst = 1.0;
    out->umean = 0.059761;
    out->precision = TMX_FP64;
    return TMX_OK;
}

int tmx_case_wlayout(int W, double u_max, double tau_f, double tau_c, double k, double rho, tmx_case* out)
{
    if (!out) return fail(TMX_E_INVALID, "tmx_case_wlayout: null output");
    if (W < 3) return fail(TMX_E_INVALID, "tmx_case_wlayout: W=%d must be >= 3", W);
    if (!(u_max > 0) || !std::isfinite(u_max)) return fail(TMX_E_INVALID, "u_max must be positive");
    tmx_case c;
    std::memset(&c, 0, sizeof c);
    c.inx = 8 * W;
    c.iny = W;
    c.nz = W;
    c.mnx = 2 * W;
    c.mny = 4 * W;
    c.ia = 3 * W + 1;
    c.tau = tau_f;
    c.tau_a = c.tau_b = c.tau_c = tau_c;
    c.rho0 = rho;
    c.rho_out = rho;
    c.c_in[0][0] = 1.0;
    c.c_in[1][1] = 1.0;
    c.rateconst = k;
    c.umean = 1.0;
    c.precision = TMX_FP64;
    std::vector<double> U1, U2;
    inlet_profile(c, U1, U2);
    double mx = 0.0;
    for (double v : U1) mx = std::max(mx, v);
    if (!(mx > 0)) return fail(TMX_E_INVALID, "degenerate inlet profile");
    c.umean = u_max / mx;
    *out = c;
    return tmx_case_check(out);
}

int tmx_case_check(const tmx_case* c)
{
    if (!c) return fail(TMX_E_INVALID, "null case");
    return check_case(*c);
}


int tmx_case_footprint(const tmx_case* c, long long* bytes)
{
    int rc = tmx_case_check(c);
    if (rc) return rc;
    if (!bytes) return fail(TMX_E_INVALID, "null output");
    Geom G;
    geometry_of(*c, G);
    *bytes = footprint(G, boundary_count(G), c->precision);
    return TMX_OK;
}

int tmx_create(const tmx_case* c, int device, tmx_handle** out)
{
    if (!out) return fail(TMX_E_INVALID, "null output handle");
    *out = nullptr;
    int rc = tmx_case_check(c);
    if (rc) return rc;
    int ndev = 0;
    TMX_CK(cudaGetDeviceCount(&ndev));
    if (device < 0 || device >= ndev) return fail(TMX_E_INVALID, "device %d out of range (%d devices)", device, ndev);
    TMX_CK(cudaSetDevice(device));

    tmx_handle* h = new tmx_handle();
    h->c = *c;
    h->device = device;
    geometry_of(*c, h->G);
    physics_of(*c, h->P);
    h->K = &kForms[c->precision];
    h->sbytes = h->K->sbytes;
    h->tbytes = h->K->tbytes;
    const Geom& G = h->G;

    // boundary node list, faces first, sorted by class then node index
    std::vector<int> nodes;
    std::vector<unsigned char> cls;
    rc = boundary_list(G, nodes, cls, h->nface, &h->class_count, &h->nswept);
    if (rc) {
        delete h;
        return rc;
    }
    h->nb = (int)nodes.size();

    auto alloc = [&](void** p, size_t n) -> cudaError_t {
        cudaError_t e = cudaMalloc(p, n);
        if (e == cudaSuccess) h->bytes += (long long)n;
        return e;
    };
    cudaError_t e = cudaStreamCreateWithFlags(&h->stream, cudaStreamNonBlocking);
    if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&h->aux, cudaStreamNonBlocking);
    if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&h->aux2, cudaStreamNonBlocking);
    if (e == cudaSuccess) e = cudaEventCreateWithFlags(&h->join2, cudaEventDisableTiming);
    if (e == cudaSuccess) e = cudaEventCreateWithFlags(&h->fork, cudaEventDisableTiming);
    if (e == cudaSuccess) e = cudaEventCreateWithFlags(&h->join, cudaEventDisableTiming);
    for (int s = 0; s < 2 && e == cudaSuccess; s++) {
        e = alloc((void**)&h->pop[s], (size_t)76 * G.ps * h->sbytes);
        if (e == cudaSuccess) e = alloc((void**)&h->rho[s], (size_t)4 * G.ps * h->tbytes);
        if (e == cudaSuccess) e = alloc((void**)&h->uin_d[s], (size_t)(G.iny + 3) * (G.nz + 3) * h->tbytes);
        if (e == cudaSuccess && h->K->moments) e = alloc((void**)&h->mom[s], (size_t)2 * G.ps * sizeof(float4));
    }
    if (e == cudaSuccess) e = alloc((void**)&h->mac, (size_t)7 * G.ps * sizeof(double));
    if (e == cudaSuccess) e = alloc((void**)&h->bnode, std::max<size_t>(1, nodes.size()) * sizeof(int));
    if (e == cudaSuccess) e = alloc((void**)&h->bcls, std::max<size_t>(1, cls.size()));
    if (e == cudaSuccess) e = alloc((void**)&h->stats, (size_t)(G.mny + G.iny) * 9 * sizeof(double));
    if (e == cudaSuccess) e = alloc((void**)&h->partial, (size_t)kSumBlocks * 6 * sizeof(double));
    if (e == cudaSuccess && h->nb)
        e = cudaMemcpy(h->bnode, nodes.data(), nodes.size() * sizeof(int), cudaMemcpyHostToDevice);
    if (e == cudaSuccess && h->nb) e = cudaMemcpy(h->bcls, cls.data(), cls.size(), cudaMemcpyHostToDevice);
    std::vector<int4> runs;
    if (h->K->run[0]) {
        h->run_nt = run_threads(c->precision, G.nnodes);
        step_runs(G, 0, h->run_nt, runs);
        h->nruns = (int)runs.size();
        if (e == cudaSuccess) e = alloc((void**)&h->runs, std::max<size_t>(1, runs.size()) * sizeof(int4));
        if (e == cudaSuccess) e = alloc((void**)&h->counters, 2 * sizeof(int));
        if (e == cudaSuccess && !(h->error = error_flag_take())) e = cudaErrorMemoryAllocation;
        if (e == cudaSuccess && !runs.empty())
            e = cudaMemcpy(h->runs, runs.data(), runs.size() * sizeof(int4), cudaMemcpyHostToDevice);
    }
    if (e != cudaSuccess) {
        const int code = (e == cudaErrorMemoryAllocation) ? TMX_E_NOMEM : TMX_E_CUDA;
        free_all(h);
        delete h;
        cudaGetLastError();
        return fail(code, "tmx_create: %s", cudaGetErrorString(e));
    }
    int sms = 148;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    h->bulk_blocks = std::max(1, std::min((G.nnodes + 255) / 256, sms * 8));
    if (h->K->run[0]) {
        const void* k = (const void*)h->K->run[h->run_nt > 128];
        const int smem = h->K->run_smem(h->run_nt);
        cudaFuncSetAttribute(k, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
        cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        int per = 1;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k, h->run_nt, smem);
        cudaGetLastError();
        h->run_slots = sms * std::max(1, per);
    }
    // the FP16 form's interior as 32 x 4 sweep tiles (the same bits as the flat
    // kernel, faster)
    if (h->K->moments) {
        const SweepShape* sh = sweep_shape(TMX_SHAPE_SWEEP4);
        int per = 4;
        if (sweep_allow_smem() == cudaSuccess)
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, (const void*)sh->single, sh->threads(), sh->smem(false));
        cudaGetLastError();
        const int nt = sh->threads(), rest = (h->nface - h->nswept + nt - 1) / nt + (h->nb - h->nface + nt / 32 - 1) / (nt / 32);
        const int rc = tmx_set_shape(h, TMX_SHAPE_SWEEP4, sweep_planes(h->G, sms * std::max(1, per), rest));
        if (rc) {
            const std::string msg = last_error();
            tmx_destroy(h);
            return fail(rc, "%s", msg.c_str());
        }
    }
    *out = h;
    return TMX_OK;
}

int tmx_set_shape(tmx_handle* h, int kind, int zchunk)
{
    if (!h) return fail(TMX_E_INVALID, "null handle");
    const SweepShape* sh = sweep_shape(kind);
    if (kind != TMX_SHAPE_FLAT && !sh) return fail(TMX_E_INVALID, "tmx_set_shape: unknown kind %d", kind);
    if (sh && !h->K->moments)
        return fail(TMX_E_INVALID, "tmx_set_shape: the sweep shapes are for the FP16 form only");
    if (sh && zchunk < 1) return fail(TMX_E_INVALID, "tmx_set_shape: zchunk must be >= 1");
    TMX_CK(cudaSetDevice(h->device));
    TMX_CK(cudaStreamSynchronize(h->stream));
    if (sh) {
        TMX_CK(sweep_allow_smem());
        std::vector<int4> t;
        sweep_tiles(h->G, 0, sh->ty, zchunk, false, t);
        int4* d = nullptr;
        if (!t.empty()) {
            cudaError_t e = cudaMalloc((void**)&d, t.size() * sizeof(int4));
            if (e == cudaSuccess) e = cudaMemcpy(d, t.data(), t.size() * sizeof(int4), cudaMemcpyHostToDevice);
            if (e == cudaSuccess) e = copies_arrived();
            if (e != cudaSuccess) {
                cudaFree(d);
                cudaGetLastError();
                return fail(e == cudaErrorMemoryAllocation ? TMX_E_NOMEM : TMX_E_CUDA, "tmx_set_shape: %s",
                            cudaGetErrorString(e));
            }
        }
        cudaFree(h->tiles);
        h->tiles = d;
        h->ntiles = (int)t.size();
        int per = 1, sms = 148;
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, h->device);
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, (const void*)sh->single, sh->threads(), sh->smem(false));
        cudaGetLastError();
        h->sweep_slots = sms * std::max(1, per);
    }
    h->shape = kind;
    h->zchunk = zchunk;
    drop_graphs(h);
    return TMX_OK;
}

int tmx_init(tmx_handle* h)
{
    if (!h) return fail(TMX_E_INVALID, "null handle");
    TMX_CK(cudaSetDevice(h->device));
    TMX_CK(cudaStreamSynchronize(h->stream));
    int rc = inlet_profile_form(h->c, h->stream, h->uin1, h->uin2);
    if (rc) return rc;
    if (h->tbytes == 8) {
        const size_t nu = h->uin1.size() * sizeof(double);
        TMX_CK(cudaMemcpy(h->uin_d[0], h->uin1.data(), nu, cudaMemcpyHostToDevice));
        TMX_CK(cudaMemcpy(h->uin_d[1], h->uin2.data(), nu, cudaMemcpyHostToDevice));
    } else {
        std::vector<float> a(h->uin1.begin(), h->uin1.end()), b(h->uin2.begin(), h->uin2.end());
        TMX_CK(cudaMemcpy(h->uin_d[0], a.data(), a.size() * sizeof(float), cudaMemcpyHostToDevice));
        TMX_CK(cudaMemcpy(h->uin_d[1], b.data(), b.size() * sizeof(float), cudaMemcpyHostToDevice));
    }
    TMX_CK(copies_arrived());
    h->cur = 0;
    h->rcur = 0;
    tmx::StepPtrs X{};
    X.pout = h->pop[0];
    X.rcur = h->rho[0];
    X.mac = h->mac;
    X.mcur = h->mom[0];
    h->K->init<<<h->bulk_blocks, 256, 0, h->stream>>>(X, h->G, h->P, h->c.rho0);
    TMX_CK(cudaGetLastError());
    // a step clears the other parity's run counter; the first finds both clear
    if (h->counters) TMX_CK(cudaMemsetAsync(h->counters, 0, 2 * sizeof(int), h->stream));
    TMX_CK(cudaStreamSynchronize(h->stream));
    if (h->error) *(volatile int*)h->error = 0;  // the earlier state's
    h->steps = 0;
    h->inited = true;
    return TMX_OK;
}

int tmx_step(tmx_handle* h, int nsteps)
{
    if (!h) return fail(TMX_E_INVALID, "null handle");
    if (!h->inited) return fail(TMX_E_STATE, "tmx_step before tmx_init");
    if (nsteps < 0) return fail(TMX_E_INVALID, "negative step count");
    TMX_CK(cudaSetDevice(h->device));
    for (int left = nsteps; left > 0;) {
        const int n = graph_length(left, h->graph_many[h->cur], h->singles);
        if (n == 1 && h->singles < kGraphWorth) h->singles++;
        const int rc = graph_steps(h, n, left == 1);
        if (rc) return rc;
        left -= n;
    }
    return TMX_OK;
}

int tmx_sync(tmx_handle* h)
{
    if (!h) return fail(TMX_E_INVALID, "null handle");
    TMX_CK(cudaSetDevice(h->device));
    TMX_CK(cudaStreamSynchronize(h->stream));
    return settled(h);
}

long long tmx_steps_done(const tmx_handle* h) { return h ? h->steps : -1; }

int tmx_checkpoint_size(const tmx_handle* h, long long* bytes)
{
    if (!h || !bytes) return fail(TMX_E_INVALID, "null argument");
    long long b[5];
    checkpoint_sections(h->G, h->c.precision, b);
    *bytes = checkpoint_total(b);
    return TMX_OK;
}

int tmx_checkpoint(tmx_handle* h, void* buf, long long size)
{
    if (!h || !buf) return fail(TMX_E_INVALID, "null argument");
    if (!h->inited) return fail(TMX_E_STATE, "tmx_checkpoint before tmx_init");
    long long b[5];
    checkpoint_sections(h->G, h->c.precision, b);
    if (size != checkpoint_total(b)) return fail(TMX_E_INVALID, "checkpoint buffer of %lld bytes, %lld needed", size,
                                                 checkpoint_total(b));
    TMX_CK(cudaSetDevice(h->device));
    TMX_CK(cudaStreamSynchronize(h->stream));
    if (const int rc = settled(h)) return rc;
    CheckpointHeader hd{};
    std::memcpy(hd.magic, kCheckpointMagic, 8);
    hd.abi = TMX_ABI_VERSION;
    hd.precision = h->c.precision;
    hd.c = h->c;
    hd.steps = h->steps;
    hd.ps = h->G.ps;
    std::memcpy(hd.bytes, b, sizeof b);
    char* p = (char*)buf;
    std::memcpy(p, &hd, sizeof hd);
    p += sizeof hd;
    const void* src[4] = {h->pop[h->cur], h->rho[h->cur], h->mom[h->cur], h->mac};
    for (int k = 0; k < 4; k++) {
        if (b[k]) TMX_CK(cudaMemcpy(p, src[k], (size_t)b[k], cudaMemcpyDeviceToHost));
        p += b[k];
    }
    std::memcpy(p, h->uin1.data(), (size_t)b[4] / 2);
    std::memcpy(p + b[4] / 2, h->uin2.data(), (size_t)b[4] / 2);
    return TMX_OK;
}

int tmx_restore(tmx_handle* h, const void* buf, long long size)
{
    if (!h || !buf) return fail(TMX_E_INVALID, "null argument");
    int rc = checkpoint_check(buf, size, h->c, h->G);
    if (rc) return rc;
    TMX_CK(cudaSetDevice(h->device));
    TMX_CK(cudaStreamSynchronize(h->stream));
    CheckpointHeader hd;
    std::memcpy(&hd, buf, sizeof hd);
    const char* p = (const char*)buf + sizeof hd;
    // the state goes into buffer set 0, which the next step then reads
    void* dst[4] = {h->pop[0], h->rho[0], h->mom[0], h->mac};
    for (int k = 0; k < 4; k++) {
        if (hd.bytes[k]) TMX_CK(cudaMemcpy(dst[k], p, (size_t)hd.bytes[k], cudaMemcpyHostToDevice));
        p += hd.bytes[k];
    }
    const size_t nu = (size_t)(h->G.iny + 3) * (h->G.nz + 3);
    h->uin1.assign((const double*)p, (const double*)p + nu);
    h->uin2.assign((const double*)p + nu, (const double*)p + 2 * nu);
    if (h->tbytes == 8) {
        TMX_CK(cudaMemcpy(h->uin_d[0], h->uin1.data(), nu * 8, cudaMemcpyHostToDevice));
        TMX_CK(cudaMemcpy(h->uin_d[1], h->uin2.data(), nu * 8, cudaMemcpyHostToDevice));
    } else {
        std::vector<float> a(h->uin1.begin(), h->uin1.end()), c(h->uin2.begin(), h->uin2.end());
        TMX_CK(cudaMemcpy(h->uin_d[0], a.data(), nu * 4, cudaMemcpyHostToDevice));
        TMX_CK(cudaMemcpy(h->uin_d[1], c.data(), nu * 4, cudaMemcpyHostToDevice));
    }
    TMX_CK(copies_arrived());
    if (h->counters) {
        TMX_CK(cudaMemsetAsync(h->counters, 0, 2 * sizeof(int), h->stream));
        TMX_CK(cudaStreamSynchronize(h->stream));
    }
    if (h->error) *(volatile int*)h->error = 0;  // the earlier state's
    h->cur = 0;
    h->rcur = 0;
    h->steps = hd.steps;
    h->inited = true;
    return TMX_OK;
}

int tmx_case_of(const tmx_handle* h, tmx_case* out)
{
    if (!h || !out) return fail(TMX_E_INVALID, "null argument");
    *out = h->c;
    return TMX_OK;
}

int tmx_fields(tmx_handle* h, int box, int field, double* host_out)
{
    if (!h || !host_out) return fail(TMX_E_INVALID, "null argument");
    if (box < 0 || box > 1 || field < 0 || field > 6) return fail(TMX_E_INVALID, "box %d / field %d out of range", box, field);
    if (!h->inited) return fail(TMX_E_STATE, "tmx_fields before tmx_init");
    TMX_CK(cudaSetDevice(h->device));
    const int rc = box_to_host(h->G, box, h->mac + (size_t)field * h->G.ps + h->G.base[box],
                               (double*)h->pop[1 - h->cur], h->stream, host_out);
    return rc ? rc : settled(h);
}

int tmx_populations(tmx_handle* h, int box, int fld, double* host_out)
{
    if (!h || !host_out) return fail(TMX_E_INVALID, "null argument");
    if (box < 0 || box > 1 || fld < 0 || fld > 3) return fail(TMX_E_INVALID, "box %d / field %d out of range", box, fld);
    if (!h->inited) return fail(TMX_E_STATE, "tmx_populations before tmx_init");
    TMX_CK(cudaSetDevice(h->device));
    const Geom& G = h->G;
    const size_t n = (size_t)G.nx[box] * G.ny[box] * G.nz;
    if (h->sbytes == 8) {
        for (int q = 0; q < 19; q++) {
            const double* src = (const double*)h->pop[h->cur] + (size_t)(fld * 19 + q) * G.ps + G.base[box];
            int rc = box_to_host(G, box, src, (double*)h->pop[1 - h->cur], h->stream, host_out + q * n);
            if (rc) return rc;
        }
        return settled(h);
    }
    // reduced precision: widen on the host; the FP16 form adds back feq of
    // the writing node's moments exactly as the kernels do (tmx_engine.cuh).  (The
    // copies below do not wait for the handle's stream by themselves.)
    TMX_CK(cudaStreamSynchronize(h->stream));
    if (const int rc = settled(h)) return rc;
    std::vector<double> wide(n);
    std::vector<unsigned char> raw(4 * n * h->sbytes);
    // moment records {(rho, cA, cB, cC), (ux, uy, uz, 1 - 1.5|u|^2)}, 8 floats per node
    std::vector<float> mr(8 * n);
    if (h->K->moments) {
        const float4* m = h->mom[h->cur];
        TMX_CK(cudaMemcpy(mr.data(), m + 2 * (size_t)G.base[box], n * 2 * sizeof(float4), cudaMemcpyDeviceToHost));
    }
    for (int q = 0; q < 19; q++) {
        // interleaved layout: the four fields of (q, node) side by side
        const unsigned char* src =
            (const unsigned char*)h->pop[h->cur] + ((size_t)q * G.ps + G.base[box]) * 4 * h->sbytes;
        TMX_CK(cudaMemcpy(raw.data(), src, raw.size(), cudaMemcpyDeviceToHost));
        const float w = (float)(q == 0 ? 1.0 / 3.0 : (q <= 6 ? 1.0 / 18.0 : 1.0 / 36.0));
        for (size_t t = 0; t < n; t++) {
            float v;
            const size_t e = (t * 4 + fld) * h->sbytes;
            if (h->sbytes == 4) {
                std::memcpy(&v, &raw[e], 4);
            } else {
                unsigned short hb;
                std::memcpy(&hb, &raw[e], 2);
                const float* rec = &mr[8 * t];
                const float r = rec[fld];
                const float pw = poly_q_host(q, rec[4], rec[5], rec[6], rec[7]) * w;
                v = std::fmaf(r, pw, half_bits_to_float(hb));
            }
            wide[t] = v;
        }
        const int nx = G.nx[box], ny = G.ny[box], nz = G.nz;
        for (int k = 0; k < nz; k++)
            for (int j = 0; j < ny; j++)
                for (int i = 0; i < nx; i++)
                    host_out[q * n + ((size_t)i * ny + j) * nz + k] = wide[((size_t)k * ny + j) * nx + i];
    }
    return TMX_OK;
}

int tmx_mixing(tmx_handle* h, double* rows_out, double* outlet_im)
{
    if (!h || !rows_out) return fail(TMX_E_INVALID, "null argument");
    if (!h->inited) return fail(TMX_E_STATE, "tmx_mixing before tmx_init");
    TMX_CK(cudaSetDevice(h->device));
    const Geom& G = h->G;
    const int nrow = G.mny + G.iny;
    tmx::k_mixing_rows<<<nrow, 3 * tmx::kRowPart, 0, h->stream>>>(h->mac, G, h->stats);
    TMX_CK(cudaGetLastError());
    std::vector<double> st((size_t)nrow * 9);
    TMX_CK(cudaMemcpyAsync(st.data(), h->stats, st.size() * sizeof(double), cudaMemcpyDeviceToHost, h->stream));
    TMX_CK(cudaStreamSynchronize(h->stream));
    if (const int rc = settled(h)) return rc;
    // running maxima over the rows in the reference's order, starting at 0
    double mx[3] = {0.0, 0.0, 0.0};
    for (int r = 0; r < nrow; r++) {
        const double* s = &st[(size_t)r * 9];
        double* o = rows_out + (size_t)r * 7;
        const bool mixing_row = r < G.mny;
        o[0] = mixing_row ? r + 1 : (r - G.mny + 1) + G.mny;
        for (int q = 0; q < 3; q++) {
            if (mx[q] < s[6 + q]) mx[q] = s[6 + q];
            o[1 + q] = s[q];
        }
        const bool ok = mixing_row ? (s[0] > 0 && s[1] > 0 && s[2] > 0) : (s[0] > 0);
        for (int q = 0; q < 3; q++) {
            if (ok) {
                const double Is = s[3 + q] / (s[q] * (mx[q] - s[q]));
                o[4 + q] = 1.0 - std::sqrt(Is);
            } else {
                o[4 + q] = 0.0;
            }
        }
    }
    if (outlet_im)
        for (int q = 0; q < 3; q++) outlet_im[q] = rows_out[4 + q];
    return TMX_OK;
}

// Scratch address of tmx_mixing_static per device, resolved by the first
// call on that device (cudaGetSymbolAddress with the device current).
namespace {
constexpr int kMixStaticDevices = 64;
std::once_flag g_mix_once[kMixStaticDevices];
double* g_mix_ptr[kMixStaticDevices];
cudaError_t g_mix_err[kMixStaticDevices];
}  // namespace

int tmx_mixing_static(tmx_handle* h, double* rows_out, double* outlet_im)
{
    if (!h || !rows_out) return fail(TMX_E_INVALID, "null argument");
    if (!h->inited) return fail(TMX_E_STATE, "tmx_mixing_static before tmx_init");
    const Geom& G = h->G;
    const int nrow = G.mny + G.iny;
    if (nrow > tmx::kMixStaticRows)
        return fail(TMX_E_INVALID,
                    "tmx_mixing_static: mny + iny = %d rows exceeds its fixed scratch of %d rows (use tmx_mixing)",
                    nrow, tmx::kMixStaticRows);
    const int d = h->device;
    if (d < 0 || d >= kMixStaticDevices)
        return fail(TMX_E_INVALID, "tmx_mixing_static: device %d is beyond its table of %d devices", d,
                    kMixStaticDevices);
    TMX_CK(cudaSetDevice(d));
    std::call_once(g_mix_once[d], [d] { g_mix_err[d] = tmx::mixing_static_scratch(&g_mix_ptr[d]); });
    if (g_mix_err[d] != cudaSuccess)
        return fail(TMX_E_CUDA, "tmx_mixing_static: cudaGetSymbolAddress on device %d: %s", d,
                    cudaGetErrorString(g_mix_err[d]));
    double* stats = g_mix_ptr[d];
    double* rows = stats + (size_t)tmx::kMixStaticRows * 9;
    tmx::k_mixing_rows<<<nrow, 3 * tmx::kRowPart, 0, h->stream>>>(h->mac, G, stats);
    tmx::k_mixing_finish<<<1, 96, 0, h->stream>>>(stats, G, rows);
    TMX_CK(cudaGetLastError());
    TMX_CK(cudaMemcpyAsync(rows_out, rows, (size_t)nrow * 7 * sizeof(double), cudaMemcpyDeviceToHost, h->stream));
    TMX_CK(cudaStreamSynchronize(h->stream));
    if (const int rc = settled(h)) return rc;
    if (outlet_im)
        for (int q = 0; q < 3; q++) outlet_im[q] = rows_out[4 + q];
    return TMX_OK;
}

int tmx_sums(tmx_handle* h, double out[8])
{
    if (!h || !out) return fail(TMX_E_INVALID, "null argument");
    if (!h->inited) return fail(TMX_E_STATE, "tmx_sums before tmx_init");
    TMX_CK(cudaSetDevice(h->device));
    tmx::k_sums<<<kSumBlocks, 256, 0, h->stream>>>(h->mac, h->G, h->partial);
    TMX_CK(cudaGetLastError());
    std::vector<double> p((size_t)kSumBlocks * 6);
    TMX_CK(cudaMemcpyAsync(p.data(), h->partial, p.size() * sizeof(double), cudaMemcpyDeviceToHost, h->stream));
    TMX_CK(cudaStreamSynchronize(h->stream));
    if (const int rc = settled(h)) return rc;
    double s[6] = {0, 0, 0, 0, 0, 0};
    for (int b = 0; b < kSumBlocks; b++)
        for (int m = 0; m < 6; m++) s[m] += p[(size_t)b * 6 + m];
    out[0] = s[0];
    out[1] = s[1];
    out[2] = s[2];
    out[3] = s[3];
    out[4] = s[1] + s[2] + s[3];
    out[5] = s[4];
    out[6] = s[5];
    out[7] = (double)h->G.nnodes;
    return TMX_OK;
}

int tmx_pressure_power(tmx_handle* h, double* pressure_rows, double* pressure_x, double* power_rows,
                       double units[2])
{
    if (!h || !pressure_rows || !pressure_x || !power_rows || !units) return fail(TMX_E_INVALID, "null argument");
    if (!h->inited) return fail(TMX_E_STATE, "tmx_pressure_power before tmx_init");
    TMX_CK(cudaSetDevice(h->device));
    const Geom& G = h->G;
    const int nrow = G.mny + G.iny, npow = G.mny - 2, nout = 1 + nrow + G.inx + 4 * npow;
    if (!h->diag) {
        cudaError_t e = cudaMalloc((void**)&h->diag, (size_t)nout * sizeof(double));
        if (e != cudaSuccess) {
            h->diag = nullptr;
            cudaGetLastError();
            return fail(e == cudaErrorMemoryAllocation ? TMX_E_NOMEM : TMX_E_CUDA, "tmx_pressure_power: %s",
                        cudaGetErrorString(e));
        }
        h->bytes += (long long)nout * sizeof(double);
    }
    const int items = 1 + nrow + G.inx + npow;
    tmx::k_pressure_power<<<items, tmx::kRowPart, 0, h->stream>>>(h->mac, G, h->c.tau, h->diag);
    TMX_CK(cudaGetLastError());
    std::vector<double> o((size_t)nout);
    TMX_CK(cudaMemcpyAsync(o.data(), h->diag, o.size() * sizeof(double), cudaMemcpyDeviceToHost, h->stream));
    TMX_CK(cudaStreamSynchronize(h->stream));
    if (const int rc = settled(h)) return rc;
    const double ptop = o[0];
    for (int r = 0; r < nrow; r++) {
        pressure_rows[3 * r] = r + 1;  // mixing rows 1..mny, then inlet row j as j + mny
        pressure_rows[3 * r + 1] = o[1 + r];
        pressure_rows[3 * r + 2] = o[1 + r] - ptop;
    }
    for (int i = 0; i < G.inx; i++) {
        pressure_x[2 * i] = i + 1;
        pressure_x[2 * i + 1] = o[1 + nrow + i];
    }
    for (int j = 0; j < npow; j++) {
        power_rows[5 * j] = j + 2;
        for (int m = 0; m < 4; m++) power_rows[5 * j + 1 + m] = o[1 + nrow + G.inx + 4 * j + m];
    }
    // the reference's unit factors (Tmixer.cpp:185-196: LENGTH 0.0008 m, PRESSURE
    // 101325 Pa, KVISCOSITY 1.004e-6 m^2/s, length = inx), as its macros expand
    const double tau = h->c.tau, rho0 = h->c.rho0;
    const double L0 = (0.0008 / (G.inx - 1));
    const double T0 = ((((2.0 * tau - 1.0) / 6.0) / 0.000001004) * (L0 * L0));
    const double M0 = ((101325.0 / (rho0 / 3.0)) * (L0 * T0 * T0));
    units[0] = ((M0) / (L0 * T0 * T0));
    units[1] = ((L0 * L0) / (T0 * T0 * T0));
    return TMX_OK;
}

int tmx_inlet_profile(tmx_handle* h, double* uin1, double* uin2)
{
    if (!h || !uin1 || !uin2) return fail(TMX_E_INVALID, "null argument");
    if (!h->inited) return fail(TMX_E_STATE, "tmx_inlet_profile before tmx_init");
    std::memcpy(uin1, h->uin1.data(), h->uin1.size() * sizeof(double));
    std::memcpy(uin2, h->uin2.data(), h->uin2.size() * sizeof(double));
    return TMX_OK;
}

int tmx_step_timed(tmx_handle* h, int nsteps, double* ms_bulk, double* ms_boundary, double* ms_total)
{
    if (!h) return fail(TMX_E_INVALID, "null handle");
    if (!h->inited) return fail(TMX_E_STATE, "tmx_step_timed before tmx_init");
    if (nsteps <= 0) return fail(TMX_E_INVALID, "nsteps must be positive");
    TMX_CK(cudaSetDevice(h->device));
    std::vector<cudaEvent_t> ev((size_t)nsteps * 4);
    for (auto& x : ev) TMX_CK(cudaEventCreate(&x));
    cudaEvent_t t0, t1;
    TMX_CK(cudaEventCreate(&t0));
    TMX_CK(cudaEventCreate(&t1));
    TMX_CK(cudaEventRecord(t0, h->stream));
    int rc = TMX_OK;
    for (int s = 0; s < nsteps && rc == TMX_OK; s++) rc = timed_step(h, s == nsteps - 1, &ev[(size_t)s * 4]);
    TMX_CK(cudaEventRecord(t1, h->stream));
    TMX_CK(cudaEventSynchronize(t1));
    double sb = 0, sbd = 0;
    for (int s = 0; s < nsteps && rc == TMX_OK; s++) {
        float a = 0, b = 0;
        TMX_CK(cudaEventElapsedTime(&a, ev[(size_t)s * 4], ev[(size_t)s * 4 + 1]));
        TMX_CK(cudaEventElapsedTime(&b, ev[(size_t)s * 4 + 2], ev[(size_t)s * 4 + 3]));
        sb += a;
        sbd += b;
    }
    float tot = 0;
    TMX_CK(cudaEventElapsedTime(&tot, t0, t1));
    for (auto& x : ev) cudaEventDestroy(x);
    cudaEventDestroy(t0);
    cudaEventDestroy(t1);
    if (rc) return rc;
    if (ms_bulk) *ms_bulk = sb;
    if (ms_boundary) *ms_boundary = sbd;
    if (ms_total) *ms_total = tot;
    return settled(h);
}

int tmx_time_steps(tmx_handle* h, int nsteps, double* ms)
{
    if (!h || !ms) return fail(TMX_E_INVALID, "null argument");
    if (!h->inited) return fail(TMX_E_STATE, "tmx_time_steps before tmx_init");
    if (nsteps <= 0) return fail(TMX_E_INVALID, "nsteps must be positive");
    TMX_CK(cudaSetDevice(h->device));
    cudaEvent_t t0, t1;
    TMX_CK(cudaEventCreate(&t0));
    TMX_CK(cudaEventCreate(&t1));
    TMX_CK(cudaEventRecord(t0, h->stream));
    int rc = tmx_step(h, nsteps);
    TMX_CK(cudaEventRecord(t1, h->stream));
    TMX_CK(cudaEventSynchronize(t1));
    float el = 0;
    TMX_CK(cudaEventElapsedTime(&el, t0, t1));
    cudaEventDestroy(t0);
    cudaEventDestroy(t1);
    if (rc) return rc;
    *ms = el;
    return settled(h);
}

int tmx_counts(const tmx_handle* h, long long out[4])
{
    if (!h || !out) return fail(TMX_E_INVALID, "null argument");
    out[0] = h->G.nnodes;
    out[1] = h->G.nnodes - h->nb;
    out[2] = h->nb;
    out[3] = h->bytes;
    return TMX_OK;
}

void tmx_destroy(tmx_handle* h)
{
    if (!h) return;
    cudaSetDevice(h->device);
    if (h->stream) cudaStreamSynchronize(h->stream);
    free_all(h);
    delete h;
}

}  // extern "C"
