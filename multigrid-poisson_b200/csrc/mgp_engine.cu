// mgp_engine.cu -- host runtime and C ABI of the multigrid engine (libmgp.so).
//
// One mgp_solver = one level hierarchy resident in HBM, one CUDA stream and a cache of
// instantiated CUDA graphs.  The V/F-cycle recursion of the reference (include/vcycle.h,
// include/fcycle.h) runs on the host only while a graph is being captured; every later
// iteration of PoissonSolver::solve is a single cudaGraphLaunch of the whole cycle plus
// the fine-level residual and its max-norm, followed by an 8-byte read-back for the
// reference's stopping rule (include/libpoisson.h:293-355).
#include <cuda_runtime.h>

#include <algorithm>
#include <chrono>
#include <cmath>
#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <fstream>
#include <functional>
#include <type_traits>
#include <iomanip>
#include <iostream>
#include <cstdlib>
#include <map>
#include <mutex>
#include <new>
#include <sstream>
#include <string>
#include <tuple>
#include <utility>
#include <vector>

#include "mgp.h"
#include "mgp_kernels.cuh"
#include "mgp_wave.cuh"
#include "mgp_tail.cuh"
#include "mgp_cluster.cuh"

using namespace mgp;

// ---------------------------------------------------------------------------------------
// errors
namespace {
thread_local std::string g_err;

int fail(int status, const char* fmt, ...) {
    char buf[512];
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(buf, sizeof(buf), fmt, ap);
    va_end(ap);
    g_err = buf;
    return status;
}

#define CK(call)                                                                                   \
    do {                                                                                           \
        cudaError_t e_ = (call);                                                                   \
        if (e_ != cudaSuccess) {                                                                   \
            return fail(e_ == cudaErrorMemoryAllocation ? MGP_ERR_OOM : MGP_ERR_CUDA, "%s: %s (%s:%d)", \
                        #call, cudaGetErrorString(e_), __FILE__, __LINE__);                        \
        }                                                                                          \
    } while (0)

#define CKS(expr)               \
    do {                        \
        int s_ = (expr);        \
        if (s_ != MGP_OK) return s_; \
    } while (0)

constexpr int kThreads = 256;

int sm_count(int dev) {
    static int cached[64] = {0};
    if (dev >= 0 && dev < 64 && cached[dev]) return cached[dev];
    int n = 148;
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    if (dev >= 0 && dev < 64) cached[dev] = n;
    return n;
}
}  // namespace

// ---------------------------------------------------------------------------------------
struct LevelState {
    Geom G;                 // device geometry (pitched, no ghosts) + relaxation bounds
    double h;
    size_t elems;           // elements per field buffer (nx*sx)
    void* ubuf[2] = {nullptr, nullptr};  // Jacobi ping-pong pair; Gauss-Seidel uses [0]
    void* f = nullptr;
    void* r = nullptr;
    void* face[6] = {};
    int64_t face_shape[6][3];
    int cur = 0;            // index of the buffer that is "u" (Domain::swap_u, domain.h:311-316)
    bool first_done = false;  // the set-up of the finer level already did this level's first sweep
    bool gs_column = false; // padded y extent even: colour depends on (j,k) only; whole columns
    mgp_level_info info;    // host (reference) layout
    // Wavefront passes (k_wave, large Jacobi levels): sweeps two at a time and the residual of
    // the last sweep in the same pass.  Two sweeps in one pass write u2 into a third level-sized
    // buffer that rotates with the two of the ping-pong pair; phys[] are the three allocations
    // in their original order, whose arrangement over (ubuf[0], ubuf[1], spare) is part of the
    // graph state.  wt[M] / wmap_*[M]: tiling and tensor maps of the M-stage passes.
    bool pair = false;
    void* spare = nullptr;
    void* phys[3] = {nullptr, nullptr, nullptr};
    bool wave = false;
    WaveTile wt[4];
    CUtensorMap wmap_u[4][3];   // u0 planes, per allocation
    CUtensorMap wmap_f[4];
    CUtensorMap wmap_bk[4][3];  // u_prev's k = 0 / nz-1 columns (V x rows boxes), per allocation
    CUtensorMap wmap_bj[3];     // u_prev's j = 0 / ny-1 rows (P x 1 boxes), per allocation
    int tune[MGP_TUNE_PARAMS] = {};  // launch shapes of this level's kernels (MGP_TUNE_*; 0 = built-in)
};

struct GraphEntry {
    cudaGraphExec_t exec = nullptr;
    uint64_t post_state = 0;
    int64_t kernels = 0;  // kernel nodes in the graph
};

// The first sweep of a correction's zero guess that the refinement residual writes along
// (RefineArgs::first): the smoothing of the correction cycle that follows.
struct RefineFirst {
    int on = 0;  // 0 none, 1 Jacobi, 2 red-black
    double omega = 0;
    bool operator==(const RefineFirst& o) const { return on == o.on && (!on || omega == o.omega); }
};

struct mgp_solver {
    mgp_desc desc{};
    int dtype = MGP_F64;
    int device = 0;
    int levels = 0;
    size_t esize = 8;
    int face_kind[6] = {};
    bool gs_alternate = true;  // GaussSeidel::alternate (include/gaussseidel.h:18)
    cudaStream_t stream = nullptr;
    std::vector<LevelState> lv;
    unsigned long long* d_norm = nullptr;  // [0] scratch for max-norms
    unsigned long long* h_norm = nullptr;  // pinned read-back
    int* err_word = nullptr;               // kernels' wait-timeout flag (8 bytes after a norm word)
    void* stage = nullptr;                 // device copy of a host-layout field (large transfers)
    size_t stage_bytes = 0;
    std::map<std::tuple<int, int64_t, uint64_t, uint64_t>, GraphEntry> graphs;
    bool capturing = false;
    int64_t launches = 0;  // kernels launched on this solver (graph replays count their nodes)
    // Iterative refinement: this solver holds level 0 in FP64 (u, f, r, boundary data) and
    // `inner` the correction hierarchy (all levels, FP32 or FP64, zero boundary data).  The
    // inner solver shares this solver's stream.
    mgp_solver* inner = nullptr;
    RefineFirst guess;  // inner solvers: the sweep that level 0's guess holds
    bool owns_stream = true;
    // Side stream of the coarse-grid set-up on large levels: the Neumann face restriction runs on
    // it, forked and joined by the two events, overlapped with the residual (own-memory solvers only).
    cudaStream_t side = nullptr;
    cudaEvent_t ev_fork = nullptr, ev_join = nullptr;
    // Problems of a batch allocate from the batch's memory pool in the batch's stream order
    // (no device-wide synchronisation when they come and go) and read norms back through the
    // batch's pinned slab.
    cudaMemPool_t pool = nullptr;
    bool owns_h_norm = true;
    unsigned wait_polls = kWaitPolls;  // bound of the wavefront passes' and the cluster's waits
};

// Where a solver's memory comes from: nullptr = its own stream, cudaMalloc, pinned read-back.
struct CreateCtx {
    cudaStream_t stream;
    cudaMemPool_t pool;
    unsigned long long* h_norm;  // 64 pinned bytes
};

namespace {

// ---- device memory: cudaMalloc, or the batch pool in stream order ------------------------
cudaError_t dev_alloc(mgp_solver* s, void** p, size_t bytes) {
    if (s->pool) return cudaMallocFromPoolAsync(p, bytes, s->pool, s->stream);
    return cudaMalloc(p, bytes);
}
void dev_free(mgp_solver* s, void* p) {
    if (!p) return;
    if (s->pool) cudaFreeAsync(p, s->stream);
    else cudaFree(p);
}
cudaError_t dev_zero(mgp_solver* s, void* p, size_t bytes) {
    if (s->pool) return cudaMemsetAsync(p, 0, bytes, s->stream);
    return cudaMemset(p, 0, bytes);
}

// ---- state helpers ----------------------------------------------------------------------
// Graph state: bit 0 GaussSeidel::alternate, bit l+1 the current buffer of level l, and from
// bit 32 four bits per level with paired sweeps: which allocations sit in ubuf[0] and ubuf[1]
// (3*i0 + i1; the spare is the third).  Pairs are enabled on at most kPairMaxLevels levels of
// solvers with at most 31 levels.
constexpr int kPairMaxLevels = 8;
int phys_index(const LevelState& L, const void* p) {
    for (int i = 0; i < 3; i++)
        if (L.phys[i] == p) return i;
    return 0;
}
uint64_t state_bits(const mgp_solver* s) {
    uint64_t b = s->gs_alternate ? 1ull : 0ull;
    for (int l = 0; l < s->levels; l++) b |= (uint64_t)(s->lv[l].cur & 1) << (l + 1);
    int pi = 0;
    for (int l = 0; l < s->levels; l++) {
        const LevelState& L = s->lv[l];
        if (!L.pair) continue;
        b |= (uint64_t)(3 * phys_index(L, L.ubuf[0]) + phys_index(L, L.ubuf[1])) << (32 + 4 * pi);
        pi++;
    }
    return b;
}
void set_state_bits(mgp_solver* s, uint64_t b) {
    s->gs_alternate = b & 1ull;
    for (int l = 0; l < s->levels; l++) s->lv[l].cur = (int)((b >> (l + 1)) & 1ull);
    int pi = 0;
    for (int l = 0; l < s->levels; l++) {
        LevelState& L = s->lv[l];
        if (!L.pair) continue;
        const int code = (int)((b >> (32 + 4 * pi)) & 15ull);
        const int i0 = code / 3, i1 = code % 3;
        L.ubuf[0] = L.phys[i0];
        L.ubuf[1] = L.phys[i1];
        L.spare = L.phys[3 - i0 - i1];
        pi++;
    }
}

void* u_ptr(mgp_solver* s, int l) { return s->lv[l].ubuf[s->lv[l].cur]; }
void* uprev_ptr(mgp_solver* s, int l) {
    LevelState& L = s->lv[l];
    return L.ubuf[1] ? L.ubuf[1 - L.cur] : L.ubuf[0];
}

template <typename T>
Faces<T> faces_of(mgp_solver* s, int l) {
    Faces<T> F;
    for (int f = 0; f < 6; f++) F.g[f] = (const T*)s->lv[l].face[f];
    return F;
}

int grid_1d(mgp_solver* s, long long n) {
    long long b = (n + kThreads - 1) / kThreads;
    long long cap = (long long)sm_count(s->device) * 8;
    return (int)std::max(1ll, std::min(b, cap));
}

int check_launch(mgp_solver* s) {
    s->launches++;
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return fail(MGP_ERR_CUDA, "kernel launch: %s", cudaGetErrorString(e));
    return MGP_OK;
}

// Programmatic dependent launches (the kernels call pdl_begin first); MGP_PDL=0 launches
// them in ordinary stream order instead.
bool pdl_enabled() {
    static const bool on = [] {
        const char* e = std::getenv("MGP_PDL");
        return !(e && e[0] == '0');
    }();
    return on;
}

template <typename... KArgs, typename... Act>
cudaError_t launch_pdl(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, Act&&... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = pdl_enabled() ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kernel, std::forward<Act>(args)...);
}

template <typename... KArgs, typename... Act>
int launch_k(mgp_solver* s, void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, Act&&... args) {
    const cudaError_t e = launch_pdl(kernel, grid, block, smem, s->stream, std::forward<Act>(args)...);
    if (e != cudaSuccess) return fail(MGP_ERR_CUDA, "kernel launch: %s", cudaGetErrorString(e));
    return check_launch(s);
}

// Ordinary stream-ordered launch (the kernel starts after everything before it completed).
template <typename... KArgs, typename... Act>
int launch_k_ordered(mgp_solver* s, void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, Act&&... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s->stream;
    cfg.numAttrs = 0;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, std::forward<Act>(args)...);
    if (e != cudaSuccess) return fail(MGP_ERR_CUDA, "kernel launch: %s", cudaGetErrorString(e));
    return check_launch(s);
}

// Blocks of `kernel` resident per SM (256 threads, static shared memory only).
template <typename K>
int resident_blocks(K kernel) {
    int n = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kernel, kThreads, 0) != cudaSuccess || n < 1) n = 1;
    return n;
}

// Planes per block of a marching kernel: bx blocks cover a plane, `chunks` split the march.
// Small levels march one plane per thread.  Large levels choose the chunk count whose whole
// grid fills the resident block slots best (a few blocks in an extra wave would run alone),
// counting the two planes each chunk re-reads at its start.
int march_chunks(int bx, int nx, int cap) {
    if ((long long)bx * nx <= cap) return nx;
    int best = 1;
    double best_eff = -1.0;
    for (int waves = 1; waves <= 8; waves++) {
        int c = (int)std::min<long long>(nx, std::max(1ll, (long long)waves * cap / bx));
        const long long blocks = (long long)bx * c;
        const long long w = (blocks + cap - 1) / cap;
        const int ichunk = (nx + c - 1) / c;
        const double fill = (double)blocks / (double)(w * cap);
        const double reread = 1.0 / (1.0 + 2.0 / (3.0 * ichunk));
        const double eff = fill * reread;
        if (eff > best_eff + 1e-9) {
            best_eff = eff;
            best = c;
        }
    }
    return best;
}

// x/hsq equals x*(1/hsq) bit for bit when hsq is a power of two (scaling by 2^k is exact);
// the kernels then multiply instead of dividing.
template <typename T>
void hsq_terms(T hsq, T& inv, int& pow2) {
    int ex = 0;
    const double m = std::frexp((double)hsq, &ex);
    pow2 = (m == 0.5) && std::isfinite((double)hsq) && std::isnormal((double)hsq);
    inv = pow2 ? (T)(1.0 / (double)hsq) : T(0);
    if (pow2 && !std::isnormal((double)inv)) pow2 = 0;
}

// ---- tensor maps ----------------------------------------------------------------------------
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_tiled() {
    static const EncodeTiledFn fn = [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess ||
            q != cudaDriverEntryPointSuccess)
            return (EncodeTiledFn) nullptr;
        return (EncodeTiledFn)p;
    }();
    return fn;
}

// A 3-D map (k, j, i) of one pitched field buffer with a (box_k, box_j, 1) box; reads outside
// the level's shape are filled with zeros.
bool encode_field_map(CUtensorMap* m, void* base, bool f64, const Geom& G, int box_k, int box_j) {
    EncodeTiledFn fn = encode_tiled();
    if (!fn) return false;
    const cuuint64_t es = f64 ? 8 : 4;
    const cuuint64_t dims[3] = {(cuuint64_t)G.nz, (cuuint64_t)G.ny, (cuuint64_t)G.nx};
    const cuuint64_t strides[2] = {(cuuint64_t)G.sy * es, (cuuint64_t)G.sx * es};
    const cuuint32_t box[3] = {(cuuint32_t)box_k, (cuuint32_t)box_j, 1};
    const cuuint32_t estr[3] = {1, 1, 1};
    return fn(m, f64 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT64 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, base, dims, strides, box,
              estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// ---- wavefront passes ---------------------------------------------------------------------
// Jacobi levels of at least kWaveMinPoints points (at least 3 per axis, nz small enough for one
// TMA box row) relax with k_wave: two sweeps per pass, and the residual that follows the last
// sweep (the coarse-grid set-up's, or the solve loop's with its max-norm) in the same pass,
// with MGP_FLAG_WAVE (opt-in: on B200 the pass is issue-bound and slower than the separate
// passes).  Solvers carved from a batch pool
// sweep with the batch engine's own kernels.
constexpr long long kWaveMinPoints = 1ll << 20;
constexpr size_t kWaveMaxSmem = 224 * 1024;  // dynamic; the static barriers and reduction slots fit beside it

// Tiling of an M-stage pass: TJ output rows per CTA (thread rows TJ + 2(M-1), one 16-byte
// k-vector each, at most kWaveMaxThreads threads and kWaveMaxSmem bytes of rings), and the
// chunk count along i.  Among those, the one with the least work per SM: CTAs per SM x steps
// per chunk (its planes plus the 2(M-1) a chunk re-computes at its ends) x thread rows (the
// TJ rows of the tile plus the halo rows it re-computes), plus one for the copied halo rows.  The CTAs of one chunk run together,
// so halo rows come from L2.
// Pipeline depths of the wavefront passes: u0 ring slots, f planes in flight, L2 prefetch
// distance and kind.  MGP_WAVE_RU / _FA / _L2A / _L2MODE override them (experiments).
struct WaveDepth {
    int ru = 6, fa = 3, l2a = 6, l2mode = 2;
};
WaveDepth wave_depth() {
    static const WaveDepth d = [] {
        WaveDepth w;
        auto env = [](const char* n, int& v, int lo, int hi) {
            const char* e = std::getenv(n);
            if (e && *e) v = std::max(lo, std::min(hi, std::atoi(e)));
        };
        env("MGP_WAVE_RU", w.ru, 3, kWaveMaxRing);
        env("MGP_WAVE_FA", w.fa, 1, kWaveMaxRing - 1);
        env("MGP_WAVE_L2A", w.l2a, 0, 32);
        env("MGP_WAVE_L2MODE", w.l2mode, 0, 2);
        return w;
    }();
    return d;
}

template <typename T>
WaveTile wave_tiling(const Geom& G, int M, int sms, const WaveDepth& d) {
    constexpr int V = VecT<T>::V;
    constexpr long long ES = sizeof(T);
    WaveTile best;
    const int nvec = (G.nz + V - 1) / V;
    const int P = nvec * V;
    if (P > kWaveMaxWidth || nvec < 3) return best;  // a row needs interior vectors besides its two ends
    auto rup = [](long long n) { return (int)((n + 127) / 128 * 128); };
    double best_cost = 1e300;
    int tj_only = 0;  // MGP_WAVE_TJ<M>: an experiment's fixed tile height
    {
        char name[16];
        std::snprintf(name, sizeof(name), "MGP_WAVE_TJ%d", M);
        if (const char* e = std::getenv(name); e && *e) tj_only = std::atoi(e);
    }
    for (int TJ = 1; TJ <= G.ny; TJ++) {
        if (tj_only > 0 && TJ != tj_only) continue;
        const int rows = TJ + 2 * (M - 1);
        if (rows * nvec > kWaveMaxThreads || rows + 2 > 256) break;
        // a u0 slot: the (rows+2) x P box, then u_prev's k = 0 and k = nz-1 columns (rows x V
        // each) and its j = 0 and j = ny-1 rows (P each)
        const int bk = rup(rows * V * ES), bj = rup(P * ES);
        const int u_box = rup((long long)(rows + 2) * P * ES);
        const int su = u_box + 2 * bk + 2 * bj, sf = rup((long long)rows * P * ES), sw = sf;
        const size_t smem = 256 + (size_t)d.ru * su + (size_t)(M + d.fa) * sf + (size_t)2 * (M - 1) * sw;
        if (smem > kWaveMaxSmem) break;
        const int tiles_j = (G.ny + TJ - 1) / TJ;
        for (int c = 1; c <= G.nx; c++) {
            const int ci = (G.nx + c - 1) / c;
            if ((G.nx + ci - 1) / ci != c) continue;
            const long long per_sm = ((long long)tiles_j * c + sms - 1) / sms;
            if (per_sm > 16) break;
            // steps of a chunk: its planes, the 2(M-1) it re-computes at its ends, and about
            // three for the copies that fill the rings before the first step
            const double cost = (double)per_sm * (ci + 2 * (M - 1) + 3) * (rows + 1);
            if (cost < best_cost * (1.0 - 1e-9)) {
                best_cost = cost;
                best.ok = true;
                best.TJ = TJ;
                best.rows = rows;
                best.nvec = nvec;
                best.P = P;
                best.tiles_j = tiles_j;
                best.ci = ci;
                best.chunks = c;
                best.slot_u = su;
                best.slot_f = sf;
                best.slot_w = sw;
                best.b_klo = u_box;
                best.b_khi = u_box + bk;
                best.b_jlo = u_box + 2 * bk;
                best.b_jhi = u_box + 2 * bk + bj;
                best.kl = (G.nz - 1) / V * V;
                best.ru = d.ru;
                best.fa = d.fa;
                best.l2a = d.l2a;
                best.l2mode = d.l2mode;
                best.smem = smem;
            }
        }
    }
    return best;
}

// A 3-D map (k, j, i) of a pitched field with a (P, rows, 1) box; reads outside the level's
// shape are zero-filled.
bool encode_wave_map(CUtensorMap* m, void* base, bool f64, const Geom& G, int P, int rows) {
    return encode_field_map(m, base, f64, G, P, rows);
}

template <typename T>
cudaError_t wave_prepare_level(mgp_solver* s, LevelState& L, int npair) {
    L.wave = false;
    L.pair = false;
    const Geom& G = L.G;
    // the k-edge tensor maps carry one vector per row: TMA needs that to be 16 bytes
    if (VecT<T>::V * sizeof(T) != 16) return cudaSuccess;
    if (s->desc.relaxation != MGP_JACOBI || !(s->desc.flags & MGP_FLAG_WAVE) || s->pool || !L.ubuf[1] ||
        s->levels > 31 || npair >= kPairMaxLevels || (long long)G.nx * G.ny * G.nz < kWaveMinPoints || G.nx < 3 ||
        G.ny < 3 || G.nz < 3 || !encode_tiled())
        return cudaSuccess;
    for (int M = 1; M <= 3; M++) {
        L.wt[M] = wave_tiling<T>(G, M, sm_count(s->device), wave_depth());
        if (!L.wt[M].ok) return cudaSuccess;
    }
    cudaError_t e = dev_alloc(s, &L.spare, L.elems * sizeof(T));
    if (e == cudaSuccess) e = dev_zero(s, L.spare, L.elems * sizeof(T));
    if (e != cudaSuccess) return e;
    L.phys[0] = L.ubuf[0];
    L.phys[1] = L.ubuf[1];
    L.phys[2] = L.spare;
    const bool f64 = sizeof(T) == 8;
    bool ok = true;
    constexpr int V = VecT<T>::V;
    for (int M = 1; M <= 3 && ok; M++) {
        const WaveTile& t = L.wt[M];
        for (int b = 0; b < 3 && ok; b++) {
            ok = encode_wave_map(&L.wmap_u[M][b], L.phys[b], f64, G, t.P, t.rows + 2) &&
                 encode_wave_map(&L.wmap_bk[M][b], L.phys[b], f64, G, V, t.rows);
        }
        if (ok) ok = encode_wave_map(&L.wmap_f[M], L.f, f64, G, t.P, t.rows);
    }
    for (int b = 0; b < 3 && ok; b++) ok = encode_wave_map(&L.wmap_bj[b], L.phys[b], f64, G, L.wt[1].P, 1);
    if (!ok) {
        dev_free(s, L.spare);
        L.spare = nullptr;
        return cudaSuccess;
    }
    L.pair = true;
    L.wave = true;
    if (const char* e = std::getenv("MGP_WAVE_VERBOSE"); e && *e == '1') {
        for (int M = 1; M <= 3; M++) {
            const WaveTile& t = L.wt[M];
            std::fprintf(stderr, "wave %dx%dx%d M=%d: TJ=%d rows=%d threads=%d grid=%dx%d ci=%d smem=%zu ru=%d fa=%d l2a=%d l2mode=%d\n",
                         G.nx, G.ny, G.nz, M, t.TJ, t.rows, t.rows * t.nvec, t.tiles_j, t.chunks, t.ci, t.smem, t.ru,
                         t.fa, t.l2a, t.l2mode);
        }
    }
    return cudaSuccess;
}

template <typename T, int NJ, int RES, bool WU1>
int launch_wave_k(mgp_solver* s, const WaveTile& t, const CUtensorMap& mu, const CUtensorMap& mf,
                  const CUtensorMap& mbk, const CUtensorMap& mbj, const WaveArgs<T>& a) {
    auto kernel = k_wave<T, NJ, RES, WU1>;
    static bool attr_set[64] = {};  // per instantiation and device
    if (s->device < 64 && !attr_set[s->device]) {
        CK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kWaveMaxSmem));
        attr_set[s->device] = true;
    }
    // the consumer threads in whole warps, then the producer warp
    const unsigned threads = (unsigned)((t.rows * t.nvec + 31) / 32 * 32 + 32);
    return launch_k(s, kernel, dim3((unsigned)(t.tiles_j * t.chunks)), dim3(threads), t.smem, mu, mf, mbk, mbj, a);
}

// nj Jacobi sweeps (1 or 2) of level l in one pass, then (res != 0) the residual of their
// result: r stored, and with res == 2 its max-norm into *norm.  Buffers as Relaxation::relax
// leaves them: one sweep -> u_prev's buffer becomes u; two sweeps -> the spare buffer takes u2
// and becomes u, u_prev takes u1 when wu1 (else its relaxed points are left stale), and the old
// u becomes the spare.
template <typename T>
int launch_wave(mgp_solver* s, int l, int nj, int res, bool wu1, T omega, unsigned long long* norm) {
    LevelState& L = s->lv[l];
    const int M = nj + (res ? 1 : 0);
    const WaveTile& t = L.wt[M];
    WaveArgs<T> a;
    a.G = L.G;
    a.A = (const T*)u_ptr(s, l);
    a.B = (T*)uprev_ptr(s, l);
    a.C = (T*)L.spare;
    a.r = (T*)L.r;
    a.f = (const T*)L.f;
    a.F = faces_of<T>(s, l);
    // the constants of launch_stencil (jacobi.h:41-44, residual.h, neumann.h:117)
    a.two_h = (T)(2.0 * L.h);
    a.hsq = (T)(L.h * L.h);
    a.one_omega = (T)(1.0 - omega);
    a.omega_sixth = (T)(omega / 6.0);
    hsq_terms(a.hsq, a.inv_hsq, a.hsq_pow2);
    a.t = t;
    a.norm = norm;
    a.err = s->err_word;
    a.wait_polls = s->wait_polls;
    const int ia = phys_index(L, a.A), ib = phys_index(L, a.B);
    const CUtensorMap& mu = L.wmap_u[M][ia];
    const CUtensorMap& mf = L.wmap_f[M];
    const CUtensorMap& mbk = L.wmap_bk[M][ib];
    const CUtensorMap& mbj = L.wmap_bj[ib];
    int st;
#define MGP_WAVE(NJ_, RES_, WU1_) launch_wave_k<T, NJ_, RES_, WU1_>(s, t, mu, mf, mbk, mbj, a)
    if (nj == 1) {
        if (res == 0) st = MGP_WAVE(1, 0, false);
        else if (res == 1) st = MGP_WAVE(1, 1, false);
        else st = MGP_WAVE(1, 2, false);
    } else if (res == 0) {
        st = wu1 ? MGP_WAVE(2, 0, true) : MGP_WAVE(2, 0, false);
    } else if (res == 1) {
        st = wu1 ? MGP_WAVE(2, 1, true) : MGP_WAVE(2, 1, false);
    } else {
        st = wu1 ? MGP_WAVE(2, 2, true) : MGP_WAVE(2, 2, false);
    }
#undef MGP_WAVE
    CKS(st);
    if (nj == 1) L.cur ^= 1;
    else std::swap(L.ubuf[L.cur], L.spare);
    return MGP_OK;
}

// ---- stencil launches -------------------------------------------------------------------
#ifndef MGP_SHORT_MARCH
#define MGP_SHORT_MARCH 1  // compile-time switch of the short-march rule in launch_stencil
#endif
constexpr long long kShortMarchMinPoints = 1ll << 22;
constexpr int kMaxGridRows = 65535;  // largest gridDim.y: boxes of more chunks keep the long march

// Large levels whose plane does not fill a wave of blocks march short chunks.  Measured on B200
// with the autotuner (F-cycles on 513x257x129 and 257^3): 3-5 planes per block were fastest in
// FP64 and 2-3 in FP32, against the 13-20 the fill rule gives -- FP32 most (four points per
// 16-byte vector, so half the threads per plane); F-cycle 513x257x129 FP32 1.164 -> 1.078 ms,
// 1025x513x257 FP32 5.90 -> 5.24 ms, FP64 1.370 -> 1.343 and 8.29 -> 8.08 ms.  Where one plane
// already fills a wave (1025x1025x513 FP64) the long march stays: short ones cost 2.5% there.
template <typename T>
int short_march_chunks(const Geom& G, int bx, int cap, int chunks) {
    constexpr int kShort = sizeof(T) == 8 ? 4 : 3;
    if (MGP_SHORT_MARCH && bx < cap && (long long)G.nx * G.ny * G.nz >= kShortMarchMinPoints &&
        (G.nx + chunks - 1) / chunks > kShort && (G.nx + kShort - 1) / kShort <= kMaxGridRows)
        return (G.nx + kShort - 1) / kShort;
    return chunks;
}

// Planes per block of the register form (k_stencil_planes), 0: the staged march.  `ichunk`: the
// march's built-in planes per block.  Measured on B200 per launch, march against registers:
// short marches on large levels, three planes -- 513x257x129 FP64 sweep 83.4 -> 77.4 us, red-black
// half-sweep 81.3 -> 77.9, FP32 sweep 52.2 -> 46.9, residual 58.3 -> 52.7, 257^3 FP32 sweep
// 43.5 -> 38.2 us; four planes are slower (80.3 us at 513x257x129), and the FP64 residual there
// keeps the march (83.9 against 85.3 us).  Longer marches on levels below that, two planes --
// 257x129x65 FP64 sweep 14.3 -> 11.0 us, half-sweep 11.9 -> 10.4, residual 14.2 -> 12.3, FP32 sweep
// 10.0 -> 8.7; one plane per block (the ONE form) 11.6.  Where one plane fills the chip the long
// march stays.  So it does for sweeps and the FP64 residual with its norm in long thin boxes, whose
// plane is one block (bx == 1), part of its threads idle, and two planes per block make more
// blocks than the chip holds (`cap`): V-cycle iteration with the sweeps in registers and as the
// march, 4097x9x9 red-black FP64 187 and 165 us (with the norm as well 159), FP32 199 and 174,
// Jacobi FP64 116 and 105, 2049x17x17 red-black 132 and 126; the plain residual is 1-3% apart, the
// FP32 residual faster in registers (with norm 199 against 202).
template <typename T, int OP>
int planes_in_registers(const Geom& G, int bx, int ichunk, int cap, bool norm) {
    if (ichunk == 1) return 0;
    auto fits = [&](int P) { return (G.nx + P - 1) / P <= kMaxGridRows ? P : 0; };
    if ((long long)G.nx * G.ny * G.nz < kShortMarchMinPoints) {
        const bool sweep_or_norm64 = OP != OP_RESIDUAL || (norm && sizeof(T) == 8);
        return bx == 1 && (G.nx + 1) / 2 > cap && sweep_or_norm64 ? 0 : fits(2);
    }
    constexpr int kShort = sizeof(T) == 8 ? 4 : 3;
    if (ichunk > kShort || (OP == OP_RESIDUAL && sizeof(T) == 8)) return 0;
    return fits(3);
}

// Arguments of a stencil over level l, but for the planes per block.
template <typename T>
StencilArgs<T> level_stencil(mgp_solver* s, int l, const void* src, void* dst, T omega, int colour, unsigned long long* norm) {
    LevelState& L = s->lv[l];
    StencilArgs<T> a;
    a.G = L.G;
    a.src = (const T*)src;
    a.dst = (T*)dst;
    a.f = (const T*)L.f;
    a.F = faces_of<T>(s, l);
    // Constants formed as in jacobi.h:41-44 / gaussseidel.h:32-34 / neumann.h:117
    // (T-typed locals computed from the double-typed settings.h).
    a.two_h = (T)(2.0 * L.h);
    a.hsq = (T)(L.h * L.h);
    a.one_omega = (T)(1.0 - omega);
    a.omega_sixth = (T)(omega / 6.0);
    hsq_terms(a.hsq, a.inv_hsq, a.hsq_pow2);
    a.colour = colour;
    a.norm = norm;
    return a;
}

// How a stencil over level l is cut: bx blocks cover a plane, `chunks` of `ichunk` planes; regs: in
// the register form (k_stencil_planes), else the march.
struct StencilShape {
    int bx = 1, chunks = 1, ichunk = 1;
    bool regs = false;
    dim3 grid() const { return dim3(bx, chunks); }
};
template <typename T, int OP>
StencilShape stencil_shape(mgp_solver* s, int l, bool norm) {
    LevelState& L = s->lv[l];
    constexpr int V = VecT<T>::V;
    StencilShape q;
    const int plane = L.G.ny * ((L.G.nz + V - 1) / V);  // threads per plane
    q.bx = (plane + kThreads - 1) / kThreads;
    int cap = 0;  // resident blocks; 0: an explicit shape
    if constexpr (OP != OP_GS_COLUMN) {
        const bool nrm = OP == OP_RESIDUAL && norm;
        const int planes = L.tune[OP == OP_RESIDUAL ? (nrm ? MGP_TUNE_NORM_PLANES : MGP_TUNE_RESID_PLANES)
                                                    : MGP_TUNE_RELAX_PLANES];
        if (planes > 0) {
            q.chunks = (L.G.nx + planes - 1) / planes;
        } else {
            cap = sm_count(s->device) * (nrm ? (std::is_same<T, double>::value ? resident_blocks(k_residual_norm64<false>)
                                                                               : resident_blocks(k_stencil<T, OP, true>))
                                             : resident_blocks(k_stencil<T, OP, false>));
            q.chunks = march_chunks(q.bx, L.G.nx, cap);
            q.chunks = short_march_chunks<T>(L.G, q.bx, cap, q.chunks);
        }
    }
    q.ichunk = (L.G.nx + q.chunks - 1) / q.chunks;
    if constexpr (OP != OP_GS_COLUMN) {
        const int P = cap ? planes_in_registers<T, OP>(L.G, q.bx, q.ichunk, cap, norm) : 0;
        q.regs = P != 0;
        if (P) q.ichunk = P;
    }
    q.chunks = (L.G.nx + q.ichunk - 1) / q.ichunk;
    return q;
}

template <typename T, int OP>
int launch_stencil(mgp_solver* s, int l, const void* src, void* dst, T omega, int colour, unsigned long long* norm) {
    const StencilShape q = stencil_shape<T, OP>(s, l, norm != nullptr);
    StencilArgs<T> a = level_stencil<T>(s, l, src, dst, omega, colour, norm);
    a.ichunk = q.ichunk;
    const dim3 grid = q.grid();
    if constexpr (OP != OP_GS_COLUMN) {
        if (q.regs) {
            if constexpr (OP == OP_RESIDUAL) {
                if (norm && q.ichunk == 2) return launch_k(s, k_stencil_planes<T, OP, true, 2>, grid, dim3(kThreads), 0, a);
                if constexpr (std::is_same<T, float>::value)
                    if (norm) return launch_k(s, k_stencil_planes<T, OP, true, 3>, grid, dim3(kThreads), 0, a);
            }
            if (q.ichunk == 2) return launch_k(s, k_stencil_planes<T, OP, false, 2>, grid, dim3(kThreads), 0, a);
            if constexpr (!(OP == OP_RESIDUAL && std::is_same<T, double>::value))
                return launch_k(s, k_stencil_planes<T, OP, false, 3>, grid, dim3(kThreads), 0, a);
        }
    }
    if constexpr (std::is_same<T, double>::value && OP == OP_RESIDUAL) {
        if (norm) {
            if (a.ichunk == 1) return launch_k(s, k_residual_norm64<true>, grid, dim3(kThreads), 0, a);
            return launch_k(s, k_residual_norm64<false>, grid, dim3(kThreads), 0, a);
        }
    }
    if (OP != OP_GS_COLUMN && a.ichunk == 1) {  // one plane per block: the one-round-trip form
        if (OP == OP_RESIDUAL && norm) return launch_k(s, k_stencil<T, OP, true, true>, grid, dim3(kThreads), 0, a);
        return launch_k(s, k_stencil<T, OP, false, true>, grid, dim3(kThreads), 0, a);
    }
    if (OP == OP_RESIDUAL && norm) return launch_k(s, k_stencil<T, OP, true>, grid, dim3(kThreads), 0, a);
    return launch_k(s, k_stencil<T, OP, false>, grid, dim3(kThreads), 0, a);
}

// Residual requests a relaxation may take over: on wavefront levels the pass of its last
// sweep also forms the residual of the result -- r stored (the coarse-grid set-up's residual),
// or r stored with its max-norm (the solve loop's).
enum { RESID_NONE = 0, RESID_STORE = 1, RESID_NORM = 2 };

// later: another relaxation of this level follows in the same cycle before anything reads
// u_prev (the pre-smoothing of a V- or F-cycle), so a sweep pair that ends the call may leave
// u_prev's relaxed points stale: that later relaxation overwrites all of them.
// resid / norm: a residual request (above); *resid_done tells whether it was taken over (the
// caller forms the residual itself otherwise).
template <typename T>
int relax_t(mgp_solver* s, int l, double omega, int64_t nsmooth, bool later = false, int resid = RESID_NONE,
            unsigned long long* norm = nullptr, bool* resid_done = nullptr) {
    // Relaxation<T>::relax (include/relaxation.h:19-94)
    LevelState& L = s->lv[l];
    if (resid_done) *resid_done = false;
    // first_done: the coarse-grid set-up that just zeroed this level also wrote its first sweep
    const bool skip_first = L.first_done;
    L.first_done = false;
    if (s->desc.relaxation == MGP_JACOBI) {
        int64_t it = 0;
        if (skip_first && nsmooth > 0) {
            L.cur ^= 1;  // that sweep's swap_u
            it = 1;
        }
        if (L.wave && L.tune[MGP_TUNE_WAVE] != 1) {
            // the fused residual multiplies by 1/h^2, which is exact where h^2 is a power of two
            T hsq = (T)(L.h * L.h), inv;
            int pow2 = 0;
            hsq_terms(hsq, inv, pow2);
            while (it < nsmooth) {
                const int nj = nsmooth - it >= 2 ? 2 : 1;
                const bool last = it + nj >= nsmooth;
                const int res = last && pow2 ? resid : RESID_NONE;
                CKS(launch_wave<T>(s, l, nj, res, nj == 2 && last && !later, (T)omega, norm));
                if (res != RESID_NONE && resid_done) *resid_done = true;
                it += nj;
            }
            return MGP_OK;
        }
        for (; it < nsmooth; it++) {
            L.cur ^= 1;  // swap_u: the previous iterate becomes the source
            CKS((launch_stencil<T, OP_JACOBI>(s, l, uprev_ptr(s, l), u_ptr(s, l), (T)omega, 0, nullptr)));
        }
    } else {
        for (int64_t it = 0; it < 2 * nsmooth; it++) {
            const int colour = s->gs_alternate ? 0 : 1;
            void* u = u_ptr(s, l);
            if (!(it == 0 && skip_first)) {
                if (L.gs_column) CKS((launch_stencil<T, OP_GS_COLUMN>(s, l, u, u, (T)omega, colour, nullptr)));
                else CKS((launch_stencil<T, OP_GS>(s, l, u, u, (T)omega, colour, nullptr)));
            }
            s->gs_alternate = !s->gs_alternate;
        }
    }
    return MGP_OK;
}

// One red-black half-sweep of a given colour (mgp_relax_colour); the alternate flag stays.
template <typename T>
int relax_colour_t(mgp_solver* s, int l, double omega, int colour) {
    LevelState& L = s->lv[l];
    L.first_done = false;
    void* u = u_ptr(s, l);
    if (L.gs_column) return launch_stencil<T, OP_GS_COLUMN>(s, l, u, u, (T)omega, colour, nullptr);
    return launch_stencil<T, OP_GS>(s, l, u, u, (T)omega, colour, nullptr);
}

template <typename T>
int residual_t(mgp_solver* s, int l, unsigned long long* norm) {
    LevelState& L = s->lv[l];
    // with a norm, the march also takes the stored r outside the relaxation bounds
    return launch_stencil<T, OP_RESIDUAL>(s, l, u_ptr(s, l), L.r, T(0), 0, norm);
}

View level_view(const LevelState& L) {
    View v;
    v.n[0] = L.G.nx; v.n[1] = L.G.ny; v.n[2] = L.G.nz;
    v.s0 = L.G.sx; v.s1 = L.G.sy;
    return v;
}
View face_view(const int64_t* fs) {
    View v;
    v.n[0] = (int)fs[0]; v.n[1] = (int)fs[1]; v.n[2] = (int)fs[2];
    v.s0 = fs[1] * fs[2]; v.s1 = fs[2];
    return v;
}

template <typename T>
RestrictArgs<T> restrict_args(mgp_solver* s, int l, bool zero_coarse_u, long long* npts) {
    LevelState& F = s->lv[l];
    LevelState& C = s->lv[l + 1];
    RestrictArgs<T> a;
    a.in = (const T*)F.r;
    a.vi = level_view(F);
    a.out = (T*)C.f;
    a.vo = level_view(C);
    a.zero_u = zero_coarse_u ? (T*)u_ptr(s, l + 1) : nullptr;
    a.fw = s->desc.restriction == MGP_FULLWEIGHTING;
    a.fs = FirstSweep<T>{};
    *npts = (long long)C.G.nx * C.G.ny * C.G.nz;
    return a;
}

// The first sweep of level l+1, written by the set-up of level l (it runs right before that
// level's relaxation in every cycle), with the constants launch_stencil would form.  Off for
// column-ordered Gauss-Seidel (a sequential sweep) and without smoothing.
template <typename T>
FirstSweep<T> first_sweep_of(mgp_solver* s, int l, double omega, int64_t ns) {
    FirstSweep<T> w{};
    LevelState& C = s->lv[l + 1];
    if (ns < 1 || C.gs_column) return w;
    w.on = 1;
    w.gs = s->desc.relaxation == MGP_GAUSSSEIDEL;
    w.colour = s->gs_alternate ? 0 : 1;
    w.uw = w.gs ? (T*)u_ptr(s, l + 1) : (T*)C.ubuf[C.cur ^ 1];
    for (int f = 0; f < 6; f++) w.gc[f] = (const T*)C.face[f];
    w.G = C.G;
    const T om = (T)omega;
    w.one_omega = (T)(1.0 - om);
    w.omega_sixth = (T)(om / 6.0);
    w.hsq = (T)(C.h * C.h);
    w.two_h = (T)(2.0 * C.h);
    return w;
}

template <typename T>
int restrict_t(mgp_solver* s, int l, bool zero_coarse_u, const FirstSweep<T>& w = FirstSweep<T>{}) {
    long long n = 0;
    RestrictArgs<T> a = restrict_args<T>(s, l, zero_coarse_u, &n);
    a.fs = w;
    const LevelState& C = s->lv[l + 1];
    const dim3 grid((C.G.ny * C.G.nz + kThreads - 1) / kThreads, C.G.nx);
    if (a.zero_u && a.fs.on) return launch_k(s, k_restrict<T, true>, grid, dim3(kThreads), 0, a);
    return launch_k(s, k_restrict<T, false>, grid, dim3(kThreads), 0, a);
}

template <typename T>
BcRestrictArgs<T> bc_args(mgp_solver* s, int l, bool* any);

template <typename T>
int restrict_bc_t(mgp_solver* s, int l, cudaStream_t on = nullptr) {
    bool any = false;
    BcRestrictArgs<T> a = bc_args<T>(s, l, &any);
    // Dirichlet faces: coarse g = 0 (dirichlet.h:101-107).  Coarse Dirichlet arrays are
    // zero from allocation and nothing in a cycle writes them, so there is nothing to launch.
    if (!any) return MGP_OK;
    LevelState& C = s->lv[l + 1];
    long long nmax = 1;
    for (int f = 0; f < 6; f++)
        nmax = std::max(nmax, (long long)(C.face_shape[f][0] * C.face_shape[f][1] * C.face_shape[f][2]));
    dim3 grid((unsigned)std::max(1ll, std::min((nmax + kThreads - 1) / kThreads, 4096ll)), 6);
    if (on) {  // the side stream: an ordinary launch after the fork event
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = grid;
        cfg.blockDim = dim3(kThreads);
        cfg.stream = on;
        const cudaError_t e = cudaLaunchKernelEx(&cfg, k_restrict_bc<T>, a);
        if (e != cudaSuccess) return fail(MGP_ERR_CUDA, "kernel launch: %s", cudaGetErrorString(e));
        return check_launch(s);
    }
    return launch_k(s, k_restrict_bc<T>, grid, dim3(kThreads), 0, a);
}

template <typename T, bool ADD>
int prolong_t(mgp_solver* s, int l) {
    LevelState& F = s->lv[l];
    LevelState& C = s->lv[l + 1];
    constexpr int V = VecT<T>::V;
    const int rows = C.G.ny * ((F.G.nz + V - 1) / V);  // one thread per coarse (j) row x fine k-vector
    dim3 grid((rows + kThreads - 1) / kThreads, C.G.nx);
    ProlongArgs<T> a{(const T*)u_ptr(s, l + 1), C.G, (T*)u_ptr(s, l), (T*)F.r, F.G};
    return launch_k(s, k_prolong<T, ADD>, grid, dim3(kThreads), 0, a);
}

// Prolongation + add and the first Jacobi sweep after it in one pass (k_prolong_sweep): Jacobi
// levels >= 1, unless tuned off or relaxed by the wavefront passes, with nsmooth even and at
// least 2.  Even: between the set-up that zeroed the coarse u and this prolongation the coarse
// level is swept 2*nsmooth (V-cycle), nsmooth (coarsest level) or 3*nsmooth (F-cycle) times, so
// with nsmooth even the prolongation reads the zeroed buffer, whose unrelaxed (Dirichlet)
// points are +0 -- the condition under which the kernel may leave u' unstored.  With nsmooth
// odd it reads the other buffer, whose Dirichlet points hold whatever they held.
// Built in only on levels of at most 2^16 points (MGP_TUNE_PROLONG_SWEEP = 2 forces it): forming
// u' at seven points per thread makes larger levels instruction-bound -- on B200 the 513x257x129
// F-cycle iteration took 1.585 ms fused on levels 1-4 against 1.453 ms separate, and the
// autotuner keeps the separate passes on its 2.15M- and 277K-point levels.  Levels of at most
// 30000 points run in the cluster, which leaves it those up to 65536 and the ones kept out; there
// the separate passes are the faster ones by now (65^3 Jacobi F-cycle, 35937 points: 186 us per
// iteration fused, 179 separate; 257x129x65, 36465 points: 333 and 327).
constexpr long long kProlongSweepMaxPoints = 1ll << 16;
bool prolong_sweep_fused(const mgp_solver* s, int l, int64_t ns) {
    const LevelState& L = s->lv[l];
    const int t = L.tune[MGP_TUNE_PROLONG_SWEEP];
    if (!(s->desc.relaxation == MGP_JACOBI && l >= 1 && ns >= 2 && (ns & 1) == 0 && !L.wave && !L.first_done) ||
        t == 1)
        return false;
    return t == 2 || (long long)L.G.nx * L.G.ny * L.G.nz <= kProlongSweepMaxPoints;
}

template <typename T>
int prolong_sweep_t(mgp_solver* s, int l, double omega) {
    LevelState& F = s->lv[l];
    LevelState& C = s->lv[l + 1];
    ProlongSweepArgs<T> a;
    a.uc = (const T*)u_ptr(s, l + 1);
    a.Gc = C.G;
    a.u = (T*)u_ptr(s, l);
    a.dst = (T*)uprev_ptr(s, l);
    a.f = (const T*)F.f;
    a.r = (T*)F.r;
    a.Gf = F.G;
    a.F = faces_of<T>(s, l);
    const T om = (T)omega;  // the relaxation takes omega as a T (jacobi.h:41-44)
    a.two_h = (T)(2.0 * F.h);
    a.hsq = (T)(F.h * F.h);
    a.one_omega = (T)(1.0 - om);
    a.omega_sixth = (T)(om / 6.0);
    const dim3 grid((F.G.ny * F.G.nz + kThreads - 1) / kThreads, F.G.nx);
    CKS(launch_k(s, k_prolong_sweep<T>, grid, dim3(kThreads), 0, a));
    F.cur ^= 1;  // the sweep's swap_u: u is now the other buffer
    return MGP_OK;
}

template <typename T>
int add_t(mgp_solver* s, int l) {
    LevelState& L = s->lv[l];
    const long long n = (long long)L.G.nx * L.G.ny * L.G.nz;
    return launch_k(s, k_add<T>, dim3(grid_1d(s, n)), dim3(kThreads), 0, (T*)u_ptr(s, l), (const T*)L.r, L.G);
}

template <typename T>
int zero_u_t(mgp_solver* s, int l) {
    CK(cudaMemsetAsync(u_ptr(s, l), 0, s->lv[l].elems * sizeof(T), s->stream));
    return MGP_OK;
}

template <typename T>
int norm_t(mgp_solver* s, const void* a, int l, unsigned long long* out) {
    LevelState& L = s->lv[l];
    const int bx = (L.G.ny * L.G.nz + kThreads - 1) / kThreads;
    const int chunks = std::max(1, std::min(L.G.nx, sm_count(s->device) * 8 / bx));
    return launch_k(s, k_norm<T>, dim3(bx, chunks), dim3(kThreads), 0, (const T*)a, L.G, out);
}

template <typename T>
BcRestrictArgs<T> bc_args(mgp_solver* s, int l, bool* any) {
    BcRestrictArgs<T> a;
    LevelState& F = s->lv[l];
    LevelState& C = s->lv[l + 1];
    *any = false;
    for (int f = 0; f < 6; f++) {
        a.gf[f] = (const T*)F.face[f];
        a.gc[f] = (T*)C.face[f];
        a.vf[f] = face_view(F.face_shape[f]);
        a.vc[f] = face_view(C.face_shape[f]);
        a.neumann[f] = s->face_kind[f] == MGP_NEUMANN;
        *any |= a.neumann[f] != 0;
    }
    a.u = (const T*)u_ptr(s, l);
    a.Gf = F.G;
    a.h = (T)F.h;
    a.fw = s->desc.restriction == MGP_FULLWEIGHTING;
    return a;
}

// Coarse-grid correction set-up (vcycle.h:34-76, fcycle.h:130-172) in one launch:
// residual(l) -> restrict -> u_{l+1}.init_zero(), plus the Neumann face restriction.
template <typename T>
int coarse_setup_fused_t(mgp_solver* s, int l, const FirstSweep<T>& w) {
    LevelState& F = s->lv[l];
    LevelState& C = s->lv[l + 1];
    constexpr int V = VecT<T>::V;
    RRArgs<T> a;
    a.fs = w;
    a.Gf = F.G;
    a.Gc = C.G;
    a.u = (const T*)u_ptr(s, l);
    a.f = (const T*)F.f;
    a.r = (const T*)F.r;
    a.fc = (T*)C.f;
    a.uc = (T*)u_ptr(s, l + 1);
    a.F = faces_of<T>(s, l);
    a.two_h = (T)(2.0 * F.h);
    a.hsq = (T)(F.h * F.h);
    hsq_terms(a.hsq, a.inv_hsq, a.hsq_pow2);
    a.fw = s->desc.restriction == MGP_FULLWEIGHTING;
    // Coarse tile: tkc points along k (balanced over the k tiles of a row; 2*tkc a multiple of
    // V keeps the fine rows' vectors aligned) by tjc rows, chosen for the fewest idle lanes
    // per coarse point in blocks of at most 384 threads (two blocks per SM).
    const int kmax = V == 2 ? 31 : 30;
    const int ntk = (C.G.nz + kmax - 1) / kmax;
    int tkc = (C.G.nz + ntk - 1) / ntk;
    tkc = (2 * tkc + V - 1) / V * V / 2;
    const int tkv = 2 * tkc / V + 1;
    int tjc = 1;
    double best = 1e30;
    for (int c = 1; c <= std::min(C.G.ny, 16); c++) {
        const int thr = tkv * (2 * c + 1);
        if (thr > 384) break;
        const double cost = (double)((thr + 31) / 32 * 32) / (double)(c * std::min(tkc, C.G.nz));
        if (cost < best - 1e-9) {
            best = cost;
            tjc = c;
        }
    }
    const int rows = 2 * tjc + 1;
    a.tkc = tkc;
    a.tjc = tjc;
    a.tiles_j = (C.G.ny + tjc - 1) / tjc;
    a.tiles_k = (C.G.nz + tkc - 1) / tkc;
    const int tiles = a.tiles_j * a.tiles_k;
    const size_t smem = rr_smem_bytes<T>(tkv, rows);
    static bool attr_set[2][64] = {};  // per dtype and device
    bool& set = attr_set[sizeof(T) == 8][s->device & 63];
    if (!set) {
        // the largest block (384 threads) needs less than 160 KB
        CK(cudaFuncSetAttribute(k_resid_restrict<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, 160 * 1024));
        set = true;
    }
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_resid_restrict<T>, tkv * rows, smem) != cudaSuccess ||
        per_sm < 1)
        per_sm = 1;
    const int tuned = s->lv[l].tune[MGP_TUNE_SETUP_PLANES];
    const int chunks = tuned > 0 ? (C.G.nx + tuned - 1) / tuned : march_chunks(tiles, C.G.nx, sm_count(s->device) * per_sm);
    a.ci = (C.G.nx + chunks - 1) / chunks;
    const int nchunks = (C.G.nx + a.ci - 1) / a.ci;
    a.main_blocks = tiles * nchunks;
    bool any = false;
    a.bc = bc_args<T>(s, l, &any);
    int extra = 0;
    a.bc_blocks_per_face = 1;
    if (any) {
        long long nmax = 1;
        for (int f = 0; f < 6; f++)
            nmax = std::max(nmax, (long long)(C.face_shape[f][0] * C.face_shape[f][1] * C.face_shape[f][2]));
        a.bc_blocks_per_face = (int)std::max(1ll, std::min(64ll, (nmax + tkv * rows - 1) / (tkv * rows)));
        extra = 6 * a.bc_blocks_per_face;
    }
    return launch_k(s, k_resid_restrict<T>, dim3(a.main_blocks + extra), dim3(tkv, rows), smem, a);
}

// The three-kernel form (large levels): residual (r stored), restriction with u_{l+1} = 0
// fused, Neumann face restriction.  The one-kernel form leaves r unstored where the residual
// is formed; nothing reads those values before the next residual overwrites them.
// The one-kernel form is built in only on levels of at most kFusedSetupMaxPoints points, the size
// up to which visits run in one cluster anyway (so it serves levels kept out of the cluster).
// Above that the residual and the restriction, now both bound by little more than their launch,
// are faster apart: with the separate kernels down to 36K points instead of 2^20, on B200 per
// solve iteration, 161x97x193 576 -> 539 us, 129x65x65 276 -> 246, 65^3 red-black 251 -> 239,
// 513x257x129 1619 -> 1600, 257x257x129 red-black 1246 -> 1225.  MGP_FLAG_FUSED_SETUP uses the
// one-kernel form on every level.
constexpr long long kFusedSetupMaxPoints = 30000;

// The set-up of level l forms its residual in a separate pass (the three-kernel form), which
// the relaxation before it may take over.
bool setup_residual_separate(const mgp_solver* s, int l) {
    const Geom& G = s->lv[l].G;
    if (s->desc.flags & MGP_FLAG_FUSED_SETUP) return false;
    const int form = s->lv[l].tune[MGP_TUNE_SETUP_FORM];
    if (form) return form == 1;
    return (long long)G.nx * G.ny * G.nz > kFusedSetupMaxPoints;
}

// The residual of level l and the Neumann face restriction to level l+1 in one launch, where the
// residual takes its built-in shape on levels below kFacesMaxPoints (*done tells).  The side
// stream adds a branch to the captured graph at every visit, which the first solve of a solver
// pays for (capture and instantiation), Neumann face or not; on B200, four iterations (three on
// 257x129x65), with the side stream on every level above 30000 points, and now: 161x97x193 3.81 ->
// 2.74 ms, 257x129x65 1.87 -> 1.31, 513x257x129 F 6.83 -> 6.17 and V 3.38 -> 3.20 (6.34 and 3.26
// with the limit at 2^20), 65^3 all Dirichlet 2.92 -> 2.50; later solves take the same time.
// Above the limit the residual is a march of its own and the side stream stays.
constexpr long long kFacesMaxPoints = kShortMarchMinPoints;
template <typename T>
int residual_faces_t(mgp_solver* s, int l, bool* done) {
    *done = false;
    const Geom& G = s->lv[l].G;
    if ((long long)G.nx * G.ny * G.nz >= kFacesMaxPoints) return MGP_OK;
    const StencilShape q = stencil_shape<T, OP_RESIDUAL>(s, l, false);
    if (!(q.regs && q.ichunk == 2) && !(q.ichunk == 1 && !s->lv[l].tune[MGP_TUNE_RESID_PLANES])) return MGP_OK;
    ResidualFacesArgs<T> a;
    bool any = false;
    a.s = level_stencil<T>(s, l, u_ptr(s, l), s->lv[l].r, T(0), 0, nullptr);
    a.s.ichunk = q.ichunk;
    a.bc = bc_args<T>(s, l, &any);
    long long nmax = 1;
    for (int f = 0; f < 6; f++) {
        const int64_t* fs = s->lv[l + 1].face_shape[f];
        nmax = std::max(nmax, (long long)(fs[0] * fs[1] * fs[2]));
    }
    a.per_face = (int)((nmax + kThreads - 1) / kThreads);
    a.rows = (6 * a.per_face + q.bx - 1) / q.bx;
    if (q.chunks + a.rows > kMaxGridRows) return MGP_OK;
    *done = true;
    const dim3 grid(q.bx, q.chunks + a.rows);
    if (q.regs) return launch_k(s, k_residual_faces<T, 2>, grid, dim3(kThreads), 0, a);
    return launch_k(s, k_residual_faces<T, 1>, grid, dim3(kThreads), 0, a);
}

// resid_done: the relaxation before the set-up already stored r (wavefront pass).
template <typename T>
int coarse_setup_t(mgp_solver* s, int l, double omega, int64_t ns, bool resid_done = false) {
    const FirstSweep<T> w = first_sweep_of<T>(s, l, omega, ns);
    if (!setup_residual_separate(s, l)) {
        CKS(coarse_setup_fused_t<T>(s, l, w));
    } else {
        // The face restriction (reads u and the fine faces) and the residual (reads u, writes r)
        // are independent: the face restriction runs in blocks of the residual's launch or, beside
        // longer ones, on the side stream, joined before the restriction, whose first coarse sweep
        // reads the coarse faces.
        bool any = false, done = false;
        for (int f = 0; f < 6; f++) any = any || s->face_kind[f] == MGP_NEUMANN;
        if (any && !resid_done) CKS(residual_faces_t<T>(s, l, &done));
        if (done) {
            // r and the coarse faces are there
        } else if (any && !resid_done && s->side) {
            CK(cudaEventRecord(s->ev_fork, s->stream));
            CK(cudaStreamWaitEvent(s->side, s->ev_fork, 0));
            CKS(restrict_bc_t<T>(s, l, s->side));
            CK(cudaEventRecord(s->ev_join, s->side));
            CKS(residual_t<T>(s, l, nullptr));
            CK(cudaStreamWaitEvent(s->stream, s->ev_join, 0));
        } else {
            if (!resid_done) CKS(residual_t<T>(s, l, nullptr));
            CKS(restrict_bc_t<T>(s, l));
        }
        CKS(restrict_t<T>(s, l, /*zero_coarse_u=*/true, w));
    }
    s->lv[l + 1].first_done = w.on != 0;
    return MGP_OK;
}

// ---- the coarsest levels in one CTA (mgp_tail.cuh) -------------------------------------
constexpr size_t kTailMaxSmem = 220 * 1024;

size_t tail_level_bytes(const mgp_solver* s, int l) {
    const LevelState& L = s->lv[l];
    const size_t n = (size_t)L.G.nx * L.G.ny * L.G.nz;
    size_t faces = 0;
    for (int f = 0; f < 6; f++) faces += (size_t)(L.face_shape[f][0] * L.face_shape[f][1] * L.face_shape[f][2]);
    const int fields = s->desc.relaxation == MGP_JACOBI ? 4 : 3;
    return (fields * n + faces) * s->esize;
}

// First level of the tail (0: none, the default): the smallest l >= 1 whose levels l..L-1 all
// fit.  Not for column-ordered Gauss-Seidel layouts (their sweep order runs along i) nor for
// levels whose Jacobi buffers rotate with a third one.  Off unless MGP_TUNE_TAIL asks for it:
// on B200 the 513x257x129 F-cycle iteration takes 1.72 ms with the tail (levels 4-5, one block
// per visit) against 1.45 ms with the grid kernels -- one SM works through the 5049-point level
// at tens of microseconds per visit where the grid launches spread each operation over all SMs.
int tail_level(const mgp_solver* s) {
    if (s->levels < 2 || s->lv[0].tune[MGP_TUNE_TAIL] != 1) return 0;
    for (int l = 1; l < s->levels; l++) {
        if (s->levels - l > kTailMaxLevels) continue;
        size_t bytes = 0;
        bool ok = true;
        for (int m = l; m < s->levels; m++) {
            bytes += tail_level_bytes(s, m);
            ok = ok && !s->lv[m].gs_column && !s->lv[m].pair;
        }
        if (ok && bytes <= kTailMaxSmem) return l;
    }
    return 0;
}

template <typename T>
int launch_tail(mgp_solver* s, int t0, bool fcycle, double omega, int64_t ns) {
    TailArgs<T> a{};
    static_assert(sizeof(TailArgs<T>) % sizeof(int) == 0, "the kernel copies its arguments as ints");
    a.nl = s->levels - t0;
    a.ns = (int)ns;
    a.jacobi = s->desc.relaxation == MGP_JACOBI;
    a.fw = s->desc.restriction == MGP_FULLWEIGHTING;
    a.alt = s->gs_alternate;
    int off = 0;
    for (int m = 0; m < a.nl; m++) {
        LevelState& L = s->lv[t0 + m];
        TailLevel<T>& q = a.L[m];
        q.G = L.G;
        q.ub[0] = (T*)L.ubuf[0];
        q.ub[1] = a.jacobi ? (T*)L.ubuf[1] : nullptr;
        q.f = (T*)L.f;
        q.r = (T*)L.r;
        // constants as launch_stencil and bc_args form them (jacobi.h:41-44, neumann.h:117):
        // the relaxation takes omega as a T, so it is rounded to T first
        const T om = (T)omega;
        q.two_h = (T)(2.0 * L.h);
        q.hsq = (T)(L.h * L.h);
        q.one_omega = (T)(1.0 - om);
        q.omega_sixth = (T)(om / 6.0);
        q.h = (T)L.h;
        hsq_terms(q.hsq, q.inv_hsq, q.pow2);
        const int n = L.G.nx * L.G.ny * L.G.nz;
        q.so_u[0] = off;
        off += n;
        q.so_u[1] = a.jacobi ? off : q.so_u[0];
        if (a.jacobi) off += n;
        q.so_f = off;
        off += n;
        q.so_r = off;
        off += n;
        for (int f = 0; f < 6; f++) {
            q.g[f] = (T*)L.face[f];
            q.gn[f] = (int)(L.face_shape[f][0] * L.face_shape[f][1] * L.face_shape[f][2]);
            q.neumann[f] = s->face_kind[f] == MGP_NEUMANN;
            q.so_g[f] = off;
            off += q.gn[f];
        }
        a.cur[m] = L.cur;
    }
    // The visit as a program (vcycle_t / fcycle_t's recursion), and the host state it leaves:
    // each Jacobi sweep swaps the pair (a skipped first one included); red-black relaxations flip
    // `alternate` 2*nsmooth times, which leaves it as it was.
    a.nops = 0;
    bool over = false;
    auto emit = [&](int op, int m) {
        if (a.nops >= kTailMaxOps) {
            over = true;
            return;
        }
        a.op[a.nops] = (unsigned char)op;
        a.lv[a.nops] = (unsigned char)m;
        a.nops++;
    };
    auto relax = [&](int m, bool skip) {
        emit(skip ? TAIL_RELAX_SKIP1 : TAIL_RELAX, m);
        if (a.jacobi) s->lv[t0 + m].cur ^= (int)(ns & 1);
    };
    const bool skip0 = s->lv[t0].first_done && ns > 0;
    std::function<void(int, bool)> v = [&](int m, bool skip) {
        relax(m, skip);
        if (m >= a.nl - 1) return;
        emit(TAIL_SETUP, m);
        v(m + 1, false);
        emit(TAIL_PROLONG, m);
        relax(m, false);
    };
    std::function<void(int, bool)> f = [&](int m, bool skip) {
        relax(m, skip);
        emit(TAIL_SETUP, m);
        if (m + 1 < a.nl - 1) f(m + 1, false);
        v(m + 1, false);
        emit(TAIL_PROLONG, m);
    };
    const uint64_t state_before = state_bits(s);
    if (fcycle) f(0, skip0);
    else v(0, skip0);
    if (over) {
        set_state_bits(s, state_before);
        return fail(MGP_ERR_UNSUPPORTED, "coarse-level visit longer than %d operations", kTailMaxOps);
    }
    for (int m = 0; m < a.nl; m++) s->lv[t0 + m].first_done = false;
    const size_t smem = (size_t)off * sizeof(T);
    static bool attr_set[2][64] = {};
    bool& set = attr_set[sizeof(T) == 8][s->device & 63];
    if (!set) {
        CK(cudaFuncSetAttribute(k_tail<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTailMaxSmem));
        set = true;
    }
    return launch_k(s, k_tail<T>, dim3(1), dim3(kTailThreads), smem, a);
}

// ---- the coarse levels in one cluster (mgp_cluster.cuh) -----------------------------------
// The cluster's finest level has at most kClMaxPoints points: its 16 SMs work a 36K-point level off
// more slowly than the grid kernels do on all of them (65^3 red-black F-cycle 239 us per iteration
// with level 1, 36K points, in the cluster and 229 without; 129x65x65 in FP32, 70K points, 276 and
// 258), while 18.5K points still gain (33x33x17 118 against 128 us).
constexpr long long kClMaxPoints = kFusedSetupMaxPoints;
constexpr size_t kClMaxSmem = 216 * 1024;  // dynamic; the argument copy and reduction slots fit beside it

// CTAs of the largest cluster this device co-schedules with that much shared memory: 16 (opt-in
// size), 8, or 0 (none).
int cluster_ctas(int dev) {
    static std::mutex mu;
    static int cached[64] = {};  // 0: not asked yet, else CTAs + 1
    std::lock_guard<std::mutex> lk(mu);
    int& c = cached[dev & 63];
    if (c) return c - 1;
    int best = 0;
    auto kernels = {(const void*)k_cluster<double, true, true>,   (const void*)k_cluster<float, true, true>,
                    (const void*)k_cluster<double, false, false>, (const void*)k_cluster<float, false, false>,
                    (const void*)k_cluster<double, false, true>,  (const void*)k_cluster<float, false, true>};
    for (int n : {16, 8}) {
        bool ok = true;
        for (const void* k : kernels) {
            cudaLaunchAttribute attr[1];
            attr[0].id = cudaLaunchAttributeClusterDimension;
            attr[0].val.clusterDim.x = n;
            attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
            cudaLaunchConfig_t cfg = {};
            cfg.gridDim = dim3(n);
            cfg.blockDim = dim3(kClMaxThreads);
            cfg.dynamicSmemBytes = kClMaxSmem;
            cfg.attrs = attr;
            cfg.numAttrs = 1;
            int active = 0;
            ok = ok && cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kClMaxSmem) == cudaSuccess &&
                 cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess &&
                 cudaOccupancyMaxActiveClusters(&active, k, &cfg) == cudaSuccess && active >= 1;
        }
        if (ok) {
            best = n;
            break;
        }
    }
    cudaGetLastError();  // a refused size leaves an error behind
    c = best + 1;
    return best;
}

unsigned div_magic(int d) { return d <= 1 ? 0u : (unsigned)(((1ull << 32) + d - 1) / d); }

// Planes of a CTA's slab: at least two in every slab, the last one included (the east and west
// face restriction reads three planes from the face inwards, two slabs' worth at most).
// Levels on which a sweep updates at most kClOnePoints points go to one CTA: their sweeps then end
// with a block barrier instead of an exchange (820 cycles, more than their arithmetic).  Ten 65^3
// red-black F-cycles 2.55 -> 2.43 ms (9^3 and 5^3 in one CTA), four 33x17x17 Jacobi ones 375 -> 363 us
// (9x5x5); Jacobi levels of 765 and 1001 points are faster in slabs (161x97x193 by 2%); nothing
// between 225 and 765 was measured for Jacobi, nor above 729 for red-black.
constexpr long long kClOnePoints = 512;
int slab_planes(const Geom& G, int nc, bool jacobi) {
    const int nx = G.nx;
    if ((long long)nx * G.ny * G.nz <= (jacobi ? kClOnePoints : 2 * kClOnePoints)) return nx;
    int P = std::max(2, (nx + nc - 1) / nc);
    while (P < nx && nx % P == 1) P++;
    return std::min(P, nx);
}

// Slab shape and shared-memory offsets of levels t..L-1 in a cluster of `nc` CTAs; false when
// they do not fit.  `lev` (may be null) receives them, *smem / *threads the launch's.
template <typename T>
bool cluster_plan(const mgp_solver* s, int t, int nc, ClArgs<T>* a, size_t* smem, int* threads) {
    const bool jac = s->desc.relaxation == MGP_JACOBI;
    long long off = 0, gather = 0;
    int nt = 256;
    for (int m = t; m < s->levels; m++) {
        const LevelState& L = s->lv[m];
        const Geom& G = L.G;
        const int P = slab_planes(G, nc, jac);
        const int rp = G.nz + (G.nz & 1);
        const long long pl = (long long)G.ny * rp;
        if (pl * (4 * P + 6) * (long long)sizeof(T) > (long long)kClMaxSmem * 2) return false;
        const int ncol = std::max(0, G.y1 - G.y0) * std::max(0, G.z1 - G.z0);
        const int nitem = jac ? ncol : (std::max(0, G.y1 - G.y0) + 1) / 2 * std::max(0, G.z1 - G.z0);
        // Threads: one per relaxation item of the finest level, or even passes over the items; an
        // operation's set-up per warp counts, so no more than that (at least 8 warps: the Neumann
        // faces are dealt out to warps).
        if (m == t) {
            const int passes = std::max(1, (nitem + kClMaxThreads - 1) / kClMaxThreads);
            nt = std::max(256, ((nitem + passes - 1) / passes + 31) / 32 * 32);
        }
        auto split = [&](int n) { return n ? std::max(1, std::min(P, nt / n)) : 1; };
        const int nseg = split(nitem), rseg = split(ncol);
        ClLevel<T> q{};
        q.G = G;
        q.P = P;
        q.nact = (G.nx + P - 1) / P;
        q.rp = rp;
        q.pl = (int)pl;
        q.m_rp = div_magic(rp);
        q.nseg = nseg;
        q.seglen = (P + nseg - 1) / nseg;
        q.m_nz = div_magic(G.nz);
        q.m_ny = div_magic(G.ny);
        q.m_yz = div_magic(G.ny * G.nz);
        q.m_pl = div_magic((int)pl);
        q.m_P = div_magic(P);
        q.ncol = ncol;
        q.m_col = div_magic(ncol);
        q.nitem = nitem;
        q.m_item = div_magic(nitem);
        q.rseg = rseg;
        q.rlen = (P + rseg - 1) / rseg;
        auto take = [&](long long n) {
            const long long o = off;
            off += n;
            return (int)o;
        };
        q.so_u[0] = take((P + 2) * pl);
        q.so_u[1] = jac ? take((P + 2) * pl) : q.so_u[0];
        q.so_f = take(P * pl);
        q.so_r = take((P + 2) * pl);
        for (int f = 0; f < 6; f++) {
            q.neumann[f] = s->face_kind[f] == MGP_NEUMANN;
            const long long n = f == MGP_EAST || f == MGP_WEST ? pl : (long long)(P + 2) * (f <= MGP_SOUTH ? G.nz : G.ny);
            q.so_g[f] = q.neumann[f] ? take(n) : 0;
        }
        if (m > t) {
            const LevelState& F = s->lv[m - 1];
            const int Pf = slab_planes(F.G, nc, jac);
            gather = std::max(gather, ((Pf + 2) / 2 + 3) * pl);
        }
        if (off * (long long)sizeof(T) > (long long)kClMaxSmem) return false;
        if (a) a->L[m - t] = q;
    }
    if (a) a->so_gather = (int)off;
    off += gather;
    long long bytes = off * (long long)sizeof(T);
    for (int m = t; m < s->levels; m++) {  // the column tables
        const Geom& G = s->lv[m].G;
        const int wy = std::max(0, G.y1 - G.y0), wz = std::max(0, G.z1 - G.z0);
        if (a) {
            a->L[m - t].so_tab = (int)bytes;
            a->L[m - t].so_pair = (int)bytes + 4 * wy * wz;
        }
        bytes += 4ll * wz * (wy + (jac ? 0 : (wy + 1) / 2));
    }
    *smem = (size_t)bytes;
    *threads = nt;
    return *smem <= kClMaxSmem;
}

// First level of the cluster's visits (s->levels: none): the finest level of at most kClMaxPoints
// points whose hierarchy fits in one cluster's shared memory.  An operation takes 0.5-1.5 us there
// against 2.5-3 us as a launch of its own: without the cluster a solve iteration takes 1588 ->
// 1645 us on 513x257x129, 229 -> 347 us on 65^3 (red-black), 81 -> 128 us on 33x17x17.  Not for
// column-ordered Gauss-Seidel (its sweep runs along x),
// levels with wavefront buffers, or levels whose launch shapes or set-up form were asked for
// (they are shapes of the per-level kernels), nor beside the one-CTA form.
int cluster_level(const mgp_solver* s) {
    if (s->levels < 2 || s->pool || (s->desc.flags & MGP_FLAG_FUSED_SETUP) || s->lv[0].tune[MGP_TUNE_TAIL]) return s->levels;
    const int nc = cluster_ctas(s->device);
    if (!nc) return s->levels;
    for (int l = std::max(0, s->levels - kClMaxLevels); l < s->levels - 1; l++) {
        const Geom& G = s->lv[l].G;
        bool ok = (long long)G.nx * G.ny * G.nz <= kClMaxPoints;
        for (int m = l; m < s->levels && ok; m++) {
            ok = !s->lv[m].gs_column && !s->lv[m].pair;
            for (int p = 0; p < MGP_TUNE_PARAMS; p++) ok = ok && !s->lv[m].tune[p];
        }
        size_t smem = 0;
        int threads = 0;
        if (ok && (s->dtype == MGP_F64 ? cluster_plan<double>(s, l, nc, nullptr, &smem, &threads)
                                       : cluster_plan<float>(s, l, nc, nullptr, &smem, &threads)))
            return l;
    }
    return s->levels;
}

// One visit of levels t..L-1: F(t) when `f`, then V(t) when `v`, then (level 0 only) the solve
// loop's residual with its max-norm into *norm when `norm`.
template <typename T>
int launch_cluster(mgp_solver* s, int t, bool f, bool v, double omega, int64_t ns, unsigned long long* norm = nullptr) {
    static_assert(sizeof(ClArgs<T>) % sizeof(int) == 0, "the kernel copies its arguments as ints");
    ClArgs<T> a{};
    size_t smem = 0;
    int threads = 0;
    const int nc = cluster_ctas(s->device);
    if (!cluster_plan<T>(s, t, nc, &a, &smem, &threads)) return fail(MGP_ERR_STATE, "coarse levels do not fit a cluster");
    const bool jac = s->desc.relaxation == MGP_JACOBI;
    a.nl = s->levels - t;
    a.ns = (int)ns;
    a.fw = s->desc.restriction == MGP_FULLWEIGHTING;
    a.alt = s->gs_alternate;
    a.norm = norm;
    a.err = s->err_word;
    a.polls = s->wait_polls;
    for (int m = 0; m < a.nl; m++) {
        LevelState& L = s->lv[t + m];
        ClLevel<T>& q = a.L[m];
        q.ub[0] = (T*)L.ubuf[0];
        q.ub[1] = jac ? (T*)L.ubuf[1] : nullptr;
        q.f = (T*)L.f;
        q.r = (T*)L.r;
        for (int c = 0; c < 6; c++) q.g[c] = (T*)L.face[c];
        // constants as launch_stencil and bc_args form them: omega is rounded to T first
        const T om = (T)omega;
        q.two_h = (T)(2.0 * L.h);
        q.hsq = (T)(L.h * L.h);
        q.one_omega = (T)(1.0 - om);
        q.omega_sixth = (T)(om / 6.0);
        q.h = (T)L.h;
        hsq_terms(q.hsq, q.inv_hsq, q.pow2);
        a.cur |= (unsigned)(L.cur & 1) << m;
    }
    auto emit = [&](int op, int m) {
        if (a.nops < kClMaxOps) {
            a.op[a.nops] = (unsigned char)op;
            a.lv[a.nops] = (unsigned char)m;
        }
        a.nops++;
    };
    // the recursion of vcycle_t / fcycle_t, and the host state it leaves (each Jacobi sweep swaps
    // the pair; red-black relaxations flip `alternate` an even number of times)
    bool skip = s->lv[t].first_done;
    auto relax = [&](int m) {
        emit(skip ? CL_RELAX_SKIP1 : CL_RELAX, m);
        skip = false;
        if (jac) s->lv[t + m].cur ^= (int)(ns & 1);
    };
    std::function<void(int)> vc = [&](int m) {
        relax(m);
        if (m >= a.nl - 1) return;
        emit(CL_SETUP, m);
        vc(m + 1);
        emit(CL_PROLONG, m);
        relax(m);
    };
    std::function<void(int)> fc = [&](int m) {
        relax(m);
        emit(CL_SETUP, m);
        if (m + 1 < a.nl - 1) fc(m + 1);
        vc(m + 1);
        emit(CL_PROLONG, m);
    };
    const uint64_t before = state_bits(s);
    if (f) fc(0);
    if (v) vc(0);
    if (norm) emit(CL_NORM, 0);
    if (a.nops > kClMaxOps) {
        set_state_bits(s, before);
        return fail(MGP_ERR_STATE, "coarse-level visit of %d operations", a.nops);
    }
    for (int m = 0; m < a.nl; m++) s->lv[t + m].first_done = false;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = nc;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(nc);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s->stream;
    cfg.attrs = attr;
    cfg.numAttrs = pdl_enabled() ? 2 : 1;
    const cudaError_t e = jac                        ? cudaLaunchKernelEx(&cfg, k_cluster<T, true, true>, a)
                          : a.polls == kWaitPolls ? cudaLaunchKernelEx(&cfg, k_cluster<T, false, false>, a)
                                                  : cudaLaunchKernelEx(&cfg, k_cluster<T, false, true>, a);
    if (e != cudaSuccess) return fail(MGP_ERR_CUDA, "kernel launch: %s", cudaGetErrorString(e));
    return check_launch(s);
}

// tail_norm: the caller's residual of level l with its max-norm, right after this cycle (the
// solve loop's); the cycle's last relaxation may take it over and then sets *tail_done.
template <typename T>
int vcycle_t(mgp_solver* s, int l, double omega, int64_t ns, unsigned long long* tail_norm = nullptr,
             bool* tail_done = nullptr) {
    // Vcycle<T> (include/vcycle.h:14-98)
    if (ns >= 1 && l >= cluster_level(s)) {
        if (tail_done) *tail_done = tail_norm != nullptr;
        return launch_cluster<T>(s, l, false, true, omega, ns, tail_norm);
    }
    if (!tail_norm && l >= 1 && l == tail_level(s)) return launch_tail<T>(s, l, false, omega, ns);
    const int tail = tail_norm ? RESID_NORM : RESID_NONE;
    if (l >= s->levels - 1) return relax_t<T>(s, l, omega, ns, false, tail, tail_norm, tail_done);
    bool rd = false;
    CKS(relax_t<T>(s, l, omega, ns, /*later=*/true, setup_residual_separate(s, l) ? RESID_STORE : RESID_NONE, nullptr,
                   &rd));
    CKS(coarse_setup_t<T>(s, l, omega, ns, rd));
    CKS(vcycle_t<T>(s, l + 1, omega, ns));
    if (!tail_norm && prolong_sweep_fused(s, l, ns)) {
        CKS(prolong_sweep_t<T>(s, l, omega));
        return relax_t<T>(s, l, omega, ns - 1, false, tail, tail_norm, tail_done);
    }
    CKS((prolong_t<T, true>(s, l)));
    CKS(relax_t<T>(s, l, omega, ns, false, tail, tail_norm, tail_done));
    return MGP_OK;
}

template <typename T>
int fcycle_t(mgp_solver* s, int l, double omega, int64_t ns, unsigned long long* tail_norm = nullptr,
             bool* tail_done = nullptr) {
    // Fcycle<T> (include/fcycle.h:13-97); the V-cycle of this level that follows relaxes it again
    if (tail_done) *tail_done = false;
    const int cl = ns >= 1 ? cluster_level(s) : s->levels;
    if (l >= cl) {
        if (tail_done) *tail_done = tail_norm != nullptr;
        return launch_cluster<T>(s, l, true, l == 0, omega, ns, tail_norm);
    }
    if (!tail_norm && l >= 1 && l == tail_level(s)) return launch_tail<T>(s, l, true, omega, ns);
    bool rd = false;
    CKS(relax_t<T>(s, l, omega, ns, /*later=*/true, setup_residual_separate(s, l) ? RESID_STORE : RESID_NONE, nullptr,
                   &rd));
    CKS(coarse_setup_t<T>(s, l, omega, ns, rd));
    if (l + 1 >= cl) {  // F(l+1) and V(l+1) in one launch
        CKS(launch_cluster<T>(s, l + 1, l < s->levels - 2, true, omega, ns));
    } else {
        if (l < s->levels - 2) CKS(fcycle_t<T>(s, l + 1, omega, ns));
        CKS(vcycle_t<T>(s, l + 1, omega, ns));
    }
    CKS((prolong_t<T, true>(s, l)));
    if (l == 0) CKS(vcycle_t<T>(s, 0, omega, ns, tail_norm, tail_done));
    return MGP_OK;
}

// dtype dispatch
#define DISPATCH(s, CALL_T)                                   \
    ((s)->dtype == MGP_F64 ? ([&]() { using T = double; return CALL_T; })() \
                           : ([&]() { using T = float; return CALL_T; })())

// One solve iteration: the cycle, then residual + max-norm of the finest level
// (include/libpoisson.h:294-330).  Captured once per (cycle, nsmooth, omega, state).
int iteration_body(mgp_solver* s, int cycle, int64_t ns, double omega) {
    // the norm word is zeroed first: the cycle's last pass may already reduce into it
    CK(cudaMemsetAsync(s->d_norm, 0, sizeof(unsigned long long), s->stream));
    bool done = false;
    if (cycle == MGP_CYCLE_V) CKS(DISPATCH(s, (vcycle_t<T>(s, 0, omega, ns, s->d_norm, &done))));
    else if (cycle == MGP_CYCLE_F) CKS(DISPATCH(s, (fcycle_t<T>(s, 0, omega, ns, s->d_norm, &done))));
    if (!done) CKS(DISPATCH(s, (residual_t<T>(s, 0, s->d_norm))));
    return MGP_OK;
}

int launch_iteration(mgp_solver* s, int cycle, int64_t ns, double omega) {
    uint64_t ob;
    memcpy(&ob, &omega, sizeof(ob));
    auto key = std::make_tuple(cycle, ns, ob, state_bits(s));
    auto it = s->graphs.find(key);
    if (it == s->graphs.end()) {
        const uint64_t pre = state_bits(s);
        const int64_t launches0 = s->launches;
        cudaGraph_t g = nullptr;
        CK(cudaStreamBeginCapture(s->stream, cudaStreamCaptureModeThreadLocal));
        s->capturing = true;
        int st = iteration_body(s, cycle, ns, omega);
        s->capturing = false;
        cudaError_t e = cudaStreamEndCapture(s->stream, &g);
        if (st != MGP_OK) {
            if (g) cudaGraphDestroy(g);
            set_state_bits(s, pre);
            return st;
        }
        if (e != cudaSuccess) {
            set_state_bits(s, pre);
            return fail(MGP_ERR_CUDA, "graph capture: %s", cudaGetErrorString(e));
        }
        GraphEntry ge;
        ge.post_state = state_bits(s);
        ge.kernels = s->launches - launches0;
        s->launches = launches0;
        cudaError_t ei = cudaGraphInstantiate(&ge.exec, g, 0);
        cudaGraphDestroy(g);
        set_state_bits(s, pre);
        if (ei != cudaSuccess) return fail(MGP_ERR_CUDA, "graph instantiate: %s", cudaGetErrorString(ei));
        it = s->graphs.emplace(key, ge).first;
    }
    CK(cudaGraphLaunch(it->second.exec, s->stream));
    s->launches += it->second.kernels;
    set_state_bits(s, it->second.post_state);
    return MGP_OK;
}

// first (may be null): the norm reduced into word 2 before.
int read_norm(mgp_solver* s, double* out, double* first = nullptr) {
    // the norm word and, 8 bytes on, the error word of the wavefront and cluster passes
    CK(cudaMemcpyAsync(s->h_norm, s->d_norm, first ? 24 : 16, cudaMemcpyDeviceToHost, s->stream));
    CK(cudaStreamSynchronize(s->stream));
    if (const int err = reinterpret_cast<const int*>(s->h_norm)[2]) {
        CK(cudaMemsetAsync(s->err_word, 0, sizeof(int), s->stream));
        CK(cudaStreamSynchronize(s->stream));
        return fail(MGP_ERR_TIMEOUT, "%s; results are invalid",
                    err == kErrCluster ? "coarse levels in a cluster: a wait for a neighbour's planes ran out"
                                       : "wavefront pass: a shared-memory ring wait ran out of time");
    }
    double v;
    unsigned long long b = *s->h_norm;
    memcpy(&v, &b, sizeof(v));
    *out = v;
    if (first) memcpy(first, s->h_norm + 2, sizeof(v));
    return MGP_OK;
}

// ---- iterative refinement ------------------------------------------------------------
// The first sweep of the corrections of (omega, ns).
RefineFirst refine_first(const mgp_solver* in, double omega, int64_t ns) {
    RefineFirst w;
    if (ns >= 1 && !in->lv[0].gs_column && !in->lv[0].wave) w.on = in->desc.relaxation == MGP_JACOBI ? 1 : 2;
    w.omega = omega;
    return w;
}

// Arguments and grid of one refinement residual; chunks as the caller cuts them.
template <typename Ti, bool R>
RefineArgs<double, Ti, R> refine_args(mgp_solver* s, const RefineFirst& w, unsigned long long* norm) {
    mgp_solver* in = s->inner;
    LevelState& L = s->lv[0];
    LevelState& I = in->lv[0];
    RefineArgs<double, Ti, R> a{};
    a.G = L.G;
    a.G.poff = I.G.poff;
    a.src = (const double*)u_ptr(s, 0);
    a.f = (const double*)L.f;
    a.dst = (double*)L.r;
    a.F = faces_of<double>(s, 0);
    a.two_h = 2.0 * L.h;
    a.hsq = L.h * L.h;
    hsq_terms(a.hsq, a.inv_hsq, a.hsq_pow2);
    a.norm = norm;
    a.sxi = I.G.sx;
    a.syi = I.G.sy;
    a.fi = (Ti*)I.f;
    a.ui = (Ti*)u_ptr(in, 0);
    a.uw = (Ti*)uprev_ptr(in, 0);
    a.first = w.on;
    a.fcolour = in->gs_alternate ? 0 : 1;
    const Ti om = (Ti)w.omega;  // the relaxation takes omega as a Ti (jacobi.h:41-44)
    a.w0 = (Ti)(1.0 - om);
    a.w1 = (Ti)(om / 6.0);
    a.hsqi = (Ti)(I.h * I.h);
    return a;
}

template <typename Ti, bool R>
int refine_residual_t(mgp_solver* s, const RefineFirst& w) {
    LevelState& L = s->lv[0];
    auto a = refine_args<Ti, R>(s, w, s->d_norm);
    constexpr int V = VecT<double>::V;
    const int plane = L.G.ny * ((L.G.nz + V - 1) / V);
    const int bx = (plane + kThreads - 1) / kThreads;
    const int cap = sm_count(s->device) * resident_blocks(k_refine_residual<double, Ti, R>);
    int chunks = short_march_chunks<double>(L.G, bx, cap, march_chunks(bx, L.G.nx, cap));
    a.ichunk = (L.G.nx + chunks - 1) / chunks;
    chunks = (L.G.nx + a.ichunk - 1) / a.ichunk;
    CK(cudaMemsetAsync(s->d_norm, 0, sizeof(unsigned long long), s->stream));
    CKS(launch_k(s, k_refine_residual<double, Ti, R>, dim3(bx, chunks), dim3(kThreads), 0, a));
    if (!R) {
        s->inner->lv[0].first_done = w.on != 0;
        s->inner->guess = w;
    }
    return MGP_OK;
}

template <typename Ti>
int refine_update_t(mgp_solver* s) {
    mgp_solver* in = s->inner;
    LevelState& L = s->lv[0];
    LevelState& I = in->lv[0];
    constexpr int V = VecT<double>::V;
    UpdateArgs<double, Ti> a{(double*)u_ptr(s, 0), L.G, (const Ti*)u_ptr(in, 0), I.G.sx, I.G.sy};
    const int bx = (L.G.ny * ((L.G.nz + V - 1) / V) + kThreads - 1) / kThreads;
    return launch_k(s, k_refine_update<double, Ti>, dim3(bx, L.G.nx), dim3(kThreads), 0, a);
}

// The FP64 residual and its norm, starting the next correction.
int refine_residual(mgp_solver* s, const RefineFirst& w = RefineFirst{}) {
    return s->inner->dtype == MGP_F32 ? refine_residual_t<float, false>(s, w) : refine_residual_t<double, false>(s, w);
}
// The FP64 residual stored in r (the user-visible residual), and its norm.
int refine_store_residual(mgp_solver* s) {
    const RefineFirst w;
    return s->inner->dtype == MGP_F32 ? refine_residual_t<float, true>(s, w) : refine_residual_t<double, true>(s, w);
}

// One refinement step, captured once per (cycle, nsmooth, omega, inner state): the
// correction cycle on the inner hierarchy, u += e, and the new FP64 residual with its norm.
int launch_refine_step(mgp_solver* s, int cycle, int64_t ns, double omega) {
    mgp_solver* in = s->inner;
    uint64_t ob;
    memcpy(&ob, &omega, sizeof(ob));
    auto key = std::make_tuple(100 + cycle, ns, ob, state_bits(in));
    auto it = s->graphs.find(key);
    const RefineFirst w = refine_first(in, omega, ns);
    if (it == s->graphs.end()) {
        const uint64_t pre = state_bits(in);
        const int64_t s0 = s->launches, i0 = in->launches;
        in->lv[0].first_done = w.on != 0;  // the residual before this step wrote the first sweep
        cudaGraph_t g = nullptr;
        CK(cudaStreamBeginCapture(s->stream, cudaStreamCaptureModeThreadLocal));
        int st;
        if (in->dtype == MGP_F32) {
            st = cycle == MGP_CYCLE_V ? vcycle_t<float>(in, 0, omega, ns) : fcycle_t<float>(in, 0, omega, ns);
            if (st == MGP_OK) st = refine_update_t<float>(s);
        } else {
            st = cycle == MGP_CYCLE_V ? vcycle_t<double>(in, 0, omega, ns) : fcycle_t<double>(in, 0, omega, ns);
            if (st == MGP_OK) st = refine_update_t<double>(s);
        }
        if (st == MGP_OK) st = refine_residual(s, w);
        in->lv[0].first_done = false;
        cudaError_t e = cudaStreamEndCapture(s->stream, &g);
        GraphEntry ge;
        ge.post_state = state_bits(in);
        ge.kernels = (s->launches - s0) + (in->launches - i0);
        s->launches = s0;  // the capture launched nothing; replays count the graph's kernels
        in->launches = i0;
        set_state_bits(in, pre);
        if (st != MGP_OK || e != cudaSuccess) {
            if (g) cudaGraphDestroy(g);
            return st != MGP_OK ? st : fail(MGP_ERR_CUDA, "graph capture: %s", cudaGetErrorString(e));
        }
        cudaError_t ei = cudaGraphInstantiate(&ge.exec, g, 0);
        cudaGraphDestroy(g);
        if (ei != cudaSuccess) return fail(MGP_ERR_CUDA, "graph instantiate: %s", cudaGetErrorString(ei));
        it = s->graphs.emplace(key, ge).first;
    }
    CK(cudaGraphLaunch(it->second.exec, s->stream));
    set_state_bits(in, it->second.post_state);
    in->guess = w;
    s->launches += it->second.kernels;
    return MGP_OK;
}

int validate(const mgp_solver* s) { return s ? MGP_OK : fail(MGP_ERR_INVALID_ARG, "null solver"); }
int validate_level(const mgp_solver* s, int l, bool need_coarser = false) {
    CKS(validate(s));
    if (l < 0 || l >= s->levels || (need_coarser && l + 1 >= s->levels))
        return fail(MGP_ERR_INVALID_ARG, "level %d out of range (levels=%d)", l, s->levels);
    return MGP_OK;
}

// 3-D strided copy between a reference-layout host array and a pitched device buffer,
// shape points only.
// Fields of at least kStageMinBytes cross PCIe as one DMA of the host array's layout: a
// device staging copy of that layout is filled by one contiguous copy (upload) or by the
// repack kernel (download), so the link sees long contiguous runs instead of one short row
// per (i, j); the repack between layouts runs at HBM speed.  The staging buffer is
// allocated on first use and kept with the solver.
constexpr size_t kStageMinBytes = 8u << 20;

template <typename T>
int repack_t(mgp_solver* s, int l, void* dev, bool to_device) {
    LevelState& L = s->lv[l];
    const mgp_level_info& I = L.info;
    const long long off = I.halo[1] * I.stride[0] + I.halo[3] * I.stride[1] + I.halo[5];
    const long long n = (long long)L.G.nx * L.G.ny * L.G.nz;
    if (to_device)
        return launch_k(s, k_repack<T, true>, dim3(grid_1d(s, n)), dim3(kThreads), 0, (T*)dev, L.G, (T*)s->stage, off,
                        (long long)I.stride[0], (long long)I.stride[1]);
    return launch_k(s, k_repack<T, false>, dim3(grid_1d(s, n)), dim3(kThreads), 0, (T*)dev, L.G, (T*)s->stage, off,
                    (long long)I.stride[0], (long long)I.stride[1]);
}

int copy_field_staged(mgp_solver* s, int l, void* dev, void* host, bool to_device) {
    LevelState& L = s->lv[l];
    const mgp_level_info& I = L.info;
    const size_t es = s->esize;
    const size_t bytes = (size_t)I.size * es;
    if (s->stage_bytes < bytes) {
        dev_free(s, s->stage);
        s->stage = nullptr;
        s->stage_bytes = 0;
        CK(dev_alloc(s, &s->stage, bytes));
        s->stage_bytes = bytes;
    }
    if (to_device) {
        CK(cudaMemcpyAsync(s->stage, host, bytes, cudaMemcpyHostToDevice, s->stream));
        CKS(DISPATCH(s, (repack_t<T>(s, l, dev, true))));
    } else {
        CKS(DISPATCH(s, (repack_t<T>(s, l, dev, false))));
        // copy the shape points back with the longest contiguous runs the host layout has:
        // k rows, whole (j, k) planes when z has no halo, the whole block when y has none too
        const size_t off = (size_t)(I.halo[1] * I.stride[0] + I.halo[3] * I.stride[1] + I.halo[5]) * es;
        size_t width = (size_t)L.G.nz * es, rows = (size_t)L.G.ny, planes = (size_t)L.G.nx;
        size_t row_pitch = (size_t)I.stride[1] * es, plane_pitch = (size_t)I.stride[0] * es;
        if (row_pitch == width) {
            width *= rows;
            rows = planes;
            row_pitch = plane_pitch;
            planes = 1;
            if (row_pitch == width) {
                width *= rows;
                rows = 1;
                row_pitch = width;
            }
        }
        char* hb = (char*)host + off;
        const char* sb = (const char*)s->stage + off;
        if (planes == 1) {
            CK(cudaMemcpy2DAsync(hb, row_pitch, sb, row_pitch, width, rows, cudaMemcpyDeviceToHost, s->stream));
        } else {
            cudaMemcpy3DParms p = {};
            p.srcPtr = make_cudaPitchedPtr(const_cast<char*>(sb), row_pitch, width, (size_t)I.pad[1]);
            p.dstPtr = make_cudaPitchedPtr(hb, row_pitch, width, (size_t)I.pad[1]);
            p.extent = make_cudaExtent(width, rows, planes);
            p.kind = cudaMemcpyDeviceToHost;
            CK(cudaMemcpy3DAsync(&p, s->stream));
        }
    }
    CK(cudaStreamSynchronize(s->stream));
    return MGP_OK;
}

int copy_field(mgp_solver* s, int l, void* dev, void* host, bool to_device) {
    LevelState& L = s->lv[l];
    const mgp_level_info& I = L.info;
    const size_t es = s->esize;
    if ((size_t)I.size * es >= kStageMinBytes) return copy_field_staged(s, l, dev, host, to_device);
    char* hbase = (char*)host + (size_t)(I.halo[1] * I.stride[0] + I.halo[3] * I.stride[1] + I.halo[5]) * es;
    cudaMemcpy3DParms p = {};
    cudaPitchedPtr hp = make_cudaPitchedPtr(hbase, (size_t)I.pad[2] * es, (size_t)L.G.nz * es, (size_t)I.pad[1]);
    cudaPitchedPtr dp = make_cudaPitchedPtr(dev, (size_t)L.G.sy * es, (size_t)L.G.nz * es, (size_t)L.G.ny);
    p.extent = make_cudaExtent((size_t)L.G.nz * es, (size_t)L.G.ny, (size_t)L.G.nx);
    if (to_device) {
        p.srcPtr = hp;
        p.dstPtr = dp;
        p.kind = cudaMemcpyHostToDevice;
    } else {
        p.srcPtr = dp;
        p.dstPtr = hp;
        p.kind = cudaMemcpyDeviceToHost;
    }
    CK(cudaMemcpy3DAsync(&p, s->stream));
    CK(cudaStreamSynchronize(s->stream));
    return MGP_OK;
}

void* field_ptr(mgp_solver* s, int field, int l) {
    switch (field) {
        case MGP_FIELD_U: return u_ptr(s, l);
        case MGP_FIELD_UPREV: return uprev_ptr(s, l);
        case MGP_FIELD_F: return s->lv[l].f;
        case MGP_FIELD_R: return s->lv[l].r;
        default: return nullptr;
    }
}

void release(mgp_solver* s) {
    if (!s) return;
    for (auto& kv : s->graphs)
        if (kv.second.exec) cudaGraphExecDestroy(kv.second.exec);
    s->graphs.clear();
    for (auto& L : s->lv) {
        // with paired sweeps the three u buffers may sit in any of the slots
        for (void* p : {L.ubuf[0], L.ubuf[1], L.spare, L.f, L.r}) dev_free(s, p);
        for (void* p : L.face) dev_free(s, p);
    }
    dev_free(s, s->d_norm);
    if (s->h_norm && s->owns_h_norm) cudaFreeHost(s->h_norm);
    dev_free(s, s->stage);
    if (s->inner) release(s->inner);
    if (s->stream && s->owns_stream) cudaStreamDestroy(s->stream);
    if (s->side) cudaStreamDestroy(s->side);
    if (s->ev_fork) cudaEventDestroy(s->ev_fork);
    if (s->ev_join) cudaEventDestroy(s->ev_join);
    delete s;
}

// Dirichlet data of level l into u and u_prev.
template <typename T>
int write_faces_t(mgp_solver* s, int l) {
    LevelState& L = s->lv[l];
    WriteFacesArgs<T> a{};
    a.u[0] = (T*)u_ptr(s, l);
    a.u[1] = L.ubuf[1] ? (T*)uprev_ptr(s, l) : nullptr;
    a.G = L.G;
    long long nmax = 0;
    for (int f = 0; f < 6; f++) {
        a.g[f] = (const T*)L.face[f];
        if (s->face_kind[f] != MGP_DIRICHLET) continue;  // Neumann write_to only fills ghosts
        a.dirichlet |= 1 << f;
        nmax = std::max(nmax, (long long)(L.face_shape[f][0] * L.face_shape[f][1] * L.face_shape[f][2]));
    }
    if (!a.dirichlet) return MGP_OK;
    return launch_k(s, k_write_faces<T>, dim3((unsigned)grid_1d(s, nmax), 6, a.u[1] ? 2 : 1), dim3(kThreads), 0, a);
}

struct DeviceGuard {
    int prev = -1;
    explicit DeviceGuard(int dev) {
        if (cudaGetDevice(&prev) != cudaSuccess) prev = -1;
        if (prev != dev) cudaSetDevice(dev);
    }
    ~DeviceGuard() {
        int now = -1;
        if (prev >= 0 && cudaGetDevice(&now) == cudaSuccess && now != prev) cudaSetDevice(prev);
    }
};

}  // namespace

// =======================================================================================
// C ABI
extern "C" {

const char* mgp_status_string(int st) {
    switch (st) {
        case MGP_OK: return "ok";
        case MGP_ERR_INVALID_ARG: return "invalid argument";
        case MGP_ERR_OOM: return "out of device memory";
        case MGP_ERR_NO_DEVICE: return "no CUDA device";
        case MGP_ERR_CUDA: return "CUDA error";
        case MGP_ERR_TIMEOUT: return "timeout";
        case MGP_ERR_DIVERGED: return "diverged";
        case MGP_ERR_UNSUPPORTED: return "unsupported";
        case MGP_ERR_STATE: return "invalid state";
        default: return "unknown status";
    }
}

const char* mgp_last_error(void) { return g_err.c_str(); }
int mgp_abi_version(void) { return MGP_ABI_VERSION; }

int mgp_device_count(int* n) {
    if (!n) return fail(MGP_ERR_INVALID_ARG, "null out pointer");
    int c = 0;
    cudaError_t e = cudaGetDeviceCount(&c);
    if (e != cudaSuccess) c = 0;
    *n = c;
    return MGP_OK;
}

int mgp_plan_level(const mgp_desc* d, int l, mgp_level_info* out) {
    if (!d || !out) return fail(MGP_ERR_INVALID_ARG, "null descriptor or out pointer");
    if (d->levels < 1 || d->levels > 30) return fail(MGP_ERR_INVALID_ARG, "levels must be in [1,30]");
    if (l < 0 || l >= d->levels) return fail(MGP_ERR_INVALID_ARG, "level %d out of range", l);
    for (int k = 0; k < 3; k++)
        if (d->dims[k] < 2 || d->dims[k] > (1 << 20)) return fail(MGP_ERR_INVALID_ARG, "dims must be in [2, 2^20]");
    if (d->restriction != MGP_INJECTION && d->restriction != MGP_FULLWEIGHTING)
        return fail(MGP_ERR_INVALID_ARG, "unknown restriction %d", d->restriction);
    if (d->prolongation != MGP_TRILINEAR) return fail(MGP_ERR_INVALID_ARG, "unknown prolongation %d", d->prolongation);
    if (d->relaxation != MGP_JACOBI && d->relaxation != MGP_GAUSSSEIDEL)
        return fail(MGP_ERR_INVALID_ARG, "unknown relaxation %d", d->relaxation);
    if (d->dtype != MGP_F64 && d->dtype != MGP_F32) return fail(MGP_ERR_INVALID_ARG, "unknown dtype %d", d->dtype);
    if (!(d->h > 0.0) || !std::isfinite(d->h)) return fail(MGP_ERR_INVALID_ARG, "h must be positive");
    for (int f = 0; f < 6; f++)
        if (d->bc[f] != MGP_DIRICHLET && d->bc[f] != MGP_NEUMANN) return fail(MGP_ERR_INVALID_ARG, "bad bc[%d]", f);
    // DomainSettings(l) (src/domainsettings.cpp:12-29): dims_l = (dims >> l) + 1, exact.
    for (int64_t m = 1; m < d->levels; m++)
        for (int k = 0; k < 3; k++) {
            int64_t n = (d->dims[k] >> m) + 1;
            if (((n - 1) << m) + 1 != d->dims[k])
                return fail(MGP_ERR_INVALID_ARG, "Invalid grid of size: (%lld,%lld,%lld)",
                            (long long)((d->dims[0] >> m) + 1), (long long)((d->dims[1] >> m) + 1),
                            (long long)((d->dims[2] >> m) + 1));
        }
    int kind[6];
    for (int f = 0; f < 6; f++) kind[f] = d->bc[f];
    if (!(d->flags & MGP_FLAG_STRICT_BC)) {
        // Domain's constructor replaces north/south by Dirichlet (domain.h:191-192) and
        // builds bottom as Dirichlet in both branches (domain.h:140-145).
        kind[MGP_NORTH] = MGP_DIRICHLET;
        kind[MGP_SOUTH] = MGP_DIRICHLET;
        kind[MGP_BOTTOM] = MGP_DIRICHLET;
    }
    // Halo widths follow the requested kinds (domain.h:102-108).
    const int64_t he = d->bc[MGP_EAST] != MGP_DIRICHLET, hw = d->bc[MGP_WEST] != MGP_DIRICHLET;
    const int64_t hn = d->bc[MGP_NORTH] != MGP_DIRICHLET, hs = d->bc[MGP_SOUTH] != MGP_DIRICHLET;
    const int64_t ht = d->bc[MGP_TOP] != MGP_DIRICHLET, hb = d->bc[MGP_BOTTOM] != MGP_DIRICHLET;
    int64_t n[3];
    for (int k = 0; k < 3; k++) n[k] = l == 0 ? d->dims[k] : (d->dims[k] >> l) + 1;
    mgp_level_info& I = *out;
    memset(&I, 0, sizeof(I));
    for (int k = 0; k < 3; k++) I.shape[k] = n[k];
    I.halo[0] = he; I.halo[1] = hw; I.halo[2] = hn; I.halo[3] = hs; I.halo[4] = ht; I.halo[5] = hb;
    I.pad[0] = n[0] + he + hw;
    I.pad[1] = n[1] + hn + hs;
    I.pad[2] = n[2] + ht + hb;
    I.stride[0] = I.pad[1] * I.pad[2];
    I.stride[1] = I.pad[2];
    I.stride[2] = 1;
    I.size = I.pad[0] * I.pad[1] * I.pad[2];
    I.h = d->h * (double)(1ll << l);
    for (int k = 0; k < 3; k++) I.origin[k] = d->origin[k];
    for (int f = 0; f < 6; f++) I.face_kind[f] = kind[f];
    const int64_t fs[6][3] = {{n[0], 1, n[2]}, {n[0], 1, n[2]}, {1, n[1], n[2]},
                              {1, n[1], n[2]}, {n[0], n[1], 1}, {n[0], n[1], 1}};
    memcpy(I.face_shape, fs, sizeof(fs));
    if (d->relaxation == MGP_GAUSSSEIDEL) {
        // The colour rule is the parity of the padded linear index (gaussseidel.h:56,81).
        // Halo widths are the same on every level, and every level's extents are odd
        // except possibly at a single-level grid; the test uses this level's extents.
        const int64_t pz = I.pad[2];
        if (pz % 2 == 0)
            return fail(MGP_ERR_UNSUPPORTED,
                        "red-black Gauss-Seidel colouring degenerates for padded z extent %lld (even): the "
                        "reference's result on this layout depends on thread timing",
                        (long long)pz);
    }
    return MGP_OK;
}

static int create_plain(const mgp_desc* d, mgp_solver** out, const CreateCtx* ctx) {
    if (!d || !out) return fail(MGP_ERR_INVALID_ARG, "null descriptor or out pointer");
    *out = nullptr;
    std::vector<mgp_level_info> plan(d->levels > 0 && d->levels <= 30 ? d->levels : 1);
    for (int l = 0; l < (int)d->levels || l == 0; l++) CKS(mgp_plan_level(d, l, &plan[l]));
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev < 1)
        return fail(MGP_ERR_NO_DEVICE, "Device array requested but no CUDA devices were detected");
    if (d->device < 0 || d->device >= ndev) return fail(MGP_ERR_NO_DEVICE, "device %d not present", d->device);

    mgp_solver* s = new (std::nothrow) mgp_solver();
    if (!s) return fail(MGP_ERR_OOM, "host allocation failed");
    s->desc = *d;
    s->dtype = d->dtype;
    s->device = d->device;
    s->levels = (int)d->levels;
    s->esize = d->dtype == MGP_F64 ? 8 : 4;
    for (int f = 0; f < 6; f++) s->face_kind[f] = plan[0].face_kind[f];
    const int64_t hw = plan[0].halo[1], hs = plan[0].halo[3], hb = plan[0].halo[5];

    DeviceGuard guard(s->device);
    if (ctx) {
        s->stream = ctx->stream;
        s->owns_stream = false;
        s->pool = ctx->pool;
        s->h_norm = ctx->h_norm;
        s->owns_h_norm = false;
    } else if (cudaStreamCreateWithFlags(&s->stream, cudaStreamNonBlocking) != cudaSuccess) {
        s->stream = nullptr;
        release(s);
        return fail(MGP_ERR_CUDA, "stream creation failed");
    }
    if (!s->pool && (cudaStreamCreateWithFlags(&s->side, cudaStreamNonBlocking) != cudaSuccess ||
                     cudaEventCreateWithFlags(&s->ev_fork, cudaEventDisableTiming) != cudaSuccess ||
                     cudaEventCreateWithFlags(&s->ev_join, cudaEventDisableTiming) != cudaSuccess)) {
        release(s);
        return fail(MGP_ERR_CUDA, "side stream creation failed");
    }
    s->lv.resize(s->levels);
    for (int l = 0; l < s->levels; l++) {
        LevelState& L = s->lv[l];
        L.info = plan[l];
        const mgp_level_info& I = L.info;
        memcpy(L.face_shape, I.face_shape, sizeof(L.face_shape));
        L.h = I.h;
        // With odd pad[1] (and odd pad[2], checked by the plan) the colour is
        // (i+j+k+hw+hs+hb)&1; with even pad[1] it is (j+k+hs+hb)&1 and each (j,k) column is
        // swept in i order, as the reference does on one thread.
        L.gs_column = s->desc.relaxation == MGP_GAUSSSEIDEL && (I.pad[1] % 2 == 0);
        Geom& G = L.G;
        G.nx = (int)I.shape[0];
        G.ny = (int)I.shape[1];
        G.nz = (int)I.shape[2];
        const int64_t align = 64 / (int64_t)s->esize;
        G.sy = (I.shape[2] + align - 1) / align * align;
        G.sx = G.sy * I.shape[1];
        G.x0 = s->face_kind[MGP_WEST] == MGP_DIRICHLET;
        G.x1 = G.nx - (s->face_kind[MGP_EAST] == MGP_DIRICHLET);
        G.y0 = s->face_kind[MGP_SOUTH] == MGP_DIRICHLET;
        G.y1 = G.ny - (s->face_kind[MGP_NORTH] == MGP_DIRICHLET);
        G.z0 = s->face_kind[MGP_BOTTOM] == MGP_DIRICHLET;
        G.z1 = G.nz - (s->face_kind[MGP_TOP] == MGP_DIRICHLET);
        L.elems = (size_t)G.sx * I.shape[0];
        const size_t bytes = L.elems * s->esize;
        const int nbuf = s->desc.relaxation == MGP_JACOBI ? 2 : 1;
        cudaError_t e = cudaSuccess;
        for (int b = 0; b < nbuf && e == cudaSuccess; b++) e = dev_alloc(s, &L.ubuf[b], bytes);
        if (e == cudaSuccess) e = dev_alloc(s, &L.f, bytes);
        if (e == cudaSuccess) e = dev_alloc(s, &L.r, bytes);
        for (int f = 0; f < 6 && e == cudaSuccess; f++)
            e = dev_alloc(s, &L.face[f], (size_t)(I.face_shape[f][0] * I.face_shape[f][1] * I.face_shape[f][2]) * s->esize);
        if (e != cudaSuccess) {
            release(s);
            return fail(e == cudaErrorMemoryAllocation ? MGP_ERR_OOM : MGP_ERR_CUDA, "allocating level %d: %s", l,
                        cudaGetErrorString(e));
        }
        for (void* p : {L.ubuf[0], L.ubuf[1], L.f, L.r})
            if (p && e == cudaSuccess) e = dev_zero(s, p, bytes);
        for (int f = 0; f < 6; f++)
            if (e == cudaSuccess)
                e = dev_zero(s, L.face[f], (size_t)(I.face_shape[f][0] * I.face_shape[f][1] * I.face_shape[f][2]) * s->esize);
        if (e != cudaSuccess) {
            release(s);
            return fail(MGP_ERR_CUDA, "zeroing level %d: %s", l, cudaGetErrorString(e));
        }
    }
    for (int l = 0; l < s->levels; l++)
        s->lv[l].G.poff = s->lv[l].gs_column ? (int)((hs + hb) & 1) : (int)((hw + hs + hb) & 1);
    {
        int npair = 0;
        for (int l = 0; l < s->levels; l++) {
            cudaError_t e = s->dtype == MGP_F64 ? wave_prepare_level<double>(s, s->lv[l], npair)
                                                : wave_prepare_level<float>(s, s->lv[l], npair);
            if (e != cudaSuccess) {
                release(s);
                return fail(e == cudaErrorMemoryAllocation ? MGP_ERR_OOM : MGP_ERR_CUDA, "wavefront buffer of level %d: %s",
                            l, cudaGetErrorString(e));
            }
            npair += s->lv[l].pair;
        }
    }
    cudaError_t e = dev_alloc(s, (void**)&s->d_norm, 64);
    if (e == cudaSuccess) e = dev_zero(s, s->d_norm, 64);
    if (e == cudaSuccess && !s->h_norm) e = cudaMallocHost(&s->h_norm, 64);
    s->err_word = reinterpret_cast<int*>(reinterpret_cast<char*>(s->d_norm) + 8);
    // a pooled solver's set-up is ordered on the shared stream; nothing to wait for here
    if (e == cudaSuccess && !s->pool) e = cudaDeviceSynchronize();
    if (e != cudaSuccess) {
        release(s);
        return fail(e == cudaErrorMemoryAllocation ? MGP_ERR_OOM : MGP_ERR_CUDA, "solver set-up: %s",
                    cudaGetErrorString(e));
    }
    *out = s;
    return MGP_OK;
}

static int create_solver(const mgp_desc* d, mgp_solver** out, const CreateCtx* ctx) {
    if (!d || !out) return fail(MGP_ERR_INVALID_ARG, "null descriptor or out pointer");
    *out = nullptr;
    const uint32_t refine = d->flags & (MGP_FLAG_REFINE_F32 | MGP_FLAG_REFINE_F64);
    if (!refine) return create_plain(d, out, ctx);
    if (refine == (MGP_FLAG_REFINE_F32 | MGP_FLAG_REFINE_F64))
        return fail(MGP_ERR_INVALID_ARG, "choose one of MGP_FLAG_REFINE_F32 / MGP_FLAG_REFINE_F64");
    if (d->dtype != MGP_F64) return fail(MGP_ERR_INVALID_ARG, "a refinement solver keeps level 0 in FP64 (dtype F64)");
    if (d->levels < 2) return fail(MGP_ERR_INVALID_ARG, "a refinement solver needs at least 2 levels");
    // the correction hierarchy: every level, the requested inner precision
    mgp_desc di = *d;
    di.flags &= ~(MGP_FLAG_REFINE_F32 | MGP_FLAG_REFINE_F64);
    di.dtype = (refine & MGP_FLAG_REFINE_F32) ? MGP_F32 : MGP_F64;
    // the outer level: FP64, level 0 only
    mgp_desc dout = *d;
    dout.flags &= ~(MGP_FLAG_REFINE_F32 | MGP_FLAG_REFINE_F64);
    dout.levels = 1;
    mgp_solver* outer = nullptr;
    CKS(create_plain(&dout, &outer, ctx));
    // the inner hierarchy shares the outer solver's stream (and memory pool)
    mgp_solver* inner = nullptr;
    CreateCtx ictx{outer->stream, outer->pool, outer->h_norm};
    int st = create_plain(&di, &inner, &ictx);
    if (st != MGP_OK) {
        release(outer);
        return st;
    }
    inner->err_word = outer->err_word;  // seen by the outer solver's norm read-back
    outer->inner = inner;
    outer->desc = *d;  // keeps the refine flag and the user's level count
    *out = outer;
    return MGP_OK;
}

int mgp_create(const mgp_desc* d, mgp_solver** out) { return create_solver(d, out, nullptr); }

int mgp_destroy(mgp_solver* s) {
    if (!s) return MGP_OK;
    DeviceGuard guard(s->device);
    cudaStreamSynchronize(s->stream);
    release(s);
    return MGP_OK;
}

int mgp_num_levels(const mgp_solver* s) { return s ? s->levels : 0; }

int mgp_level_info_get(const mgp_solver* s, int l, mgp_level_info* out) {
    CKS(validate_level(s, l));
    if (!out) return fail(MGP_ERR_INVALID_ARG, "null out pointer");
    *out = s->lv[l].info;
    return MGP_OK;
}

int mgp_upload_field(mgp_solver* s, int field, int l, const void* host, int64_t count) {
    CKS(validate_level(s, l));
    void* dev = field_ptr(s, field, l);
    if (!dev || !host) return fail(MGP_ERR_INVALID_ARG, "bad field %d or null host pointer", field);
    if (count != s->lv[l].info.size)
        return fail(MGP_ERR_INVALID_ARG, "count %lld != level size %lld", (long long)count,
                    (long long)s->lv[l].info.size);
    DeviceGuard guard(s->device);
    return copy_field(s, l, dev, const_cast<void*>(host), true);
}

int mgp_download_field(mgp_solver* s, int field, int l, void* host, int64_t count) {
    CKS(validate_level(s, l));
    void* dev = field_ptr(s, field, l);
    if (!dev || !host) return fail(MGP_ERR_INVALID_ARG, "bad field %d or null host pointer", field);
    if (count != s->lv[l].info.size)
        return fail(MGP_ERR_INVALID_ARG, "count %lld != level size %lld", (long long)count,
                    (long long)s->lv[l].info.size);
    DeviceGuard guard(s->device);
    return copy_field(s, l, dev, host, false);
}

static int face_io(mgp_solver* s, int face, int l, void* host, int64_t count, bool up) {
    CKS(validate_level(s, l));
    if (face < 0 || face > 5 || !host) return fail(MGP_ERR_INVALID_ARG, "bad face %d or null pointer", face);
    const int64_t* fs = s->lv[l].face_shape[face];
    const int64_t n = fs[0] * fs[1] * fs[2];
    if (count != n) return fail(MGP_ERR_INVALID_ARG, "count %lld != face size %lld", (long long)count, (long long)n);
    DeviceGuard guard(s->device);
    if (up) CK(cudaMemcpyAsync(s->lv[l].face[face], host, n * s->esize, cudaMemcpyHostToDevice, s->stream));
    else CK(cudaMemcpyAsync(host, s->lv[l].face[face], n * s->esize, cudaMemcpyDeviceToHost, s->stream));
    CK(cudaStreamSynchronize(s->stream));
    return MGP_OK;
}

int mgp_upload_face(mgp_solver* s, int face, int l, const void* host, int64_t count) {
    return face_io(s, face, l, const_cast<void*>(host), count, true);
}
int mgp_field_device(mgp_solver* s, int field, int l, void** ptr, int64_t layout[5]) {
    CKS(validate_level(s, l));
    if (!ptr || !layout) return fail(MGP_ERR_INVALID_ARG, "null out pointer");
    void* dev = field_ptr(s, field, l);
    if (!dev) return fail(MGP_ERR_INVALID_ARG, "bad field %d", field);
    const Geom& G = s->lv[l].G;
    *ptr = dev;
    layout[0] = G.nx;
    layout[1] = G.ny;
    layout[2] = G.nz;
    layout[3] = G.sx;
    layout[4] = G.sy;
    return MGP_OK;
}

int mgp_face_device(mgp_solver* s, int face, int l, void** ptr, int64_t shape[3]) {
    CKS(validate_level(s, l));
    if (!ptr || !shape) return fail(MGP_ERR_INVALID_ARG, "null out pointer");
    if (face < 0 || face > 5) return fail(MGP_ERR_INVALID_ARG, "bad face %d", face);
    *ptr = s->lv[l].face[face];
    for (int k = 0; k < 3; k++) shape[k] = s->lv[l].face_shape[face][k];
    return MGP_OK;
}

int mgp_download_face(mgp_solver* s, int face, int l, void* host, int64_t count) {
    return face_io(s, face, l, host, count, false);
}

int mgp_write_bc(mgp_solver* s, int l) {
    CKS(validate_level(s, l));
    DeviceGuard guard(s->device);
    CKS(DISPATCH(s, (write_faces_t<T>(s, l))));
    CK(cudaStreamSynchronize(s->stream));
    return MGP_OK;
}

int mgp_set_wait_polls(mgp_solver* s, int64_t polls) {
    CKS(validate(s));
    if (polls < 0 || polls > (int64_t)UINT32_MAX) return fail(MGP_ERR_INVALID_ARG, "polls must be in [0, 2^32)");
    const unsigned p = polls == 0 ? kWaitPolls : (unsigned)polls;
    DeviceGuard guard(s->device);
    CK(cudaStreamSynchronize(s->stream));
    // the captured iterations carry the bound in their kernels' parameters
    for (mgp_solver* x : {s, s->inner}) {
        if (!x) continue;
        x->wait_polls = p;
        for (auto& kv : x->graphs)
            if (kv.second.exec) cudaGraphExecDestroy(kv.second.exec);
        x->graphs.clear();
    }
    return MGP_OK;
}

int mgp_set_iteration_limits(mgp_solver* s, int64_t maxiter, int64_t miniter, double tolerance) {
    CKS(validate(s));
    s->desc.maxiter = maxiter;
    s->desc.miniter = miniter;
    s->desc.tolerance = tolerance;
    return MGP_OK;
}

// ---- operators ----------------------------------------------------------------------
int mgp_relax(mgp_solver* s, int l, double omega, int64_t nsmooth) {
    CKS(validate_level(s, l));
    DeviceGuard guard(s->device);
    if (omega < 0) omega = s->desc.relaxation == MGP_JACOBI ? 6.0 / 7.0 : 8.0 / 9.0;
    return DISPATCH(s, (relax_t<T>(s, l, omega, nsmooth)));
}
int mgp_relax_colour(mgp_solver* s, int l, double omega, int colour) {
    CKS(validate_level(s, l));
    if (s->desc.relaxation != MGP_GAUSSSEIDEL)
        return fail(MGP_ERR_UNSUPPORTED, "mgp_relax_colour: the solver relaxes with Jacobi");
    if (colour != 0 && colour != 1) return fail(MGP_ERR_INVALID_ARG, "colour must be 0 or 1");
    DeviceGuard guard(s->device);
    if (omega < 0) omega = 8.0 / 9.0;
    return DISPATCH(s, (relax_colour_t<T>(s, l, omega, colour)));
}
int mgp_relax_residual(mgp_solver* s, int l, double omega, int64_t nsmooth, double* norm) {
    CKS(validate_level(s, l));
    DeviceGuard guard(s->device);
    if (omega < 0) omega = s->desc.relaxation == MGP_JACOBI ? 6.0 / 7.0 : 8.0 / 9.0;
    unsigned long long* nw = norm ? s->d_norm : nullptr;
    if (nw) CK(cudaMemsetAsync(s->d_norm, 0, sizeof(unsigned long long), s->stream));
    bool done = false;
    CKS(DISPATCH(s, (relax_t<T>(s, l, omega, nsmooth, false, nw ? RESID_NORM : RESID_STORE, nw, &done))));
    if (!done) CKS(DISPATCH(s, (residual_t<T>(s, l, nw))));
    if (nw) return read_norm(s, norm);
    return MGP_OK;
}
int mgp_residual(mgp_solver* s, int l) {
    CKS(validate_level(s, l));
    DeviceGuard guard(s->device);
    return DISPATCH(s, (residual_t<T>(s, l, nullptr)));
}
int mgp_restrict(mgp_solver* s, int l) {
    CKS(validate_level(s, l, true));
    DeviceGuard guard(s->device);
    return DISPATCH(s, (restrict_t<T>(s, l, false)));
}
int mgp_zero_u(mgp_solver* s, int l) {
    CKS(validate_level(s, l));
    DeviceGuard guard(s->device);
    return DISPATCH(s, (zero_u_t<T>(s, l)));
}
int mgp_restrict_bc(mgp_solver* s, int l) {
    CKS(validate_level(s, l, true));
    DeviceGuard guard(s->device);
    // Dirichlet coarse faces are re-zeroed here for callers that wrote them directly.
    for (int f = 0; f < 6; f++)
        if (s->face_kind[f] == MGP_DIRICHLET) {
            const int64_t* fs = s->lv[l + 1].face_shape[f];
            CK(cudaMemsetAsync(s->lv[l + 1].face[f], 0, (size_t)(fs[0] * fs[1] * fs[2]) * s->esize, s->stream));
        }
    return DISPATCH(s, (restrict_bc_t<T>(s, l)));
}
int mgp_prolong(mgp_solver* s, int l) {
    CKS(validate_level(s, l, true));
    DeviceGuard guard(s->device);
    return DISPATCH(s, (prolong_t<T, false>(s, l)));
}
int mgp_prolong_add(mgp_solver* s, int l) {
    CKS(validate_level(s, l, true));
    DeviceGuard guard(s->device);
    return DISPATCH(s, (prolong_t<T, true>(s, l)));
}
int mgp_add(mgp_solver* s, int l) {
    CKS(validate_level(s, l));
    DeviceGuard guard(s->device);
    return DISPATCH(s, (add_t<T>(s, l)));
}
int mgp_vcycle(mgp_solver* s, int l, double omega, int64_t nsmooth) {
    CKS(validate_level(s, l));
    DeviceGuard guard(s->device);
    if (omega < 0) omega = s->desc.relaxation == MGP_JACOBI ? 6.0 / 7.0 : 8.0 / 9.0;
    return DISPATCH(s, (vcycle_t<T>(s, l, omega, nsmooth)));
}
int mgp_fcycle(mgp_solver* s, int l, double omega, int64_t nsmooth) {
    CKS(validate_level(s, l, true));
    DeviceGuard guard(s->device);
    if (omega < 0) omega = s->desc.relaxation == MGP_JACOBI ? 6.0 / 7.0 : 8.0 / 9.0;
    return DISPATCH(s, (fcycle_t<T>(s, l, omega, nsmooth)));
}
int mgp_norm(mgp_solver* s, int field, int l, double* out) {
    CKS(validate_level(s, l));
    void* a = field_ptr(s, field, l);
    if (!a || !out) return fail(MGP_ERR_INVALID_ARG, "bad field %d or null out", field);
    DeviceGuard guard(s->device);
    CK(cudaMemsetAsync(s->d_norm, 0, sizeof(unsigned long long), s->stream));
    CKS(DISPATCH(s, (norm_t<T>(s, a, l, s->d_norm))));
    return read_norm(s, out);
}
int mgp_synchronize(mgp_solver* s) {
    CKS(validate(s));
    DeviceGuard guard(s->device);
    CK(cudaStreamSynchronize(s->stream));
    return MGP_OK;
}

int mgp_get_stream(mgp_solver* s, void** stream) {
    CKS(validate(s));
    if (!stream) return fail(MGP_ERR_INVALID_ARG, "null out pointer");
    *stream = (void*)s->stream;
    return MGP_OK;
}

// ---- launch-shape tuning ------------------------------------------------------------------
namespace {

void drop_graphs(mgp_solver* s) {
    for (auto& kv : s->graphs)
        if (kv.second.exec) cudaGraphExecDestroy(kv.second.exec);
    s->graphs.clear();
}

// Process cache of searched configurations: key -> levels x MGP_TUNE_PARAMS values.
std::mutex g_tune_mu;
std::map<std::string, std::vector<int>> g_tune_cache;
bool g_tune_file_loaded = false;

const char* tune_file() {
    const char* p = std::getenv("MGP_TUNE_CACHE");
    return p && p[0] ? p : nullptr;
}

// One line per configuration: the key, then the values.
void tune_cache_load_locked() {
    if (g_tune_file_loaded) return;
    g_tune_file_loaded = true;
    const char* path = tune_file();
    if (!path) return;
    std::ifstream in(path);
    std::string line;
    while (std::getline(in, line)) {
        std::istringstream ls(line);
        std::string key;
        if (!(ls >> key)) continue;
        std::vector<int> v;
        int x;
        while (ls >> x) v.push_back(x);
        g_tune_cache[key] = v;
    }
}

// Version of the built-in launch rules, part of a configuration's key.  Values searched against
// other rules are not taken from a file: any of them on a coarse level keeps it, and the finer
// ones, out of the cluster, and set planes keep a level off the register form, so a file written
// before these were built in made 33x17x17 solves slower than the built-in choices do.
constexpr int kTuneRules = 2;

std::string tune_key(const mgp_solver* s, int cycle, int64_t ns, uint32_t flags_used) {
    cudaDeviceProp p{};
    cudaGetDeviceProperties(&p, s->device);
    std::ostringstream k;
    k << "v" << kTuneRules << "/sm" << p.major << p.minor << "x" << p.multiProcessorCount << "/" << (s->dtype == MGP_F64 ? "f64" : "f32")
      << "/" << s->desc.dims[0] << "x" << s->desc.dims[1] << "x" << s->desc.dims[2] << "/L" << s->levels << "/bc";
    for (int f = 0; f < 6; f++) k << s->face_kind[f];
    k << "/r" << s->desc.relaxation << "p" << s->desc.prolongation << "q" << s->desc.restriction << "/c" << cycle
      << "n" << ns << "/f" << flags_used;
    return k.str();
}

void apply_tuning(mgp_solver* s, const std::vector<int>& v) {
    for (int l = 0; l < s->levels; l++)
        for (int p = 0; p < MGP_TUNE_PARAMS; p++) s->lv[l].tune[p] = v[(size_t)l * MGP_TUNE_PARAMS + p];
    drop_graphs(s);
}

std::vector<int> current_tuning(const mgp_solver* s) {
    std::vector<int> v((size_t)s->levels * MGP_TUNE_PARAMS);
    for (int l = 0; l < s->levels; l++)
        for (int p = 0; p < MGP_TUNE_PARAMS; p++) v[(size_t)l * MGP_TUNE_PARAMS + p] = s->lv[l].tune[p];
    return v;
}

// Device copy of every field buffer of every level (u pair, spare, f, r) and the host state
// that says which buffer is which.
struct SavedFields {
    void* buf = nullptr;
    uint64_t bits = 0;
    std::vector<std::pair<void*, size_t>> parts;  // (buffer, bytes), in copy order
};

int save_fields(mgp_solver* s, SavedFields& sv) {
    size_t total = 0;
    for (auto& L : s->lv)
        for (void* p : {L.phys[0] ? L.phys[0] : L.ubuf[0], L.phys[0] ? L.phys[1] : L.ubuf[1], L.phys[2], L.f, L.r})
            if (p) {
                sv.parts.emplace_back(p, L.elems * s->esize);
                total += L.elems * s->esize;
            }
    size_t free_b = 0, tot_b = 0;
    CK(cudaMemGetInfo(&free_b, &tot_b));
    if (total + (64u << 20) > free_b)
        return fail(MGP_ERR_OOM, "autotune: %zu bytes needed for the saved fields, %zu free", total, free_b);
    CK(cudaMalloc(&sv.buf, total));
    size_t off = 0;
    for (auto& pr : sv.parts) {
        CK(cudaMemcpyAsync((char*)sv.buf + off, pr.first, pr.second, cudaMemcpyDeviceToDevice, s->stream));
        off += pr.second;
    }
    sv.bits = state_bits(s);
    return MGP_OK;
}

int restore_fields(mgp_solver* s, SavedFields& sv) {
    size_t off = 0;
    for (auto& pr : sv.parts) {
        CK(cudaMemcpyAsync(pr.first, (char*)sv.buf + off, pr.second, cudaMemcpyDeviceToDevice, s->stream));
        off += pr.second;
    }
    set_state_bits(s, sv.bits);
    for (auto& L : s->lv) L.first_done = false;
    CK(cudaStreamSynchronize(s->stream));
    CK(cudaFree(sv.buf));
    sv.buf = nullptr;
    return MGP_OK;
}

// Milliseconds per solve iteration of the current tuning: graphs captured afresh, two
// iterations to warm up, then the best of `trials` runs of `reps` iterations.
int time_iteration(mgp_solver* s, int cycle, int64_t ns, double omega, int reps, int trials, cudaEvent_t e0,
                   cudaEvent_t e1, double* ms) {
    drop_graphs(s);
    for (int i = 0; i < 2; i++) CKS(launch_iteration(s, cycle, ns, omega));
    double best = 1e30;
    for (int t = 0; t < trials; t++) {
        CK(cudaEventRecord(e0, s->stream));
        for (int i = 0; i < reps; i++) CKS(launch_iteration(s, cycle, ns, omega));
        CK(cudaEventRecord(e1, s->stream));
        CK(cudaEventSynchronize(e1));
        float t_ms = 0.f;
        CK(cudaEventElapsedTime(&t_ms, e0, e1));
        best = std::min(best, (double)t_ms / reps);
    }
    CK(cudaGetLastError());
    *ms = best;
    return MGP_OK;
}

// Coordinate descent over the levels' parameters, finest level first.  A candidate replaces
// the current value only when it is faster by more than 0.5%, so timing noise does not move
// a choice.
int autotune_search(mgp_solver* s, int cycle, int64_t ns, double omega, double* untuned_ms, double* tuned_ms) {
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    CK(cudaEventCreate(&e0));
    CK(cudaEventCreate(&e1));
    auto done = [&](int st) {
        cudaEventDestroy(e0);
        cudaEventDestroy(e1);
        return st;
    };
    // iterations per timed run: about 20 ms of work
    double probe = 0;
    const std::vector<int> builtin((size_t)s->levels * MGP_TUNE_PARAMS, 0);
    apply_tuning(s, builtin);
    int st = time_iteration(s, cycle, ns, omega, 2, 1, e0, e1, &probe);
    if (st != MGP_OK) return done(st);
    const int reps = (int)std::max(3.0, std::min(200.0, 20.0 / std::max(probe, 1e-3)));
    double best = 0;
    st = time_iteration(s, cycle, ns, omega, reps, 3, e0, e1, &best);
    if (st != MGP_OK) return done(st);
    const double untuned = best;
    static const int kPlanes[] = {1, 2, 3, 4, 5, 6, 7, 8, 12, 16, 24, 32};
    for (int l = 0; l < s->levels; l++) {
        LevelState& L = s->lv[l];
        const bool coarser = l < s->levels - 1;
        for (int p = 0; p < MGP_TUNE_PARAMS; p++) {
            std::vector<int> cand;
            switch (p) {
                case MGP_TUNE_RELAX_PLANES:
                    if (L.gs_column || (L.wave && L.tune[MGP_TUNE_WAVE] != 1)) break;
                    // fall through
                case MGP_TUNE_RESID_PLANES:
                    for (int c : kPlanes)
                        if (c < L.G.nx) cand.push_back(c);
                    break;
                case MGP_TUNE_NORM_PLANES:
                    if (l == 0)
                        for (int c : kPlanes)
                            if (c < L.G.nx) cand.push_back(c);
                    break;
                case MGP_TUNE_SETUP_FORM:
                    if (coarser && !(s->desc.flags & MGP_FLAG_FUSED_SETUP)) cand = {1, 2};
                    break;
                case MGP_TUNE_SETUP_PLANES:
                    if (coarser && !setup_residual_separate(s, l))
                        for (int c : kPlanes)
                            if (c < s->lv[l + 1].G.nx) cand.push_back(c);
                    break;
                case MGP_TUNE_WAVE:
                    if (L.wave) cand = {1};
                    break;
                case MGP_TUNE_TAIL:
                    if (l == 0 && s->levels >= 2) cand = {1};
                    break;
                case MGP_TUNE_PROLONG_SWEEP:
                    if (coarser && l >= 1 && s->desc.relaxation == MGP_JACOBI && ns >= 2 && !(ns & 1)) cand = {1, 2};
                    break;
            }
            const int keep = L.tune[p];
            int chosen = keep;
            for (int c : cand) {
                if (c == keep) continue;
                L.tune[p] = c;
                double t = 0;
                st = time_iteration(s, cycle, ns, omega, reps, 2, e0, e1, &t);
                if (st != MGP_OK) return done(st);
                if (t < best * 0.995) {
                    best = t;
                    chosen = c;
                }
            }
            L.tune[p] = chosen;
        }
    }
    // final comparison, alternating the two settings
    const std::vector<int> tuned = current_tuning(s);
    double tu = 1e30, tt = 1e30;
    for (int r = 0; r < 2; r++) {
        double t = 0;
        apply_tuning(s, builtin);
        if ((st = time_iteration(s, cycle, ns, omega, reps, 2, e0, e1, &t)) != MGP_OK) return done(st);
        tu = std::min(tu, t);
        apply_tuning(s, tuned);
        if ((st = time_iteration(s, cycle, ns, omega, reps, 2, e0, e1, &t)) != MGP_OK) return done(st);
        tt = std::min(tt, t);
    }
    tu = std::min(tu, untuned);
    if (tt > tu) {  // the search found nothing that holds up: keep the built-in choices
        apply_tuning(s, builtin);
        tt = tu;
    }
    if (untuned_ms) *untuned_ms = tu;
    if (tuned_ms) *tuned_ms = tt;
    return done(MGP_OK);
}

}  // namespace

int mgp_set_tuning(mgp_solver* s, int level, int param, int64_t value) {
    CKS(validate(s));
    mgp_solver* t = s->inner ? s->inner : s;
    if (level < 0 || level >= t->levels) return fail(MGP_ERR_INVALID_ARG, "level %d out of range", level);
    if (param < 0 || param >= MGP_TUNE_PARAMS) return fail(MGP_ERR_INVALID_ARG, "unknown tuning parameter %d", param);
    const int64_t hi = param == MGP_TUNE_SETUP_FORM ? 2
                       : (param == MGP_TUNE_WAVE || param == MGP_TUNE_TAIL) ? 1
                       : param == MGP_TUNE_PROLONG_SWEEP ? 2
                                                           : (int64_t)1 << 20;
    if (value < 0 || value > hi) return fail(MGP_ERR_INVALID_ARG, "tuning value %lld out of range", (long long)value);
    DeviceGuard guard(t->device);
    CK(cudaStreamSynchronize(t->stream));
    t->lv[level].tune[param] = (int)value;
    drop_graphs(t);
    return MGP_OK;
}

int mgp_get_tuning(mgp_solver* s, int level, int param, int64_t* value) {
    CKS(validate(s));
    const mgp_solver* t = s->inner ? s->inner : s;
    if (!value) return fail(MGP_ERR_INVALID_ARG, "null out pointer");
    if (level < 0 || level >= t->levels) return fail(MGP_ERR_INVALID_ARG, "level %d out of range", level);
    if (param < 0 || param >= MGP_TUNE_PARAMS) return fail(MGP_ERR_INVALID_ARG, "unknown tuning parameter %d", param);
    *value = t->lv[level].tune[param];
    return MGP_OK;
}

int mgp_autotune(mgp_solver* s, int cycle, int64_t nsmooth, double omega, uint32_t flags, double* untuned_ms,
                 double* tuned_ms) {
    CKS(validate(s));
    if (cycle != MGP_CYCLE_V && cycle != MGP_CYCLE_F)
        return fail(MGP_ERR_INVALID_ARG, "autotune: cycle must be MGP_CYCLE_V or MGP_CYCLE_F");
    if (nsmooth < 0) return fail(MGP_ERR_INVALID_ARG, "nsmooth must be >= 0");
    mgp_solver* t = s->inner ? s->inner : s;
    if (cycle == MGP_CYCLE_F && t->levels < 2) return fail(MGP_ERR_INVALID_ARG, "an F-cycle needs at least 2 levels");
    DeviceGuard guard(t->device);
    if (omega < 0) omega = t->desc.relaxation == MGP_JACOBI ? 6.0 / 7.0 : 8.0 / 9.0;
    if (untuned_ms) *untuned_ms = 0;
    if (tuned_ms) *tuned_ms = 0;
    const std::string key = tune_key(t, cycle, nsmooth, t->desc.flags & (MGP_FLAG_WAVE | MGP_FLAG_FUSED_SETUP));
    if (!(flags & MGP_AUTOTUNE_FORCE)) {
        std::lock_guard<std::mutex> lk(g_tune_mu);
        tune_cache_load_locked();
        auto it = g_tune_cache.find(key);
        if (it != g_tune_cache.end() && it->second.size() == (size_t)t->levels * MGP_TUNE_PARAMS) {
            CK(cudaStreamSynchronize(t->stream));
            apply_tuning(t, it->second);
            return MGP_OK;
        }
    }
    CK(cudaStreamSynchronize(t->stream));
    SavedFields sv;
    CKS(save_fields(t, sv));
    const std::vector<int> before = current_tuning(t);
    int st = autotune_search(t, cycle, nsmooth, omega, untuned_ms, tuned_ms);
    const int rs = restore_fields(t, sv);
    drop_graphs(t);
    if (st != MGP_OK) {
        apply_tuning(t, before);
        return st;
    }
    CKS(rs);
    const std::vector<int> v = current_tuning(t);
    std::lock_guard<std::mutex> lk(g_tune_mu);
    g_tune_cache[key] = v;
    if (const char* path = tune_file()) {
        std::ofstream out(path, std::ios::app);
        out << key;
        for (int x : v) out << ' ' << x;
        out << '\n';
    }
    return MGP_OK;
}

// ---- solve ----------------------------------------------------------------------------
// Iterative refinement (MGP_FLAG_REFINE_F32 / _F64): r = f - A u in FP64 on level 0, one
// correction cycle A e ~= r on the inner hierarchy (zero initial guess, zero boundary data),
// u += e; repeated until ||r||inf / ||f||inf < tolerance, maxiter steps or maxtime.  The
// correction equation uses the same discrete operator as the reference, so the converged u is
// the reference discretisation's solution; unlike the reference's own cycle loop the
// Neumann boundary data enter only through the FP64 residual, which removes the
// reference's stagnation on Neumann problems.
static int solve_refined(mgp_solver* s, int cycle, int64_t ns, double omega, double maxtime, uint32_t flags,
                         mgp_stats* out) {
    using clock = std::chrono::steady_clock;
    const auto t0 = clock::now();
    auto since = [&](clock::time_point a) { return std::chrono::duration<double>(clock::now() - a).count(); };
    if (cycle != MGP_CYCLE_V && cycle != MGP_CYCLE_F)
        return fail(MGP_ERR_INVALID_ARG, "refinement uses \"Vcycle\" or \"Fcycle\" corrections");
    if (ns < 0) return fail(MGP_ERR_INVALID_ARG, "nsmooth must be >= 0");
    DeviceGuard guard(s->device);
    if (omega < 0) omega = s->desc.relaxation == MGP_JACOBI ? 6.0 / 7.0 : 8.0 / 9.0;
    const int64_t launches_at_start = s->launches + s->inner->launches;
    double fnorm = 0.0, rnorm = 0.0;
    CK(cudaMemsetAsync(s->d_norm + 2, 0, sizeof(unsigned long long), s->stream));
    CKS(norm_t<double>(s, s->lv[0].f, 0, s->d_norm + 2));
    CKS(refine_residual(s, refine_first(s->inner, omega, ns)));
    s->inner->lv[0].first_done = false;  // consumed by the steps' graphs
    CKS(read_norm(s, &rnorm, &fnorm));
    double rel = rnorm / fnorm;
    const double first = rel;
    if (flags & MGP_SOLVE_VERBOSE)
        std::cout << std::setw(4) << 0 << ": Initial residual: " << std::setw(8) << rel << std::endl;
    int64_t it = 0;
    while (it < s->desc.maxiter && !(rel < s->desc.tolerance)) {
        if (since(t0) > maxtime) {
            std::cout << "WARNING: Solver reached maximum wall time without converging!" << std::endl;
            break;
        }
        CKS(launch_refine_step(s, cycle, ns, omega));
        CKS(read_norm(s, &rnorm));
        rel = rnorm / fnorm;
        it++;
        if (flags & MGP_SOLVE_VERBOSE)
            std::cout << std::setw(4) << it << ": Relative residual: " << std::setw(8) << rel << std::endl;
    }
    CKS(refine_store_residual(s));  // the user-visible FP64 residual of the returned u
    CK(cudaStreamSynchronize(s->stream));
    if (out) {
        out->rel_res = rel;
        out->iterations = (double)it;
        out->seconds = since(t0);
        out->cycles_run = it;
        out->first_rel_res = first;
        out->kernel_launches = s->launches + s->inner->launches - launches_at_start;
    }
    return MGP_OK;
}

int mgp_solve(mgp_solver* s, int cycle, int64_t nsmooth, double omega, const char* ofile, double maxtime,
              uint32_t flags, mgp_stats* out) {
    CKS(validate(s));
    if (s->inner) return solve_refined(s, cycle, nsmooth, omega, maxtime, flags, out);
    using clock = std::chrono::steady_clock;
    const auto t0 = clock::now();
    auto since = [&](clock::time_point a) { return std::chrono::duration<double>(clock::now() - a).count(); };
    if (cycle != MGP_CYCLE_RELAXATION && cycle != MGP_CYCLE_V && cycle != MGP_CYCLE_F)
        return fail(MGP_ERR_INVALID_ARG, "solver must be \"Relaxation\", \"Vcycle\" or \"Fcycle\"");
    if (cycle == MGP_CYCLE_F && s->levels < 2)
        return fail(MGP_ERR_INVALID_ARG, "an F-cycle needs at least 2 levels");
    if (nsmooth < 0) return fail(MGP_ERR_INVALID_ARG, "nsmooth must be >= 0");
    DeviceGuard guard(s->device);
    if (omega < 0) omega = s->desc.relaxation == MGP_JACOBI ? 6.0 / 7.0 : 8.0 / 9.0;
    const bool verbose = flags & MGP_SOLVE_VERBOSE;
    const int64_t launches_at_start = s->launches;
    const bool print_cycle = flags & MGP_SOLVE_PRINT_CYCLE_TIME;
    const char* cname = cycle == MGP_CYCLE_V ? "Vcycle" : "Fcycle";

    // initial relative residual (include/libpoisson.h:253-284)
    double fnorm = 0.0, rnorm = 0.0;
    // (both norms in one read-back: words 0 and 2, word 1 holds the passes' error flag)
    CK(cudaMemsetAsync(s->d_norm, 0, sizeof(unsigned long long), s->stream));
    CK(cudaMemsetAsync(s->d_norm + 2, 0, sizeof(unsigned long long), s->stream));
    CKS(DISPATCH(s, (norm_t<T>(s, s->lv[0].f, 0, s->d_norm + 2))));
    CKS(DISPATCH(s, (residual_t<T>(s, 0, s->d_norm))));
    CKS(read_norm(s, &rnorm, &fnorm));
    double rel_res = rnorm / fnorm;
    const double first = rel_res;
    if (verbose) std::cout << std::setw(4) << 0 << ": Initial residual: " << std::setw(8) << rel_res << std::endl;
    std::ofstream log;
    const bool use_log = ofile && ofile[0];
    if (use_log) {
        log.open(ofile, std::ios::app);
        log << "#    seconds     rel_res" << std::endl;
    }
    int64_t iter = 0, cycles = 0;
    for (iter = 0; iter < s->desc.maxiter; iter++) {
        const auto tc = clock::now();
        CKS(launch_iteration(s, cycle, nsmooth, omega));
        double norm = 0.0;
        CKS(read_norm(s, &norm));
        if (cycle != MGP_CYCLE_RELAXATION) {
            cycles++;
            if (print_cycle) std::cout << cname << " took " << since(tc) << " seconds" << std::endl;
        }
        // T norm (include/libpoisson.h:309-331)
        if (s->dtype == MGP_F32) norm = (double)(float)((float)norm / fnorm);
        else norm /= fnorm;
        if (use_log) {  // logs the previous iteration's value, as :332-336 does
            log << std::setw(12) << since(t0);
            log << std::setw(12) << rel_res;
            log << std::endl;
        }
        if (verbose) std::cout << std::setw(4) << iter + 1 << ": Relative residual: " << std::setw(8) << norm << std::endl;
        if (iter >= s->desc.miniter) {
            if (norm > 2.0 * rel_res) {
                rel_res = norm;
                break;
            } else if (std::abs(norm - rel_res) < s->desc.tolerance) {
                rel_res = norm;
                break;
            }
            if (since(t0) > maxtime) {
                std::cout << "WARNING: Solver reached maximum wall time without converging!" << std::endl;
                break;
            }
        }
        rel_res = norm;
    }
    if (out) {
        out->rel_res = rel_res;
        out->iterations = (double)iter;
        out->seconds = since(t0);
        out->cycles_run = cycles;
        out->first_rel_res = first;
        out->kernel_launches = s->launches - launches_at_start;
    }
    return MGP_OK;
}

int mgp_mem_info(int device, size_t* free_bytes, size_t* total_bytes) {
    if (!free_bytes || !total_bytes) return fail(MGP_ERR_INVALID_ARG, "null out pointer");
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || device < 0 || device >= ndev)
        return fail(MGP_ERR_NO_DEVICE, "device %d not present", device);
    DeviceGuard guard(device);
    CK(cudaMemGetInfo(free_bytes, total_bytes));
    return MGP_OK;
}

int mgp_fill_sine_modes(mgp_solver* s, int n_modes, const double* amp, const double* kx, const double* ky,
                        const double* kz, const double L[3]) {
    CKS(validate(s));
    if (s->dtype != MGP_F64) return fail(MGP_ERR_INVALID_ARG, "the sine-mode fill writes an FP64 right-hand side");
    if (n_modes < 0 || n_modes > 64 || (n_modes && (!amp || !kx || !ky || !kz)) || !L)
        return fail(MGP_ERR_INVALID_ARG, "need 0..64 modes and L[3]");
    const double pi = 3.14159265358979323846;
    SineModes m{};
    m.n = n_modes;
    for (int i = 0; i < n_modes; i++) {
        m.amp[i] = amp[i];
        m.wx[i] = kx[i] * pi / L[0];
        m.wy[i] = ky[i] * pi / L[1];
        m.wz[i] = kz[i] * pi / L[2];
    }
    DeviceGuard guard(s->device);
    LevelState& L0 = s->lv[0];
    const Geom& G = L0.G;
    dim3 grid((G.nz + 31) / 32, (G.ny + 7) / 8, 1);
    const int tiles = (int)(grid.x * grid.y);
    const int chunks = std::max(1, std::min(G.nx, (sm_count(s->device) * 8 + tiles - 1) / tiles));
    const int ichunk = (G.nx + chunks - 1) / chunks;
    grid.z = (G.nx + ichunk - 1) / ichunk;
    k_fill_sine<<<grid, kThreads, 0, s->stream>>>((double*)L0.f, G, L0.h, m, ichunk);
    cudaError_t e = cudaGetLastError();
    s->launches++;
    if (e == cudaSuccess) e = cudaStreamSynchronize(s->stream);
    if (e != cudaSuccess) return fail(MGP_ERR_CUDA, "sine-mode fill: %s", cudaGetErrorString(e));
    return MGP_OK;
}

int mgp_fill_problem(mgp_solver* s, int problem) {
    CKS(validate(s));
    if (s->dtype != MGP_F64) return fail(MGP_ERR_INVALID_ARG, "the problem fill writes FP64 level-0 data");
    if (problem < 1 || problem > 3) return fail(MGP_ERR_INVALID_ARG, "problem must be 1, 2 or 3");
    DeviceGuard guard(s->device);
    LevelState& L0 = s->lv[0];
    ProblemFill pf{problem, s->desc.origin[0], s->desc.origin[1], s->desc.origin[2], L0.h};
    const long long n = (long long)L0.G.nx * L0.G.ny * L0.G.nz;
    k_fill_problem_f<<<grid_1d(s, n), kThreads, 0, s->stream>>>((double*)L0.f, (double*)u_ptr(s, 0), L0.G, pf);
    CKS(check_launch(s));
    for (int f = 0; f < 6; f++) {
        const int64_t* fs = L0.face_shape[f];
        const long long nf = fs[0] * fs[1] * fs[2];
        k_fill_problem_face<<<grid_1d(s, nf), kThreads, 0, s->stream>>>((double*)L0.face[f], L0.G, pf, f,
                                                                          s->face_kind[f] == MGP_NEUMANN);
        CKS(check_launch(s));
    }
    if (L0.ubuf[1]) CK(cudaMemsetAsync(uprev_ptr(s, 0), 0, L0.elems * sizeof(double), s->stream));
    CK(cudaStreamSynchronize(s->stream));
    return mgp_write_bc(s, 0);
}

int mgp_u_error(mgp_solver* s, mgp_solver* ref, int problem, double out[4]) {
    CKS(validate(s));
    if (!out) return fail(MGP_ERR_INVALID_ARG, "null out pointer");
    if (s->dtype != MGP_F64 || (ref && ref->dtype != MGP_F64)) return fail(MGP_ERR_INVALID_ARG, "FP64 solvers only");
    LevelState& L0 = s->lv[0];
    if (ref && (ref->lv[0].G.nx != L0.G.nx || ref->lv[0].G.ny != L0.G.ny || ref->lv[0].G.nz != L0.G.nz))
        return fail(MGP_ERR_INVALID_ARG, "shapes differ");
    if (!ref && (problem < 1 || problem > 3)) return fail(MGP_ERR_INVALID_ARG, "problem must be 1, 2 or 3");
    DeviceGuard guard(s->device);
    unsigned long long* dm = nullptr;
    CK(cudaMallocAsync((void**)&dm, 64, s->stream));
    cudaError_t e = cudaMemsetAsync(dm, 0, 64, s->stream);
    ProblemFill pf{problem, s->desc.origin[0], s->desc.origin[1], s->desc.origin[2], L0.h};
    const long long n = (long long)L0.G.nx * L0.G.ny * L0.G.nz;
    if (e == cudaSuccess) {
        k_u_error<<<grid_1d(s, n), kThreads, 0, s->stream>>>((const double*)u_ptr(s, 0),
                                                            ref ? (const double*)u_ptr(ref, 0) : nullptr, L0.G,
                                                            ref ? ref->lv[0].G : L0.G, pf, dm, (double*)(dm + 2));
        e = cudaGetLastError();
        s->launches++;
    }
    unsigned long long h[4] = {0, 0, 0, 0};
    if (e == cudaSuccess) e = cudaMemcpyAsync(h, dm, 32, cudaMemcpyDeviceToHost, s->stream);
    cudaFreeAsync(dm, s->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s->stream);
    if (e != cudaSuccess) return fail(MGP_ERR_CUDA, "u error: %s", cudaGetErrorString(e));
    double v[4];
    memcpy(v, h, 32);
    out[0] = v[0];
    out[1] = std::sqrt(v[2]);
    out[2] = std::sqrt(v[3]);
    out[3] = v[1];
    return MGP_OK;
}

int mgp_fill_uniform(mgp_solver* s, uint64_t seed, double lo, double hi) {
    CKS(validate(s));
    if (s->dtype != MGP_F64) return fail(MGP_ERR_INVALID_ARG, "the uniform fill writes an FP64 right-hand side");
    DeviceGuard guard(s->device);
    LevelState& L0 = s->lv[0];
    const long long n = (long long)L0.G.nx * L0.G.ny * L0.G.nz;
    k_fill_uniform<<<grid_1d(s, n), kThreads, 0, s->stream>>>((double*)L0.f, L0.G, (unsigned long long)seed, lo, hi);
    CKS(check_launch(s));
    CK(cudaStreamSynchronize(s->stream));
    return MGP_OK;
}

int mgp_host_alloc(void** p, size_t bytes) {
    if (!p) return fail(MGP_ERR_INVALID_ARG, "null out pointer");
    CK(cudaMallocHost(p, bytes));
    return MGP_OK;
}
int mgp_host_free(void* p) {
    if (p) CK(cudaFreeHost(p));
    return MGP_OK;
}

}  // extern "C"

#include "mgp_batch.cuh"
#include "mgp_norm_static.cuh"
