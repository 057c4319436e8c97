// ewfd_batch.cu -- the batched solver (ewf_batch_*) and the z-chunk autotuner.
//
// The reference runs one model and one source per process (README.md:86-102; one scenario
// directory per run).  A batch holds several problems (models, possibly of different sizes and
// model families) with several right-hand sides each, advanced together: the launches of a right-hand
// side, or of all of a large model's, form a chain of their own -- two per step -- and the chains of a run
// of steps are captured in one CUDA graph, one after the other (which leaves a model's fields in L2 for
// its whole run of steps) or on parallel branches.
#include "ewfd.h"
#include "ewfd_internal.h"
#include "ewfd_batch.cuh"
#include "ewfd_step.h"

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <map>
#include <tuple>
#include <vector>

using namespace ewf;

#define CK(call)                                                                                     \
    do {                                                                                             \
        cudaError_t e_ = (call);                                                                     \
        if (e_ != cudaSuccess)                                                                       \
            return ewf_fail(e_ == cudaErrorMemoryAllocation ? EWF_ERR_NOMEM : EWF_ERR_CUDA,          \
                            "%s: %s (%s:%d)", #call, cudaGetErrorString(e_), __FILE__, __LINE__);     \
    } while (0)

namespace {

struct Prob {
    ewf_params p;
    int R = 1;
    int sx = 0;             // materials / damping box
    long long sy = 0;
    size_t box = 0;
    long long base_off = 0;
    size_t sbox = 0;        // the R state boxes (the material box's pitches)
    long long sbase_off = 0;
    void *state[9] = {};
    void *mats[12] = {};
    void *w1[3] = {};
    void *w3 = nullptr;
    bool m_set[12] = {};
    bool w_set[4] = {};
    int kchunk = 0;                         // planes per CTA (0: by size, split_shape)
    const SrcEntry *d_sent = nullptr;       // source entries, right-hand side by right-hand side
    const int *d_sstart = nullptr;          // first entry of each right-hand side, R + 1
    int group0 = 0;                         // the problem's first (problem, RHS) group of k_binject
    RecFuse rf{};                           // receivers in the velocity kernel
    bool rec_fuse = true;
    bool fdiv = false;                      // div_spacing verified for dx, dy, dz
    std::vector<int32_t> rec;               // n x (i,j,k,comp)
    std::vector<std::vector<BatchSrc>> src;  // per RHS
    std::vector<double> stf;
};

// Tables for the device, gathered on the host: one allocation and one copy for all of them (one each took the host
// 42 us a problem: 8 ms for 200 problems of 16^3, which take 45 us a step).
struct Tables {
    std::vector<unsigned char> h;
    unsigned char *d = nullptr;
    template <typename T>
    size_t add(const std::vector<T> &v)  // its place, for at()
    {
        const size_t at = (h.size() + 255) / 256 * 256;
        h.resize(at + v.size() * sizeof(T));
        if (!v.empty()) memcpy(h.data() + at, v.data(), v.size() * sizeof(T));
        return at;
    }
    int send()
    {
        if (h.empty()) return EWF_OK;
        CK(cudaMalloc(&d, h.size()));
        CK(cudaMemcpy(d, h.data(), h.size(), cudaMemcpyHostToDevice));
        h = std::vector<unsigned char>();
        return EWF_OK;
    }
    template <typename T>
    const T *at(size_t place) const { return reinterpret_cast<const T *>(d + place); }
    void free()
    {
        cudaFree(d);
        d = nullptr;
        h.clear();
    }
};

// What one sequence of launches advances: right-hand sides [r0, r0 + R) of a problem
struct Chain {
    int prob = 0, r0 = 0, R = 1;
    int branch = -1;          // its branch (balanced by cell-updates), -1: the batch's stream
    int ty = 4;               // CTA tile height
    bool pair = false;        // two cells per thread
    bool stream_l2 = false;   // its kernels: materials and new velocities first to leave L2
    StepArgs<float> a;        // of right-hand side r0
    StressSrc ss{};           // sources in the stress kernel (nsrc 0: k_binject)
    int nsrc = 0;
    RecFuse rf{};
    double work = 0;          // cells
    std::vector<int> many;    // the chains of tiny problems it stands for (k_stress_many), and for each step parity
    const ManyProb *d_many[2] = {nullptr, nullptr};  // their arguments,
    const int2 *d_map = nullptr;  // and the problem of each CTA
    int blocks = 0;
    const int *d_groups = nullptr;  // the (problem, RHS) groups of theirs that k_binject applies,
    const int2 *d_rows = nullptr;   // the receivers (row, problem) that k_brecord_many samples
    int groups = 0, rows = 0;
};

float *bptr(const Prob &q, void *alloc) { return alloc ? (float *)alloc + q.base_off : nullptr; }
// Right-hand sides of a model between these many cells run apart, each its own chain: by itself one keeps its
// fields in L2 from step to step.  On larger grids they share launches, and the materials' way from HBM; on
// smaller ones a step of many chains is bound by their launches, about 1 us each.  us per step of 2, 3 and 6
// right-hand sides of ortho n^3 in shared launches and apart:
//   64^3 13 17 33 and 10 14 31        96^3 35 56 116 and 34 52 103      112^3 66 101 198 and 61 91 182
//   128^3 92 136 260 and 84 126 251   144^3 142 206 396 and 142 213 426   160^3 182 265 513 and 186 278 556
// and of 6 with a small isotropic model: 30^3 11.4 and 14.5, 40^3 16.1 and 17.9, 50^3 28.1 and 23.6, 64^3 40.3 and 30.7.
// More of them change nothing: 64 of iso 50^3 180 and 129, 64^3 304 and 203, 80^3 667 and 369, of ortho 50^3 221 and 169, 64^3 361
// and 279; 32 of iso 100^3 699 and 502, of ortho 100^3 821 and 738; 12 of ortho 128^3 520 and 488.
constexpr double APART_FROM = 1e5, APART_TO = 2.5e6;

float *sptr(const Prob &q, void *alloc) { return alloc ? (float *)alloc + q.sbase_off : nullptr; }

}  // namespace

struct ewf_batch {
    int device = 0;
    int nt = 0;
    cudaStream_t stream = nullptr;
    cudaEvent_t ev0 = nullptr, ev1 = nullptr;
    std::vector<Prob> probs;
    std::vector<Chain> chains;
    Tables tables, many_tables;          // what the pointers below and those of the problems and chains point into
    const BatchProb<float> *d_all = nullptr;  // every problem, indexed by problem id
    std::vector<BatchProb<float>> h_all;  // host copy of d_all
    int nrhs_total = 0;
    // sources
    const BatchSrc *d_src = nullptr;
    const int *d_src_start = nullptr;
    const double *d_stf = nullptr;
    const int *d_stf_off = nullptr;
    const int *d_order = nullptr;
    // receivers
    const long long *d_rec_off = nullptr;
    const int *d_rec_comp = nullptr;
    int nrec_total = 0;
    std::vector<int> rec_base;  // per problem: first trace row
    double *d_traces = nullptr;
    int *d_it = nullptr;
    int it = 0;
    void *d_stage = nullptr;
    size_t stage_bytes = 0;
    bool dirty = true;   // device tables need a rebuild
    int ty = 4;          // CTA tile height (4, 8 or 16 rows of 32 columns; two-cell kernels: twice as many, 16 at most)
    int l2pf = 0;        // the velocity kernels' L2 prefetch distance (autotuned; 0: by size)
    int own = 0;         // the problems' chains on parallel streams: those that do not fill the GPU (0), all (1) (autotuned)
    bool pdl = true;     // kernels launched as programmatic dependents (off if capture refuses)
    static constexpr int BRANCHES = 8;
    cudaStream_t branch[BRANCHES] = {};
    cudaEvent_t fork_ev = nullptr, join_ev[BRANCHES] = {};
    cudaGraphExec_t gexec = nullptr, gexec_short = nullptr;  // of gsteps and of SHORT_GRAPH steps
    int gsteps = 64;     // steps per graph (even: the step counters alternate between two locations)
    long long ran = 0;   // steps run since the tables were made
    float last_ms = 0.f;
};

static void free_tables(ewf_batch *b)
{
    b->chains.clear();
    b->ran = 0;
    b->tables.free();
    b->many_tables.free();
    for (cudaGraphExec_t *x : {&b->gexec, &b->gexec_short}) {
        if (*x) cudaGraphExecDestroy(*x);
        *x = nullptr;
    }
}

extern "C" void ewf_batch_destroy(ewf_batch *b)
{
    if (!b) return;
    cudaSetDevice(b->device);
    if (b->stream) cudaStreamSynchronize(b->stream);
    free_tables(b);
    for (auto &q : b->probs) {
        for (auto &x : q.state) cudaFree(x);
        for (auto &x : q.mats) cudaFree(x);
        for (auto &x : q.w1) cudaFree(x);
        cudaFree(q.w3);
    }
    cudaFree(b->d_traces);
    cudaFree(b->d_it);
    cudaFree(b->d_stage);
    if (b->ev0) cudaEventDestroy(b->ev0);
    if (b->ev1) cudaEventDestroy(b->ev1);
    if (b->fork_ev) cudaEventDestroy(b->fork_ev);
    for (auto &e : b->join_ev)
        if (e) cudaEventDestroy(e);
    for (auto &x : b->branch)
        if (x) cudaStreamDestroy(x);
    if (b->stream) cudaStreamDestroy(b->stream);
    delete b;
}

extern "C" int ewf_batch_create(int32_t n, const ewf_params *p, const int32_t *n_rhs, ewf_batch **out)
{
    if (!out || !p || n < 1 || n > 4096) return ewf_fail(EWF_ERR_ARG, "bad batch size");
    *out = nullptr;
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev < 1) {
        cudaGetLastError();
        return ewf_fail(EWF_ERR_NODEVICE, "no CUDA device visible");
    }
    for (int i = 0; i < n; ++i) {
        const ewf_params &q = p[i];
        if (q.nx < 4 || q.ny < 4 || q.nz < 4) return ewf_fail(EWF_ERR_ARG, "problem %d: grid must be >= 4", i);
        if (q.precision != EWF_PREC_F32) return ewf_fail(EWF_ERR_UNSUPPORTED, "problem %d: batches are FP32", i);
        if (q.nt != p[0].nt) return ewf_fail(EWF_ERR_ARG, "problem %d: every problem of a batch runs the same nt", i);
        if ((q.model == EWF_MODEL_ISO) != (q.damping == EWF_DAMP_PML1D))
            return ewf_fail(EWF_ERR_UNSUPPORTED, "problem %d: model/damping combination", i);
        if (q.model == EWF_MODEL_ISO_HET || q.vdamp != 0.0)
            return ewf_fail(EWF_ERR_UNSUPPORTED, "problem %d: batches run models 0 and 1 without vdamp", i);
        if (q.nx > q.ny && q.over_y > 0) return ewf_fail(EWF_ERR_UNSUPPORTED, "problem %d: nx > ny with over_y > 0", i);
        if (n_rhs && (n_rhs[i] < 1 || n_rhs[i] > 64)) return ewf_fail(EWF_ERR_ARG, "problem %d: 1..64 right-hand sides", i);
        if (!(q.dx > 0 && q.dy > 0 && q.dz > 0 && q.dt > 0)) return ewf_fail(EWF_ERR_ARG, "problem %d: spacing/dt", i);
    }
    ewf_batch *b = new (std::nothrow) ewf_batch();
    if (!b) return ewf_fail(EWF_ERR_NOMEM, "host allocation");
    cudaGetDevice(&b->device);
    b->nt = p[0].nt;
    b->probs.resize(n);
    size_t stage = 0;
#define CKB(call)                                                                                    \
    do {                                                                                             \
        cudaError_t e_ = (call);                                                                     \
        if (e_ != cudaSuccess) {                                                                     \
            int s_ = ewf_fail(e_ == cudaErrorMemoryAllocation ? EWF_ERR_NOMEM : EWF_ERR_CUDA,         \
                              "%s: %s", #call, cudaGetErrorString(e_));                              \
            ewf_batch_destroy(b);                                                                    \
            return s_;                                                                               \
        }                                                                                            \
    } while (0)
    CKB(cudaStreamCreateWithFlags(&b->stream, cudaStreamNonBlocking));
    CKB(cudaEventCreate(&b->ev0));
    CKB(cudaEventCreate(&b->ev1));
    CKB(cudaEventCreateWithFlags(&b->fork_ev, cudaEventDisableTiming));
    for (int k = 0; k < ewf_batch::BRANCHES; ++k) {
        CKB(cudaStreamCreateWithFlags(&b->branch[k], cudaStreamNonBlocking));
        CKB(cudaEventCreateWithFlags(&b->join_ev[k], cudaEventDisableTiming));
    }
    for (int i = 0; i < n; ++i) {
        Prob &q = b->probs[i];
        q.p = p[i];
        q.p.workdir = nullptr;
        q.R = n_rhs ? n_rhs[i] : 1;
        q.kchunk = p[i].kchunk > 0 ? p[i].kchunk : 0;
        if (q.p.model == EWF_MODEL_ORTHO)
            q.fdiv = ewf_fdiv_verified((float)q.p.dx) && ewf_fdiv_verified((float)q.p.dy) &&
                     ewf_fdiv_verified((float)q.p.dz);
        const int hx = 32;
        q.sx = hx + ((q.p.nx + 2 + 31) / 32) * 32;
        q.sy = (long long)q.sx * (q.p.ny + 3);
        q.box = (size_t)q.sy * (q.p.nz + 3);
        q.base_off = hx + (long long)q.sx + q.sy;
        q.sbox = q.box * q.R;      // R boxes back to back
        q.sbase_off = q.base_off;
        q.src.resize(q.R);
        for (int f = 0; f < 9; ++f) {
            CKB(cudaMalloc(&q.state[f], q.sbox * 4));
            CKB(cudaMemsetAsync(q.state[f], 0, q.sbox * 4, b->stream));
        }
        const int nm = q.p.model == EWF_MODEL_ISO ? 2 : 12;
        for (int f = 0; f < nm; ++f) {
            CKB(cudaMalloc(&q.mats[f], q.box * 4));
            CKB(cudaMemsetAsync(q.mats[f], 0, q.box * 4, b->stream));
        }
        if (q.p.damping == EWF_DAMP_W3D) {
            CKB(cudaMalloc(&q.w3, q.box * 4));
            CKB(cudaMemsetAsync(q.w3, 0, q.box * 4, b->stream));
        } else {
            const int n1[3] = {q.p.nx + 2, q.p.ny + 2, q.p.nz + 2};
            for (int a = 0; a < 3; ++a) {
                CKB(cudaMalloc(&q.w1[a], n1[a] * 4));
                CKB(cudaMemsetAsync(q.w1[a], 0, n1[a] * 4, b->stream));
            }
        }
        stage = std::max(stage, (size_t)(q.p.nx + 1) * (q.p.ny + 1) * (q.p.nz + 1) * 8);
        b->nrhs_total += q.R;
    }
    CKB(cudaMalloc(&b->d_stage, stage));
    b->stage_bytes = stage;
    // graphs of two launches per chain and step, of some 16 thousand nodes at most
    const size_t nch = b->nrhs_total;  // chains, at most
    while (b->gsteps > 2 && b->gsteps * 2 * nch > 16384) b->gsteps -= 2;
    CKB(cudaMalloc(&b->d_it, 2 * nch * sizeof(int)));
    CKB(cudaMemsetAsync(b->d_it, 0, 2 * nch * sizeof(int), b->stream));
    CKB(cudaStreamSynchronize(b->stream));
#undef CKB
    *out = b;
    return EWF_OK;
}

static int check_prob(const ewf_batch *b, int32_t prob)
{
    if (!b) return ewf_fail(EWF_ERR_ARG, "NULL batch");
    if (prob < 0 || prob >= (int)b->probs.size()) return ewf_fail(EWF_ERR_ARG, "problem %d out of range", prob);
    return EWF_OK;
}

static int mat_slot(int model, int id)
{
    static const int ortho[] = {EWF_M_C11, EWF_M_C22, EWF_M_C33, EWF_M_C12, EWF_M_C13, EWF_M_C23,
                                EWF_M_C66XY, EWF_M_C55XZ, EWF_M_C44YZ, EWF_M_BX, EWF_M_BY, EWF_M_BZ};
    if (model == EWF_MODEL_ISO) return id == EWF_M_C11 ? 0 : id == EWF_M_C12 ? 1 : -1;
    for (int q = 0; q < 12; ++q)
        if (ortho[q] == id) return q;
    return -1;
}

extern "C" int ewf_batch_set_field(ewf_batch *b, int32_t prob, int32_t field, const void *host, size_t n,
                                   int32_t dtype_bytes)
{
    int st = check_prob(b, prob);
    if (st) return st;
    if (!host || (dtype_bytes != 4 && dtype_bytes != 8)) return ewf_fail(EWF_ERR_ARG, "bad host buffer");
    Prob &q = b->probs[prob];
    int ex, ey, ez;
    if (!ewf_field_extent(q.p, field, &ex, &ey, &ez)) return ewf_fail(EWF_ERR_ARG, "field %d not in this problem", field);
    if (n != (size_t)ex * ey * ez) return ewf_fail(EWF_ERR_ARG, "field %d: %zu elements, %d expected", field, n, ex * ey * ez);
    float *dst;
    int sx = q.sx;
    long long sy = q.sy;
    const int ms = mat_slot(q.p.model, field);
    if (ms >= 0) dst = bptr(q, q.mats[ms]);
    else if (field == EWF_D_W3D) dst = bptr(q, q.w3);
    else if (field >= EWF_D_WX && field <= EWF_D_WZ) { dst = (float *)q.w1[field - EWF_D_WX]; sx = 0; sy = 0; }
    else return ewf_fail(EWF_ERR_ARG, "field %d: batches take materials and damping (state starts at zero)", field);
    CK(cudaMemcpyAsync(b->d_stage, host, n * dtype_bytes, cudaMemcpyHostToDevice, b->stream));
    const unsigned nb = (unsigned)std::min<size_t>((n + 255) / 256, 152 * 16);
    if (dtype_bytes == 4) k_pack<float, float><<<nb, 256, 0, b->stream>>>(dst, (const float *)b->d_stage, ex, ey, ez, sx, sy);
    else k_pack<float, double><<<nb, 256, 0, b->stream>>>(dst, (const double *)b->d_stage, ex, ey, ez, sx, sy);
    CK(cudaGetLastError());
    CK(cudaStreamSynchronize(b->stream));
    if (ms >= 0) q.m_set[ms] = true;
    if (field >= EWF_D_WX && field <= EWF_D_W3D) q.w_set[field - EWF_D_WX] = true;
    return EWF_OK;
}

extern "C" int ewf_batch_set_stf(ewf_batch *b, int32_t prob, const double *stf, size_t n)
{
    int st = check_prob(b, prob);
    if (st) return st;
    if (!stf || n < (size_t)b->nt) return ewf_fail(EWF_ERR_ARG, "Src needs %d samples", b->nt);
    b->probs[prob].stf.assign(stf, stf + b->nt);
    b->dirty = true;
    return EWF_OK;
}

extern "C" int ewf_batch_set_sources(ewf_batch *b, int32_t prob, int32_t rhs, int32_t n, const int32_t *cijk,
                                     const double *coef)
{
    int st = check_prob(b, prob);
    if (st) return st;
    Prob &q = b->probs[prob];
    if (rhs < 0 || rhs >= q.R) return ewf_fail(EWF_ERR_ARG, "rhs %d out of range", rhs);
    if (n < 0 || n > MAXSRC || (n > 0 && (!cijk || !coef))) return ewf_fail(EWF_ERR_ARG, "0..%d sources", MAXSRC);
    std::vector<BatchSrc> v;
    for (int e = 0; e < n; ++e) {
        const int c = cijk[4 * e], i = cijk[4 * e + 1], j = cijk[4 * e + 2], k = cijk[4 * e + 3];
        int ex, ey, ez;
        if (c < EWF_F_SXX || c > EWF_F_SYZ || !ewf_field_extent(q.p, c, &ex, &ey, &ez))
            return ewf_fail(EWF_ERR_ARG, "source %d: not a stress field", e);
        if (i < 0 || j < 0 || k < 0 || i >= ex || j >= ey || k >= ez) return ewf_fail(EWF_ERR_ARG, "source %d outside the grid", e);
        v.push_back(BatchSrc{prob, rhs, c, i, j, k, coef[e]});
    }
    q.src[rhs] = v;
    b->dirty = true;
    return EWF_OK;
}

extern "C" int ewf_batch_set_moment_tensor(ewf_batch *b, int32_t prob, int32_t rhs, const double mt[6], int32_t xs,
                                           int32_t ys, int32_t zs, int32_t stencil)
{
    if (!mt) return ewf_fail(EWF_ERR_ARG, "NULL tensor");
    int32_t cijk[24];
    double coef[6];
    static const int ok4[6][3] = {{1, 1, 1}, {1, 1, 1}, {1, 1, 1}, {3, 3, 1}, {3, 3, 1}, {2, 2, 1}};
    static const int ani[6][3] = {{1, 1, 1}, {1, 1, 1}, {1, 1, 1}, {2, 2, 1}, {-1, 1, 1}, {3, 2, 1}};
    static const int comp[6] = {EWF_F_SXX, EWF_F_SYY, EWF_F_SZZ, EWF_F_SXY, EWF_F_SXZ, EWF_F_SYZ};
    // statement order of the reference: OK4:336-342 (xx yy zz yz xz xy), ANISO:233-247 (xx yy zz xy yz xz)
    static const int ord_ok4[6] = {0, 1, 2, 5, 4, 3};
    static const int ord_ani[6] = {0, 1, 2, 3, 5, 4};
    if (stencil != 0 && stencil != 1) return ewf_fail(EWF_ERR_ARG, "stencil must be 0 or 1");
    for (int e = 0; e < 6; ++e) {
        const int m = stencil == 0 ? ord_ok4[e] : ord_ani[e];
        const int *o = stencil == 0 ? ok4[m] : ani[m];
        cijk[4 * e] = comp[m];
        cijk[4 * e + 1] = xs + o[0];
        cijk[4 * e + 2] = ys + o[1];
        cijk[4 * e + 3] = zs + o[2];
        coef[e] = mt[m];
    }
    return ewf_batch_set_sources(b, prob, rhs, 6, cijk, coef);
}

extern "C" int ewf_batch_set_receivers(ewf_batch *b, int32_t prob, int32_t n, const int32_t *ijkc)
{
    int st = check_prob(b, prob);
    if (st) return st;
    Prob &q = b->probs[prob];
    if (n < 0 || (n > 0 && !ijkc)) return ewf_fail(EWF_ERR_ARG, "bad receiver list");
    for (int r = 0; r < n; ++r) {
        const int i = ijkc[4 * r], j = ijkc[4 * r + 1], k = ijkc[4 * r + 2], c = ijkc[4 * r + 3];
        int ex, ey, ez;
        if (c < 0 || c > 8 || !ewf_field_extent(q.p, c, &ex, &ey, &ez)) return ewf_fail(EWF_ERR_ARG, "receiver %d field", r);
        if (i < 0 || j < 0 || k < 0 || i >= ex || j >= ey || k >= ez) return ewf_fail(EWF_ERR_ARG, "receiver %d outside", r);
    }
    q.rec.assign(ijkc, ijkc + 4 * (size_t)n);
    b->dirty = true;
    return EWF_OK;
}

// Chains below BRANCH_CELLS cells share the GPU on parallel branches; a larger one
// fills it, and alone keeps its fields in L2.  us per step of six problems n^3, one after another and on
// four branches:
//   iso    32^3 30 10   64^3 40 22   80^3 62 50   96^3 76 88     128^3 198 222   160^3 432 441
//   ortho  32^3 30 11   64^3 50 30   80^3 75 76   96^3 104 122   128^3 296 287   160^3 571 565
// As many branches (two at least) as hold BRANCH_SHARE cells between them, which L2 still keeps.  us per step on 2, 4 and
// 8 branches (these and the above with chunks by each problem's own size):
//   12 iso 24^3 29 16 11    6 iso 40^3 17 14 12     8 iso 50^3 29 24 25    8 iso 64^3 32 28 39
//   8 ortho 64^3 40 40 54   8 iso 72^3 52 61 82     8 iso 80^3 50 74 91    6 ortho 80^3 64 76 85
constexpr double BRANCH_CELLS = 6e5, BRANCH_SHARE = 1.1e6;
// MANY_MIN or more problems of one scheme below MANY_CELLS cells share two launches a step (k_stress_many), and one more each for
// sources and receivers that those do not take: more chains than there are branches wait for one another's launches.  A few of
// the largest run better as chains, so those up to MANY_CELLS_2 have to be MANY_MIN_2, and fit L2 together where the model has
// twelve material arrays (MANY_ORTHO cells).  us per step of chains and of shared launches by number of problems:
//   iso 12^3  8 5.7 8.2   16 11.1 8.2   100 71 19       iso 16^3  8 5.5 7.7   15 10.7 8.0   50 36 13.6   200 134 45
//   iso 24^3  8 5.8 8.0   15 11.2 9.3   50 38 22   200 143 103      iso 28^3  8 6.4 11.8   16 12.6 14.1   50 43 28   200 159 144
//   iso 27^3  9 11.0 12.2   12 11.8 10.6     iso 32^3  16 13.2 14.9   50 44.5 42.9   200 165 178
//   ortho 24^3  9 10.9 11.4   15 11.9 11.0   50 40 30     ortho 28^3  33 30.8 27.3   100 84 93     ortho 32^3  100 91 120
// and of problems with a stress receiver each: iso 16^3  15 17.4 9.6   50 60 15.8   200 253 48     iso 28^3  50 74 31   200 277 147.
constexpr double MANY_CELLS = 2e4, MANY_CELLS_2 = 2.8e4, MANY_ORTHO = 1.2e6;
constexpr int MANY_MIN = 12, MANY_MIN_2 = 32;
// A chunk that is asked for is the most planes that the rule by size may take.  It takes no more than 6 by itself, and chains
// want no more: one model after another, or few at a time, they do not fill the GPU in longer chunks.  us per step by the rule and in 16, 32 and 64
// planes: 4 iso 100^3 63 137 186 293     6 iso 64^3 22 46 71 124     6 rhs of ortho 80^3 55 131 173 295     4 rhs of iso 144^3 221 232 239 251
// (64 planes in the shared launches of before 147, 93, 266, 306).  8 stands for the rule where the autotuner returns it.
constexpr int KCHUNK_BY_SIZE = 8;
static int scheme(const ewf_params &p) { return p.model == EWF_MODEL_ISO ? 0 : p.damping == EWF_DAMP_W3D ? 1 : 2; }

// Rebuilds the device tables (problem descriptors, sources, receivers, traces).
static int build_tables(ewf_batch *b)
{
    CK(cudaStreamSynchronize(b->stream));
    free_tables(b);
    const int n = (int)b->probs.size();
    std::vector<BatchProb<float>> all(n);
    for (int i = 0; i < n; ++i) {
        Prob &q = b->probs[i];
        const ewf_params &p = q.p;
        BatchProb<float> &bp = all[i];
        memset(&bp, 0, sizeof(bp));
        StepArgs<float> &d = bp.a;
        for (int f = 0; f < 9; ++f) d.f[f] = sptr(q, q.state[f]);
        for (int f = 0; f < 12; ++f) d.m[f] = bptr(q, q.mats[f]);
        for (int a = 0; a < 3; ++a) d.w1[a] = (const float *)q.w1[a];
        d.w3 = bptr(q, q.w3);
        d.sy = q.sy;
        d.sx = q.sx;
        bp.rhs_stride = (long long)q.box;
        d.nx = p.nx; d.ny = p.ny; d.nz = p.nz;
        d.bc1_rows = std::min(p.ny, std::min(p.nx, p.ny + std::max(0, p.over_y)));
        d.dt = (float)p.dt;
        d.rdt = 1.0f / d.dt;
        d.dx = (float)p.dx; d.dy = (float)p.dy; d.dz = (float)p.dz;
        d.rdx = 1.0f / d.dx; d.rdy = 1.0f / d.dy; d.rdz = 1.0f / d.dz;
        d.c66 = (float)p.c66; d.bx = (float)p.bx; d.by = (float)p.by; d.bz = (float)p.bz;
        d.third = 1.0f / 3.0f;
        d.one = 1.0f;
        d.minus_one = -1.0f;
        d.fdiv = q.fdiv ? 1 : 0;
        d.bc1 = p.free_surface == EWF_FS_BC1 ? 1 : 0;
        d.smu_on = p.surface_mu > 0.0 ? 1 : 0;
        d.smu = (float)p.surface_mu;
    }
    Tables &tab = b->tables;
    struct Places {
        size_t ent, from, grp, off, rent;
    };
    std::vector<Places> at(n);
    const size_t at_all = tab.add(all);
    // sources grouped by (problem, rhs)
    std::vector<BatchSrc> src;
    std::vector<int> start;
    std::vector<double> stf((size_t)n * b->nt, 0.0);
    std::vector<int> stf_off(n), order(n);
    for (int i = 0; i < n; ++i) {
        Prob &q = b->probs[i];
        q.group0 = (int)start.size();
        std::vector<SrcEntry> ent;
        std::vector<int> from;
        for (int r = 0; r < q.R; ++r) {
            start.push_back((int)src.size());
            from.push_back((int)ent.size());
            for (auto &e : q.src[r]) {
                src.push_back(e);
                ent.push_back(SrcEntry{e.comp, e.i, e.j, e.k, e.coef});
            }
            if (!q.src[r].empty() && q.stf.empty()) return ewf_fail(EWF_ERR_STATE, "problem %d has sources but no Src", i);
        }
        from.push_back((int)ent.size());
        at[i].ent = tab.add(ent);
        at[i].from = tab.add(from);
        stf_off[i] = i * b->nt;
        if (!q.stf.empty()) std::copy(q.stf.begin(), q.stf.end(), stf.begin() + (size_t)i * b->nt);
        order[i] = q.p.src_order;
    }
    start.push_back((int)src.size());
    b->h_all = all;
    const size_t at_src = tab.add(src), at_start = tab.add(start), at_stf = tab.add(stf), at_stf_off = tab.add(stf_off), at_order = tab.add(order);
    // receivers: per problem, RHS-major
    std::vector<int> rc;
    std::vector<long long> ro;
    b->rec_base.assign(n, 0);
    for (int i = 0; i < n; ++i) {
        Prob &q = b->probs[i];
        b->rec_base[i] = (int)rc.size();
        const int nr = (int)q.rec.size() / 4;
        for (int r = 0; r < q.R; ++r)
            for (int e = 0; e < nr; ++e) {
                rc.push_back(q.rec[4 * e + 3]);
                ro.push_back((long long)q.rec[4 * e] + (long long)q.rec[4 * e + 1] * q.sx +
                             (long long)q.rec[4 * e + 2] * q.sy + (long long)r * (long long)q.box);
            }
    }
    const int nrec = (int)rc.size();
    if (nrec != b->nrec_total || !b->d_traces) {
        cudaFree(b->d_traces);
        b->d_traces = nullptr;
        if (nrec) {
            CK(cudaMalloc(&b->d_traces, (size_t)nrec * b->nt * sizeof(double)));
            CK(cudaMemset(b->d_traces, 0, (size_t)nrec * b->nt * sizeof(double)));
        }
    }
    b->nrec_total = nrec;
    const size_t at_rec_off = tab.add(ro), at_rec_comp = tab.add(rc);
    for (int i = 0; i < n; ++i) {
        Prob &q = b->probs[i];
        const RecTables t = make_rec_tables((int)q.rec.size() / 4, q.rec.data(), q.p.nx, q.p.ny, q.p.nz);
        q.rec_fuse = t.fuse;
        q.rf = RecFuse{};
        at[i].grp = tab.add(t.grp);
        at[i].off = tab.add(t.off);
        at[i].rent = tab.add(t.ent);
        if (t.fuse && !t.ent.empty()) {
            q.rf.ngx = (q.p.nx + 31) / 32;
            q.rf.kmin = t.kmin;
            q.rf.kmax = t.kmax;
            q.rf.traces = b->d_traces + (size_t)b->rec_base[i] * b->nt;
            q.rf.trace_len = b->nt;
        }
    }
    if (int st = tab.send()) return st;
    b->d_all = tab.at<BatchProb<float>>(at_all);
    b->d_src = tab.at<BatchSrc>(at_src);
    b->d_src_start = tab.at<int>(at_start);
    b->d_stf = tab.at<double>(at_stf);
    b->d_stf_off = tab.at<int>(at_stf_off);
    b->d_order = tab.at<int>(at_order);
    b->d_rec_off = tab.at<long long>(at_rec_off);
    b->d_rec_comp = tab.at<int>(at_rec_comp);
    for (int i = 0; i < n; ++i) {
        Prob &q = b->probs[i];
        q.d_sent = tab.at<SrcEntry>(at[i].ent);
        q.d_sstart = tab.at<int>(at[i].from);
        if (q.rf.traces) {
            q.rf.grp = tab.at<uint2>(at[i].grp);
            q.rf.off = tab.at<int>(at[i].off);
            q.rf.ent = tab.at<int2>(at[i].rent);
        }
    }
    // the chains, and which of them are tiny problems whose launches take sources and receivers
    auto fuses = [&](const Chain &c, std::vector<SrcEntry> *ent, int *before, StressSrc *f, bool *plane1) {
        const Prob &q = b->probs[c.prob];
        *before = 0;
        for (int r = 0; r < c.r0 + c.R; ++r) {
            if (r < c.r0) *before += (int)q.src[r].size();
            else
                for (auto &e : q.src[r]) ent->push_back(SrcEntry{e.comp, e.i, e.j, e.k, e.coef});
        }
        return make_stress_src(*ent, q.p.nx, q.p.ny, q.p.nz, f, plane1);
    };
    std::vector<Chain> singles;
    std::vector<int> tiny[3][2];  // by scheme, up to MANY_CELLS and above
    for (int i = 0; i < n; ++i) {
        const Prob &q = b->probs[i];
        const double cells = (double)q.p.nx * q.p.ny * q.p.nz;
        Chain c;
        c.prob = i;
        if (cells >= APART_FROM && cells < APART_TO) {
            c.work = cells;
            for (c.r0 = 0; c.r0 < q.R; ++c.r0) singles.push_back(c);
            continue;
        }
        c.R = q.R;
        c.work = cells * q.R;
        if (cells < MANY_CELLS_2 && q.R == 1) tiny[scheme(q.p)][cells < MANY_CELLS ? 0 : 1].push_back((int)singles.size());
        singles.push_back(c);
    }
    std::vector<char> grouped(singles.size(), 0);
    auto share_launches = [&](const std::vector<int> &list) {
        Chain c;
        c.prob = singles[list[0]].prob;
        c.many = list;
        for (int q : list) {
            c.work += singles[q].work;
            grouped[q] = 1;
        }
        b->chains.push_back(c);
    };
    for (auto &t : tiny) {
        std::vector<int> list;
        double cells = 0;
        for (int q : t[1]) cells += singles[q].work;
        if (t[0].size() + t[1].size() >= MANY_MIN_2 && (&t == &tiny[0] || cells <= MANY_ORTHO)) list = t[1];
        if (t[0].size() + list.size() >= MANY_MIN) list.insert(list.begin(), t[0].begin(), t[0].end());
        if (!list.empty()) share_launches(list);
    }
    // their list of CTAs also takes a model of more rows than a grid of 65535 CTAs of 16
    for (int q = 0; q < (int)singles.size(); ++q)
        if (singles[q].R == 1 && b->probs[singles[q].prob].p.ny > 65535 * 16) share_launches({q});
    for (size_t q = 0; q < singles.size(); ++q)
        if (!grouped[q]) b->chains.push_back(singles[q]);
    // branches: largest chains first, each to the least loaded branch
    int share = 1;  // chains that run at the same time
    for (auto &c : b->chains) c.branch = -1;
    if (b->chains.size() > 1) {
        std::vector<Chain *> idx;
        for (auto &c : b->chains)
            if (b->own || c.work < BRANCH_CELLS) idx.push_back(&c);
        std::stable_sort(idx.begin(), idx.end(), [](const Chain *x, const Chain *y) { return x->work > y->work; });
        int branches = std::min(2, (int)idx.size());
        double held = 0;
        for (int k = 0; k < (int)idx.size() && k < ewf_batch::BRANCHES; ++k) {
            held += idx[k]->work;
            if (held <= BRANCH_SHARE) branches = std::max(branches, k + 1);
        }
        share = std::max(1, branches);
        double load[ewf_batch::BRANCHES] = {};
        for (Chain *c : idx) {
            c->branch = (int)(std::min_element(load, load + branches) - load);
            load[c->branch] += c->work;
        }
    }
    auto prepare = [&](Chain &c, double together) {
        const Prob &q = b->probs[c.prob];
        const ewf_params &p = q.p;
        const SplitShape shape = split_shape(p.nx, p.ny, p.nz, c.R);
        c.ty = std::max(b->ty, shape.ty);
        c.stream_l2 = shape.stream;
        c.a = all[c.prob].a;
        for (auto &f : c.a.f) f += c.r0 * (long long)q.box;
        c.a.l2pf = b->l2pf ? b->l2pf : shape.l2pf;
        // Chunks as long as for one problem of all the cells that run at the same time.  us per step with chunks by
        // the problem's own size, and so: 6 iso 40^3 12.0 and 8.8, 16 iso 40^3 32.4 and 22.9, 8 iso 50^3 24.5 and
        // 16.8, 8 ortho 64^3 40.6 and 38.1, 8 iso 80^3 50.1 and 49.2.
        c.a.kchunk = split_shape(p.nx, p.ny, p.nz, (int)std::min(1e6, c.R * together)).kchunk;
        if (q.kchunk > 0) c.a.kchunk = std::min(q.kchunk, c.a.kchunk);
        c.a.kchunk = std::max(c.a.kchunk, (p.nz + 65534) / 65535);  // a grid has at most 65535 CTAs along z
        c.pair = c.R > 1 || (shape.pair && enough_pairs(p.model, together * p.nx * p.ny * p.nz, c.a.kchunk));
        std::vector<SrcEntry> ent;
        int before = 0;
        bool plane1 = false;
        const bool fused = fuses(c, &ent, &before, &c.ss, &plane1);
        c.nsrc = (int)ent.size();
        if (fused) {
            c.ss.src = q.d_sent + before;
            if (c.R > 1) c.ss.inl = 0;
            // plane 2's thread applies a shear entry on plane 1, so it has to store that plane too
            if (plane1) c.a.kchunk = std::max(c.a.kchunk, 4);
        }
        c.ss.stf = b->d_stf + (size_t)c.prob * b->nt;
        c.ss.nstf = b->nt;
        c.ss.order = p.src_order;
        c.rf = q.rf;
        if (c.rf.grp) c.rf.traces += (size_t)c.r0 * (q.rec.size() / 4) * b->nt;
    };
    struct ManyPlaces {
        Chain *c;
        size_t many[2], map, groups, rows;
    };
    std::vector<ManyPlaces> many_at;
    for (auto &c : b->chains) {
        if (c.many.empty()) {
            prepare(c, c.branch >= 0 ? share : 1);
            continue;
        }
        std::vector<ManyProb> mp[2];
        std::vector<int2> map, rows;
        std::vector<int> groups;
        const int at = (int)(&c - b->chains.data());
        for (int q : c.many) {
            Chain &o = singles[q];
            prepare(o, c.work / o.work);
            const Prob &pr = b->probs[o.prob];
            if (o.nsrc > 0 && o.ss.nsrc == 0) groups.push_back(pr.group0);
            if (!pr.rec_fuse)
                for (int e = 0; e < (int)pr.rec.size() / 4; ++e) rows.push_back(make_int2(b->rec_base[o.prob] + e, o.prob));
            ManyProb m;
            m.a = o.a;
            m.ss = o.ss;
            m.rf = o.rf;
            const ewf_params &p = b->probs[o.prob].p;
            m.ntx = (p.nx + TX - 1) / TX;
            m.nty = (p.ny + b->ty - 1) / b->ty;
            const int ctas = m.ntx * m.nty * ((p.nz + o.a.kchunk - 1) / o.a.kchunk);
            for (int k = 0; k < ctas; ++k) map.push_back(make_int2((int)mp[0].size(), k));
            for (int par = 0; par < 2; ++par) {
                m.ss.it_ptr = b->d_it + 2 * at + par;
                m.rf.it_rd = b->d_it + 2 * at + par;
                m.rf.it_wr = nullptr;
                mp[par].push_back(m);
            }
        }
        c.blocks = (int)map.size();
        c.groups = (int)groups.size();
        c.rows = (int)rows.size();
        many_at.push_back({&c, {b->many_tables.add(mp[0]), b->many_tables.add(mp[1])}, b->many_tables.add(map), b->many_tables.add(groups), b->many_tables.add(rows)});
    }
    if (int st = b->many_tables.send()) return st;
    for (auto &m : many_at) {
        for (int par = 0; par < 2; ++par) m.c->d_many[par] = b->many_tables.at<ManyProb>(m.many[par]);
        m.c->d_map = b->many_tables.at<int2>(m.map);
        m.c->d_groups = b->many_tables.at<int>(m.groups);
        m.c->d_rows = b->many_tables.at<int2>(m.rows);
    }
    // every chain's counters at the batch's step
    const std::vector<int> its(2 * b->chains.size(), b->it);
    CK(cudaMemcpy(b->d_it, its.data(), its.size() * sizeof(int), cudaMemcpyHostToDevice));
    b->dirty = false;
    return EWF_OK;
}

// One step of chain i on a stream; `parity` = the step number's: its counter is at d_it[2 i + parity], the
// next step's at d_it[2 i + 1 - parity].
template <int MODEL, int DAMP, bool ST>
static void chain_step_t(ewf_batch *b, int i, int parity, bool first, cudaStream_t s)
{
    const Chain &c = b->chains[i];
    const Prob &q = b->probs[c.prob];
    const StepArgs<float> &a = c.a;
    int *const it_rd = b->d_it + 2 * i + parity, *const it_wr = b->d_it + 2 * i + 1 - parity;
    if (!c.many.empty()) {
        launch_on(k_stress_many<MODEL, DAMP>, dim3(c.blocks), dim3(TX, b->ty), s, b->pdl && !first, (const ManyProb *)c.d_many[parity],
                  (const int2 *)c.d_map);
        if (c.groups)
            k_binject<float><<<(c.groups + 31) / 32, 32, 0, s>>>(b->d_all, b->d_src, b->d_src_start, c.d_groups, 0, c.groups, b->d_stf, b->d_stf_off,
                                                                 b->d_order, b->nt, it_rd);
        launch_on(k_velocity_many<MODEL, DAMP>, dim3(c.blocks), dim3(TX, b->ty), s, b->pdl, (const ManyProb *)c.d_many[parity],
                  (const int2 *)c.d_map, (const int *)it_rd, it_wr);
        if (c.rows)
            k_brecord_many<float><<<std::min((c.rows + 255) / 256, 1024), 256, 0, s>>>(b->d_all, c.d_rows, c.rows, b->d_rec_off, b->d_rec_comp,
                                                                                       b->d_traces, b->nt, it_rd);
        return;
    }
    StressSrc ss = c.ss;
    ss.it_ptr = it_rd;
    RecFuse rf = c.rf;
    rf.it_rd = it_rd;
    if (q.rec_fuse) rf.it_wr = it_wr;
    const int rows = c.pair ? pair_rows(c.ty) : c.ty, tiles_x = (q.p.nx + TX - 1) / TX;
    const dim3 blk(c.pair ? PAIR_TX : TX, rows), grd(tiles_x * c.R, (q.p.ny + rows - 1) / rows, (q.p.nz + a.kchunk - 1) / a.kchunk);
    const long long stride = (long long)q.box, nr = (long long)q.rec.size() / 4;
    // (a problem with several right-hand sides in one launch has all of them: r0 = 0)
    if (c.R > 1) launch_on(k_stress_pair_mr<MODEL, DAMP, ST>, grd, blk, s, b->pdl && !first, a, c.R, stride, ss, (const int *)q.d_sstart);
    else if (c.pair) launch_on(k_stress_pair<MODEL, DAMP, ST>, grd, blk, s, b->pdl && !first, a, ss);
    else launch_on(k_stress<float, MODEL, DAMP>, grd, blk, s, b->pdl && !first, a, ss);
    if (c.nsrc > 0 && ss.nsrc == 0)
        k_binject<float><<<(c.R + 31) / 32, 32, 0, s>>>(b->d_all, b->d_src, b->d_src_start, nullptr, q.group0 + c.r0, c.R, b->d_stf, b->d_stf_off,
                                                        b->d_order, b->nt, it_rd);
    if (c.R > 1) launch_on(k_velocity_pair_mr<MODEL, DAMP, ST>, grd, blk, s, b->pdl, a, c.R, stride, rf, nr * b->nt);
    else if (c.pair) launch_on(k_velocity_pair<MODEL, DAMP, false, ST>, grd, blk, s, b->pdl, a, rf);
    else launch_on(k_velocity<float, MODEL, DAMP, false>, grd, blk, s, b->pdl, a, rf);
    if (!q.rec_fuse) {
        const int nrow = (int)nr * c.R;
        k_brecord<float><<<std::min((nrow + 255) / 256, 1024), 256, 0, s>>>(b->h_all[c.prob].a, b->d_rec_off, b->d_rec_comp,
                                                                            b->rec_base[c.prob] + c.r0 * (int)nr, nrow, b->d_traces, b->nt, it_rd);
        k_advance<<<1, 1, 0, s>>>(it_rd, it_wr);
    }
}

template <int MODEL, int DAMP>
static void chain_step(ewf_batch *b, int i, int parity, bool first, cudaStream_t s)
{
    if (b->chains[i].stream_l2) chain_step_t<MODEL, DAMP, true>(b, i, parity, first, s);
    else chain_step_t<MODEL, DAMP, false>(b, i, parity, first, s);
}

// `steps` steps of every chain from step parity `parity` on, one chain after the other: the branches' on
// streams forked from the batch's and joined, then the others on the batch's stream.
static void batch_steps(ewf_batch *b, int steps, int parity)
{
    auto chain = [&](size_t i, cudaStream_t s) {
        const ewf_params &p = b->probs[b->chains[i].prob].p;
        for (int k = 0; k < steps; ++k) {
            const int par = (parity + k) & 1;
            // nothing of another chain's to overlap with: a chain's first launch is a plain one
            if (p.model == EWF_MODEL_ISO) chain_step<MODEL_ISO, DAMP_PML1D>(b, (int)i, par, k == 0, s);
            else if (p.damping == EWF_DAMP_W3D) chain_step<MODEL_ORTHO, DAMP_W3D>(b, (int)i, par, k == 0, s);
            else chain_step<MODEL_ORTHO, DAMP_SEP>(b, (int)i, par, k == 0, s);
        }
    };
    bool used[ewf_batch::BRANCHES] = {};
    for (const Chain &c : b->chains)
        if (c.branch >= 0) used[c.branch] = true;
    bool forked = false;
    for (int k = 0; k < ewf_batch::BRANCHES; ++k) {
        if (!used[k]) continue;
        if (!forked) cudaEventRecord(b->fork_ev, b->stream);
        forked = true;
        cudaStreamWaitEvent(b->branch[k], b->fork_ev, 0);
    }
    for (size_t i = 0; i < b->chains.size(); ++i)
        if (b->chains[i].branch >= 0) chain(i, b->branch[b->chains[i].branch]);
    for (int k = 0; k < ewf_batch::BRANCHES; ++k) {
        if (!used[k]) continue;
        cudaEventRecord(b->join_ev[k], b->branch[k]);
        cudaStreamWaitEvent(b->stream, b->join_ev[k], 0);
    }
    for (size_t i = 0; i < b->chains.size(); ++i)
        if (b->chains[i].branch < 0) chain(i, b->stream);
}

static int batch_graph(ewf_batch *b, int steps, cudaGraphExec_t *exec)
{
    cudaGraph_t g = nullptr;
    CK(cudaStreamBeginCapture(b->stream, cudaStreamCaptureModeThreadLocal));
    batch_steps(b, steps, 0);
    const cudaError_t le = cudaGetLastError();
    const cudaError_t ce = cudaStreamEndCapture(b->stream, &g);
    if (le != cudaSuccess || ce != cudaSuccess) {
        if (g) cudaGraphDestroy(g);
        return ewf_fail(EWF_ERR_CUDA, "batch graph capture: %s", cudaGetErrorString(le != cudaSuccess ? le : ce));
    }
    const cudaError_t ie = cudaGraphInstantiate(exec, g, 0);
    cudaGraphDestroy(g);
    if (ie != cudaSuccess) {
        *exec = nullptr;
        return ewf_fail(EWF_ERR_CUDA, "batch graph instantiate: %s", cudaGetErrorString(ie));
    }
    return EWF_OK;
}

static int ready_graph(ewf_batch *b, int steps, cudaGraphExec_t *exec)
{
    if (*exec) return EWF_OK;
    int st = batch_graph(b, steps, exec);
    if (st && b->pdl) {  // a driver that cannot capture dependent launches: plain ones
        cudaGetLastError();
        b->pdl = false;
        st = batch_graph(b, steps, exec);
    }
    return st;
}

// Steps go in graphs of SHORT_GRAPH steps where the chains are small on average (SHORT_CELLS): launched one by one, a
// step of n chains takes the host some 5 n us.  Larger chains hide that.
static double chain_cells(const ewf_batch *b)
{
    double cells = 0;
    for (auto &c : b->chains) cells += c.work;
    return cells / std::max<size_t>(1, b->chains.size());
}
static int short_graph(const ewf_batch *b) { return chain_cells(b) < SHORT_CELLS ? std::min(SHORT_GRAPH, b->gsteps) : 0; }
// A graph of gsteps steps leaves fewer gaps, but takes the host as long to make as launching its steps would (2.6 us
// a launch), so one is made once the batch has run, or is about to run, steps that take four times as long,
// at least 256 and at most 768 of them (a step of a chain: 0.9 us, or 6e4 cells a us).  us per step in graphs of 8 (*: launches) and of 64, and ms of the first
// 64 steps that way: 64 rhs of iso 50^3 134.5 129.0, 11.2 29.8     100 iso 40^3 143.4 135.2, 14.2 45     100 ortho 32^3 99.8 90.7, 11.9 46
//   12 iso 72^3 80.1 76.3, 5.9 9.5     12 rhs of iso 50^3 26.2 25.0, 2.4 5.4     12 rhs of ortho 100^3* 288 278, 18.2 22
static long long long_from(const ewf_batch *b)
{
    const double step_us = std::max(0.9, chain_cells(b) / 6e4);
    return (long long)std::min(768.0, std::max(256.0, 4 * 2.6 * 2 * b->gsteps / step_us));
}

static int batch_ready(ewf_batch *b)
{
    for (size_t i = 0; i < b->probs.size(); ++i) {
        const Prob &q = b->probs[i];
        const int nm = q.p.model == EWF_MODEL_ISO ? 2 : 12;
        for (int f = 0; f < nm; ++f)
            if (!q.m_set[f]) return ewf_fail(EWF_ERR_STATE, "problem %zu: material slot %d not set", i, f);
        if (q.p.damping == EWF_DAMP_W3D ? !q.w_set[3] : !(q.w_set[0] && q.w_set[1] && q.w_set[2]))
            return ewf_fail(EWF_ERR_STATE, "problem %zu: damping not set", i);
    }
    if (b->dirty) return build_tables(b);
    return EWF_OK;
}

extern "C" int ewf_batch_reset(ewf_batch *b)
{
    if (!b) return ewf_fail(EWF_ERR_ARG, "NULL batch");
    std::vector<ZeroBuf> z;
    for (auto &q : b->probs)
        for (auto &x : q.state) z.push_back({x, q.sbox * 4});
    if (b->d_traces) z.push_back({b->d_traces, (size_t)b->nrec_total * b->nt * sizeof(double)});
    z.push_back({b->d_it, 2 * (size_t)b->nrhs_total * sizeof(int)});
    if (int st = zero_buffers(z, b->stream)) return st;
    CK(cudaStreamSynchronize(b->stream));
    b->it = 0;
    return EWF_OK;
}

extern "C" int ewf_batch_run(ewf_batch *b, int32_t nsteps)
{
    if (!b || nsteps < 0) return ewf_fail(EWF_ERR_ARG, "bad argument");
    int st = batch_ready(b);
    if (st) return st;
    if (b->it + nsteps > b->nt) return ewf_fail(EWF_ERR_ARG, "step %d + %d exceeds nt = %d", b->it, nsteps, b->nt);
    // graphs start from an even step
    const int odd = b->it & 1, rest = std::max(0, nsteps - odd), brief = short_graph(b);
    const int nlong = b->gexec || b->ran + nsteps >= long_from(b) ? rest / b->gsteps : 0, nshort = brief > 0 ? (rest - nlong * b->gsteps) / brief : 0;
    if (nlong && (st = ready_graph(b, b->gsteps, &b->gexec))) return st;
    if (nshort && (st = ready_graph(b, brief, &b->gexec_short))) return st;
    CK(cudaEventRecord(b->ev0, b->stream));
    int done = 0;
    if ((nlong || nshort) && odd) {
        batch_steps(b, 1, 1);
        done = 1;
    }
    for (int q = 0; q < nlong; ++q, done += b->gsteps) CK(cudaGraphLaunch(b->gexec, b->stream));
    for (int q = 0; q < nshort; ++q, done += brief) CK(cudaGraphLaunch(b->gexec_short, b->stream));
    for (int n = 0; done < nsteps; done += n) {
        n = std::min(nsteps - done, b->gsteps);
        batch_steps(b, n, (b->it + done) & 1);
    }
    CK(cudaGetLastError());
    CK(cudaEventRecord(b->ev1, b->stream));
    CK(cudaStreamSynchronize(b->stream));
    CK(cudaEventElapsedTime(&b->last_ms, b->ev0, b->ev1));
    b->it += nsteps;
    b->ran += nsteps;
    return EWF_OK;
}

extern "C" int ewf_batch_last_run_ms(const ewf_batch *b, double *ms)
{
    if (!b || !ms) return ewf_fail(EWF_ERR_ARG, "NULL argument");
    *ms = b->last_ms;
    return EWF_OK;
}

extern "C" int ewf_batch_get_seismograms(ewf_batch *b, int32_t prob, int32_t rhs, double *out, size_t n)
{
    int st = check_prob(b, prob);
    if (st) return st;
    const Prob &q = b->probs[prob];
    if (rhs < 0 || rhs >= q.R) return ewf_fail(EWF_ERR_ARG, "rhs out of range");
    const int nr = (int)q.rec.size() / 4;
    if (n != (size_t)nr * b->nt || (!out && n)) return ewf_fail(EWF_ERR_ARG, "%zu samples, %d expected", n, nr * b->nt);
    if (b->dirty) return ewf_fail(EWF_ERR_STATE, "receivers changed since the last run");
    if (n)
        CK(cudaMemcpy(out, b->d_traces + ((size_t)b->rec_base[prob] + (size_t)rhs * nr) * b->nt, n * sizeof(double),
                      cudaMemcpyDeviceToHost));
    return EWF_OK;
}

extern "C" int ewf_batch_get_field(ewf_batch *b, int32_t prob, int32_t rhs, int32_t field, void *host, size_t n,
                                   int32_t dtype_bytes)
{
    int st = check_prob(b, prob);
    if (st) return st;
    const Prob &q = b->probs[prob];
    if (rhs < 0 || rhs >= q.R || field < 0 || field > 8 || !host || (dtype_bytes != 4 && dtype_bytes != 8))
        return ewf_fail(EWF_ERR_ARG, "bad argument");
    int ex, ey, ez;
    ewf_field_extent(q.p, field, &ex, &ey, &ez);
    if (n != (size_t)ex * ey * ez) return ewf_fail(EWF_ERR_ARG, "field size");
    const float *src = sptr(q, q.state[field]) + (size_t)rhs * q.box;
    const unsigned nb = (unsigned)std::min<size_t>((n + 255) / 256, 152 * 16);
    if (dtype_bytes == 4) k_unpack<float, float><<<nb, 256, 0, b->stream>>>((float *)b->d_stage, src, ex, ey, ez, q.sx, q.sy);
    else k_unpack<double, float><<<nb, 256, 0, b->stream>>>((double *)b->d_stage, src, ex, ey, ez, q.sx, q.sy);
    CK(cudaGetLastError());
    CK(cudaMemcpyAsync(host, b->d_stage, n * dtype_bytes, cudaMemcpyDeviceToHost, b->stream));
    CK(cudaStreamSynchronize(b->stream));
    return EWF_OK;
}

// Times `nsteps` steps for each launch form and tile height, then for each prefetch distance, with CUDA events, keeps the
// fastest, and leaves the batch reset (the tuning steps advance the state).
extern "C" int ewf_batch_autotune(ewf_batch *b, int32_t nsteps, int32_t *kchunk_out)
{
    if (!b || nsteps < 1) return ewf_fail(EWF_ERR_ARG, "bad argument");
    static const int ty_cand[] = {4, 8};
    const int steps = std::min(nsteps, b->nt - 1);
    int best_ty = 4, best_pf = 0, best_own = 0;
    auto apply = [&](int ty, int own, int pf) {
        for (auto &q : b->probs) q.kchunk = KCHUNK_BY_SIZE;
        b->ty = ty;
        b->own = own;
        b->l2pf = pf;
        b->dirty = true;
    };
    // ms per step.  Batches of small chains are timed in the graphs that they run in: the host does not keep up with their
    // launches one by one, and every setting would take what it takes.
    auto time = [&](float *ms) {
        int st = batch_ready(b);
        if (!st) st = ewf_batch_reset(b);
        if (st) return st;
        const int brief = std::min(short_graph(b), std::max(2, steps & ~1)), n = std::max(4, steps / std::max(1, brief));  // (past the last step nothing is sampled or injected)
        cudaGraphExec_t exec = nullptr;
        if (brief > 0) {
            if ((st = ready_graph(b, brief, &exec))) return st;
            cudaError_t e = cudaGraphLaunch(exec, b->stream);  // warm
            if (e == cudaSuccess) e = cudaEventRecord(b->ev0, b->stream);
            for (int q = 0; q < n && e == cudaSuccess; ++q) e = cudaGraphLaunch(exec, b->stream);
            if (e == cudaSuccess) e = cudaEventRecord(b->ev1, b->stream);
            if (e == cudaSuccess) e = cudaStreamSynchronize(b->stream);
            cudaGraphExecDestroy(exec);
            CK(e);
        } else {
            batch_steps(b, 1, 0);  // warm
            CK(cudaEventRecord(b->ev0, b->stream));
            if (steps > 0) batch_steps(b, steps, 1);
            CK(cudaEventRecord(b->ev1, b->stream));
            CK(cudaStreamSynchronize(b->stream));
        }
        CK(cudaEventElapsedTime(ms, b->ev0, b->ev1));
        *ms /= brief > 0 ? n * brief : std::max(1, steps);
        return (int)EWF_OK;
    };
    // the setting by default is timed twice; with small chains another one has to be faster by more than those two differ
    apply(best_ty, best_own, best_pf);
    float t[2] = {}, ms = 0.f;
    for (float &x : t)
        if (int st = time(&x)) return st;
    const float margin = short_graph(b) ? std::max(0.01f * std::min(t[0], t[1]), std::fabs(t[0] - t[1])) : 0.f;
    float best = std::min(t[0], t[1]) - margin;
    bool other = false;
    for (int own = 0; own < 2; ++own)
        for (int ty : ty_cand) {
            if (own == 0 && ty == 4) continue;
            apply(ty, own, 0);
            if (int st = time(&ms)) return st;
            if (ms < best) {
                best = ms;
                best_ty = ty;
                best_own = own;
                other = true;
            }
        }
    if (other) best -= margin;
    for (int pf : {2, 3, 4}) {  // then the velocity kernels' L2 prefetch distance at that setting
        apply(best_ty, best_own, pf);
        if (int st = time(&ms)) return st;
        if (ms < best) {
            best = ms;
            best_pf = pf;
        }
    }
    apply(best_ty, best_own, best_pf);
    if (int st = batch_ready(b)) return st;
    if (kchunk_out) *kchunk_out = KCHUNK_BY_SIZE;
    return ewf_batch_reset(b);
}

extern "C" int ewf_batch_set_tile(ewf_batch *b, int32_t tile_y)
{
    if (!b) return ewf_fail(EWF_ERR_ARG, "NULL batch");
    if (tile_y != 4 && tile_y != 8 && tile_y != 16) return ewf_fail(EWF_ERR_ARG, "tile_y must be 4, 8 or 16 (got %d)", tile_y);
    b->ty = tile_y;
    b->dirty = true;
    return EWF_OK;
}

extern "C" int ewf_batch_set_launch(ewf_batch *b, int32_t own)
{
    if (!b) return ewf_fail(EWF_ERR_ARG, "NULL batch");
    if (own != 0 && own != 1) return ewf_fail(EWF_ERR_ARG, "own must be 0 or 1 (got %d)", own);
    b->own = own;
    b->dirty = true;
    return EWF_OK;
}

extern "C" int ewf_batch_get_launch(const ewf_batch *b, int32_t *own)
{
    if (!b || !own) return ewf_fail(EWF_ERR_ARG, "NULL argument");
    *own = b->own;
    return EWF_OK;
}

extern "C" int ewf_batch_set_l2_prefetch(ewf_batch *b, int32_t planes)
{
    if (!b) return ewf_fail(EWF_ERR_ARG, "NULL batch");
    if (planes < 0 || planes > 8) return ewf_fail(EWF_ERR_ARG, "planes must be in [0, 8] (got %d)", planes);
    b->l2pf = planes;
    b->dirty = true;
    return EWF_OK;
}

extern "C" int ewf_batch_get_l2_prefetch(const ewf_batch *b, int32_t *planes)
{
    if (!b || !planes) return ewf_fail(EWF_ERR_ARG, "NULL argument");
    *planes = b->l2pf;
    return EWF_OK;
}

extern "C" int ewf_batch_get_tile(const ewf_batch *b, int32_t *tile_y)
{
    if (!b || !tile_y) return ewf_fail(EWF_ERR_ARG, "NULL argument");
    *tile_y = b->ty;
    return EWF_OK;
}
