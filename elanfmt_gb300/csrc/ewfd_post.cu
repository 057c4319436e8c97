// ewfd_post.cu -- seismogram post-processing: a cascade of second-order IIR sections (the
// Butterworth band-pass the isotropic MATLAB driver applies before comparing traces,
// vizme_FastBiotED_GPU3D_OK_2024_final.m:551-558, 579-582, 604-607, "sosfilt(sos, x)").
//
// Each section is the direct form II transposed recursion
//     y = b0 x + s1;   s1 = b1 x - a1 y + s2;   s2 = b2 x - a2 y
// with zero initial state, the sections applied one after the other (section 0 first).  The
// host and device versions perform the same operations in the same order (the library is built
// without FMA contraction), so they give the same bits.
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <cmath>

#include "ewfd.h"
#include "ewfd_internal.h"

namespace {

constexpr int MAXSEC = EWF_SOS_MAX_SECTIONS;

struct Sos {
    double c[MAXSEC][5];  // b0 b1 b2 a1 a2, normalised by a0
    int n;
};

int make_sos(const double *sos, int32_t nsec, Sos *out)
{
    if (!sos || nsec < 1 || nsec > MAXSEC) return ewf_fail(EWF_ERR_ARG, "sosfilt: 1..%d sections (got %d)", MAXSEC, nsec);
    out->n = nsec;
    for (int s = 0; s < nsec; ++s) {
        const double *r = sos + 6 * s;
        const double a0 = r[3];
        if (!(a0 != 0.0)) return ewf_fail(EWF_ERR_ARG, "sosfilt: section %d has a0 = 0", s);
        out->c[s][0] = r[0] / a0;
        out->c[s][1] = r[1] / a0;
        out->c[s][2] = r[2] / a0;
        out->c[s][3] = r[4] / a0;
        out->c[s][4] = r[5] / a0;
    }
    return EWF_OK;
}

// one trace in place: the host path, and a device thread of k_sosfilt_trace
__host__ __device__ inline void filter_trace(const Sos &q, double *x, int64_t n)
{
    double s1[MAXSEC], s2[MAXSEC];
    for (int s = 0; s < q.n; ++s) s1[s] = s2[s] = 0.0;
    for (int64_t t = 0; t < n; ++t) {
        double v = x[t];
        for (int s = 0; s < q.n; ++s) {
            const double *c = q.c[s];
            const double y = c[0] * v + s1[s];
            s1[s] = c[1] * v - c[3] * y + s2[s];
            s2[s] = c[2] * v - c[4] * y;
            v = y;
        }
        x[t] = v;
    }
}

// ---------------------------------------------------------------------------------------------
// The same recursion on device-resident traces.  It is serial in time: a pass is bound by FP64
// instructions following one another, not by the 16 bytes a sample moves.  Measured on GB300, a warp
// takes 64 cycles per FP64 instruction, dependent or not and however many lanes are active, and an SM
// 19 cycles per instruction over four or more warps.  So what counts is how many FP64 instructions one
// warp issues per sample: 36 for four sections in one thread, 9 with a section per lane.  Here a pair
// of warps shares those 9 on two of the SM's four units: lane l of both stands for section l % G of
// trace l / G, the second warp forms the feed-forward products b0 v, b1 v, b2 v of U samples at a time,
// the first runs the feedback (y, a1 y, a2 y and three sums: 6 instructions), and they hand over
// through shared memory with one barrier per U samples.  A section's output is the next section's
// input two phases later.  Each section performs the host path's operations in its order, so the
// bits are the same.  (Spreading the feedback's chain of four over lanes with shuffles was
// no faster: a lane's FP64 result reaches a shuffle or a select only 25 to 50 cycles after the next
// FP64 instruction could have had it.)
// 192 traces x 4000 samples x 4 sections: 5.98 ms with a thread per trace, 1.33 with a section per lane
// in one warp, 0.86 as here (450 cycles per sample).
// ---------------------------------------------------------------------------------------------
constexpr int U = 16;  // samples per phase

template <int G>
__global__ void __launch_bounds__(64) k_sosfilt(const Sos q, double *__restrict__ x, int64_t ntr, int64_t n)
{
    constexpr int ROWS = 32 / G, PER = ROWS * U / 32;  // traces per pair of warps; samples a lane moves per phase
    __shared__ double prod[2][3][U][32];  // products of a phase
    __shared__ double outs[2][U][32];     // the sections' outputs of a phase
    __shared__ double ins[2][U][ROWS];    // samples of a phase, by trace
    const int lane = threadIdx.x & 31, s = lane % G, row = lane / G;
    const int64_t tr0 = (int64_t)blockIdx.x * ROWS;
    const int64_t groups = (n + U - 1) / U, phases = groups + 2 * q.n;
    const double *c = q.c[s < q.n ? s : 0];

    if (threadIdx.x >= 32) {
        const double c0 = c[0], c1 = c[1], c2 = c[2];
        double next[PER];
        // e = lane + 32 k is sample e % U of trace e / U: coalesced along the samples
        auto fetch = [&](int64_t g) {
#pragma unroll
            for (int k = 0; k < PER; ++k) {
                const int e = lane + 32 * k;
                const int64_t tr = tr0 + e / U, t = g * U + e % U;
                next[k] = (tr < ntr && t < n) ? x[tr * n + t] : 0.0;
            }
        };
        auto stage = [&](int buf) {
#pragma unroll
            for (int k = 0; k < PER; ++k) {
                const int e = lane + 32 * k;
                ins[buf][e % U][e / U] = next[k];
            }
        };
        fetch(0);
        stage(0);
        __syncwarp();
        for (int64_t ph = 0; ph < phases; ++ph) {
            const int now = (int)(ph & 1);
            fetch(ph + 1);
            const int64_t g = ph - 2 * s;
            if (s < q.n && g >= 0 && g < groups) {
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const double v = s == 0 ? ins[now][u][row] : outs[1 - now][u][lane - 1];
                    prod[now][0][u][lane] = c0 * v;
                    prod[now][1][u][lane] = c1 * v;
                    prod[now][2][u][lane] = c2 * v;
                }
            }
            const int64_t go = ph - 2 * q.n;  // the last section finished this group in the phase before
            if (go >= 0) {
#pragma unroll
                for (int k = 0; k < PER; ++k) {
                    const int e = lane + 32 * k;
                    const int64_t tr = tr0 + e / U, t = go * U + e % U;
                    if (tr < ntr && t < n) x[tr * n + t] = outs[1 - now][e % U][(e / U) * G + q.n - 1];
                }
            }
            stage(1 - now);
            __syncthreads();
        }
    } else {
        const double c3 = c[3], c4 = c[4];
        double s1 = 0.0, s2 = 0.0;
        for (int64_t ph = 0; ph < phases; ++ph) {
            const int now = (int)(ph & 1);
            const int64_t g = ph - 1 - 2 * s;
            if (s < q.n && g >= 0 && g < groups) {
                // (the samples after a trace's end, in its last group, change nothing that is stored)
                double p[3][U];
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    p[0][u] = prod[1 - now][0][u][lane];
                    p[1][u] = prod[1 - now][1][u][lane];
                    p[2][u] = prod[1 - now][2][u][lane];
                }
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const double y = p[0][u] + s1;
                    s1 = p[1][u] - c3 * y + s2;
                    s2 = p[2][u] - c4 * y;
                    outs[now][u][lane] = y;
                }
            }
            __syncthreads();
        }
    }
}

// A thread per trace: its latency is that of all the sections' instructions in a row, but every lane of a warp issues for
// a trace of its own, whatever the number of sections.
__global__ void __launch_bounds__(64) k_sosfilt_trace(const Sos q, double *x, int64_t ntr, int64_t n)
{
    const int64_t tr = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (tr < ntr) filter_trace(q, x + tr * n, n);
}

// Which of the two is faster, by their measured times: a pair of warps takes 0.21 us per sample alone and 0.095 (one
// section 0.14) times the pairs per SM when there are many, over the samples and two phases per section; a thread
// 0.2 us and 0.315 per section, and 0.15 and 1.8e-5 times the traces per section when there are many.  ms by pairs and by threads:
//   192 x 4000, 4 sections 0.86 and 5.9     4864 x 2000, 5 sections 2.1 and 3.7     9728 x 1000, 9 sections 3.8 and 3.0
//   20000 x 1000: 4 sections 1.7 and 2.1, 5 sections 3.4 and 2.6     40000 x 500, 8 sections 4.1 and 3.4     1e6 x 16, 4 sections 4.5 and 1.1
bool trace_per_thread(int nsec, int lanes, double ntr, double n)
{
    const double pairs = ntr * lanes / 32, len = U * (std::ceil(n / U) + 2 * nsec);
    const double by_pairs = len * std::max(0.212, (lanes == 1 ? 0.14 : 0.095) * pairs / 152);
    const double by_threads = n * std::max(0.2 + 0.315 * nsec, nsec * (0.15 + 1.78e-5 * ntr));
    return by_threads < by_pairs;
}

template <int G>
void launch_sosfilt(const Sos &q, double *x, int64_t ntr, int64_t n, cudaStream_t stream)
{
    if (trace_per_thread(q.n, G, (double)ntr, (double)n)) {
        k_sosfilt_trace<<<(unsigned)((ntr + 63) / 64), 64, 0, stream>>>(q, x, ntr, n);
        return;
    }
    k_sosfilt<G><<<(unsigned)((ntr * G + 31) / 32), 64, 0, stream>>>(q, x, ntr, n);
}

}  // namespace

extern "C" int ewf_sosfilt(const double *sos, int32_t nsec, double *x, int64_t ntr, int64_t n)
{
    Sos q;
    int st = make_sos(sos, nsec, &q);
    if (st) return st;
    if ((!x && ntr * n > 0) || ntr < 0 || n < 0) return ewf_fail(EWF_ERR_ARG, "sosfilt: bad trace array");
    for (int64_t tr = 0; tr < ntr; ++tr) filter_trace(q, x + tr * n, n);
    return EWF_OK;
}

extern "C" int ewf_sosfilt_device(const double *sos, int32_t nsec, double *x, int64_t ntr, int64_t n, void *stream)
{
    Sos q;
    int st = make_sos(sos, nsec, &q);
    if (st) return st;
    if ((!x && ntr * n > 0) || ntr < 0 || n < 0) return ewf_fail(EWF_ERR_ARG, "sosfilt: bad trace array");
    if (ntr == 0 || n == 0) return EWF_OK;
    // the smallest power of two that holds the sections
    const cudaStream_t st_ = (cudaStream_t)stream;
    if (q.n == 1) launch_sosfilt<1>(q, x, ntr, n, st_);
    else if (q.n == 2) launch_sosfilt<2>(q, x, ntr, n, st_);
    else if (q.n <= 4) launch_sosfilt<4>(q, x, ntr, n, st_);
    else if (q.n <= 8) launch_sosfilt<8>(q, x, ntr, n, st_);
    else launch_sosfilt<16>(q, x, ntr, n, st_);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return ewf_fail(EWF_ERR_CUDA, "sosfilt launch: %s", cudaGetErrorString(e));
    return EWF_OK;
}
