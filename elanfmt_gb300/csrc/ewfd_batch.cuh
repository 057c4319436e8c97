// ewfd_batch.cuh -- batched time step: many problems (models of uneven size) x many right-hand
// sides (sources) advanced together.
//
// A problem is one model (grid, materials, damping) with R right-hand sides (source sets); its R
// state sets are separate boxes (rhs_stride elements apart) sharing the material arrays.  Problems do
// not depend on one another, nor do right-hand sides, so each chain -- a right-hand side, or all of a
// large model -- runs the solver's launches by itself (k_stress / k_velocity or their two-cell forms, with
// sources, receivers and step counter inside); k_stress_pair_mr / k_velocity_pair_mr advance several
// right-hand sides, their CTAs of a tile reading its material planes from HBM once.
// Here: the problem descriptor, and the separate injection and recording kernels for the entries
// those launches do not take (sources outside the stress cells, receivers of other fields or cells).
#pragma once
#include "ewfd_pair.cuh"

namespace ewf {

template <typename T>
struct BatchProb {
    StepArgs<T> a;                        // the problem, state of RHS 0
    long long rhs_stride;                 // elements between the state boxes of consecutive RHS
};

// Point injection: one thread per (problem, RHS), entries in order, as k_inject.  `list`: which of them (else `groups` from
// group0 on).
struct BatchSrc {
    int prob, rhs, comp, i, j, k;
    double coef;
};

template <typename T>
__global__ void k_binject(const BatchProb<T> *__restrict__ probs, const BatchSrc *__restrict__ src,
                          const int *__restrict__ src_start, const int *__restrict__ list, int group0, int groups, const double *__restrict__ stf,
                          const int *__restrict__ stf_off, const int *__restrict__ order, int nstf,
                          const int *__restrict__ it_ptr)
{
    const int n = blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= groups) return;
    const int g = list ? list[n] : group0 + n;
    const int it = *it_ptr;
    if (it < 0 || it >= nstf) return;
    for (int e = src_start[g]; e < src_start[g + 1]; ++e) {
        const BatchSrc q = src[e];
        const StepArgs<T> &P = probs[q.prob].a;
        const T s = (T)stf[stf_off[q.prob] + it];
        inject_entry(P, SrcEntry{q.comp, q.i, q.j, q.k, q.coef}, s, order[q.prob], (long long)q.rhs * probs[q.prob].rhs_stride);
    }
}

// Tiny problems of one scheme in one launch (separate ones would be bound by the launch rate): a CTA looks up its problem and its place in it (map: problem,
// CTA of the problem) and runs the one-cell update with that problem's arguments, sources and receivers.
struct ManyProb {
    StepArgs<float> a;
    StressSrc ss;
    RecFuse rf;
    int ntx, nty;
};
template <int MODEL, int DAMP>
__global__ void __launch_bounds__(split_max_threads<float>(), split_min_ctas<float>()) k_stress_many(const ManyProb *__restrict__ probs,
                                                                                                    const int2 *__restrict__ map)
{
    pdl_trigger();
    const int2 m = map[blockIdx.x];
    const ManyProb &p = probs[m.x];
    const int t = m.y / p.ntx, k0 = (t / p.nty) * p.a.kchunk;
    stress_column<float, MODEL, DAMP, 1, true>(p.a, (m.y % p.ntx) * TX + threadIdx.x, (t % p.nty) * blockDim.y + threadIdx.y, k0,
                                               min(k0 + p.a.kchunk, p.a.nz), p.ss);
}
template <int MODEL, int DAMP>
__global__ void __launch_bounds__(split_max_threads<float>(), split_min_ctas<float>())
    k_velocity_many(const ManyProb *__restrict__ probs, const int2 *__restrict__ map, const int *it_rd, int *it_wr)
{
    pdl_trigger();
    if (blockIdx.x == 0 && threadIdx.x == 0 && threadIdx.y == 0) {
        pdl_wait();
        *it_wr = *it_rd + 1;
    }
    const int2 m = map[blockIdx.x];
    const ManyProb &p = probs[m.x];
    const int t = m.y / p.ntx, k0 = (t / p.nty) * p.a.kchunk;
    velocity_column<float, MODEL, DAMP, false, 1, true>(p.a, (m.y % p.ntx) * TX + threadIdx.x, (t % p.nty) * blockDim.y + threadIdx.y, k0,
                                                        min(k0 + p.a.kchunk, p.a.nz), p.rf);
}

// Receiver gather of one chain's right-hand sides: rows [row0, row0 + nrow) of the traces.
template <typename T>
__global__ void k_brecord(const StepArgs<T> a, const long long *__restrict__ rec_off, const int *__restrict__ rec_comp, int row0,
                          int nrow, double *__restrict__ traces, int nt, const int *it_rd)
{
    const int it = *it_rd;
    if (it >= 0 && it < nt)
        for (int r = row0 + blockIdx.x * blockDim.x + threadIdx.x; r < row0 + nrow; r += gridDim.x * blockDim.x)
            traces[(long long)r * nt + it] = (double)a.f[rec_comp[r]][rec_off[r]];
}

// The same for rows of several problems: (row, problem) each.
template <typename T>
__global__ void k_brecord_many(const BatchProb<T> *__restrict__ probs, const int2 *__restrict__ rows, int nrow,
                               const long long *__restrict__ rec_off, const int *__restrict__ rec_comp, double *__restrict__ traces, int nt,
                               const int *it_rd)
{
    const int it = *it_rd;
    if (it >= 0 && it < nt)
        for (int n = blockIdx.x * blockDim.x + threadIdx.x; n < nrow; n += gridDim.x * blockDim.x) {
            const int r = rows[n].x;
            traces[(long long)r * nt + it] = (double)probs[rows[n].y].a.f[rec_comp[r]][rec_off[r]];
        }
}

__global__ void k_advance(const int *it_rd, int *it_wr) { *it_wr = *it_rd + 1; }

}  // namespace ewf
