// ewfd_step.h -- host side of the two-kernel step shared by the solver and the batch (ewfd.cu).
#pragma once
#include <limits.h>
#include <stdint.h>
#include <string.h>

#include <vector>

#include "ewfd.h"
#include "ewfd_kernels.cuh"

// Sources for the stress kernel (false: the injection kernel applies them)
bool make_stress_src(const std::vector<ewf::SrcEntry> &v, int nx, int ny, int nz, ewf::StressSrc *f, bool *plane1);

// Receivers for the velocity kernel (fuse false: the recording kernel samples them)
struct RecTables {
    bool fuse = true;
    int kmin = INT32_MAX, kmax = -1;
    std::vector<uint2> grp;
    std::vector<int> off;
    std::vector<int2> ent;
};
RecTables make_rec_tables(int n, const int32_t *ijkc, int nx, int ny, int nz);

// Graphs of a few steps for small grids: the steps a long graph leaves over (even), and up to how many
// cells (on average, in a batch) the host's launches are what a step takes
constexpr int SHORT_GRAPH = 8;
constexpr double SHORT_CELLS = 4e5;

// Launch shape by the cells a launch updates (R right-hand sides)
struct SplitShape {
    int kchunk, ty, l2pf;
    bool pair;
    bool stream;
};
SplitShape split_shape(int nx, int ny, int nz, int R = 1);

// Two cells per thread halve the threads: chunks longer than the rule's (a caller's own) can leave too few of them.  us per step of one
// and of two cells by planes per chunk, where they part:
//   iso 128^3  8 37.6 37.9  16 42.5 45.7  64 127 138     200x190x150  32 142 124  64 155 181     97x83x71  8 19.2 19.8  64 77 94
//   iso-het 128^3  16 58.9 53.3  32 87.7 90.5     200x190x150  32 169 154  64 196 205     97x83x71  16 33.1 33.4  64 88 107
//   ortho 128^3  16 63.1 51.7  32 96.6 88.9     97x83x71  8 24.7 24.3  16 39.6 39.1  32 59 71     80x80x70  8 20.8 23.9  16 25.7 41.6
inline bool enough_pairs(int model, double cells, int kchunk)
{
    return cells / (2.0 * kchunk) >= (model == EWF_MODEL_ISO ? 7.5e4 : model == EWF_MODEL_ISO_HET ? 5e4 : 3e4);
}

// Buffers (16-byte aligned) set to zero in stream order, ZERO_GROUP of them per launch
struct ZeroBuf {
    void *p;
    size_t bytes;
};
int zero_buffers(const std::vector<ZeroBuf> &v, cudaStream_t stream);

// A launch on a stream; `pdl`: as a programmatic dependent of the stream's previous
// kernel (the kernel waits for it with griddepcontrol.wait before touching any state).
template <typename... P, typename... A>
inline void launch_on(void (*kern)(P...), dim3 grid, dim3 block, cudaStream_t stream, bool pdl, A... args)
{
    cudaLaunchConfig_t cfg;
    memset(&cfg, 0, sizeof(cfg));
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.stream = stream;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = pdl ? 1 : 0;
    cudaLaunchKernelEx(&cfg, kern, args...);
}
