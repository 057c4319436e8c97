// ewfd_pair.cuh -- the two-kernel step's FP32 kernels with two cells per thread.
//
// k_stress and k_velocity (ewfd_kernels.cuh) spend most of their instructions on addresses, loads and
// stores of single values: 215 and 197 per 32 cells of the isotropic scheme against 82 floating-point
// operations per cell.  On grids whose fields stay in L2, where the memory does not set the pace, that
// is what a step takes.  Here a thread owns the cells (i, i+1), i even: aligned values move as 8-byte
// pairs, the two shifted neighbours per field a pair needs beside its own come as one value each,
// and the arithmetic runs on packed pairs (mul / fma .rn.f32x2: two IEEE operations per instruction,
// subnormals kept), operation by operation in the order of stress_math and vel_math, so
// the results are the same bits.  A warp covers 16 pairs of two rows, a CTA 32 columns x 2 ty rows.
#pragma once
#include "ewfd_kernels.cuh"

namespace ewf {

typedef unsigned long long f2;  // two floats: the pair's first cell in the low half

__device__ __forceinline__ f2 pk(float lo, float hi)
{
    f2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ f2 dup(float v) { return pk(v, v); }
__device__ __forceinline__ float lo(f2 a) { return __uint_as_float((unsigned)a); }
__device__ __forceinline__ float hi(f2 a) { return __uint_as_float((unsigned)(a >> 32)); }
__device__ __forceinline__ f2 mul2(f2 a, f2 b)
{
    f2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c)
{
    f2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
// Sums and differences are a * 1 + b and b * -1 + a, one rounding each (the product is exact, the signs of
// zeros those of a + b and a - b), with the 1 and -1 a value the assembler does not know: it contracts
// a packed product whose only use is a packed sum into fma.f32x2, .rn and --fmad=false notwithstanding.
struct PairOps {
    f2 one, minus;
    __device__ __forceinline__ f2 add(f2 a, f2 b) const { return fma2(a, one, b); }
    __device__ __forceinline__ f2 sub(f2 a, f2 b) const { return fma2(b, minus, a); }
};
__device__ __forceinline__ f2 neg2(f2 a) { return a ^ 0x8000000080000000ull; }

// NC: the read-only path, for what no launch writes; the state is read plainly (lds)
template <bool NC = true>
__device__ __forceinline__ f2 ld2(const float *p)
{
    return NC ? __ldg(reinterpret_cast<const f2 *>(p)) : *reinterpret_cast<const f2 *>(p);
}
// ST: a line that the step does not need again soon, the first to leave L2 (split_shape).
template <bool ST>
__device__ __forceinline__ f2 ldm(const float *p)
{
    return ST ? __ldcs(reinterpret_cast<const f2 *>(p)) : ld2(p);
}
template <bool ST = false>
__device__ __forceinline__ void st2(float *p, f2 v, bool m0, bool m1)
{
    if (m0 && m1) {
        if (ST) __stcs(reinterpret_cast<f2 *>(p), v);
        else *reinterpret_cast<f2 *>(p) = v;
    } else {
        if (m0) p[0] = lo(v);
        if (m1) p[1] = hi(v);
    }
}

// The six shear quotients of both cells (div_shear): x[0..5] by dy dx dz dx dz dy.
__device__ __forceinline__ void div_shear2(const StepArgs<float> &a, const f2 (&x)[6], f2 (&q)[6])
{
    // the smallest key (2 |x| bits - 1: zero last) and the largest magnitude of the twelve
    unsigned key = 0xffffffffu;
    float top = 0.f;
#pragma unroll
    for (int e = 0; e < 6; ++e) {
        const float u = lo(x[e]), v = hi(x[e]);
        key = min(key, min(2u * __float_as_uint(u) - 1u, 2u * __float_as_uint(v) - 1u));
        top = fmaxf(top, fmaxf(fabsf(u), fabsf(v)));
    }
    const float d[6] = {a.dy, a.dx, a.dz, a.dx, a.dz, a.dy}, r[6] = {a.rdy, a.rdx, a.rdz, a.rdx, a.rdz, a.rdy};
    const bool ok = a.fdiv != 0 && top <= 0x1p100f;  // a NaN is none of the others' business: its quotient is NaN either way
    if (ok && key >= 2u * 0x12800000u - 1u) {
#pragma unroll
        for (int e = 0; e < 6; ++e) {
            const f2 p = mul2(x[e], dup(r[e]));
            const f2 n = fma2(p, dup(d[e]), neg2(x[e]));
            q[e] = fma2(neg2(n), dup(r[e]), p);
        }
    } else if (ok) {
#pragma unroll
        for (int e = 0; e < 6; ++e) q[e] = pk(div_small(lo(x[e]), d[e], r[e]), div_small(hi(x[e]), d[e], r[e]));
    } else {
#pragma unroll
        for (int e = 0; e < 6; ++e) q[e] = pk(__fdiv_rn(lo(x[e]), d[e]), __fdiv_rn(hi(x[e]), d[e]));
    }
}

template <int MODEL, int DAMP>
struct StressIn2 {
    f2 vx, vx_jm, vy, vy_jp, vz_p, vz_jm;
    float vx_i2, vy_im, vz_im;  // Vx(i+2), Vy(i-1), Vz(i-1) at plane k
    f2 s[6];
    f2 c[MODEL == MODEL_ISO ? 2 : (MODEL == MODEL_ISOHET ? 5 : 9)];
    f2 w3;
    float w;
};

template <int MODEL, int DAMP, bool ST>
__device__ __forceinline__ void stress_mat2(const StepArgs<float> &a, long long cm, int k, StressIn2<MODEL, DAMP> &q)
{
    if (MODEL == MODEL_ISO) {
        q.c[0] = ldm<ST>(a.m[0] + cm);
        q.c[1] = ldm<ST>(a.m[1] + cm);
        q.w = ld(a.w1[2] + k + 1);
    } else {
        if (MODEL == MODEL_ISOHET) {
            q.c[0] = ldm<ST>(a.m[0] + cm);
            q.c[1] = ldm<ST>(a.m[3] + cm);
#pragma unroll
            for (int f = 0; f < 3; ++f) q.c[2 + f] = ldm<ST>(a.m[6 + f] + cm);
        } else {
#pragma unroll
            for (int f = 0; f < 9; ++f) q.c[f] = ldm<ST>(a.m[f] + cm);
        }
        if (DAMP == DAMP_W3D) q.w3 = ldm<ST>(a.w3 + cm);
        else q.w = ld(a.w1[2] + k);
    }
}
template <int MODEL, int DAMP>
__device__ __forceinline__ void stress_state2(const StepArgs<float> &a, long long c, StressIn2<MODEL, DAMP> &q)
{
    q.vx = ld2<false>(a.f[0] + c);
    q.vx_i2 = a.f[0][c + 2];
    q.vx_jm = ld2<false>(a.f[0] + c - a.sx);
    q.vy = ld2<false>(a.f[1] + c);
    q.vy_jp = ld2<false>(a.f[1] + c + a.sx);
    q.vy_im = a.f[1][c - 1];
    q.vz_p = ld2<false>(a.f[2] + c + a.sy);
    q.vz_im = a.f[2][c - 1];
    q.vz_jm = ld2<false>(a.f[2] + c - a.sx);
#pragma unroll
    for (int f = 0; f < 6; ++f) q.s[f] = ld2<false>(a.f[3 + f] + c);
}

// The pair (i, i+1) of row j over planes [k0, k1).  soff, start, r: right-hand side r of several -- its state
// lies soff elements after the materials' index, its sources are entries start[r] .. start[r+1] - 1.
// The orthorhombic update loads a plane ahead (PF), in 128 registers; the others have fewer loads per plane
// and do better with 85 registers and half as many warps again (iso-het 203x151x97 72.5 -> 68.0 us a step, 96^3 15.7 ->
// 14.4; ortho 128^3 in 85 without the prefetch 52.2 -> 54.9, 320x320x256 596 -> 603).
template <int MODEL>
__host__ __device__ constexpr bool pair_prefetch() { return MODEL == MODEL_ORTHO; }
template <int MODEL, int DAMP, bool ST>
__device__ __forceinline__ void stress_pair(const StepArgs<float> &a, int i, int j, int k0, int k1, long long soff, const StressSrc &ss,
                                            const int *start = nullptr, int r = 0)
{
    constexpr bool PF = pair_prefetch<MODEL>();
    if (i >= a.nx || j >= a.ny) return;
    const bool in1 = i + 1 < a.nx, row_bc = j < a.bc1_rows;
    f2 hx = 0, wxi = 0, wxy = 0, pxy = 0;
    float hy = 0.f, wyj = 0.f;
    if (DAMP == DAMP_PML1D) {
        const float w0 = ld(a.w1[0] + i), w1 = ld(a.w1[0] + i + 1), w2 = in1 ? ld(a.w1[0] + i + 2) : 0.f;
        wyj = ld(a.w1[1] + j);
        hx = pk(0.5f * (w1 + w0), 0.5f * (w2 + w1));
        hy = 0.5f * (ld(a.w1[1] + j + 1) + wyj);
        wxi = pk(w0, w1);
        wxy = mul2(wxi, dup(wyj));
    } else if (DAMP == DAMP_SEP) {
        const float py = ld(a.w1[1] + j);
        pxy = pk(ld(a.w1[0] + i) * py, in1 ? ld(a.w1[0] + i + 1) * py : 0.f);
    }
    long long cm = (long long)i + (long long)j * a.sx + (long long)k0 * a.sy;
    long long c = cm + soff;
    float wz_k = 0.f;
    if (DAMP == DAMP_PML1D) wz_k = ld(a.w1[2] + k0);
    StressIn2<MODEL, DAMP> nxt;
    stress_mat2<MODEL, DAMP, ST>(a, cm, k0, nxt);
    pdl_wait();  // nothing above depends on an earlier launch
    f2 vx_m = ld2<false>(a.f[0] + c - a.sy), vy_m = ld2<false>(a.f[1] + c - a.sy), vz_k = ld2<false>(a.f[2] + c);
    stress_state2<MODEL, DAMP>(a, c, nxt);
    bool src_col = false;
    float s_src = 0.f;
    int e0 = 0, e1 = ss.nsrc;
    if (ss.nsrc > 0 && i + 1 >= ss.i0 && i <= ss.i1 && j >= ss.j0 && j <= ss.j1 && k0 <= ss.k1 && k1 > ss.k0) {
        const int it = *ss.it_ptr;
        src_col = it >= 0 && it < ss.nstf;
        if (src_col) s_src = (float)ss.stf[it];
        if (start) {
            e0 = start[r];
            e1 = start[r + 1];
        }
    }
    const PairOps op = {dup(a.one), dup(a.minus_one)};
    const f2 dt = dup(a.dt), rdx = dup(a.rdx), rdy = dup(a.rdy), rdz = dup(a.rdz);
    const bool guard = MODEL != MODEL_ISO;  // the isotropic scheme updates the shear components of edge cells too
    const bool g0 = !guard || i > 0;

    for (int k = k0; k < k1; ++k, c += a.sy, cm += a.sy) {
        if (!PF && k > k0) {
            stress_mat2<MODEL, DAMP, ST>(a, cm, k, nxt);
            stress_state2<MODEL, DAMP>(a, c, nxt);
        }
        const StressIn2<MODEL, DAMP> q = nxt;
        if (PF && k + 1 < k1) {
            stress_mat2<MODEL, DAMP, ST>(a, cm + a.sy, k + 1, nxt);
            stress_state2<MODEL, DAMP>(a, c + a.sy, nxt);
        }
        const f2 vx_ip = pk(hi(q.vx), q.vx_i2), vy_im = pk(q.vy_im, lo(q.vy)), vz_im = pk(q.vz_im, lo(vz_k));
        const f2 Vxx = mul2(op.sub(vx_ip, q.vx), rdx), Vyy = mul2(op.sub(q.vy_jp, q.vy), rdy), Vzz = mul2(op.sub(q.vz_p, vz_k), rdz);
        // differences of the shear terms: dVx/dy dVy/dx dVx/dz dVz/dx dVy/dz dVz/dy
        const f2 x[6] = {op.sub(q.vx, q.vx_jm), op.sub(q.vy, vy_im), op.sub(q.vx, vx_m), op.sub(vz_k, vz_im), op.sub(q.vy, vy_m), op.sub(vz_k, q.vz_jm)};
        f2 o[6];
        if (MODEL == MODEL_ISO) {
            const f2 c11 = q.c[0], c12 = q.c[1];
            const f2 hz = dup(0.5f * (q.w + wz_k)), c66dt = dup(((a.smu_on && k == 1) ? a.smu : a.c66) * a.dt);
            const f2 xy = mul2(dup(wz_k * wyj), wxi), yz = mul2(wxy, dup(wz_k));
            const f2 t12y = mul2(c12, Vyy), t12z = mul2(c12, Vzz), t12x = mul2(c12, Vxx);
            o[0] = mul2(hx, op.add(q.s[0], mul2(dt, op.add(op.add(mul2(c11, Vxx), t12y), t12z))));
            o[1] = mul2(dup(hy), op.add(q.s[1], mul2(dt, op.add(op.add(t12x, mul2(c11, Vyy)), t12z))));
            o[2] = mul2(hz, op.add(q.s[2], mul2(dt, op.add(op.add(t12x, t12y), mul2(c11, Vzz)))));
            o[3] = mul2(xy, op.add(q.s[3], mul2(c66dt, op.add(mul2(x[1], rdx), mul2(x[0], rdy)))));
            o[4] = mul2(xy, op.add(q.s[4], mul2(c66dt, op.add(mul2(x[3], rdx), mul2(x[2], rdz)))));
            o[5] = mul2(yz, op.add(q.s[5], mul2(c66dt, op.add(mul2(x[4], rdz), mul2(x[5], rdy)))));
        } else {
            const f2 W = DAMP == DAMP_W3D ? q.w3 : mul2(pxy, dup(q.w));
            if (MODEL == MODEL_ISOHET) {
                const f2 c11 = q.c[0], c12 = q.c[1];
                const f2 t12y = mul2(c12, Vyy), t12z = mul2(c12, Vzz), t12x = mul2(c12, Vxx);
                o[0] = op.add(mul2(q.s[0], W), mul2(dt, op.add(op.add(mul2(c11, Vxx), t12y), t12z)));
                o[1] = op.add(mul2(q.s[1], W), mul2(dt, op.add(op.add(t12x, mul2(c11, Vyy)), t12z)));
                o[2] = op.add(mul2(q.s[2], W), mul2(dt, op.add(op.add(t12x, t12y), mul2(c11, Vzz))));
                o[3] = op.add(mul2(q.s[3], W), mul2(mul2(q.c[2], dt), op.add(mul2(x[1], rdx), mul2(x[0], rdy))));
                o[4] = op.add(mul2(q.s[4], W), mul2(mul2(q.c[3], dt), op.add(mul2(x[3], rdx), mul2(x[2], rdz))));
                o[5] = op.add(mul2(q.s[5], W), mul2(mul2(q.c[4], dt), op.add(mul2(x[4], rdz), mul2(x[5], rdy))));
            } else {
                o[0] = op.add(mul2(q.s[0], W), mul2(dt, op.add(op.add(mul2(q.c[0], Vxx), mul2(q.c[3], Vyy)), mul2(q.c[4], Vzz))));
                o[1] = op.add(mul2(q.s[1], W), mul2(dt, op.add(op.add(mul2(q.c[3], Vxx), mul2(q.c[1], Vyy)), mul2(q.c[5], Vzz))));
                o[2] = op.add(mul2(q.s[2], W), mul2(dt, op.add(op.add(mul2(q.c[4], Vxx), mul2(q.c[5], Vyy)), mul2(q.c[2], Vzz))));
                f2 d[6];
                div_shear2(a, x, d);
                o[3] = op.add(mul2(q.s[3], W), mul2(mul2(dt, q.c[6]), op.add(d[1], d[0])));
                o[4] = op.add(mul2(q.s[4], W), mul2(mul2(dt, q.c[7]), op.add(d[3], d[2])));
                o[5] = op.add(mul2(q.s[5], W), mul2(mul2(dt, q.c[8]), op.add(d[4], d[5])));
            }
        }
        // stress_store<BC1OWN>
        const bool bc0 = a.bc1 && k == 0 && row_bc, bc1 = a.bc1 && k == 1;
        const bool gj = !guard || j > 0, gk = !guard || k > 0;
        st2(a.f[3] + c, o[0], true, in1);
        st2(a.f[4] + c, o[1], true, in1);
        st2(a.f[5] + c, bc0 ? 0ull : o[2], true, in1);
        st2(a.f[6] + c, o[3], g0 && gj, gj && in1);
        st2(a.f[7] + c, o[4], g0 && gk && !(bc1 && i > 0 && row_bc), gk && in1 && !(bc1 && row_bc));
        st2(a.f[8] + c, o[5], gj && gk && !(bc1 && j > 0), gj && gk && in1 && !(bc1 && j > 0));
        if (k == 2 && a.bc1) {
            if (row_bc) st2(a.f[7] + c - a.sy, mul2(dup(a.third), o[4]), i > 0, in1);
            if (j > 0) st2(a.f[8] + c - a.sy, mul2(dup(a.third), o[5]), true, in1);
        }
        if (src_col && k >= ss.k0 && k <= ss.k1) {
            for (int e = e0; e < e1; ++e) {
                const SrcEntry q_e = ss.inl ? ss.e[e] : ss.src[e];
                if ((q_e.i == i || (q_e.i == i + 1 && in1)) && q_e.j == j && fused_src_plane(q_e.comp, q_e.k) == k)
                    inject_entry(a, q_e, s_src, ss.order, soff);
            }
        }
        wz_k = q.w;
        vx_m = q.vx;
        vy_m = q.vy;
        vz_k = q.vz_p;
    }
}

template <int MODEL, int DAMP, bool KAHAN>
struct VelIn2 {
    f2 sxx, syy, syy_jm, szz, sxy, sxy_jp, sxz_p, syz_p, syz_jp;
    float sxx_im, sxy_i2, sxz_i2;  // sxx(i-1), sxy(i+2), sxz(i+2) at plane k
    f2 v[3];
    f2 b[MODEL == MODEL_ISO ? 1 : 3];
    f2 w3;
    float w;
    f2 cp[KAHAN ? 3 : 1];
};
template <int MODEL, int DAMP, bool KAHAN, bool ST>
__device__ __forceinline__ void vel_mat2(const StepArgs<float> &a, long long cm, int k, VelIn2<MODEL, DAMP, KAHAN> &q)
{
    if (MODEL == MODEL_ISO) {
        q.w = ld(a.w1[2] + k - 1);
    } else {
#pragma unroll
        for (int f = 0; f < 3; ++f) q.b[f] = ldm<ST>(a.m[9 + f] + cm);
        if (DAMP == DAMP_W3D) q.w3 = ldm<ST>(a.w3 + cm);
        else q.w = ld(a.w1[2] + k);
    }
}
template <int MODEL, int DAMP, bool KAHAN>
__device__ __forceinline__ void vel_state2(const StepArgs<float> &a, long long c, VelIn2<MODEL, DAMP, KAHAN> &q)
{
    q.sxx = ld2<false>(a.f[3] + c);
    q.sxx_im = a.f[3][c - 1];
    q.syy = ld2<false>(a.f[4] + c);
    q.syy_jm = ld2<false>(a.f[4] + c - a.sx);
    q.szz = ld2<false>(a.f[5] + c);
    q.sxy = ld2<false>(a.f[6] + c);
    q.sxy_jp = ld2<false>(a.f[6] + c + a.sx);
    q.sxy_i2 = a.f[6][c + 2];
    q.sxz_p = ld2<false>(a.f[7] + c + a.sy);
    q.sxz_i2 = a.f[7][c + 2];
    q.syz_p = ld2<false>(a.f[8] + c + a.sy);
    q.syz_jp = ld2<false>(a.f[8] + c + a.sx);
#pragma unroll
    for (int f = 0; f < 3; ++f) q.v[f] = ld2<false>(a.f[f] + c);
    if (KAHAN) {
#pragma unroll
        for (int f = 0; f < 3; ++f) q.cp[f] = ld2<false>(a.comp[f] + c);
    }
}

template <int MODEL, bool KAHAN>
__device__ __forceinline__ f2 vel_update2(const StepArgs<float> &a, const PairOps &op, f2 V, f2 dS, f2 w, f2 b, f2 &cp)
{
    const f2 dt = dup(a.dt), bd = mul2(b, dS);
    if (!KAHAN) {
        const f2 vr = mul2(V, dup(a.rdt));
        if (MODEL == MODEL_ISO) return mul2(mul2(w, op.add(vr, bd)), dt);
        const f2 r = mul2(op.add(mul2(vr, w), bd), dt);
        return a.vdamp_on ? op.sub(r, mul2(dup(a.vdamp), V)) : r;
    }
    const f2 inc = MODEL == MODEL_ISO ? mul2(mul2(w, bd), dt) : mul2(bd, dt);
    const f2 y = op.sub(inc, mul2(w, cp));
    const f2 av = mul2(w, V);
    const f2 t = op.add(av, y);
    cp = op.sub(op.sub(t, av), y);
    return t;
}

template <int MODEL, int DAMP, bool KAHAN, bool ST>
__device__ __forceinline__ void velocity_pair(const StepArgs<float> &a, int i, int j, int kc0, int k1, long long soff, const RecFuse &rf,
                                              double *traces)
{
    const int k0 = max(1, kc0);
    if (j < 1 || i >= a.nx || j >= a.ny || k0 >= k1) return;
    const bool in0 = i >= 1, in1 = i + 1 < a.nx;
    f2 ax = 0, pxy = 0;
    float ay = 0.f;
    if (DAMP == DAMP_PML1D) {
        ax = pk(ld(a.w1[0] + max(i - 1, 0)), ld(a.w1[0] + i));
        ay = ld(a.w1[1] + j - 1);
    } else if (DAMP == DAMP_SEP) {
        const float py = ld(a.w1[1] + j);
        pxy = pk(ld(a.w1[0] + i) * py, in1 ? ld(a.w1[0] + i + 1) * py : 0.f);
    }
    long long cm = (long long)i + (long long)j * a.sx + (long long)k0 * a.sy;
    long long c = cm + soff;
    VelIn2<MODEL, DAMP, KAHAN> nxt;
    vel_mat2<MODEL, DAMP, KAHAN, ST>(a, cm, k0, nxt);
    pdl_wait();  // nothing above depends on an earlier launch
    f2 szz_m = ld2<false>(a.f[5] + c - a.sy), sxz_k = ld2<false>(a.f[7] + c), syz_k = ld2<false>(a.f[8] + c);
    vel_state2<MODEL, DAMP, KAHAN>(a, c, nxt);
    // L2 prefetch: lane l of a row's 16 asks for the row's line of input field l
    const float *pf_row = nullptr;
    if (a.l2pf > 0) {
        const int l = (int)threadIdx.x;
        pf_row = soff ? vel_prefetch_field<float, MODEL, DAMP, KAHAN, true>(a, l) : vel_prefetch_field<float, MODEL, DAMP, KAHAN>(a, l);
        if (pf_row) pf_row += c - 2 * (long long)l + (long long)a.l2pf * a.sy;
    }
    // receivers on the pair's columns
    int slot0 = -1, slot1 = -1, r_it = 0;
    if (rf.grp && k0 <= rf.kmax && k1 > rf.kmin) {
        const uint2 g = rf.grp[j * rf.ngx + (i >> 5)];
        if ((g.x >> (i & 31)) & 3u) {
            r_it = *rf.it_rd;
            if (r_it >= 0 && r_it < rf.trace_len) {
                const int s = (int)g.y + __popc(g.x & ((1u << (i & 31)) - 1u)), first = (g.x >> (i & 31)) & 1u;
                if (first) slot0 = s;
                if ((g.x >> (i & 31)) & 2u) slot1 = s + first;
            }
        }
    }
    const PairOps op = {dup(a.one), dup(a.minus_one)};
    const f2 rdx = dup(a.rdx), rdy = dup(a.rdy), rdz = dup(a.rdz);

    for (int k = k0; k < k1; ++k, c += a.sy, cm += a.sy) {
        if (k > k0) {
            vel_mat2<MODEL, DAMP, KAHAN, ST>(a, cm, k, nxt);
            vel_state2<MODEL, DAMP, KAHAN>(a, c, nxt);
        }
        const VelIn2<MODEL, DAMP, KAHAN> q = nxt;
        if (pf_row && k + a.l2pf < k1) l2_prefetch_line(pf_row + (long long)(k - k0) * a.sy);
        const f2 sxx_im = pk(q.sxx_im, lo(q.sxx)), sxy_ip = pk(hi(q.sxy), q.sxy_i2), sxz_ip = pk(hi(sxz_k), q.sxz_i2);
        const f2 dSx = op.add(op.add(mul2(op.sub(q.sxx, sxx_im), rdx), mul2(op.sub(q.sxy_jp, q.sxy), rdy)), mul2(op.sub(q.sxz_p, sxz_k), rdz));
        const f2 dSy = op.add(op.add(mul2(op.sub(q.syy, q.syy_jm), rdy), mul2(op.sub(sxy_ip, q.sxy), rdx)), mul2(op.sub(q.syz_p, syz_k), rdz));
        const f2 dSz = op.add(op.add(mul2(op.sub(q.szz, szz_m), rdz), mul2(op.sub(sxz_ip, sxz_k), rdx)), mul2(op.sub(q.syz_jp, syz_k), rdy));
        f2 wx, wy, wz, v[3], cp[3] = {KAHAN ? q.cp[0] : 0ull, KAHAN ? q.cp[1] : 0ull, KAHAN ? q.cp[2] : 0ull};
        f2 bx, by, bz;
        if (MODEL == MODEL_ISO) {
            wx = ax;
            wy = dup(ay);
            wz = dup(q.w);
            bx = dup(a.bx);
            by = dup(a.by);
            bz = dup(a.bz);
        } else {
            wx = wy = wz = DAMP == DAMP_W3D ? q.w3 : mul2(pxy, dup(q.w));
            bx = q.b[0];
            by = q.b[MODEL == MODEL_ISO ? 0 : 1];
            bz = q.b[MODEL == MODEL_ISO ? 0 : 2];
        }
        v[0] = vel_update2<MODEL, KAHAN>(a, op, q.v[0], dSx, wx, bx, cp[0]);
        v[1] = vel_update2<MODEL, KAHAN>(a, op, q.v[1], dSy, wy, by, cp[1]);
        v[2] = vel_update2<MODEL, KAHAN>(a, op, q.v[2], dSz, wz, bz, cp[2]);
        // vel_store's ranges, for cells 1 <= i < nx
        const bool jn = j < a.ny - 1, kn = k < a.nz - 1, l0 = i < a.nx - 1, l1 = i + 1 < a.nx - 1;
        const bool m0[3] = {in0 && jn && kn, in0 && l0 && kn, in0 && l0 && jn}, m1[3] = {in1 && jn && kn, l1 && kn, l1 && jn};
#pragma unroll
        for (int f = 0; f < 3; ++f) {
            st2<ST>(a.f[f] + c, v[f], m0[f], m1[f]);
            if (KAHAN) st2(a.comp[f] + c, cp[f], m0[f], m1[f]);
        }
        if ((slot0 >= 0 || slot1 >= 0) && k >= rf.kmin && k <= rf.kmax) {
            for (int h = 0; h < 2; ++h) {
                const int slot = h ? slot1 : slot0;
                if (slot < 0) continue;
                const int *po = rf.off + (long long)slot * (rf.kmax - rf.kmin + 2) + (k - rf.kmin);
                const int e1 = po[1];
                for (int e = po[0]; e < e1; ++e) {
                    const int2 re = rf.ent[e];
                    const f2 nv = re.x == 0 ? v[0] : re.x == 1 ? v[1] : v[2], ov = re.x == 0 ? q.v[0] : re.x == 1 ? q.v[1] : q.v[2];
                    const bool upd = h ? (re.x == 0 ? m1[0] : re.x == 1 ? m1[1] : m1[2]) : (re.x == 0 ? m0[0] : re.x == 1 ? m0[1] : m0[2]);
                    const f2 val = upd ? nv : ov;
                    traces[(long long)re.y * rf.trace_len + r_it] = (double)(h ? hi(val) : lo(val));
                }
            }
        }
        szz_m = q.szz;
        sxz_k = q.sxz_p;
        syz_k = q.syz_p;
    }
}

constexpr int PAIR_TX = TX / 2;                           // pairs per row of a CTA
constexpr int PAIR_MAX_THREADS = 256;                     // CTAs of at most 16 rows
__host__ __device__ constexpr int pair_rows(int ty) { return 2 * ty < PAIR_MAX_THREADS / PAIR_TX ? 2 * ty : PAIR_MAX_THREADS / PAIR_TX; }

template <int MODEL, int DAMP, bool ST>
__global__ void __launch_bounds__(PAIR_MAX_THREADS, pair_prefetch<MODEL>() ? 2 : 3) k_stress_pair(const StepArgs<float> a, const __grid_constant__ StressSrc ss)
{
    pdl_trigger();
    const int k0 = blockIdx.z * a.kchunk;
    stress_pair<MODEL, DAMP, ST>(a, blockIdx.x * TX + 2 * threadIdx.x, blockIdx.y * blockDim.y + threadIdx.y, k0, min(k0 + a.kchunk, a.nz), 0, ss);
}

template <int MODEL, int DAMP, bool KAHAN, bool ST>
__global__ void __launch_bounds__(PAIR_MAX_THREADS, 3) k_velocity_pair(const StepArgs<float> a, const RecFuse rf)
{
    pdl_trigger();
    if (rf.it_wr && blockIdx.x == 0 && blockIdx.y == 0 && blockIdx.z == 0 && threadIdx.x == 0 && threadIdx.y == 0) {
        pdl_wait();
        *rf.it_wr = *rf.it_rd + 1;
    }
    const int k0 = ((int)gridDim.z - 1 - (int)blockIdx.z) * a.kchunk;
    velocity_pair<MODEL, DAMP, KAHAN, ST>(a, blockIdx.x * TX + 2 * threadIdx.x, blockIdx.y * blockDim.y + threadIdx.y, k0,
                                      min(k0 + a.kchunk, a.nz), 0, rf, rf.traces);
}

// Several right-hand sides of one model, their state boxes rhs_stride elements apart: the index of the
// right-hand side is the fastest part of blockIdx.x, so the CTAs of a tile are dispatched together and read
// its material planes from HBM once (the others' reads hit L2).  start: their source entries in ss.src;
// trace_stride: elements between their trace blocks.  A batch of 6 right-hand sides on ortho 128^3 and 6 isotropic
// models of 96^3 to 160^3 with these: 493 us a step, 640 with one cell per thread and separate injection and receiver launches
// for all problems; its fields and materials move in 425 us at the copy bandwidth.
template <int MODEL, int DAMP, bool ST>
__global__ void __launch_bounds__(PAIR_MAX_THREADS, pair_prefetch<MODEL>() ? 2 : 3)
    k_stress_pair_mr(const StepArgs<float> a, int R, long long rhs_stride, const __grid_constant__ StressSrc ss, const int *start)
{
    pdl_trigger();
    const int r = blockIdx.x % R, k0 = blockIdx.z * a.kchunk;
    stress_pair<MODEL, DAMP, ST>(a, (blockIdx.x / R) * TX + 2 * threadIdx.x, blockIdx.y * blockDim.y + threadIdx.y, k0, min(k0 + a.kchunk, a.nz),
                             (long long)r * rhs_stride, ss, start, r);
}

template <int MODEL, int DAMP, bool ST>
__global__ void __launch_bounds__(PAIR_MAX_THREADS, 3)
    k_velocity_pair_mr(const StepArgs<float> a, int R, long long rhs_stride, const RecFuse rf, long long trace_stride)
{
    pdl_trigger();
    if (rf.it_wr && blockIdx.x == 0 && blockIdx.y == 0 && blockIdx.z == 0 && threadIdx.x == 0 && threadIdx.y == 0) {
        pdl_wait();
        *rf.it_wr = *rf.it_rd + 1;
    }
    const int r = blockIdx.x % R, k0 = ((int)gridDim.z - 1 - (int)blockIdx.z) * a.kchunk;
    velocity_pair<MODEL, DAMP, false, ST>(a, (blockIdx.x / R) * TX + 2 * threadIdx.x, blockIdx.y * blockDim.y + threadIdx.y, k0,
                                      min(k0 + a.kchunk, a.nz), (long long)r * rhs_stride, rf, rf.traces + r * trace_stride);
}

}  // namespace ewf
